"""The neighbour passes at the sizes where their staging and bit words end.

Sets are the oracle's bit for bit; phase rates are held to the plain form's
contract, 1e-12 * max(|value|, (sigma / n_i) sum |sin|).  The angle-difference
terms are within ~4e-16 of the exact sines and a sum of n terms within
n * 1.1e-16 per unit, so the contract leaves a factor of some hundred.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from spc2_langevin_integration_gb300 import abi
from tests._helpers import alignment_scale, init_state

pytestmark = pytest.mark.gpu

RHS_TOL = 1e-12


def check_rates(o, st, prm, d):
    off, idx = o.neighbour_lists(st)
    scale, _ = alignment_scale(st, off, idx, prm["sigma"], prm["alpha"])
    ref = o.rhs_srk(st)[0][2::3]
    assert np.all(np.abs(d[2::3] - ref) <= RHS_TOL * np.maximum(np.abs(ref), scale) + 1e-300)
    return off, idx


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 703, 704, 705, 1409])
def test_all_pairs_rounds_and_positions_outside_the_box(n):
    """Rounds of 704 candidates in words of 32; a tenth of the positions lies
    outside the box or on its edges, where the reference's minimum image of
    the unwrapped positions decides."""
    L, prm = 1.3, dict(v0=0.01, sigma=1.2, rho=0.45, alpha=0.7, D_phi=0.01)
    st = init_state(n, L, 200 + n)
    rng = np.random.default_rng(n)
    for k in rng.choice(n, max(1, n // 10), replace=False):
        st[3 * k + int(rng.integers(2))] = rng.choice([-0.0, 0.0, L, L - 2e-16, -0.3 * L, 1.7 * L, -1.2 * L])
    o = po.OracleSystem(n, L, **prm)
    with abi.System(n, abi.make_params(L=L, stepper=abi.STEPPER_SRK, **prm)) as s:
        s.upload_state(st)
        off, idx = s.neighbours()
        d, _ = s.rhs_srk()
    off_ref, idx_ref = check_rates(o, st, prm, d)
    assert np.array_equal(off, off_ref) and np.array_equal(idx, idx_ref)


def test_all_pairs_block_widths_agree_bitwise():
    """A batch with enough all-pairs blocks takes 128-thread blocks, a system
    alone one warp per block."""
    L, n = 1.0, 1000
    par = [abi.make_params(L=L, stepper=abi.STEPPER_SRK, v0=0.01, sigma=1.0, rho=0.26 + 0.005 * k, alpha=1.4,
                           D_phi=0.01, seed=3, system_id=k) for k in range(40)]
    with abi.Batch(abi.STEPPER_SRK, abi.PRECISION_FP64, 40, 40 * n, 40) as b:
        slots = [b.admit(n, p, init_state(n, L, 300 + k)) for k, p in enumerate(par)]
        b.step(0.01, 3)
        got = [b.download(s) for s in slots]
    for k in (0, 17, 39):
        with abi.System(n, par[k]) as s:
            s.upload_state(init_state(n, L, 300 + k))
            s.step(0.01, 3)
            assert np.array_equal(s.download_state(), got[k])


@pytest.mark.parametrize("total", [33, 703, 704, 705, 1409])
@pytest.mark.parametrize("neighbour", [abi.NEIGHBOUR_CELL, abi.NEIGHBOUR_VERLET])
def test_fp64_staging_rounds(total, neighbour):
    """All particles in 3 x 3 cells of 7 x 7: the middle cell's stencil list
    has exactly `total` candidates (Verlet rows: its 25 cells)."""
    L, prm = 7.0, dict(v0=0.01, sigma=1.2, rho=1.0, alpha=0.7, D_phi=0.01)
    st = init_state(total, 3.0, 400 + total)
    st[0::3] += 2.0
    st[1::3] += 2.0
    o = po.OracleSystem(total, L, **prm)
    p = abi.make_params(L=L, stepper=abi.STEPPER_SRK, neighbour=neighbour, skin=0.2, **prm)
    for sparse in (0.0, 1e9):
        with abi.System(total, p) as s:
            s.set_tuning(abi.TUNE_SPARSE_BELOW, sparse)
            s.upload_state(st)
            d, a = s.rhs_srk()
            check_rates(o, st, prm, d)
            off, idx = s.neighbours()
        if sparse == 0.0:
            first = d, a
        elif neighbour == abi.NEIGHBOUR_CELL:
            assert np.array_equal(first[0], d) and np.array_equal(first[1], a)
    off_ref, idx_ref = o.neighbour_lists(st)
    assert np.array_equal(off, off_ref) and np.array_equal(idx, idx_ref)
