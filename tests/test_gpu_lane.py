"""The particle-per-lane passes against the cell-tile ones and the oracle, at
column counts where a row's candidates split into two runs (box edge, blocks
of 16 to 31 columns) and at lists longer than a lane keeps."""
import numpy as np
import pytest

from oracle import pyoracle as po
from spc2_langevin_integration_gb300 import abi
from tests._helpers import alignment_scale, init_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [4, 5, 15, 16, 17, 31, 32, 33, 47, 64])
@pytest.mark.parametrize("per_cell", [0.7, 9.0])
def test_lane_passes_over_columns(nc, per_cell):
    """FP64 and FP32X are bitwise the cell-tile passes'; FP64 rates hold the
    plain form's 1e-12 contract against the oracle."""
    L = 1.7
    prm = dict(v0=0.02, sigma=1.1, rho=L / (nc + 0.37), alpha=1.3, D_phi=0.01)
    n = max(40, int(per_cell * nc * nc))
    st = init_state(n, L, 500 + nc)
    # (no position that copy-wraps to exactly L beside one at 0: the float test
    # of every cell-list kernel has those two at distance 0, the reference at L)
    st[0:21:3] = [-0.0, 0.0, L, L - 3e-16, L / nc, np.nextafter(L / nc, 0), 0.5 * L]
    for precision in (abi.PRECISION_FP64, abi.PRECISION_FP32X):
        out = []
        for sparse in (0.0, 1e9):
            p = abi.make_params(L=L, stepper=abi.STEPPER_SRK, precision=precision, seed=4, **prm)
            with abi.System(n, p) as s:
                s.set_tuning(abi.TUNE_SPARSE_BELOW, sparse)
                s.upload_state(st)
                d, a = s.rhs_srk()
                s.step(0.01, 4)
                out.append((d, a, s.download_state()))
        assert all(np.array_equal(x, y) for x, y in zip(*out))
        if precision == abi.PRECISION_FP64:
            o = po.OracleSystem(n, L, **prm)
            off, idx = o.neighbour_lists(st)
            scale, _ = alignment_scale(st, off, idx, prm["sigma"], prm["alpha"])
            ref = o.rhs_srk(st)[0][2::3]
            assert np.all(np.abs(out[1][0][2::3] - ref) <= 1e-12 * np.maximum(np.abs(ref), scale) + 1e-300)


@pytest.mark.parametrize("n", [31, 32, 33, 480, 513, 3000])
def test_lane_lists_and_batches(n):
    """All particles in a few cells: lists of up to 3,000 neighbours (more than
    a lane's 16 words), bitwise the cell-tile passes' and, in a batch with a
    dense and an all-pairs system, bitwise the system alone."""
    L, prm = 4.0, dict(v0=0.01, sigma=1.0, rho=0.5, alpha=0.3, D_phi=0.01)
    st = init_state(n, 0.9, 600 + n)
    for precision in (abi.PRECISION_FP64, abi.PRECISION_FP32X, abi.PRECISION_FP32C):
        def par(k, **kw):
            return abi.make_params(L=L, stepper=abi.STEPPER_SRK, precision=precision, seed=6, system_id=k,
                                   **dict(prm, **kw))
        alone = []
        for sparse in (0.0, 1e9):
            with abi.System(n, par(1)) as s:
                s.set_tuning(abi.TUNE_SPARSE_BELOW, sparse)
                s.upload_state(st)
                s.step(0.01, 3)
                alone.append(s.download_state())
        if precision == abi.PRECISION_FP32C:
            assert np.abs(alone[0] - alone[1]).max() <= 1e-6
        else:
            assert np.array_equal(alone[0], alone[1])
        with abi.Batch(abi.STEPPER_SRK, precision, 3, n + 5200, 64 + 64 + 1) as b:
            b.set_tuning(abi.TUNE_SPARSE_BELOW, 60.0 if n < 3840 else 24.0)
            b.admit(5000, par(0), init_state(5000, L, 1))
            slot = b.admit(n, par(1), st)
            b.admit(200, par(2, rho=1.2), init_state(200, L, 2))
            b.step(0.01, 3)
            assert np.array_equal(b.download(slot), alone[1])


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_FP32X, abi.PRECISION_FP32C])
def test_four_lanes_and_one_lane_per_particle_agree_bitwise(precision):
    """A system alone takes four lanes per particle; in a batch of 89,000
    particles it takes one.  Rows of up to 90 neighbours (three words), and a
    system whose rows have more words than the first pass keeps."""
    L, n = 3.0, 3000
    par = [abi.make_params(L=L, stepper=abi.STEPPER_SRK, precision=precision, seed=9, system_id=k, v0=0.02,
                           sigma=1.3, rho=rho, alpha=1.1, D_phi=0.01) for k, rho in ((0, 0.2), (1, 0.3), (2, 0.6))]
    states = [init_state(n, L, 700), init_state(n, L, 701), init_state(n, 1.5, 702)]
    big = abi.make_params(L=8.0, stepper=abi.STEPPER_SRK, precision=precision, v0=0.02, sigma=1.0, rho=0.1,
                          alpha=1.0, D_phi=0.01)
    with abi.Batch(abi.STEPPER_SRK, precision, 4, 3 * n + 80000, 225 + 100 + 25 + 6400) as b:
        b.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9)
        slots = [b.admit(n, p, st) for p, st in zip(par, states)]
        b.admit(80000, big, init_state(80000, 8.0, 703))
        b.step(0.01, 4)
        got = [b.download(s) for s in slots]
    for p, st, want in zip(par, states, got):
        with abi.System(n, p) as s:
            s.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9)
            s.upload_state(st)
            s.step(0.01, 4)
            assert np.array_equal(s.download_state(), want)
