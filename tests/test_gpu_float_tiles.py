"""The float cell-tile passes (tensor cores) at the edges of their tiles: row
tiles of 32 in groups of 128, blocks of 32 candidates, staging rounds of 1,024
(FP32C) and 768 (FP32X).

FP32X sums are exact integers, so the lane kernels' results are matched bit for
bit.  FP32C is held to its own inputs' rounding against FP64: phases to 1.9e-7
(a float of a reduced phase) and cosines and sines to 1.2e-7 on both sides of a
term, products and the sum to 1.8e-7: 1e-6 sigma on a mean of sines, and on a
mean of rate differences times cosines (rates up to sigma, both sides) 5e-6
sigma.
"""
import numpy as np
import pytest

from spc2_langevin_integration_gb300 import abi

pytestmark = pytest.mark.gpu


L, RHO, SIGMA = 1.0, 0.249, 1.3
PRM = dict(v0=0.01, sigma=SIGMA, rho=RHO, alpha=0.6, D_phi=0.02)


def _state(counts, seed):
    """counts[k] particles in cell k of the 4 x 4 grid, in mixed order."""
    rng = np.random.default_rng(seed)
    cell = np.repeat(np.arange(16), counts)
    rng.shuffle(cell)
    st = np.empty(3 * cell.size)
    st[0::3] = (cell % 4 + rng.uniform(0.001, 0.999, cell.size)) * L / 4
    st[1::3] = (cell // 4 + rng.uniform(0.001, 0.999, cell.size)) * L / 4
    st[2::3] = rng.uniform(-np.pi, np.pi, cell.size)
    return cell.size, st


def _counts(case):
    if case == "rows":  # one cell per row-tile and group edge
        return [1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 0, 96, 127, 128, 129, 257]
    return [case] + 15 * [5]  # one crowded cell: its list is case + 40 long


def _system(n, precision, st, lane=False, units=False):
    s = abi.System(n, abi.make_params(L=L, stepper=abi.STEPPER_SRK, precision=precision, seed=5, **PRM))
    s.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9 if lane else 0)
    if units:
        s.set_tuning(abi.TUNE_CELL_UNITS, 1)
    s.upload_state(st)
    return s


@pytest.mark.parametrize("case", ["rows", 24, 55, 56, 57, 727, 728, 729, 983, 984, 985, 2100])
def test_tiles_match_the_lane_kernels_and_fp64(case):
    n, st = _state(_counts(case), 7)
    with _system(n, abi.PRECISION_FP32X, st, lane=True) as s:
        rates, extra = s.rhs_srk()
        s.step(0.01, 3)
        after = s.download_state()
    for units in (False, True):
        with _system(n, abi.PRECISION_FP32X, st, units=units) as s:
            got = s.rhs_srk()
            assert np.array_equal(got[0], rates) and np.array_equal(got[1], extra)
            s.step(0.01, 3)
            assert np.array_equal(s.download_state(), after)
    with _system(n, abi.PRECISION_FP64, st) as s:
        rates, extra = s.rhs_srk()
    first = None
    for units in (False, True):
        with _system(n, abi.PRECISION_FP32C, st, units=units) as s:
            got = s.rhs_srk()
        first = first or got
        assert np.array_equal(got[0], first[0]) and np.array_equal(got[1], first[1])
    assert np.max(np.abs(first[0][2::3] - rates[2::3])) <= 1e-6 * SIGMA
    assert np.max(np.abs(first[1][1::2] - extra[1::2])) <= 5e-6 * SIGMA


def test_a_phase_that_is_not_finite_reaches_its_neighbours_only():
    n, st = _state(_counts("rows"), 11)
    for k, v in ((3, np.nan), (500, np.inf)):
        st[3 * k + 2] = v
    with _system(n, abi.PRECISION_FP32C, st, lane=True) as s:
        want = s.rhs_srk()
    for units in (False, True):
        with _system(n, abi.PRECISION_FP32C, st, units=units) as s:
            got = s.rhs_srk()
        for g, w in zip(got, want):
            assert np.array_equal(np.isnan(g), np.isnan(w))
            assert 0 < np.isnan(g).sum() < g.size
