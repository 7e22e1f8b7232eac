"""Phases that are not finite: a right-hand side passes them on to a particle's
neighbours, and to theirs, as the plain FP64 form does, whatever kernel and
precision run.  A diverged state must not look like an isolated particle."""
import numpy as np
import pytest

from spc2_langevin_integration_gb300 import abi

pytestmark = pytest.mark.gpu

PRM = dict(L=1.0, v0=0.01, sigma=1.3, rho=0.249, alpha=0.6, D_phi=0.02, stepper=abi.STEPPER_SRK, seed=5)


def _system(st, precision, stepper=abi.STEPPER_SRK, lane=False, units=False):
    s = abi.System(st.size // 3, abi.make_params(precision=precision, **dict(PRM, stepper=stepper)))
    s.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9 if lane else 0)
    if units:
        s.set_tuning(abi.TUNE_CELL_UNITS, 1)
    s.upload_state(st)
    return s


def _crowded(seed, bad):
    """4,000 particles in one cell (several staging rounds of every float form)
    within a cutoff of each other; bad: indices whose phase is not finite."""
    rng = np.random.default_rng(seed)
    st = np.empty(3 * 4000)
    st[0::3] = rng.uniform(0.05, 0.2, 4000)
    st[1::3] = rng.uniform(0.05, 0.2, 4000)
    st[2::3] = rng.uniform(-np.pi, np.pi, 4000)
    st[3 * np.asarray(bad) + 2] = np.nan
    return st


def test_fp32c_units_keep_the_count_of_a_round_with_a_bad_neighbour():
    # one such phase in each staging round (indices ascend with the list)
    st = _crowded(1, [100, 700, 1300, 1800, 2500, 3000, 3300, 3900])
    for units in (False, True):
        with _system(st, abi.PRECISION_FP32C, units=units) as s:
            rates, extra = s.rhs_srk()
        assert np.isnan(rates[2::3]).all() and np.isnan(extra[1::2]).all()
    for units in (False, True):  # an RK4 stage of an isolated particle keeps its old rate
        with _system(st, abi.PRECISION_FP32C, stepper=abi.STEPPER_RK4, units=units) as s:
            s.step(0.01, 1)
            assert np.isnan(s.download_state()[2::3]).all()


def _spread(n, seed):
    rng = np.random.default_rng(seed)
    L = np.sqrt(n / 1500.0)
    st = np.empty(3 * n)
    st[0::3] = rng.uniform(0.0, L, n)
    st[1::3] = rng.uniform(0.0, L, n)
    st[2::3] = rng.uniform(-np.pi, np.pi, n)
    return L, st


@pytest.mark.parametrize("n,value,stepper", [  # four lanes per particle and one
    (n, v, abi.STEPPER_SRK) for n in (6000, 40000) for v in (np.nan, np.inf, -np.inf)
] + [(6000, np.nan, abi.STEPPER_EULER), (6000, np.inf, abi.STEPPER_RK4)])
def test_fp32x_passes_on_what_fp64_does(n, value, stepper):
    L, st = _spread(n, 3)
    for k in (7, n // 2, n - 1):
        st[3 * k + 2] = value

    def run(precision, lane=False, units=False):
        p = abi.make_params(L=L, v0=0.01, sigma=1.3, rho=0.1, alpha=0.6, D_phi=0.02, stepper=stepper, seed=5,
                            precision=precision)
        with abi.System(n, p) as s:
            s.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9 if lane else 0)
            if units:
                s.set_tuning(abi.TUNE_CELL_UNITS, 1)
            s.upload_state(st)
            out = list(s.rhs_srk())
            s.step(0.01, 1)
            return out + [s.download_state()]

    want = run(abi.PRECISION_FP64)
    for got in (run(abi.PRECISION_FP32X), run(abi.PRECISION_FP32X, units=True), run(abi.PRECISION_FP32X, lane=True)):
        for g, w in zip(got, want):
            assert np.array_equal(np.isnan(g), np.isnan(w))
            assert 0 < np.isnan(g).sum() < g.size


def test_fp32x_rounds_with_bad_neighbours():
    st = _crowded(2, [50, 800, 1600, 2400, 3200, 3950])
    for units in (False, True):
        with _system(st, abi.PRECISION_FP32X, units=units) as s:
            rates, extra = s.rhs_srk()
        assert np.isnan(rates[2::3]).all() and np.isnan(extra[1::2]).all()
