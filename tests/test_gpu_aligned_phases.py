"""FP64 phase rates between aligned phases, against 64 bits and more (long double).

Where phases agree to a small spread and alpha is small, a pair's sine is small
and the reference's rounding of it is too.  The yardstick is the reference's own
formula (the sine of the rounded difference, added in order) in numpy: the mean
error may be 1.6 times its, which covers two roundings of a term for one (1.42)
and the resolution of what is kept of a phase's sine and cosine (2^-64)."""
import numpy as np
import pytest

from spc2_langevin_integration_gb300 import abi

pytestmark = pytest.mark.gpu

N, L, ROWS = 1000, 1.0, 300


def _state(sd, seed):
    rng = np.random.default_rng(seed)
    st = np.empty(3 * N)
    st[0::3] = rng.uniform(0.0, L, N)
    st[1::3] = rng.uniform(0.0, L, N)
    st[2::3] = rng.uniform(-np.pi, np.pi) + 2 * np.pi * rng.integers(0, 20) + sd * rng.normal(size=N)
    return st


def _separation(st, dtype=np.float64):
    """|r_j - r_i| of the first ROWS particles i (rows) and all j, and j != i."""
    d = []
    for c in (0, 1):
        x = st[c::3].astype(dtype)
        v = x[None, :] - x[:ROWS, None]
        d.append(v - np.round(v.astype(np.float64)) * L)
    return np.sqrt(d[0] ** 2 + d[1] ** 2), np.arange(N)[None, :] != np.arange(ROWS)[:, None]


def _errors(got, st, inside, alpha, weight=None, wide_weight=None):
    """Mean errors of the rates `got` and of the reference's formula."""
    phi = st[2::3]
    diff = phi[None, :] - phi[:ROWS, None] - alpha
    wide = phi.astype(np.longdouble)[None, :] - phi.astype(np.longdouble)[:ROWS, None] - np.longdouble(alpha)
    t, e = np.sin(diff), np.sin(wide)
    if weight is not None:
        t, e = t * weight, e * wide_weight
    n = inside.sum(1)
    ref = np.cumsum(np.where(inside, t, 0.0), axis=1)[:, -1] / n
    exact = np.where(inside, e, 0.0).sum(1) / n
    return np.abs(got[:ROWS] - exact).mean(), np.abs(ref - exact).mean()


@pytest.mark.parametrize("form", ["tile", "lane", "verlet", "allpairs"])
@pytest.mark.parametrize("alpha", [0.0, 0.02, -0.3])
@pytest.mark.parametrize("sd", [3e-4, 1e-3, 1e-2, 1e-1])
def test_rates_are_as_close_as_the_reference_formula(sd, alpha, form):
    rho = 0.3 if form == "allpairs" else 0.249
    mine = theirs = 0.0
    for seed in range(3):
        st = _state(sd, seed)
        p = abi.make_params(L=L, v0=0.01, sigma=1.0, rho=rho, alpha=alpha, D_phi=0.02, stepper=abi.STEPPER_SRK,
                            skin=0.05, neighbour=abi.NEIGHBOUR_VERLET if form == "verlet" else abi.NEIGHBOUR_CELL)
        with abi.System(N, p) as s:
            if form in ("tile", "lane"):
                s.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9 if form == "lane" else 0)
            s.upload_state(st)
            rates = s.rhs_srk()[0][2::3]
        r, other = _separation(st)
        a, b = _errors(rates, st, other & (r <= rho), alpha)
        mine, theirs = mine + a, theirs + b
    assert mine <= 1.6 * theirs


@pytest.mark.parametrize("sd", [3e-4, 1e-3, 1e-2, 1e-1])
def test_vortex_arrays(sd):
    prm = dict(velocity=0.1, mu_plus=1.0, mu_minus=1.0, xi_a=0.249, xi_r=0.0, D_phi=0.01, kappa=1.0, rho=0.249)
    mine = theirs = 0.0
    for seed in range(3):
        st = _state(sd, 10 + seed)
        with abi.System(N, abi.make_va_params(L=L, stepper=abi.STEPPER_SRK, **prm)) as s:
            s.upload_state(st)
            rates = s.rhs_srk()[0][2::3]
        r, other = _separation(st)
        w, _ = _separation(st, np.longdouble)
        x2, w2 = prm["xi_a"] * prm["xi_a"], np.longdouble(prm["xi_a"]) ** 2
        a, b = _errors(rates, st, other & (r <= prm["rho"]), 0.0, 1.0 - r * r / x2, 1.0 - w * w / w2)
        mine, theirs = mine + a, theirs + b
    assert mine <= 1.6 * theirs


def test_kernels_give_the_same_bits():
    """Cell tiles, and four lanes and one per particle (by the batch's size)."""
    st = _state(2e-3, 30)
    p = abi.make_params(L=L, v0=0.01, sigma=1.0, rho=0.249, alpha=0.01, D_phi=0.02, stepper=abi.STEPPER_SRK)
    out = []
    for sparse in (0, 1e9):
        with abi.System(N, p) as s:
            s.set_tuning(abi.TUNE_SPARSE_BELOW, sparse)
            s.upload_state(st)
            s.step(0.01, 3)
            out.append(s.download_state())
    big = abi.make_params(L=5.0, v0=0.01, sigma=1.0, rho=0.1, alpha=0.0, D_phi=0.02, stepper=abi.STEPPER_SRK,
                          system_id=1)
    rng = np.random.default_rng(4)
    other = rng.uniform(0.0, 5.0, 3 * 40000)
    with abi.Batch(abi.STEPPER_SRK, abi.PRECISION_FP64, 2, N + 40000,
                   abi.cells_of(L, 0.249) + abi.cells_of(5.0, 0.1)) as b:
        b.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9)
        slot = b.admit(N, p, st)
        b.admit(40000, big, other)
        b.step(0.01, 3)
        out.append(b.download(slot))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
