"""Vortex arrays where the pair terms' shortcuts end: a copy that wraps to
exactly L, whose distance to x = 0 is L by the reference's minimum image
(PeriodicBoundaryConditions.cpp:22-35) and not 0; and separations down to those
whose squares are subnormal, where the reference's bearing is still atan2's."""
import numpy as np
import pytest

from oracle import pyoracle as po
from spc2_langevin_integration_gb300 import abi
from tests._helpers import init_state

pytestmark = pytest.mark.gpu

PRM = dict(velocity=0.1, mu_plus=20.0, mu_minus=10.0, xi_a=0.05, xi_r=0.03, D_phi=0.01, kappa=5.0, rho=0.12)
SIZES = [(400, 1.2), (21000, 8.4)]  # four lanes per particle and one


def _rhs(n, L, st):
    """Right-hand sides as (derivative, first and second additional terms), ours
    and the oracle's."""
    p = abi.make_va_params(L=L, stepper=abi.STEPPER_SRK, seed=3, **PRM)
    with abi.System(n, p) as s:
        s.upload_state(st)
        d, a = s.rhs_srk()
    ref_d, ref_a = po.OracleVortexArrays(n, L, **PRM).rhs_srk(st)[:2]
    return (d, ref_d), (a[0::2], ref_a[0::2]), (a[1::2], ref_a[1::2])


@pytest.mark.parametrize("n,L", SIZES)
@pytest.mark.parametrize("axes", [(0,), (1,), (0, 1)])
def test_pair_across_the_whole_box(axes, n, L):
    st = init_state(n, L, 5)
    for c in (0, 1):
        st[c:12:3] = 0.31
    for c in axes:  # the copy of the first one wraps to L
        st[c:12:3] = [-1e-17, 0.0, 0.004, L - 0.003]
    for got, ref in _rhs(n, L, st):
        # 0 / 0 where the oracle has it too: two of them at distance 0
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        ok = ~np.isnan(ref)
        assert np.abs(got - ref)[ok].max() <= 1e-11 * np.abs(ref[ok]).max()


@pytest.mark.parametrize("n,L", SIZES)
@pytest.mark.parametrize("r", [1e-9, 1e-15, 1e-30, 1e-120, 1e-135, 1e-136, 1e-150, 1e-153, 1e-155, 1e-160, 1e-162])
def test_close_pair(r, n, L):
    st = init_state(n, L, 5)
    st[0:6:3] = [0.0, r]  # the positions next to 0 resolve such distances
    st[1:6:3] = [0.0, 0.5 * r]
    st[2:6:3] = [0.3, 1.1]
    for got, ref in _rhs(n, L, st):
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        # the two themselves turn at a rate of one over their distance (whose
        # square holds only a few bits when it is subnormal)
        pair = np.abs(ref) > 1e6
        pair[pair.size // n * 2:] = False
        if r > 1e-150:
            assert np.abs(got - ref)[pair].max(initial=0.0) <= 1e-11 * np.abs(ref[pair]).max(initial=0.0)
        else:
            assert np.abs(np.log2(np.abs(got[pair] / ref[pair]))).max(initial=0.0) <= 1.0
        ok = ~np.isnan(ref) & ~pair
        assert np.abs(got - ref)[ok].max() <= 1e-11 * np.abs(ref[ok]).max()
