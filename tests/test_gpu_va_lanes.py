"""The vortex-arrays passes at the sizes where their lane layouts change: a
system alone (four lanes per particle) against the same in a batch of 30,000
(one lane), bitwise; rows of more words than a lane lists; all pairs; a cohesion
cutoff beyond the alignment cutoff; and the oracle's right-hand sides within the
model's 1e-11 of the largest value."""
import numpy as np
import pytest

from oracle import pyoracle as po
from spc2_langevin_integration_gb300 import abi
from tests._helpers import init_state

pytestmark = pytest.mark.gpu

PRM = dict(velocity=0.1, mu_plus=20.0, mu_minus=10.0, xi_a=0.05, xi_r=0.03, D_phi=0.01, kappa=5.0, rho=0.12)


@pytest.mark.parametrize("n,L,spread,kw", [
    (33, 1.2, 1.2, {}), (1500, 1.2, 1.2, {}), (1200, 2.0, 0.3, {}),  # up to 1,200 in a few cells
    (1, 0.4, 0.4, {}), (31, 0.4, 0.4, {}), (700, 0.4, 0.4, {}),      # all pairs (rho > L / 4)
    (600, 1.2, 1.2, dict(xi_r=0.2)),                                 # cohesion beyond rho
    (600, 0.5, 0.5, dict(xi_r=0.14)),                                # and beyond L / 4
])
def test_lane_layouts_and_oracle(n, L, spread, kw):
    prm = dict(PRM, **kw)
    st = init_state(n, spread, 800 + n)
    p = abi.make_va_params(L=L, stepper=abi.STEPPER_SRK, seed=3, system_id=1, **prm)
    with abi.System(n, p) as s:
        s.upload_state(st)
        d, a = s.rhs_srk()
        s.step(0.002, 3)
        alone = s.download_state()
    ref_d, ref_a = po.OracleVortexArrays(n, L, **prm).rhs_srk(st)[:2]
    for got, ref in ((d, ref_d), (a[0::2], ref_a[0::2]), (a[1::2], ref_a[1::2])):
        assert np.abs(got - ref).max() <= 1e-11 * max(np.abs(ref).max(), 1e-300)
    big = abi.make_va_params(L=6.0, stepper=abi.STEPPER_SRK, seed=3, system_id=2, **PRM)
    with abi.Batch(abi.STEPPER_SRK, abi.PRECISION_FP64, 2, n + 30000, abi.cells_of(L, p.rho) + 2500) as b:
        slot = b.admit(n, p, st)
        b.admit(30000, big, init_state(30000, 6.0, 9))
        b.step(0.002, 3)
        assert np.array_equal(b.download(slot), alone)
