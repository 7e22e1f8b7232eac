"""FP32X with large couplings: the second pass's phase rates keep their 52 bits
at any sigma, so the right-hand sides stay within 1e-12 sigma of FP64's."""
import numpy as np
import pytest

from spc2_langevin_integration_gb300 import abi
from tests._helpers import init_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lane", [False, True])
@pytest.mark.parametrize("sigma", [1.0, 2.0 ** 41, 2.0 ** 43 + 5.0, -3e14, 1e40, 1e200])
def test_second_pass_at_large_sigma(sigma, lane):
    n, L = 3000, 1.5
    st = init_state(n, L, 17)
    out = {}
    for precision in (abi.PRECISION_FP64, abi.PRECISION_FP32X):
        p = abi.make_params(L=L, v0=0.01, sigma=sigma, rho=0.1, alpha=0.4, D_phi=0.02, stepper=abi.STEPPER_SRK,
                            precision=precision)
        with abi.System(n, p) as s:
            s.set_tuning(abi.TUNE_SPARSE_BELOW, 1e9 if lane else 0)
            s.upload_state(st)
            out[precision] = s.rhs_srk()
    for got, want in zip(out[abi.PRECISION_FP32X], out[abi.PRECISION_FP64]):
        assert np.abs(got - want).max() <= 1e-12 * abs(sigma)
