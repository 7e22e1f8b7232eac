"""FP32C cell tiles over thousands of neighbours of one phase.  Every term of a
particle of that phase cancels in the sums of cosines and sines, so what is left
shows the rounding of the sums: a digit form keeps a cosine or sine to 2^-36 and
the sums exactly, and turning a sum into two floats, the products and their sum
keep 2^-45 of it.  The mean is within 2^-36 (|cos| + |sin|) + 2^-43 < 2^-35.4 of
zero however many neighbours there are."""
import numpy as np
import pytest

from spc2_langevin_integration_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units", [False, True])
@pytest.mark.parametrize("n", [500, 2040, 3001, 6007, 20011])
def test_equal_phases_do_not_turn(n, units):
    rng = np.random.default_rng(n)
    for phi in rng.uniform(-np.pi, np.pi, 4):
        st = np.empty(3 * n)
        st[0::3] = rng.uniform(0.05, 0.2, n)
        st[1::3] = rng.uniform(0.05, 0.2, n)
        st[2::3] = phi
        p = abi.make_params(L=1.0, v0=0.01, sigma=1.0, rho=0.249, alpha=0.0, D_phi=0.02, stepper=abi.STEPPER_SRK,
                            precision=abi.PRECISION_FP32C)
        with abi.System(n, p) as s:
            if units:
                s.set_tuning(abi.TUNE_CELL_UNITS, 1)
            s.upload_state(st)
            rates, _ = s.rhs_srk()
        assert np.abs(rates[2::3]).max() <= 2.0 ** -35.4
