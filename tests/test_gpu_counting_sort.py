"""The counting sort by cell where its launches change: the particles one CTA
places itself (1,024), counters 16 bytes apart (up to 4,096 keys), one CTA's
scan (up to 12,288 keys), and two keys per cell with sub-cells.  Neighbour sets
are the oracle's; sub-cells only order a cell's particles, so the FP32X results
(exact sums) are those without them.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from spc2_langevin_integration_gb300 import abi
from tests._helpers import init_state

pytestmark = pytest.mark.gpu

PRM = dict(v0=0.01, sigma=1.1, alpha=0.8, D_phi=0.01)


@pytest.mark.parametrize("n,nc", [(1023, 10), (1024, 10), (1025, 10), (2047, 10), (2048, 44), (2049, 10), (2000, 110), (2000, 111), (3000, 64), (3000, 65), (3000, 110), (3000, 111)])
def test_neighbour_sets_across_the_sorts_branches(n, nc):
    L, rho = 1.0, 1.0 / (nc + 0.25)
    st = init_state(n, L, 40 + nc)
    off_ref, idx_ref = po.OracleSystem(n, L, rho=rho, **PRM).neighbour_lists(st)
    with abi.System(n, abi.make_params(L=L, rho=rho, stepper=abi.STEPPER_SRK, **PRM)) as s:
        s.upload_state(st)
        for _ in range(2):  # the counters are left clear for the next evaluation
            off, idx = s.neighbours()
            assert np.array_equal(off, off_ref) and np.array_equal(idx, idx_ref)
            s.rhs_srk()


@pytest.mark.parametrize("nc", [45, 46, 78, 79])
def test_sub_cell_keys_give_the_same_sums(nc):
    L, n = 1.0, 20000
    p = abi.make_params(L=L, rho=1.0 / (nc + 0.25), stepper=abi.STEPPER_SRK, precision=abi.PRECISION_FP32X, seed=2, **PRM)
    got = []
    for sub in (0, 1):
        with abi.System(n, p) as s:
            s.set_tuning(abi.TUNE_SPARSE_BELOW, 0)
            s.set_tuning(abi.TUNE_CELL_UNITS, 1)
            s.set_tuning(abi.TUNE_SUBCELLS, sub)
            s.upload_state(init_state(n, L, 50 + nc))
            s.step(0.01, 3)
            got.append(s.download_state())
    assert np.array_equal(got[0], got[1])
