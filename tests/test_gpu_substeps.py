"""The kernels of the mixed form's linear ENE/MIX sub-steps against the oracle and against one
another: the one on a thread-block cluster a member and the grid-barrier kernels that such a
grid has otherwise (which of them a call launches is checked in test_launches.py)."""
import numpy as np
import pytest

from harness import ACC_2D
from test_gpu_parity import _spg_compare, _spg_pair

pytestmark = pytest.mark.gpu
CASES = [dict(), dict(nvor_scheme=5), dict(ln_bt_fw=0), dict(nn_bt_flt=2), dict(ln_bt_av=0), dict(nn_bt_flt=0)]


def three_calls(case, cluster, oracle, **shape):
    p = _spg_pair("mixed", case, **shape)
    p.ctx.set_spg_cluster(cluster)
    for kt in (5, 6, 7):
        for o in p.ora if oracle else ():
            o.dyn_spg_ts(kt)
        p.ctx.dyn_spg_ts(kt)
        p.ctx.synchronize()
    if oracle:
        _spg_compare(p, "mixed")
    out = {n: np.asarray(p.ctx.to_host(p.dev[n], p.s2)) for n in ACC_2D}
    out.update({n: np.asarray(p.ctx.to_host(p.dev[n], p.s3)) for n in ("UA", "VA", "UN", "VN")})
    return out


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("nn,nmem", [(1, 2), (4, 1), (5, 3), (7, 1)])
def test_cluster_and_grid_barrier_kernels(case, nn, nmem):
    """Members on one block and on clusters with one, two and four points a thread: the bits
    of k_spg_p2_ene; both checked against the oracle at the smallest grid of each kind."""
    a = three_calls(case, 2, True, nn=nn, nmem=nmem)
    b = three_calls(case, 0, nn in (1, 4), nn=nn, nmem=nmem)
    for n in a:
        assert np.array_equal(a[n], b[n]), n


@pytest.mark.parametrize("case", [dict(), dict(nvor_scheme=5), dict(ln_bt_av=0), dict(ln_bt_fw=0)])
def test_cluster_and_general_kernel_of_many_members(case):
    """More members than the combined constants serve: the bits of k_spg_p2 without its
    constant cache."""
    case = dict(case, sample=[0, 79])
    a = three_calls(case, 2, True, nn=3, nmem=80)
    b = three_calls(case, 0, False, nn=3, nmem=80)
    for n in a:
        assert np.array_equal(a[n], b[n]), n
