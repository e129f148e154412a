"""Several contexts of one process: what a kernel is set up with on the device does not
depend on which context was used last."""
import threading

import pytest

from harness import Pair

pytestmark = pytest.mark.gpu


def column_physics(jpk, prec):
    """A context with the fields of zdf_phy, dyn_zdf and dyn_nxt bound."""
    from test_zdf_tke import TKE, VFIELDS, vphys_state
    p = Pair(nn=1, prec=prec, seed=47, jpk=jpk, **TKE)
    p.states = [vphys_state(p.dom, p.nam, st) for st in p.states]
    p.bind_hotpath()
    for n in VFIELDS:
        p.bind(n)
    return p


@pytest.mark.parametrize("prec,few,many", [("mixed", 31, 60), ("fp64", 46, 62)])
def test_column_kernels_of_two_threads(prec, few, many):
    """A context with few levels beside one with many, each on a thread of its own: the
    column kernels of both keep the shared memory that they need."""
    errors = []
    ctxs = [column_physics(k, prec).ctx for k in (few, many)]

    def work(c):
        try:
            for _ in range(1500):
                c.zdf_phy(3)
                c.dyn_zdf_step(3)
                c.dyn_nxt(3)
            c.synchronize()
        except Exception as e:  # the thread's failure is the test's
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(c,)) for c in ctxs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
