"""Kernels that work on tiles or chunks of levels, against the oracle at sizes on both
sides of a tile's edge, with remainders of columns, rows and levels."""
import numpy as np
import pytest

import adj_cases
from adj_cases import Case, GpuCase
from harness import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jpi,jpj,jpk", [(30, 14, 9), (32, 17, 10), (61, 29, 18), (91, 43, 25)])
def test_tracer_adjoints(monkeypatch, jpi, jpj, jpk):
    """FCT 2/2 (tiles of 30 x 14 columns and 8 levels), iso-neutral and vertical diffusion:
    FP64 with the oracle's expressions, so the tolerance of the FP64 parity tests."""
    real = adj_cases.shelf.domain
    monkeypatch.setattr(adj_cases.shelf, "domain", lambda *a, **k: real(jpi, jpj, jpk=jpk, seed=5, e1=1000.0))
    c = Case("shelf", seed=16)
    g = GpuCase(c)
    kt, tol = c.kit + 2, 1e-12
    tape, _ = c.fct_record()
    lam = c.rand4(masked=False)
    g.ctx.bind("FCT_TAPE", g.dev(tape))
    tb_ad, tn_ad = g.dev(np.zeros(c.s4, order="F")), g.dev(np.zeros(c.s4, order="F"))
    g.ctx.tra_adv_fct_adj(kt, c.kit, "TRA", c.p2dt, g.zun, g.zvn, g.zwn, tb_ad, tn_ad, g.dev(lam), 2, 2, 2)
    for ref, got in zip(c.fct_adj(tape, lam), (tb_ad, tn_ad)):
        assert relerr(ref, g.host(got, c.s4)[0]) <= tol
    g.ctx.bind("FCT_TAPE", None)
    c.iso_coefficients()
    g.iso_coefficients()
    rtb, tb_ad = np.zeros(c.s4, order="F"), g.dev(np.zeros(c.s4, order="F"))
    c.o.tra_ldf_iso_adj(kt, c.kit, "TRA", None, None, c.gtsu, c.gtsv, None, None, rtb, None, lam, 2, 1)
    g.ctx.tra_ldf_iso_adj(kt, c.kit, "TRA", None, None, g.gtsu, g.gtsv, None, None, tb_ad, None, g.dev(lam), 2, 1)
    assert relerr(rtb, g.host(tb_ad, c.s4)[0]) <= tol
    rtb, rta = np.zeros(c.s4, order="F"), lam.copy(order="F")
    tb_ad, ta_ad = g.dev(rtb), g.dev(lam)
    c.o.tra_zdf_imp_adj(kt, c.kit, "TRA", c.p2dt, rtb, rta, 2)
    g.ctx.tra_zdf_imp_adj(kt, c.kit, "TRA", c.p2dt, tb_ad, ta_ad, 2)
    assert relerr(rtb, g.host(tb_ad, c.s4)[0]) <= tol and relerr(rta, g.host(ta_ad, c.s4)[0]) <= tol
