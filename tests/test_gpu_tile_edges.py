"""Kernels that work on tiles or chunks of levels, against the oracle at sizes on both
sides of a tile's edge, with remainders of columns, rows and levels."""
import numpy as np
import pytest

import adj_cases
from adj_cases import Case, GpuCase
from nemo_gpu import gyre, shelf
from harness import Pair, relerr

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


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nn,jpk,flat", [(2, 9, True), (8, 18, True), (8, 18, False), (17, 26, True)])
def test_level_march(prec, nn, jpk, flat):
    """The momentum trends and the time stepping of velocities and tracers with 1 to 32
    levels a thread (by the grid's size), with 1-D and with 3-D scale factors. Tolerances
    of the routines' own parity tests."""
    dom = gyre.domain(nn, jpk=jpk)
    rng = np.random.default_rng(9)
    if not flat:
        f = 1.0 + 0.1 * rng.random((dom["jpi"], dom["jpj"], 1))
        for n in "tuvwf":
            dom[f"e3{n}_0"] = np.asfortranarray(dom[f"e3{n}_0"] * f)
    p = Pair(dom=dom, nam=gyre.namelist(), prec=prec, seed=23)
    st = p.states[0]
    _, um, vm, wm = gyre.masks(dom)
    st["ahmt"], st["ahmf"] = gyre.viscosity(dom)
    st["avm"] = np.asfortranarray(2e-2 * (1.0 + rng.random(p.s3)) * wm)
    st["avm"][:, :, [0, -1]] = 0.0
    st["rhd"] = np.asfortranarray(1e-3 * rng.standard_normal(p.s3))
    p.bind_spg()
    for n in ("AHMT", "AHMF", "AVM", "RHD", "WN", "TSB", "TSN"):
        p.bind(n)
    p.bind("TSA", key="tsn")
    p.set("UA_B", [np.asfortranarray(0.05 * rng.standard_normal(p.s2) * um[:, :, 0])])
    p.set("VA_B", [np.asfortranarray(0.05 * rng.standard_normal(p.s2) * vm[:, :, 0])])
    o, h, c = p.ora[0], p.host[0], p.ctx
    for kvor in (1, 2, 4):
        o.vor_ene(3, kvor, h["UN"], h["VN"], h["UA"], h["VA"])
        c.vor_ene(3, kvor, p.dev["UN"], p.dev["VN"], p.dev["UA"], p.dev["VA"])
    o.dyn_ldf_lap(3, h["UB"], h["VB"], h["UA"], h["VA"], 1)
    c.dyn_ldf_lap(3, p.dev["UB"], p.dev["VB"], p.dev["UA"], p.dev["VA"], 1)
    for f in ("dyn_keg", "dyn_zad", "dyn_hpg"):
        getattr(o, f)(3)
        getattr(c, f)(3)
    c.synchronize()
    t = 1e-12 if prec == "fp64" else 5e-5
    p.compare("UA", p.s3, t)
    p.compare("VA", p.s3, t)
    for f in ("wzv", "dyn_zdf_step", "dyn_nxt", "tra_nxt"):
        getattr(o, f)(3)
        getattr(c, f)(3)
    c.synchronize()
    for n in ("WN", "UA", "VA", "UN", "VN", "UB", "VB"):
        p.compare(n, p.s3, t)
    for n in ("UN_B", "VN_B", "UB_B", "VB_B"):
        p.compare(n, p.s2, t)
    for n in ("TSB", "TSN"):
        p.compare(n, p.s4, t)


@pytest.mark.parametrize("nn,nmem,case", [(1, 3, dict()), (2, 1, dict(ln_bt_av=0)), (3, 2, dict(nvor_scheme=5)),
                                          (4, 5, dict(ln_bt_fw=0)), (5, 1, dict(ln_bt_av=0)), (6, 1, dict()),
                                          (9, 1, dict()), (3, 80, dict(sample=[0, 41, 79]))])
def test_sub_steps_of_a_cluster(nn, nmem, case):
    """The mixed form's linear ENE/MIX sub-steps with a member on one block (nn 1), on
    clusters of several sizes and points a thread, past the largest (nn 9: the grid
    barrier's kernel) and with more members than the combined constants serve (80); three calls, the second and third from the levels of the one before
    without time averaging. Tolerance of the routine's mixed parity tests."""
    from test_gpu_parity import _spg_compare, _spg_pair
    p = _spg_pair("mixed", case, nn=nn, nmem=nmem)
    for kt in (5, 6, 7):
        for o in p.ora:
            o.dyn_spg_ts(kt)
        p.ctx.dyn_spg_ts(kt)
        p.ctx.synchronize()
    _spg_compare(p, "mixed")


def test_sub_steps_of_one_tile_a_block():
    """The variable-volume sub-steps of a shelf whose tiles fit five blocks an SM and not
    four. Tolerance of the routine's mixed parity tests."""
    from test_gpu_parity import _spg_compare
    dom, nam = shelf.domain(421, 363, jpk=8, seed=3), shelf.namelist()
    p = Pair(prec="mixed", dom=dom, nam=nam, states=[shelf.state(dom, nam, seed=4)])
    p.bind_spg()
    p.bind("SSH_IB")
    p.ora[0].dyn_spg_ts(5)
    p.ctx.dyn_spg_ts(5)
    p.ctx.synchronize()
    _spg_compare(p, "mixed")


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("jpi,jpj,jpk", [(43, 37, 19), (64, 33, 33), (45, 17, 5)])
def test_shelf_tracers(prec, jpi, jpj, jpk):
    """The tracer routines of a step with variable volume and partial steps, with and
    without tensor copies (jpi a multiple of 4 or not), at few levels and with
    remainders of chunks. Tolerances of the hot path's parity tests."""
    dom, nam = shelf.domain(jpi, jpj, jpk=jpk, seed=7), shelf.namelist()
    p = Pair(prec=prec, dom=dom, nam=nam, states=[shelf.state(dom, nam, seed=8)])
    p.bind_hotpath()
    for n in ("GTSU", "GTSV", "SSH_IB"):
        p.bind(n)
    for kt in (5, 6):
        p.ora[0].stp_hotpath(kt)
        p.ctx.stp_hotpath(kt)
        p.ctx.synchronize()
    t = 1e-12 if prec == "fp64" else 5e-6
    p.compare("TSA", p.s4, t)
    p.compare("AH_WSLP2", p.s3, t)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_column_physics_of_a_larger_grid(monkeypatch, prec):
    """zdf_phy and ldf_slp with more than one level a thread, by their own parity tests."""
    import test_ldf_slp
    import test_zdf_tke
    real = gyre.domain
    monkeypatch.setattr(gyre, "domain", lambda nn, **k: real(11, jpk=18))
    test_ldf_slp.test_ldf_slp_gpu_matches_oracle(prec)
    for nn_mxl in (0, 2, 3):
        test_zdf_tke.test_gpu_zdf_phy(prec, nn_mxl, 1, 1)


@pytest.mark.parametrize("nk", [1, 7, 62])
@pytest.mark.parametrize("spread", [0, 3, 40])
def test_glob_sum_of_floats(nk, spread):
    """The FP32 sum against the exactly rounded one: values of one binary place, within the
    exact passes' range, and far outside it; a pass of zeros; two members. The compensated
    sum is off by at most n 2^-104 of the sum of magnitudes."""
    import math
    p = Pair(nn=2, prec="mixed", seed=3, nmem=2)
    rng = np.random.default_rng(spread)
    x = rng.standard_normal((2, nk, p.s2[1], p.s2[0])) * 2.0 ** rng.integers(-spread, spread + 1, (2, nk, 1, 1))
    x = x.astype(np.float32)
    if nk > 2:
        x[:, 1] = 0
    t = p.torch.from_numpy(x).cuda()
    p.torch.cuda.synchronize()
    mask = p.ora[0].array("tmask_i", 2).T
    for m, got in enumerate(p.ctx.glob_sum(t, nk)):
        v = (x[m].astype(np.float64) * mask).ravel()
        assert abs(got - math.fsum(v)) <= 2.0**-52 * abs(math.fsum(v)) + 2.0**-85 * np.abs(v).sum()
    bad = x.copy()
    bad[1, 0, 5, 5] = np.inf
    t.copy_(p.torch.from_numpy(bad))
    p.torch.cuda.synchronize()
    out = p.ctx.glob_sum(t, nk)
    assert np.isfinite(out[0]) and not np.isfinite(out[1])


@pytest.mark.parametrize("nn,jpk", [(6, 9), (8, 20), (8, 31)])
def test_ragged_rows(nn, jpk):
    """Rows that are no multiple of 16 bytes long: the tracer planes copied into shared
    memory by the threads. The specialised kernels without shared memory do the same
    operations in the same order, so the results are the same bits; both within the mixed
    tolerance of the oracle. A wait that gives up at once is reported and leaves the
    context usable."""
    from nemo_gpu.api import NemoError
    dom = gyre.domain(nn, jpk=jpk)
    assert dom["jpi"] % 4
    res = []
    for tma in (1, 0):
        p = Pair(dom=dom, nam=gyre.namelist(), prec="mixed", seed=31)
        p.bind_hotpath()
        p.ctx.set_tma(tma)
        for kt in (5, 6):
            p.ora[0].stp_hotpath(kt)
            p.ctx.stp_hotpath(kt)
            p.ctx.synchronize()
        p.compare("TSA", p.s4, 5e-6)
        res.append([np.asarray(p.ctx.to_host(p.dev[n], s)) for n, s in (("TSA", p.s4), ("AH_WSLP2", p.s3))])
    for x, y in zip(*res):
        assert np.array_equal(x, y)
    p.ctx.set_tma(1)
    p.ctx.set_tma_poll_limit(0)
    p.ctx.stp_hotpath(7)
    with pytest.raises(NemoError, match="tensor copy"):
        p.ctx.synchronize()
    p.ctx.set_tma_poll_limit(1 << 16)
    p.ctx.stp_hotpath(8)
    p.ctx.synchronize()


def kinds(x):
    """where x is +inf, -inf and NaN"""
    return np.stack([np.isposinf(x), np.isneginf(x), np.isnan(x)])


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_fct_of_a_value_that_is_not_finite(value):
    """tra_adv_fct with given transports in FP64 on a tracer with one infinite or undefined value:
    what the specialised kernels leave infinite and undefined is what the general ones (a
    bound tape asks for them) do."""
    p = Pair(nn=2, prec="fp64", seed=5)
    st, o, c = p.states[0], p.ora[0], p.ctx
    tb = np.array(st["tsb"], order="F")
    tb[20, 15, 6, 0] = value
    zun, zvn, zwn = o.tra_adv_trp(*[np.array(st[n], order="F") for n in ("un", "vn", "wn")])
    out = []
    for general in (0, 1):
        d = [p.to_dev([x]) for x in (zun, zvn, zwn, tb, st["tsn"], np.zeros(p.s4, order="F"))]
        c.bind("FCT_TAPE", p.to_dev([np.zeros(6 * tb.size // 2)]) if general else None)
        c.tra_adv_fct(5, 1, "TRA", 14400.0, *d, 2, 2, 2)
        out.append(kinds(c.to_host(d[5], p.s4)))
    assert out[1].any() and np.array_equal(*out)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_tracer_adjoints_of_a_value_that_is_not_finite(value):
    """The tracer adjoints of a sensitivity with one infinite or undefined value are infinite
    and undefined where the oracle's are."""
    c = Case("gyre", seed=22)
    g = GpuCase(c)
    c.iso_coefficients()
    g.iso_coefficients()
    kt = c.kit + 2
    lam = c.rand4(masked=False)
    lam[15, 10, 6, 0] = value
    zero = np.zeros(c.s4, order="F")
    rb, ra, tb, ta = zero.copy(order="F"), lam.copy(order="F"), g.dev(zero), g.dev(lam)
    c.o.tra_zdf_imp_adj(kt, c.kit, "TRA", c.p2dt, rb, ra, 2)
    g.ctx.tra_zdf_imp_adj(kt, c.kit, "TRA", c.p2dt, tb, ta, 2)
    pairs = [(rb, tb), (ra, ta)]
    ri, ti = zero.copy(order="F"), g.dev(zero)
    c.o.tra_ldf_iso_adj(kt, c.kit, "TRA", None, None, c.gtsu, c.gtsv, None, None, ri, None, lam, 2, 1)
    g.ctx.tra_ldf_iso_adj(kt, c.kit, "TRA", None, None, g.gtsu, g.gtsv, None, None, ti, None, g.dev(lam), 2, 1)
    pairs.append((ri, ti))
    tape, _ = c.fct_record()
    g.ctx.bind("FCT_TAPE", g.dev(tape))
    fb, fn = g.dev(zero), g.dev(zero)
    g.ctx.tra_adv_fct_adj(kt, c.kit, "TRA", c.p2dt, g.zun, g.zvn, g.zwn, fb, fn, g.dev(lam), 2, 2, 2)
    pairs += zip(c.fct_adj(tape, lam), (fb, fn))
    for ref, got in pairs:
        ref = kinds(ref)
        assert ref.any() and np.array_equal(ref, kinds(g.host(got, c.s4)[0]))


@pytest.mark.parametrize("nn_mxl", [0, 2, 3])
@pytest.mark.parametrize("nmem", [1, 4, 12])
def test_tke_columns_of_many_levels(nmem, nn_mxl):
    """zdf_phy in FP64 with 62 levels and so many columns that four, two and none of a level's
    values stay in shared memory. Tolerance of its own parity test."""
    from test_zdf_tke import OUT, TOL_TKE, tke_pair
    p = tke_pair("fp64", nmem=nmem, jpk=62, nn_mxl=nn_mxl, sample=sorted({0, nmem - 1}))
    for kt in (1, 2):
        for o in p.ora:
            o.zdf_phy(kt)
        p.ctx.zdf_phy(kt)
    p.ctx.synchronize()
    for n in OUT:
        p.compare(n, p.s3, TOL_TKE["fp64"])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("eos", ["seos", "eos80"])
def test_densities_of_a_larger_grid(monkeypatch, prec, eos):
    """The equations of state and bn2 with chunks of several levels a thread and a remainder of
    levels, by their own parity test."""
    import test_eos_hpg
    real = gyre.domain
    monkeypatch.setattr(gyre, "domain", lambda nn, **k: real(5, jpk=16))
    test_eos_hpg.test_gpu_eos_bn2_hpg(prec, eos)


@pytest.mark.parametrize("nmem,nk", [(1, 1), (1, 62), (5, 31), (12, 3)])
def test_glob_sum_of_doubles(nmem, nk):
    """The FP64 sum of one member and of an ensemble (whose members share the blocks) against
    the exactly rounded one; the compensated sum is off by at most n 2^-104 of the sum of
    magnitudes."""
    import math
    p = Pair(nn=2, prec="fp64", seed=3, nmem=nmem, sample=[0])
    x = np.random.default_rng(nk).standard_normal((nmem, nk, p.s2[1], p.s2[0])) * 1e3
    t = p.torch.from_numpy(x).cuda()
    p.torch.cuda.synchronize()
    mask = p.ora[0].array("tmask_i", 2).T
    for m, got in enumerate(p.ctx.glob_sum(t, nk)):
        v = (x[m] * mask).ravel()
        assert abs(got - math.fsum(v)) <= 2.0**-52 * abs(math.fsum(v)) + 2.0**-85 * np.abs(v).sum()


@pytest.mark.parametrize("jpi,jpj,jpk,order", [(302, 202, 31, 2), (302, 202, 31, 4), (332, 222, 18, 4), (320, 220, 31, 4),
                                               (62, 42, 9, 4)])
def test_advection_of_given_transports(jpi, jpj, jpk, order):
    """tra_adv_fct of given transports in the mixed form, 2nd and 4th order in the horizontal,
    at sizes of each instance of its stages. Tolerance of the mixed tracer fields."""
    dom = gyre.domain(int(-(-max((jpi - 2) / 30, (jpj - 2) / 20) // 1)), jpk=jpk)
    dom = {k: (np.asfortranarray(v[:jpi, :jpj]) if isinstance(v, np.ndarray) and v.ndim > 1 else v) for k, v in dom.items()}
    for n in ("k_top", "k_bot"):
        dom[n][0], dom[n][-1], dom[n][:, 0], dom[n][:, -1] = 0, 0, 0, 0
    dom.update(jpi=jpi, jpj=jpj)
    p = Pair(dom=dom, nam=gyre.namelist(), prec="mixed", seed=6)
    st, o, c = p.states[0], p.ora[0], p.ctx
    tr = o.tra_adv_trp(*[np.array(st[n], order="F") for n in ("un", "vn", "wn")])
    tb, tn, ta = (np.array(x, order="F") for x in (st["tsb"], st["tsn"], np.zeros(p.s4)))
    d = [p.to_dev([x]) for x in list(tr) + [tb, tn, ta]]
    o.tra_adv_fct(5, 1, "TRA", 14400.0, *tr, tb, tn, ta, 2, order, 2)
    c.tra_adv_fct(5, 1, "TRA", 14400.0, *d, 2, order, 2)
    e = relerr(14400.0 * ta + tb, 14400.0 * c.to_host(d[5], p.s4) + tb)
    assert e <= 5e-6 and np.abs(ta).max() > 0
