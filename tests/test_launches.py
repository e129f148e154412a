"""What the library launches, checked without a GPU over a stand-in for the CUDA runtime."""
import fakedev
import pytest


def test_shared_memory_on_a_second_device():
    """A process with contexts on two devices: each kernel that needs more than 48 KB of
    shared memory is opted in on both."""
    out = fakedev.run(r"""
seen = []
for device in (0, 1):
    fake.cudaSetDevice(device)
    for prec, jpk, order, fused in (("mixed", 31, 2, 0), ("mixed", 31, 2, 1), ("mixed", 64, 4, 0), ("fp64", 64, 4, 0)):
        dom = gyre.domain(1, jpk=jpk)
        c = Ctx(dom, gyre.namelist(), prec, nmem=140 if fused else 1)  # enough columns for each form of tra_zdf
        c.bind("AVT", "AH_WSLP2", "AKZ", "TSB", "TSN", "TSA", "UN", "VN", "WN", "USLP", "VSLP", "WSLPI", "WSLPJ")
        c.bind("UA", "VA", "UB", "VB", "SSHN", "SSHB", "UN_B", "VN_B", "UB_B", "VB_B", "UTAU", "VTAU", "EMP", "RCDU_BOT",
               "SSHA", "UA_B", "VA_B", "UN_ADV", "VN_ADV", "UB2_B", "VB2_B", "UN_BF", "VN_BF")
        c("set_fct_fused", fused)
        t = [c.array(2 * c.n3) for _ in range(6)]
        launches()
        c("tra_adv_fct", 10, 1, b"TRA", 14400.0, *t, 2, order, order)
        c("tra_zdf_imp", 10, 1, b"TRA", 14400.0, t[3], t[5], 2)
        if order == 2:
            c("stp_hotpath", 10)
        seen += [[device, k[0]] for k in launches() if k[-1] > 48 * 1024]
        c.close()
print(json.dumps(seen))
""")
    first, second = ({k for d, k in out if d == dev} for dev in (0, 1))
    assert first == second
    for k in ("k_fct_b_tma", "k_fct_fused_tma", "k_interp4IdE", "k_zdf_imp_async", "k_zdf_imp32"):
        assert any(k in name for name in second), k


def test_sub_step_kernels():
    """The sub-step kernel of a call by the cluster setting: 0 the grid-barrier kernel (with
    the constants combined, or with many members in the general form without its cache), 2
    the cluster kernel with one, two and four points a thread, or in its general form."""
    out = fakedev.run(r"""
seen = []
for nn, nmem in ((1, 2), (4, 1), (5, 3), (7, 1), (3, 80)):
    for mode in (0, 2):
        c = Ctx(gyre.domain(nn, jpk=4), gyre.namelist(), "mixed", nmem)
        c.bind("UA", "VA", "UB", "VB", "UN", "VN", "SSHN", "SSHB", "UN_B", "VN_B", "UB_B", "VB_B", "UTAU", "VTAU", "EMP",
               "RCDU_BOT", "SSHA", "UA_B", "VA_B", "UN_ADV", "VN_ADV", "UB2_B", "VB2_B", "UN_BF", "VN_BF")
        c("set_spg_cluster", mode)
        launches()
        c("dyn_spg_ts", 10)
        seen.append([k[0] for k in launches() if "spg_p2" in k[0]])
        c.close()
print(json.dumps(seen))
""")
    want = ["k_spg_p2_ene", "k_spg_p2_resILi512ELi1ELb0E", "k_spg_p2_ene", "k_spg_p2_resILi512ELi2ELb0E", "k_spg_p2_ene",
            "k_spg_p2_resILi512ELi4ELb0E", "k_spg_p2_ene", "k_spg_p2_resILi512ELi4ELb0E", "k_spg_p2IfLb0ELi4E",
            "ELb1EEEvNS_3DomIfEENS_7SpgArgsIfEEii"]
    assert [len(x) for x in out] == [1] * len(want)
    assert all(w in x[0] for w, x in zip(want, out)), out


def test_rule_of_the_cluster_kernel():
    """With four points a thread the cluster kernel only takes calls whose sub-steps are
    enough to pay its start; with fewer points a thread it takes all."""
    out = fakedev.run(r"""
seen = []
for jpi, jpj, nmem, nb in ((212, 142, 1, 6), (212, 142, 1, 60), (182, 122, 3, 6), (182, 122, 3, 60), (152, 102, 12, 6), (62, 42, 1, 6)):
    dom = gyre.domain((jpi - 2) // 30, jpk=4)
    c = Ctx(dom, gyre.namelist(ln_bt_auto=0, nn_baro=nb), "mixed", nmem)
    c.bind("UA", "VA", "UB", "VB", "UN", "VN", "SSHN", "SSHB", "UN_B", "VN_B", "UB_B", "VB_B", "UTAU", "VTAU", "EMP",
           "RCDU_BOT", "SSHA", "UA_B", "VA_B", "UN_ADV", "VN_ADV", "UB2_B", "VB2_B", "UN_BF", "VN_BF")
    launches()
    c("dyn_spg_ts", 10)
    seen.append(["spg_p2_res" in k[0] for k in launches() if "spg_p2" in k[0]])
    c.close()
print(json.dumps(seen))
""")
    assert out == [[False], [True], [False], [True], [True], [True]]


def test_rule_of_five_blocks_an_sm():
    """The variable-volume sub-steps take the instance for five blocks an SM where one round
    of tiles then takes the place of two, and the second of four blocks an SM is not nearly
    empty; elsewhere four."""
    out = fakedev.run(r"""
seen = []
for jpi, jpj in ((421, 363), (288, 552), (449, 328), (672, 228), (321, 449), (577, 316), (669, 465), (366, 508)):
    dom = shelf.domain(jpi, jpj, jpk=4, seed=3)
    c = Ctx(dom, shelf.namelist(), "mixed")
    c.bind("UA", "VA", "UB", "VB", "UN", "VN", "SSHN", "SSHB", "UN_B", "VN_B", "UB_B", "VB_B", "UTAU", "VTAU", "EMP",
           "RCDU_BOT", "SSHA", "UA_B", "VA_B", "UN_ADV", "VN_ADV", "UB2_B", "VB2_B", "UN_BF", "VN_BF", "SSH_IB", "SSH_IBB",
           "E3T_B", "E3T_N", "E3T_A", "E3U_N", "E3V_N", "E3W_N", "E3F_N", "HT_N", "HU_N", "HV_N", "R1_HU_N", "R1_HV_N",
           "HU_B", "HV_B", "R1_HU_B", "R1_HV_B")
    launches()
    c("dyn_spg_ts", 10)
    seen.append(["Li5E" in k[0] for k in launches() if "spg_p2" in k[0]])
    c.close()
print(json.dumps(seen))
""")
    assert out == [[True], [True], [False], [False], [False], [True], [False], [False]]


def test_forms_of_the_tke_columns():
    """FP64 zdf_phy: four, two or none of a level's values in shared memory, by which needs
    the fewest rounds of blocks."""
    out = fakedev.run(r"""
seen = []
for nmem in (1, 4, 12):
    c = Ctx(gyre.domain(2, jpk=62), gyre.namelist(ln_zdftke=1, ln_zdfevd=1), "fp64", nmem)
    c.bind("UB", "VB", "UN", "VN", "AVM_K", "AVT_K", "AVM", "AVT", "EN", "DISSL", "RN2", "RN2B", "TAUM", "GDEPW_N")
    launches()
    c("zdf_phy", 3)
    seen.append([k[0] for k in launches() if "zdf_tke" in k[0]])
    c.close()
print(json.dumps(seen))
""")
    assert ["Li4E" in out[0][0], "Li2E" in out[1][0], "Li0E" in out[2][0]] == [True] * 3, out


def test_work_memory_of_the_vertical_physics():
    """zdf_phy in the mixed form keeps one work array, the shear production; the FP64 form
    the system of the columns beside it."""
    out = fakedev.run(r"""
seen = []
for prec, b in (("mixed", 4), ("fp64", 8)):
    c = Ctx(gyre.domain(2), gyre.namelist(ln_zdftke=1, ln_zdfevd=1), prec, 3)
    c.bind("UB", "VB", "UN", "VN", "AVM_K", "AVT_K", "AVM", "AVT", "EN", "DISSL", "RN2", "RN2B", "TAUM", "GDEPW_N")
    before = fake.fake_held()
    c("zdf_phy", 3)
    c("zdf_phy", 4)
    seen.append((fake.fake_held() - before) / (b * c.n3 * 3))
    c.close()
print(json.dumps(seen))
""")
    assert out == [1.0, 5.0]


def test_chunks_of_the_fct_adjoint():
    """The FCT adjoint's levels a chunk: one on a tiny grid, so that a call waits for one level,
    eight on a large one."""
    out = fakedev.run(r"""
seen = []
for nn in (1, 3, 8):
    c = Ctx(gyre.domain(nn), gyre.namelist(), "fp64")
    c.bind("FCT_TAPE")
    t = [c.array(2 * c.n3) for _ in range(6)]
    launches()
    c("tra_adv_fct_adj", 10, 1, b"TRA", 14400.0, *t, 2, 2, 2)
    seen += [[k[1], k[2], k[3]] for k in launches() if "k_fct_adj2" in k[0]]
    c.close()
print(json.dumps(seen))
""")
    assert out == [[2, 2, 30], [4, 5, 8], [9, 12, 4]]


def test_rule_of_the_vertical_diffusion():
    """tra_zdf_imp in the mixed form with 31 levels: a block a row of columns where those
    blocks are few for the rounds that one thread a column would take."""
    out = fakedev.run(r"""
seen = []
for nn, nmem in ((2, 1), (6, 1), (7, 1), (9, 1), (10, 1), (14, 1), (1, 60), (2, 20)):
    c = Ctx(gyre.domain(nn), gyre.namelist(), "mixed", nmem)
    c.bind("AVT", "AH_WSLP2", "AKZ")
    t = [c.array(2 * c.n3) for _ in range(2)]
    launches()
    c("tra_zdf_imp", 10, 1, b"TRA", 14400.0, *t, 2)
    seen += ["async" in k[0] for k in launches() if "zdf_imp" in k[0]]
    c.close()
print(json.dumps(seen))
""")
    assert out == [False, False, True, True, False, True, True, True]


def test_instances_of_the_advection():
    """tra_adv_fct in the mixed form with given transports: stage a for six, seven or eight
    blocks an SM by the rounds that the grid takes, stage b with copied planes but where its
    second round is the plain kernel's first."""
    out = fakedev.run(r"""
seen = []
def domain(jpi, jpj):
    dom = gyre.domain(-(-max((jpi - 2) // 30, (jpj - 2) // 20) // 1) + 1)
    import numpy as np
    dom = {k: (np.asfortranarray(v[:jpi, :jpj]) if isinstance(v, np.ndarray) and v.ndim > 1 else v) for k, v in dom.items()}
    dom.update(jpi=jpi, jpj=jpj)
    return dom
for jpi, jpj, h in ((200, 151, 4), (302, 202, 4), (480, 320, 4), (320, 220, 4), (352, 260, 4), (250, 180, 2), (302, 202, 2)):
    c = Ctx(domain(jpi, jpj), gyre.namelist(), "mixed")
    t = [c.array(2 * c.n3) for _ in range(6)]
    launches()
    c("tra_adv_fct", 10, 1, b"TRA", 14400.0, *t, 2, h, 2)
    seen.append([k[0][:40] for k in launches() if "fct_" in k[0]][:2])
    c.close()
print(json.dumps(seen))
""")
    a = ["Lb0ELi6E", "Lb0ELi7E", "Lb0ELi8E", "Lb0ELi8E", "Lb0ELi6E", "Lb0ELb1ELi6E", "Lb0ELb1ELi8E"]
    b = ["tma", "fct_bI", "tma", "fct_bI", "tma", "fct_b_hot", "fct_b_hot"]
    assert all(x in k[0] and y in k[1] for x, y, k in zip(a, b, out)), out


def test_autotune_of_kernels_without_a_height():
    """nemo_gpu_autotune with timings that get shorter from one candidate to the next: it picks
    the last for the kernels that have a block height, and leaves those whose form in the
    configuration has none (the vertical diffusion of a small grid, and with tensor copies the
    tracer fluxes) as they are."""
    out = fakedev.run(r"""
seen = []
for nn in (1, 9):
    c = Ctx(gyre.domain(nn), gyre.namelist(), "mixed")
    c.bind("AVT", "AH_WSLP2", "AKZ", "TSB", "TSN", "TSA", "UN", "VN", "WN", "USLP", "VSLP", "WSLPI", "WSLPJ", "UA", "VA",
           "UB", "VB", "SSHN", "SSHB", "UN_B", "VN_B", "UB_B", "VB_B", "UTAU", "VTAU", "EMP", "RCDU_BOT", "SSHA", "UA_B",
           "VA_B", "UN_ADV", "VN_ADV", "UB2_B", "VB2_B", "UN_BF", "VN_BF")
    c("autotune", 10, 1)
    ty = (C.c_int * 64)()
    c("get_launch_shape", ty, 64)
    from nemo_gpu._ffi import K
    seen.append([ty[K[n]] for n in ("ZDF_IMP", "ISO_FLUX", "FCT_C", "SPG_P3")])
    c.close()
print(json.dumps(seen))
""")
    assert out == [[4, 4, 1, 1], [1, 4, 1, 1]]


def test_graph_after_work_arrays_grow():
    """A call with more tracers than before replaces the work arrays that a captured step points
    at; the next step is captured again, with what its own vertical scheme needs."""
    out = fakedev.run(r"""
seen = []
for routine, over in (("tra_adv_fct", {}), ("tra_adv_fct", dict(nn_fct_v=4)), ("tra_ldf_iso", {}),
                      ("tra_ldf_blp", dict(ln_traldf_lap=0, ln_traldf_blp=1, ln_traldf_iso=0, rn_aht_0=1.e11))):
    c = Ctx(gyre.domain(1, jpk=6), gyre.namelist(**over), "fp64")
    c.bind(*HOTPATH)
    t = [c.array(3 * c.n3) for _ in range(6)]
    for kt in (10, 11):
        launches()
        c("stp_hotpath", kt)
        seen.append([k[0] for k in launches()])
    for n in (2, 3):
        if routine == "tra_adv_fct":
            c(routine, 12, 1, b"TRC", 14400.0, *t, n, 2, 2)
        elif routine == "tra_ldf_iso":
            c(routine, 12, 1, b"TRC", None, None, None, None, None, None, t[0], t[0], t[1], n, 1)
        else:
            c(routine, 12, 1, b"TRC", None, None, None, None, None, None, t[0], t[1], n, 20)
        launches()
        c("stp_hotpath", 13)
        seen.append([k[0] for k in launches()])
    c.close()
print(json.dumps(seen))
""")
    for first, second, same, more in (out[:4], out[4:8], out[8:12], out[12:]):
        assert len(first) > 5 and first[-1] == "graph" and second == ["graph"] and same == ["graph"]
        assert more == first


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("fields", ["FULL_3D + gyre.FULL_2D", "FULL_3D[1:] + gyre.FULL_2D"])
def test_model_step_captured_first(prec, fields):
    """The first step asked of a context is a captured one: the closure's and the slopes' work
    arrays are made before the capture."""
    out = fakedev.run(f"""
dom, base = gyre.domain(1), gyre.namelist()
c = Ctx(dom, gyre.full_physics(dom, base, gyre.state(dom, base, seed=5))[0], "{prec}")
c.bind(*HOTPATH, "NMLN", *(n.upper() for n in gyre.{fields}))
c("stp_model", 10)
first = [k[0] for k in launches()]
c("stp_model", 11)
print(json.dumps([first, [k[0] for k in launches()]]))
""")
    # the forcing's scalars are put ahead of the graph
    assert out[0][-1] == "graph" and len(out[1]) == 2 and "usr_put" in out[1][0] and out[1][1] == "graph"
    assert ("FULL_3D[" in fields) == (not any("zdf_sh2" in k for k in out[0]))


@pytest.mark.parametrize("routine,arrays", [("tra_adv_fct", 6), ("tra_ldf_iso", 3), ("tra_ldf_blp", 1),
                                            ("tra_ldf_iso_adj", 4), ("dia_hsb_init", 4)])
def test_device_memory_runs_out(routine, arrays):
    """A call that has not the memory for its work arrays is refused and keeps none of them; a
    smaller call after it has all of its own, and so has the same call once there is memory."""
    out = fakedev.run(rf"""
c = Ctx(gyre.domain(1, jpk=6), gyre.namelist(), "fp64")
c.bind(*HOTPATH)
t = [c.array(3 * c.n3) for _ in range(6)]
call = dict(
    tra_adv_fct=lambda n: c("tra_adv_fct", 12, 1, b"TRC", 14400.0, *t, n, 2, 2),
    tra_ldf_iso=lambda n: c("tra_ldf_iso", 12, 1, b"TRC", *[None] * 6, t[0], t[0], t[1], n, 1),
    tra_ldf_blp=lambda n: c("tra_ldf_blp", 12, 1, b"TRC", *[None] * 6, t[0], t[1], n, 20),
    tra_ldf_iso_adj=lambda n: c("tra_ldf_iso_adj", 12, 1, b"TRC", *[None] * 6, t[0], t[0], t[1], n, 1),
    dia_hsb_init=lambda n: n > 2 and c("dia_hsb_init"))["{routine}"]
call(2)
held, refused = [fake.fake_held()], []
for room in range({arrays}):
    fake.fake_mallocs_left(C.c_long(room))
    try:
        call(3)
    except AssertionError as e:
        refused.append(str(e))
    fake.fake_mallocs_left(C.c_long(-1))
    call(2)
    held.append(fake.fake_held())
call(3)
held.append(fake.fake_held())
print(json.dumps([refused, held]))
""")
    refused, held = out
    assert len(refused) == arrays and all("array" in e for e in refused), refused
    assert held[1:-1] == held[:1] * arrays and held[-1] > held[0]
