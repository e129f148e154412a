"""Performance cases: the work that an ocean-model host has this library do.

Every case goes through nemo_gpu.api, the mirror of the C ABI: whole hot-path steps, single
routines of the path (dyn_spg_ts, the tracer routines, laplacian diffusion with lbc_lnk and
glob_sum), the blocks that close the path into a model step (equation of state, vertical
physics and slopes, momentum trends, time stepping), and the adjoint tracer routines. Grids are
the two of the package: the GYRE double gyre (31 z-levels, 1-D scale factors, linear free
surface) and the synthetic shelf (56 z* levels, partial bottom cells, 3-D scale factors).

`exact` restates each block in 64 bits with plain torch, from the published formulas of NEMO 4.0.
Arrays are (member, [tracer,] level, j, i), i contiguous: the memory of the Fortran arrays.
"""
import functools
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "nemo-fmi-devel_gb300"))
from nemo_gpu import _ffi, api, gyre, shelf  # noqa: E402

KT = 10               # a step of a run in progress (leap-frog, Asselin filter on)
DEV = "cuda"
F64 = torch.float64

# --------------------------------------------------------------------------- cases


def listed():
    return [
        # the headline benchmark: one hot-path step of GYRE nn_GYRE=25 in the mixed form
        dict(name="step_gyre25", kind="step", grid="gyre", jpi=752, jpj=502, jpk=31, members=1, prec="mixed"),
        # the smallest configuration, GYRE nn_GYRE=1: a step is a handful of short launches
        dict(name="step_gyre1", kind="step", grid="gyre", jpi=32, jpj=22, jpk=31, members=1, prec="mixed"),
        # the barotropic sub-steps of an ensemble: 64 members of GYRE nn_GYRE=5
        dict(name="spg_ens64", kind="spg", grid="gyre", jpi=152, jpj=102, jpk=31, members=64, prec="mixed"),
        # the barotropic sub-steps of a regional shelf (z*, EEN, flux form) on an odd grid
        dict(name="spg_shelf", kind="spg", grid="shelf", jpi=421, jpj=363, jpk=56, members=1, prec="mixed"),
        # the tracer routines called one by one on the shelf: FCT 4/4, iso-neutral, partial steps
        dict(name="tracers_shelf", kind="tracers", grid="shelf", jpi=500, jpj=400, jpk=56, members=1, prec="mixed",
             fct=4),
        # the same routines in the plain FP64 form on GYRE nn_GYRE=12 (jpi not a multiple of 4)
        dict(name="tracers_fp64", kind="tracers", grid="gyre", jpi=362, jpj=242, jpk=31, members=1, prec="fp64",
             fct=2),
        # small single calls: a laplacian trend, its halo and a global tracer sum, two members, odd sizes
        dict(name="lap_small", kind="lap", grid="gyre", jpi=93, jpj=61, jpk=31, members=2, prec="mixed"),
        # the blocks that close the path into GYRE's model step, at nn_GYRE=25 or a ragged grid
        dict(name="momentum_gyre25", kind="momentum", grid="gyre", jpi=752, jpj=502, jpk=31, members=1, prec="mixed"),
        dict(name="density_gyre25", kind="density", grid="gyre", jpi=752, jpj=502, jpk=31, members=1, prec="mixed"),
        dict(name="physics_gyre16", kind="physics", grid="gyre", jpi=481, jpj=323, jpk=31, members=1, prec="mixed"),
        dict(name="stepping_gyre25", kind="stepping", grid="gyre", jpi=752, jpj=502, jpk=31, members=1, prec="mixed"),
        # one adjoint step of the tracer window of GYRE nn_GYRE=10 (FP64 only)
        dict(name="adjoint_gyre10", kind="adjoint", grid="gyre", jpi=302, jpj=202, jpk=31, members=1, prec="fp64"),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "spg", "tracers", "tracers", "lap", "momentum", "density", "physics",
                       "stepping", "adjoint"])
    grid = rng.choice(["gyre", "gyre", "shelf"]) if kind in ("step", "spg", "tracers", "lap") else "gyre"
    prec = "fp64" if kind == "adjoint" else rng.choice(["mixed", "mixed", "mixed", "fp64"])
    jpk = 56 if grid == "shelf" else rng.choice([31, 31, 31, rng.randint(18, 40)])
    top = {"adjoint": 1.8e6}.get(kind, 3e6 if prec == "fp64" else 11e6)
    cells = math.exp(rng.uniform(math.log(3e4), math.log(top)))
    members = rng.choice([1, 1, 1, 2, rng.randint(2, 16)])
    aspect = rng.uniform(0.8, 1.7)
    n2 = max(cells / jpk / members, 400.0)
    jpi = max(16, int(math.sqrt(n2 * aspect)))
    if rng.random() < 0.4:
        jpi -= jpi % 4
    jpj = max(16, int(n2 / jpi))
    case = dict(kind=kind, grid=grid, jpi=jpi, jpj=jpj, jpk=jpk, members=members, prec=prec)
    if kind == "tracers":
        case["fct"] = rng.choice([2, 4])
    return case


def namelist(case):
    nam = shelf.namelist() if case["grid"] == "shelf" else gyre.namelist()
    if case["kind"] in ("momentum", "density", "physics"):
        nam.update(gyre.FULL_NAMELIST)
    return nam


# --------------------------------------------------------------------------- grid


@functools.lru_cache(maxsize=3)
def _domain(grid, jpi, jpj, jpk):
    if grid == "shelf":
        return shelf.domain(jpi, jpj, jpk, seed=3)
    nn = max(1, math.ceil(max((jpi - 2) / 30, (jpj - 2) / 20)))
    dom = gyre.domain(nn, jpk=jpk)
    if (dom["jpi"], dom["jpj"]) != (jpi, jpj):   # a window of the next larger GYRE grid, closed on its own frame
        dom = {k: (np.asfortranarray(v[:jpi, :jpj]) if isinstance(v, np.ndarray) and v.ndim > 1 else v)
               for k, v in dom.items()}
        for n in ("k_top", "k_bot"):
            dom[n][0], dom[n][-1], dom[n][:, 0], dom[n][:, -1] = 0, 0, 0, 0
        dom["jpi"], dom["jpj"] = jpi, jpj
    return dom


def domain(case):
    return _domain(case["grid"], case["jpi"], case["jpj"], case["jpk"])


def sh(a, di=0, dj=0, dk=0):
    """b(i,j,k) = a(i+di, j+dj, k+dk), zero outside the array."""
    return F.pad(a, (-di, di, -dj, dj, -dk, dk) if dk else (-di, di, -dj, dj))


class Grid:
    """Masks and metrics of a domain in 64 bits on the device, and the rest-state depths."""

    def __init__(self, dom):
        self.dom = dom
        self.jpi, self.jpj, self.jpk = jpi, jpj, jpk = dom["jpi"], dom["jpj"], dom["jpk"]
        for n in ("e1t", "e2t", "e1u", "e2u", "e1v", "e2v", "e1f", "e2f", "ff_f", "ff_t", "gphit", "gphiu", "gphiv"):
            setattr(self, n, self.put(dom[n]))
        for n in ("t", "u", "v", "w", "f"):
            a = dom["e3%s_0" % n]
            one = np.asfortranarray(a[:1, :1])
            self_n = self.put(one).expand(jpk, jpj, jpi) if dom.get("_flat", self.flat(dom)) else self.put(a)
            setattr(self, "e3%s_0" % n, self_n)
        kt, kb = self.put(dom["k_top"]), self.put(dom["k_bot"])
        self.lev = torch.arange(jpk, device=DEV, dtype=F64)[:, None, None]
        self.inn = torch.zeros(jpj, jpi, device=DEV, dtype=F64)
        self.inn[1:-1, 1:-1] = 1
        self.tm = ((kt != 0) & (self.lev >= kt - 1) & (self.lev <= kb - 1)).to(F64) * self.inn
        self.um = self.tm * sh(self.tm, 1) * self.inn
        self.vm = self.tm * sh(self.tm, 0, 1) * self.inn
        self.wm = self.tm * torch.cat([torch.ones_like(self.tm[:1]), self.tm[:-1]])
        self.ssm, self.ssum, self.ssvm = self.tm.amax(0), self.um.amax(0), self.vm.amax(0)
        self.mbkt = kb.clamp(min=1)
        edge = self.inn == 0
        self.mbku = torch.minimum(self.mbkt, sh(self.mbkt, 1)).clamp(min=1).masked_fill(edge, 1)
        self.mbkv = torch.minimum(self.mbkt, sh(self.mbkt, 0, 1)).clamp(min=1).masked_fill(edge, 1)
        self.up = (self.lev < jpk - 1).to(F64)                       # levels 1 .. jpk-1
        self.mid = self.up * (self.lev > 0)                          # levels 2 .. jpk-1
        self.e12t, self.e12u, self.e12v = self.e1t * self.e2t, self.e1u * self.e2u, self.e1v * self.e2v
        self.ht_0, self.hu_0, self.hv_0 = [(e * m).sum(0) for e, m in (
            (self.e3t_0, self.tm), (self.e3u_0, self.um), (self.e3v_0, self.vm))]
        self.r1_hu_0 = self.ssum / (self.hu_0 + 1 - self.ssum)
        self.r1_hv_0 = self.ssvm / (self.hv_0 + 1 - self.ssvm)
        self.dept = torch.tensor(dom["gdept_1d"], device=DEV)[:, None, None]
        self.gdept = self.dept.expand(jpk, jpj, jpi)
        self.gdepw = torch.cat([torch.zeros_like(self.e3t_0[:1]), self.e3t_0[:-1].cumsum(0)])

    @staticmethod
    def flat(dom):
        if "_flat" not in dom:
            dom["_flat"] = all(bool((dom["e3%s_0" % n] == dom["e3%s_0" % n][:1, :1]).all()) for n in "tuvwf")
        return dom["_flat"]

    @staticmethod
    def put(a):
        return torch.from_numpy(np.ascontiguousarray(a.T)).to(DEV, F64)


@functools.lru_cache(maxsize=2)
def _grid(grid, jpi, jpj, jpk):
    return Grid(_domain(grid, jpi, jpj, jpk))


def grid_of(case):
    return _grid(case["grid"], case["jpi"], case["jpj"], case["jpk"])


# ------------------------------------------------------------------ equation of state
# EOS-80 polynomials of Roquet et al., Ocean Modelling 90 (2015), as NEMO 4.0 uses them: the
# coefficients of zs^i zt^j for each power of the depth, rows by i
EOS = [
    [[9.5356891948e+02, 1.0087518651e+01, -2.5579830599e+01, 1.6846451198e+01, -8.0812310102, 1.2079167803,
      -2.4520288837e-01],
     [1.7136499189e+02, -1.3647741861e+01, 2.4043512327e+01, -2.1482926901e+01, 1.0102374985e+01, 1.1515380987e-01],
     [-3.7501039454e+02, 8.8478359933, -1.6807503990e+01, 1.0108954054e+01, -4.8340368631],
     [5.1856810420e+02, -7.2329388377, 8.3811577084, -6.2675951440e-01],
     [-3.7264470465e+02, 1.4774410611, -1.9771060192], [1.4302533998e+02, 2.0036720553e-01], [-2.2856621162e+01]],
    [[1.0748601068e+01, -1.5852644587e+01, 9.9994861860, -3.4866102017, 5.9503008642e-01],
     [-1.7817043500e+01, -7.6639383522e-01, -1.9467067787e-01, 2.2229155620e-01],
     [2.2181366768e+01, 4.1144627302, -1.2177554330], [-1.6750916338e+01, -6.6955877448e-01], [4.1202230403]],
    [[1.0375676547, 2.1836324814, -1.2548163097], [-3.4249470629, -3.4453674320e-01], [2.0542026429]],
    [[1.8729078427e-02, 3.8306136687e-01], [-5.7238495240e-02]]]
ALP = [
    [[-2.5218796628e-01, 1.2789915300, -1.2634838399, 8.0812310102e-01, -1.5098959754e-01, 3.6780433255e-02],
     [3.4119354654e-01, -1.2021756164, 1.6112195176, -1.0102374985, -1.4394226233e-02],
     [-2.2119589983e-01, 8.4037519952e-01, -7.5817155402e-01, 4.8340368631e-01],
     [1.8082347094e-01, -4.1905788542e-01, 4.7006963580e-02], [-3.6936026529e-02, 9.8855300959e-02],
     [-5.0091801383e-03]],
    [[3.9631611467e-01, -4.9997430930e-01, 2.6149576513e-01, -5.9503008642e-02],
     [1.9159845880e-02, 9.7335338937e-03, -1.6671866715e-02], [-1.0286156825e-01, 6.0887771651e-02],
     [1.6738969362e-02]],
    [[-5.4590812035e-02, 6.2740815484e-02], [8.6134185799e-03]], [[-9.5765341718e-03]]]
BET = [
    [[2.1420623987, -1.7059677327e-01, 3.0054390409e-01, -2.6853658626e-01, 1.2627968731e-01, 1.4394226233e-03],
     [-9.3752598635, 2.2119589983e-01, -4.2018759976e-01, 2.5272385134e-01, -1.2085092158e-01],
     [1.9446303907e+01, -2.7123520642e-01, 3.1429341406e-01, -2.3503481790e-02],
     [-1.8632235232e+01, 7.3872053057e-02, -9.8855300959e-02], [8.9390837485, 1.2522950346e-02], [-1.7142465871]],
    [[-2.2271304375e-01, -9.5799229402e-03, -2.4333834734e-03, 2.7786444526e-03],
     [5.5453416919e-01, 1.0286156825e-01, -3.0443885826e-02], [-6.2815936268e-01, -2.5108454043e-02],
     [2.0601115202e-01]],
    [[-4.2811838287e-02, -4.3067092900e-03], [5.1355066072e-02]], [[-7.1548119050e-04]]]


def poly(table, t, s, depth, surface=False):
    zt, zs, zh = t / 40, ((s + 20).abs() / 40).sqrt(), depth * 1e-4
    out = 0
    for k in range(0 if surface else len(table) - 1, -1, -1):
        z = 0
        for row in reversed(table[k]):
            h = 0
            for c in reversed(row):
                h = h * zt + c
            z = z * zs + h
        out = out * zh + z
    return out


def density(G, nam, ts):
    """The in situ density anomaly and the potential density of T, S (member, 2, ...)."""
    t, s = ts[:, 0], ts[:, 1]
    m = G.tm * G.up
    return (poly(EOS, t, s, G.gdept32) / nam["rau0"] - 1) * m, poly(EOS, t, s, G.gdept32, surface=True) * m


def expansion(G, nam, ts):
    t, s = ts[:, 0], ts[:, 1]
    zs = ((s + 20).abs() / 40).sqrt()
    m = G.tm * G.up / nam["rau0"]
    return torch.stack([poly(ALP, t, s, G.gdept32) * m, poly(BET, t, s, G.gdept32) / zs * m], 1)


def brunt(G, nam, ts, ab):
    d, w = G.gdept32, G.gdepw32
    zrw = torch.where(G.mid > 0, (w - d) / (sh(d, dk=-1) - d), torch.zeros_like(d))
    a = ab * (1 - zrw) + sh(ab, dk=-1) * zrw
    dt = sh(ts, dk=-1) - ts
    return nam["grav"] * (a[:, 0] * dt[:, 0] - a[:, 1] * dt[:, 1]) / G.e3w_0 * G.wm * G.mid


# --------------------------------------------------------------------------- state


def state(G, case, nam, seed):
    """A seeded state like gyre.state / shelf.state (stratified T and S with noise, a double gyre,
    w from continuity, small trends, slopes, a mixed layer with a few convecting columns), in 64 bits
    but of the values that the fields hold in the case's precision."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    m, jpk, jpj, jpi = case["members"], G.jpk, G.jpj, G.jpi
    on_shelf = case["grid"] == "shelf"

    def rn(*shape):
        return torch.randn(m, *shape, generator=g, device=DEV, dtype=F64)

    s3, s2 = (jpk, jpj, jpi), (jpj, jpi)
    t1, s1 = gyre._istate(G.dom["gdept_1d"])
    base = torch.stack([torch.tensor(t1, device=DEV), torch.tensor(s1, device=DEV)])[..., None, None]
    amp = torch.tensor([1.0, 0.2], device=DEV, dtype=F64)[:, None, None, None] * (0.002 + 0.05 * torch.exp(-G.dept / 300))
    S = {"tsb": (base + amp * rn(2, *s3)) * G.tm}
    S["tsn"] = (S["tsb"] + 0.2 * amp * rn(2, *s3)) * G.tm
    x = (torch.arange(jpi, device=DEV, dtype=F64) / max(jpi - 2, 1)).clamp(0, 1)
    y = (torch.arange(jpj, device=DEV, dtype=F64) / max(jpj - 2, 1)).clamp(0, 1)
    u0, nu = (0.03, 0.003) if on_shelf else (0.5, 0.03)
    psi = torch.sin(math.pi * x)[None, :] * torch.sin(2 * math.pi * y)[:, None] * (
        u0 * float(G.e1t.mean()) * (jpj - 2) / (2 * math.pi))
    prof = torch.exp(-G.dept / 600)
    un = (-(psi - sh(psi, 0, -1)) / G.e2u * prof + nu * rn(*s3)) * G.um
    vn = ((psi - sh(psi, -1)) / G.e1v * prof + nu * rn(*s3)) * G.vm
    S["un"], S["vn"] = un, vn
    S["ub"], S["vb"] = (un + 0.3 * nu * rn(*s3)) * G.um, (vn + 0.3 * nu * rn(*s3)) * G.vm
    S["ua"], S["va"] = 1e-6 * rn(*s3) * G.um, 1e-6 * rn(*s3) * G.vm
    if on_shelf:
        ssh = 0.05 * torch.sin(math.pi * x)[None, :] * torch.sin(2 * math.pi * y)[:, None] + 0.002 * rn(*s2)
        S["sshn"], S["sshb"] = ssh * G.ssm, (0.999 * ssh + 0.0005 * rn(*s2)) * G.ssm
    else:
        ssh = 0.3 * rn(*s2)
        for _ in range(4):
            ssh = 0.25 * (sh(ssh, 1) + sh(ssh, -1) + sh(ssh, 0, 1) + sh(ssh, 0, -1))
        S["sshn"] = ssh * G.ssm
        S["sshb"] = (ssh + 0.01 * rn(*s2)) * G.ssm
    S["avt"] = (1.2e-5 + 1e-3 * torch.exp(-G.dept / 50) * (1 + torch.rand(m, *s3, generator=g, device=DEV, dtype=F64))
                + 10.0 * (torch.rand(m, 1, *s2, generator=g, device=DEV, dtype=F64) < 0.02) * (G.dept < 300)) * G.wm * G.mid
    for n, k in (("uslp", G.um), ("vslp", G.vm), ("wslpi", G.wm), ("wslpj", G.wm)):
        S[n] = (0.004 * rn(*s3)).clamp(-0.01, 0.01) * k * (G.lev > 0)
    S["rcdu_bot"] = -1e-3 * (0.05 + 0.1 * rn(*s2).abs()) * G.ssm
    S["utau"] = (-0.08 * torch.sin(math.pi * (G.gphiu - 15) / 14)).expand(m, *s2)
    S["vtau"] = (0.08 * torch.sin(math.pi * (G.gphiv - 15) / 14)).expand(m, *s2)
    S["emp"] = 2e-5 * rn(*s2) * G.ssm
    if on_shelf:
        S["ssh_ib"] = (0.02 * torch.sin(2 * math.pi * x)[None, :] + 0 * y[:, None]).expand(m, *s2)
        for n, k in (("gtsu", G.ssum), ("gtsv", G.ssvm)):
            S[n] = 1e-3 * rn(2, *s2) * k
        S.update(zstar(G, S))
        e3u, e3v = S["e3u_n"], S["e3v_n"]
    else:
        e3u, e3v = G.e3u_0, G.e3v_0
    div = G.inn * (G.e2u * e3u * un - sh(G.e2u * e3u * un, -1) + G.e1v * e3v * vn - sh(G.e1v * e3v * vn, 0, -1)) / G.e12t * G.tm
    if on_shelf:
        r2dt = 2 * nam["rn_rdt"]
        ssha = (S["sshb"] - r2dt * (div * G.up).sum(1)) * G.ssm
        S["e3t_a"] = stretch(G, ssha)
        div = div + (S["e3t_a"] - S["e3t_b"]) / r2dt * G.tm
    S["wn"] = -torch.flip(torch.flip(div * G.up, (1,)).cumsum(1), (1,)) * G.up
    hu, hv = (S["hu_n"], S["hv_n"]) if on_shelf else (G.hu_0, G.hv_0)
    for n, a, e3, k, h, s in (("un_b", un, e3u, G.um, hu, G.ssum), ("vn_b", vn, e3v, G.vm, hv, G.ssvm),
                              ("ub_b", S["ub"], e3u, G.um, hu, G.ssum), ("vb_b", S["vb"], e3v, G.vm, hv, G.ssvm)):
        S[n] = (e3 * a * k * G.up).sum(1) / (h + 1 - s) * s
    S["ub2_b"], S["vb2_b"] = S["un_b"] * hu, S["vn_b"] * hv
    for n in ("ssha", "ua_b", "va_b", "un_adv", "vn_adv", "un_bf", "vn_bf"):
        S[n] = torch.zeros(m, *s2, device=DEV, dtype=F64)
    if case["kind"] == "stepping":
        S["ua_b"], S["va_b"] = S["un_b"] * 1.001, S["vn_b"] * 1.001
        S["ssha"] = S["sshn"] + 0.001 * rn(*s2) * G.ssm
        S["tsa"] = (S["tsn"] + 0.2 * amp * rn(2, *s3)) * G.tm
        S["avm"] = (1.2e-4 + 1e-2 * torch.exp(-G.dept / 50)) * (1 + 0.2 * rn(*s3).abs()) * G.wm * G.mid
    for n in S:   # the values that the bound arrays hold
        if case["prec"] == "mixed" and n.upper() not in _ffi.FP64_FIELDS:
            S[n] = S[n].float().to(F64)
    r32 = (lambda a: a.float().to(F64)) if case["prec"] == "mixed" else (lambda a: a)
    G.gdept32, G.gdepw32 = r32(G.gdept), r32(G.gdepw)
    if case["kind"] == "physics":
        rab = expansion(G, nam, S["tsb"])
        S["rn2b"] = r32(brunt(G, nam, S["tsb"], rab))
        S["rn2"] = r32(brunt(G, nam, S["tsn"], expansion(G, nam, S["tsn"])))
        S["rhd"] = r32(density(G, nam, S["tsb"])[0])
        S["taum"] = r32((0.1 * (1 + 0.2 * rn(*s2))).abs() * G.ssm)
        en = 1e-6 + 1e-3 * torch.exp(-G.dept / 60) * torch.rand(m, *s3, generator=g, device=DEV, dtype=F64)
        S["en"], S["dissl"] = r32(en * G.wm), r32(1e-3 * en.sqrt() * G.wm + 1e-12)
        S["avm_k"], S["avt_k"] = r32((1.2e-4 + en) * G.wm), r32((1.2e-5 + en) * G.wm)
    if case["kind"] == "adjoint":
        S["ab"], S["an"] = rn(2, *s3) * G.tm, rn(2, *s3) * G.tm
    return S


def stretch(G, ssh):
    s = ((G.ht_0 + ssh) / (G.ht_0 + 1 - G.ssm))[:, None]
    return G.e3t_0 * s * G.tm + G.e3t_0 * (1 - G.tm)


def zstar(G, S):
    """z* scale factors and depths of sshb, sshn (domvvl.F90)."""
    b, n = stretch(G, S["sshb"]), stretch(G, S["sshn"])

    def uv(e3t):
        d = G.e12t * (e3t - G.e3t_0)
        return (G.e3u_0 + G.um * 0.5 * (d + sh(d, 1)) / G.e12u, G.e3v_0 + G.vm * 0.5 * (d + sh(d, 0, 1)) / G.e12v)

    ub, vb = uv(b)
    un, vn = uv(n)
    d = n - G.e3t_0
    lower = 0.5 * G.tm
    e3w = G.e3w_0 + torch.where(G.lev == 0, d, (1 - lower) * sh(d, dk=-1) + lower * d)
    du = G.e12u * (un - G.e3u_0)
    e3f = G.e3f_0 + G.um * sh(G.um, 0, 1) * 0.5 * (du + sh(du, 0, 1)) / (G.e1f * G.e2f)
    out = dict(e3t_b=b, e3t_n=n, e3u_n=un, e3v_n=vn, e3w_n=e3w, e3f_n=e3f, ht_n=(n * G.tm * G.up).sum(1))
    for t, u, v in (("n", un, vn), ("b", ub, vb)):
        out["hu_" + t], out["hv_" + t] = (u * G.um * G.up).sum(1), (v * G.vm * G.up).sum(1)
        out["r1_hu_" + t] = G.ssum / (out["hu_" + t] + 1 - G.ssum)
        out["r1_hv_" + t] = G.ssvm / (out["hv_" + t] + 1 - G.ssvm)
    return out


ZSTAR = ("e3t_b", "e3t_n", "e3t_a", "e3u_n", "e3v_n", "e3w_n", "e3f_n", "ht_n", "hu_n", "hv_n", "r1_hu_n", "r1_hv_n",
         "hu_b", "hv_b", "r1_hu_b", "r1_hv_b", "gtsu", "gtsv", "ssh_ib")
SPG = ("ua", "va", "un", "vn", "ub", "vb", "sshn", "sshb", "un_b", "vn_b", "ub_b", "vb_b", "utau", "vtau", "emp",
       "rcdu_bot", "ssha", "ua_b", "va_b", "un_adv", "vn_adv", "ub2_b", "vb2_b", "un_bf", "vn_bf")
SPG_OUT = ("ua", "va", "un", "vn", "ssha", "ua_b", "va_b", "un_adv", "vn_adv", "ub2_b", "vb2_b", "un_bf", "vn_bf")
SLOPES = ("uslp", "vslp", "wslpi", "wslpj")
TRACERS = ("tsb", "tsn", "avt") + SLOPES
BOUND = {
    "step": SPG + TRACERS + ("wn",), "spg": SPG, "tracers": TRACERS + ("un", "vn", "wn"), "lap": ("tsb",),
    "momentum": ("un", "vn", "wn", "ub", "vb", "ua", "va"), "density": ("tsb", "tsn"),
    "physics": ("ub", "vb", "un", "vn", "avm_k", "avt_k", "avt", "en", "dissl", "rn2", "rn2b", "taum"),
    "stepping": ("un", "vn", "wn", "ua", "va", "ub", "vb", "avm", "ua_b", "va_b", "rcdu_bot", "utau", "vtau", "tsb",
                 "tsn", "tsa", "un_b", "vn_b", "ub_b", "vb_b", "sshn", "sshb", "ssha"),
    "adjoint": TRACERS,
}


@functools.lru_cache(maxsize=1)
def work_stream():
    """The program's one stream: its contexts' steps follow one another on it."""
    return torch.cuda.Stream()


def prepare(case, seed):
    nam = namelist(case)
    G = grid_of(case)
    S = state(G, case, nam, seed)
    m, s3, s2 = case["members"], (G.jpk, G.jpj, G.jpi), (G.jpj, G.jpi)
    stream = work_stream()
    ctx = api.Context(domain(case), nam, nmembers=m, prec=case["prec"], stream=stream)
    dt = ctx.dtype
    D = {}

    def bind(n, t):
        D[n] = t
        ctx.bind(n.upper(), t)

    kind = case["kind"]
    for n in BOUND[kind] + (ZSTAR if case["grid"] == "shelf" else ()):
        bind(n, S[n].to(ctx.field_dtype(n.upper())).contiguous().clone())
    z3 = lambda *lead: torch.zeros(m, *lead, *s3, device=DEV, dtype=dt)  # noqa: E731
    z2 = lambda: torch.zeros(m, *s2, device=DEV, dtype=dt)  # noqa: E731
    if kind in ("step", "tracers", "adjoint"):
        bind("tsa", z3(2))
        bind("ah_wslp2", z3())
        bind("akz", z3())
    if kind in ("tracers", "adjoint"):
        for n in ("zun", "zvn", "zwn"):
            D[n] = z3()
    if kind == "lap":
        D["tsa"] = z3(2)
    if kind == "momentum":
        ahm_t, ahm_f = 1e5 * G.tm * G.up, 1e5 * G.tm * sh(G.tm, 1) * sh(G.tm, 0, 1) * sh(G.tm, 1, 1) * G.up
        bind("ahmt", ahm_t.expand(m, *s3).to(dt).contiguous().clone())
        bind("ahmf", ahm_f.expand(m, *s3).to(dt).contiguous().clone())
        bind("rhd", density(G, nam, S["tsn"])[0].to(dt).contiguous())
    if kind in ("density", "physics"):
        bind("gdept_n", G.gdept.expand(m, *s3).to(dt).contiguous().clone())
        bind("gdepw_n", G.gdepw.expand(m, *s3).to(dt).contiguous().clone())
    if kind == "density":
        for n in ("rhd", "rhop", "rn2b", "rn2"):
            D[n] = z3()
        for n in ("rab_b", "rab_n"):
            D[n] = z3(2)
    if kind == "physics":
        for n in ("avm", "avs") + SLOPES:
            bind(n, z3())
        D["rhd"] = S["rhd"].to(dt).contiguous()
        bind("nmln", torch.zeros(m, *s2, device=DEV, dtype=torch.int32))
        bind("hmlp", z2())
        bind("hmlpt", z2())
    if kind == "adjoint":
        D["ab"], D["an"], D["aa"] = S["ab"].clone(), S["an"].clone(), z3(2)
        torch.cuda.synchronize()
        p2dt = 2 * nam["rn_rdt"]
        tape = torch.zeros(m, 2, 3, *s3, device=DEV, dtype=F64)
        ctx.tra_adv_trp(*[S[n].to(dt).contiguous() for n in ("un", "vn", "wn")], D["zun"], D["zvn"], D["zwn"])
        ctx.bind("FCT_TAPE", tape)
        ctx.tra_adv_fct(KT, 1, "TRA", p2dt, D["zun"], D["zvn"], D["zwn"], D["tsb"], D["tsn"], D["tsa"], 2, 2, 2)
        ctx.tra_ldf_iso(KT, 1, "TRA", None, None, None, None, None, None, D["tsb"], D["tsb"], D["tsa"], 2, 1)
        ctx.synchronize()
        D["tape"] = tape
    torch.cuda.synchronize()
    return dict(case=case, nam=nam, ctx=ctx, D=D, stream=stream, kt=KT, outs=outputs(case, D))


def outputs(case, D):
    kind = case["kind"]
    names = {"step": ("tsa", "ah_wslp2", "akz") + SPG_OUT, "spg": SPG_OUT,
             "tracers": ("zun", "zvn", "zwn", "tsa", "ah_wslp2", "akz"), "momentum": ("ua", "va"),
             "density": ("rab_b", "rab_n", "rn2b", "rn2", "rhd", "rhop"),
             "physics": ("en", "dissl", "avm_k", "avt_k", "avm", "avt", "avs", "nmln", "hmlp", "hmlpt") + SLOPES,
             "stepping": ("wn", "ua", "va", "ub", "vb", "un", "vn", "tsb", "tsn", "tsa", "un_b", "vn_b", "ub_b", "vb_b",
                          "sshb", "sshn"),
             "adjoint": ("ab", "an"), "lap": ("tsa",)}[kind]
    return {n: D[n] for n in names}


def run(state):
    c, D, case, kt = state["ctx"], state["D"], state["case"], state["kt"]
    kind, out = case["kind"], dict(state["outs"])
    state["kt"] = kt + 1
    if kind == "step":
        c.stp_hotpath(kt)
    elif kind == "spg":
        c.dyn_spg_ts(kt)
    elif kind == "tracers":
        zps = case["grid"] == "shelf"
        gu, gv = (D["gtsu"], D["gtsv"]) if zps else (None, None)
        p2dt = 2 * state["nam"]["rn_rdt"]
        with torch.cuda.stream(state["stream"]):
            D["tsa"].zero_()
        c.tra_adv_trp(D["un"], D["vn"], D["wn"], D["zun"], D["zvn"], D["zwn"])
        c.tra_adv_fct(kt, 1, "TRA", p2dt, D["zun"], D["zvn"], D["zwn"], D["tsb"], D["tsn"], D["tsa"], 2, case["fct"],
                      case["fct"])
        c.tra_ldf_iso(kt, 1, "TRA", None, None, gu, gv, None, None, D["tsb"], D["tsb"], D["tsa"], 2, 1)
        c.tra_zdf_imp(kt, 1, "TRA", p2dt, D["tsb"], D["tsa"], 2)
    elif kind == "lap":
        zps = case["grid"] == "shelf"
        gu, gv = (D["gtsu"], D["gtsv"]) if zps else (None, None)
        with torch.cuda.stream(state["stream"]):
            D["tsa"].zero_()
        c.tra_ldf_lap(kt, 1, "TRA", None, None, gu, gv, None, None, D["tsb"], D["tsa"], 2, 1)
        c.lbc_lnk(D["tsa"], case["jpk"], "T", nl=2)
        out["sum"] = c.glob_sum(D["tsb"], 2 * case["jpk"])
    elif kind == "momentum":
        with torch.cuda.stream(state["stream"]):
            D["ua"].zero_()
            D["va"].zero_()
        c.dyn_keg(kt)
        c.dyn_zad(kt)
        c.vor_ene(kt, 4, D["un"], D["vn"], D["ua"], D["va"])
        c.dyn_ldf_lap(kt, D["ub"], D["vb"], D["ua"], D["va"])
        c.dyn_hpg(kt)
    elif kind == "density":
        c.rab_3d(D["tsb"], D["rab_b"])
        c.bn2(D["tsb"], D["rab_b"], D["rn2b"])
        c.rab_3d(D["tsn"], D["rab_n"])
        c.bn2(D["tsn"], D["rab_n"], D["rn2"])
        c.eos_insitu(D["tsb"], D["rhd"], D["gdept_n"])
        c.eos_insitu_pot(D["tsn"], D["rhd"], D["rhop"], D["gdept_n"])
    elif kind == "physics":
        c.zdf_phy(kt)
        c.zdf_mxl(kt)
        c.ldf_slp(kt, D["rhd"], D["rn2b"])
    elif kind == "stepping":
        with torch.cuda.stream(state["stream"]):
            D["ua"].zero_()
            D["va"].zero_()
        c.wzv(kt)
        c.dyn_zdf_step(kt)
        c.tra_nxt(kt)
        c.dyn_nxt(kt)
        c.ssh_swp(kt)
    elif kind == "adjoint":
        with torch.cuda.stream(state["stream"]):
            D["aa"].zero_()
        p2dt = 2 * state["nam"]["rn_rdt"]
        c.tra_nxt_adj(kt, D["ab"], D["an"], D["aa"])
        c.tra_zdf_imp_adj(kt, 1, "TRA", p2dt, D["ab"], D["aa"], 2)
        c.tra_ldf_iso_adj(kt, 1, "TRA", None, None, None, None, None, None, D["ab"], None, D["aa"], 2, 1)
        c.bind("FCT_TAPE", D["tape"])
        c.tra_adv_fct_adj(kt, 1, "TRA", p2dt, D["zun"], D["zvn"], D["zwn"], D["ab"], D["an"], D["aa"], 2, 2, 2)
        c.bind("FCT_TAPE", None)
    return out


def work(case):
    """Bytes: each 3-D and 2-D field read once, each written once (masks and 1-D profiles are small);
    operations: what the formulas need a cell (a division or a minimum counted as one)."""
    n2 = case["jpi"] * case["jpj"] * case["members"]
    n3 = n2 * case["jpk"]
    w = 8 if case["prec"] == "fp64" else 4
    on_shelf = case["grid"] == "shelf"
    kind = case["kind"]
    # 3-D fields read + written, 2-D values, operations per cell
    f3, f2, ops = {
        "step": (14 + 8, 25 + 18, 700), "spg": (4 + 4, 25 + 18, 30),
        "tracers": (4 + 3 + 1 + 4 + 3 + 2 + 2, 4, 660), "lap": (4, 3, 30), "momentum": (8 + 2, 6, 130),
        "density": (6 + 8, 0, 500), "physics": (12 + 11, 6, 300), "stepping": (13 + 11, 20, 110),
        "adjoint": (4 + 6 + 3 + 6 + 4, 3, 500)}[kind]
    if on_shelf:
        f3 += {"step": 6, "spg": 2, "tracers": 6, "lap": 3}.get(kind, 0)
        ops += 60
    sub = 0
    if kind in ("step", "spg"):   # the sub-steps: some 90 operations a column each
        sub = 90.0 * n2 * (44 if on_shelf else 37)
    return {"bytes": float(w * (f3 * n3 + f2 * n2)), "flops": float(ops * n3 + sub)}


# --------------------------------------------------------------------------- 64-bit references


def spg_weights(G, nam):
    """nn_baro and the boxcar weights of a forward integration (ts_wgt, dynspg_ts.F90)."""
    if nam["ln_bt_auto"]:
        c = (nam["grav"] * G.ht_0.clamp(min=0) * (1 / G.e1t**2 + 1 / G.e2t**2)).sqrt().max().item()
        n = max(1, math.ceil(nam["rn_rdt"] / nam["rn_bt_cmax"] * c))
    else:
        n = nam["nn_baro"]
    w1 = [1.0 if abs(j - n) / n < 0.5 else 0.0 for j in range(1, 3 * n + 1)]
    last = max(j for j, w in enumerate(w1) if w) + 1
    w1 = w1[:last]
    w2 = [sum(w1[j:]) for j in range(last)]
    return n, [w / sum(w1) for w in w1], [w / sum(w2) for w in w2]


def ex_spg(G, S, nam):
    """dyn_spg_ts of a step in progress: forward, time-averaged; GYRE's linear free surface with the ENE
    scheme, or the shelf's z*, EEN, flux form and atmospheric pressure."""
    vvl = not nam["ln_linssh"]
    een = nam["nvor_scheme"] == _ffi.VOR["EEN"]
    rdt, grav, rau0, atfp = nam["rn_rdt"], nam["grav"], nam["rau0"], nam["rn_atfp"]
    n, w1, w2 = spg_weights(G, nam)
    dtb = rdt / n
    e3u, e3v = (S["e3u_n"], S["e3v_n"]) if vvl else (G.e3u_0, G.e3v_0)
    hu_n, hv_n, r1hu, r1hv = (S["hu_n"], S["hv_n"], S["r1_hu_n"], S["r1_hv_n"]) if vvl else (
        G.hu_0, G.hv_0, G.r1_hu_0, G.r1_hv_0)
    I, E, W, N, So = G.inn, lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, 1), lambda a: sh(a, 0, -1)
    frame = torch.ones_like(G.inn)
    frame[-1], frame[:, -1] = 0, 0
    if een:
        h = S["ht_n"]
        z = (N(h) + sh(h, 1, 1) + h + E(h)) / (N(G.ssm) + sh(G.ssm, 1, 1) + G.ssm + E(G.ssm)).clamp(min=1) * frame
        z = torch.where(z != 0, G.ff_f / torch.where(z != 0, z, 1.0), 0.0)
        ne, nw, se, sw = W(z) + z + So(z), sh(z, -1, -1) + W(z) + z, z + So(z) + sh(z, -1, -1), So(z) + sh(z, -1, -1) + W(z)
    else:
        hf = (G.e3f_0 * G.um * N(G.um) * G.up).sum(0) * frame
        z = torch.where(hf != 0, G.ff_f / torch.where(hf != 0, hf, 1.0), 0.0)

    def coriolis(fx, fy):
        if een:
            return ((ne * fy + E(nw * fy) + se * So(fy) + E(sw * So(fy))) / (12 * G.e1u),
                    -(N(sw * W(fx)) + N(se * fx) + nw * W(fx) + ne * fx) / (12 * G.e2v))
        y1, y2 = (So(fy) + sh(fy, 1, -1)) / G.e1u, (fy + E(fy)) / G.e1u
        x1, x2 = (W(fx) + sh(fx, -1, 1)) / G.e2v, (fx + N(fx)) / G.e2v
        return 0.25 * (So(z) * y1 + z * y2), -0.25 * (W(z) * x1 + z * x2)

    zu = (e3u * S["ua"] * G.um * G.up).sum(1) * r1hu
    zv = (e3v * S["va"] * G.vm * G.up).sum(1) * r1hv
    ua = S["ua"] - (zu * I)[:, None] * G.um * G.up
    va = S["va"] - (zv * I)[:, None] * G.vm * G.up
    tu, tv = coriolis(S["un_b"] * hu_n * G.e2u, S["vn_b"] * hv_n * G.e1v)
    if vvl:
        tu = tu - grav * (E(S["sshn"]) - S["sshn"]) / G.e1u
        tv = tv - grav * (N(S["sshn"]) - S["sshn"]) / G.e2v
    cu, cv = 0.5 * (E(S["rcdu_bot"]) + S["rcdu_bot"]), 0.5 * (N(S["rcdu_bot"]) + S["rcdu_bot"])
    m = S["un"].shape[0]
    bot = lambda a, k: a.gather(1, (k.long() - 1).expand(m, 1, G.jpj, G.jpi))[:, 0]  # noqa: E731
    zu = zu - tu * G.ssum + r1hu * cu * (bot(S["un"], G.mbku) - S["un_b"]) + S["utau"] * r1hu / rau0
    zv = zv - tv * G.ssvm + r1hv * cv * (bot(S["vn"], G.mbkv) - S["vn_b"]) + S["vtau"] * r1hv / rau0
    if nam["ln_apr_dyn"]:
        zu = zu + grav * (E(S["ssh_ib"]) - S["ssh_ib"]) / G.e1u
        zv = zv + grav * (N(S["ssh_ib"]) - S["ssh_ib"]) / G.e2v
    frc = S["emp"] / rau0
    o = torch.zeros_like(S["sshn"])
    sn, sb, sbb = S["sshn"], o, o
    u, ub, ubb, v, vb, vbb = S["un_b"], o, o, S["vn_b"], o, o
    hu, hv, hur, hvr = hu_n, hv_n, r1hu, r1hv
    ua_b, va_b, ssha, ua_adv, va_adv = o, o, o, o, o
    at_u = lambda a: I * 0.5 * G.ssum / G.e12u * (G.e12t * a + E(G.e12t * a))  # noqa: E731
    at_v = lambda a: I * 0.5 * G.ssvm / G.e12v * (G.e12t * a + N(G.e12t * a))  # noqa: E731
    for j in range(1, len(w1) + 1):
        a1, a2, a3 = (1.0, 0.0, 0.0) if j < 3 else (1.781105, -1.06221, 0.281105)
        ue, ve = a1 * u + a2 * ub + a3 * ubb, a1 * v + a2 * vb + a3 * vbb
        if vvl:
            p = a1 * sn + a2 * sb + a3 * sbb
            hup, hvp = G.hu_0 + at_u(p), G.hv_0 + at_v(p)
        else:
            hup, hvp = hu_n, hv_n
        fx, fy = G.e2u * ue * hup, G.e1v * ve * hvp
        ua_adv, va_adv = ua_adv + w2[j - 1] * fx / G.e2u, va_adv + w2[j - 1] * fy / G.e1v
        sa = (sn - dtb * (frc + (fx - W(fx) + fy - So(fy)) / G.e12t)) * G.ssm * I
        su, sv = (at_u(sa), at_v(sa)) if vvl else (0, 0)
        if j == 1:
            b = (1.0, 0.0, 0.0, 0.0)
        elif j == 2:
            b = (1.0833333333333, -0.1666666666666, 0.0833333333333, 0.0)
        else:
            b = (0.614, 0.285, 0.088, 0.013)
        p = b[0] * sa + b[1] * sn + b[2] * sb + b[3] * sbb
        tu, tv = coriolis(fx, fy)
        tu, tv = tu + cu * u * hur, tv + cv * v * hvr
        gu, gv = -grav * (E(p) - p) / G.e1u, -grav * (N(p) - p) / G.e2v
        if vvl:
            hura, hvra = G.ssum / (G.hu_0 + su + 1 - G.ssum), G.ssvm / (G.hv_0 + sv + 1 - G.ssvm)
            nu = (hu * u + dtb * ((G.hu_0 + at_u(p)) * gu + hup * tu + hu_n * zu)) * hura * I
            nv = (hv * v + dtb * ((G.hv_0 + at_v(p)) * gv + hvp * tv + hv_n * zv)) * hvra * I
            hu, hv = G.hu_0 + su, G.hv_0 + sv
            hur, hvr = G.ssum / (hu + 1 - G.ssum), G.ssvm / (hv + 1 - G.ssvm)
        else:
            nu = (u + dtb * (gu + tu + zu)) * G.ssum * I
            nv = (v + dtb * (gv + tv + zv)) * G.ssvm * I
        ubb, ub, u, vbb, vb, v, sbb, sb, sn = ub, u, nu, vb, v, nv, sb, sn, sa
        ua_b, va_b = ua_b + w1[j - 1] * u * (hu if vvl else 1), va_b + w1[j - 1] * v * (hv if vvl else 1)
        ssha = ssha + w1[j - 1] * sa
    out = {"ub2_b": ua_adv, "vb2_b": va_adv}
    out["un_adv"] = 0.5 * (S["ub2_b"] + ua_adv - atfp * S["un_bf"])
    out["vn_adv"] = 0.5 * (S["vb2_b"] + va_adv - atfp * S["vn_bf"])
    out["un_bf"] = atfp * S["un_bf"] + (ua_adv - S["ub2_b"])
    out["vn_bf"] = atfp * S["vn_bf"] + (va_adv - S["vb2_b"])
    r = 1 / (2 * rdt)
    if vvl:
        du, dv = r1hu * (ua_b - S["ub_b"] * S["hu_b"]) * r, r1hv * (va_b - S["vb_b"] * S["hv_b"]) * r
        ua_b = ua_b / (G.hu_0 + at_u(ssha) + 1 - G.ssum)
        va_b = va_b / (G.hv_0 + at_v(ssha) + 1 - G.ssvm)
    else:
        du, dv = (ua_b - S["ub_b"]) * r, (va_b - S["vb_b"]) * r
    out["ua"], out["va"] = ua + du[:, None] * G.up, va + dv[:, None] * G.up
    out["un"] = torch.where(G.up > 0, (S["un"] + (out["un_adv"] * r1hu - S["un_b"])[:, None]) * G.um, S["un"])
    out["vn"] = torch.where(G.up > 0, (S["vn"] + (out["vn_adv"] * r1hv - S["vn_b"])[:, None]) * G.vm, S["vn"])
    out.update(ua_b=ua_b, va_b=va_b, ssha=ssha)
    return out


def e3_of(G, S, nam):
    if nam["ln_linssh"]:
        return dict(b=G.e3t_0, n=G.e3t_0, a=G.e3t_0, u=G.e3u_0, v=G.e3v_0, w=G.e3w_0)
    return dict(b=S["e3t_b"], n=S["e3t_n"], a=S["e3t_a"], u=S["e3u_n"], v=S["e3v_n"], w=S["e3w_n"])


def interp4(G, t):
    """The compact 4th-order value at w-points (interp_4th_cpt, traadv_fct.F90), one system a column."""
    one, zero = torch.ones_like(G.wm), torch.zeros_like(G.wm)
    special = (G.lev == 1) | (G.lev == G.mbkt - 1)
    d = torch.where(special, one, 3 * G.wm + 1)
    s = torch.where(special, zero, G.wm)
    r = torch.where(special, 0.5, 3 * G.wm) * (sh(t, dk=-1) + t)
    K = G.jpk
    piv, x = [None, d[1]], [None, r[..., 1, :, :]]
    for k in range(2, K - 1):
        piv.append(d[k] - s[k] * s[k - 1] / piv[k - 1])
        x.append(r[..., k, :, :] - s[k] / piv[k - 1] * x[k - 1])
    x[K - 2] = x[K - 2] / piv[K - 2]
    for k in range(K - 3, 0, -1):
        x[k] = (x[k] - s[k] * x[k + 1]) / piv[k]
    return torch.stack([torch.zeros_like(x[1])] + x[1:] + [torch.zeros_like(x[1])], -3)


def ex_fct(G, S, nam, e3, un, vn, wn, tb, tn, order, frozen=None):
    """The advective trend (tra_adv_fct) with transports un, vn, wn of tracers (member, 2, ...); with the
    multipliers `frozen` the linear operator. Returns the trend and the multipliers."""
    un, vn, wn = un[:, None], vn[:, None], wn[:, None]
    lin, p2dt = nam["ln_linssh"], 2 * nam["rn_rdt"]
    e3 = {k: (v[:, None] if v.dim() == 4 else v) for k, v in e3.items()}
    I = G.inn * G.up
    E, W, N, So = lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, 1), lambda a: sh(a, 0, -1)
    U, D = lambda a: sh(a, dk=-1), lambda a: sh(a, dk=1)
    fx = 0.5 * ((un + un.abs()) * tb + (un - un.abs()) * E(tb)) * G.up
    fy = 0.5 * ((vn + vn.abs()) * tb + (vn - vn.abs()) * N(tb)) * G.up
    fz = 0.5 * ((wn + wn.abs()) * tb + (wn - wn.abs()) * U(tb)) * G.wm * G.mid
    if lin:
        fz = fz + wn * tb * (G.lev == 0)
    tra = -(fx - W(fx) + fy - So(fy) + fz - D(fz)) / G.e12t * I
    ta = tra / e3["n"] * G.tm
    aft = (e3["b"] * tb + p2dt * tra) / e3["a"] * G.tm * I
    if order == 2:
        cx, cy, cz = tn + E(tn), tn + N(tn), 0.5 * (tn + U(tn))
    else:
        gu, gv = (E(tn) - tn) * G.um, (N(tn) - tn) * G.vm
        lu, lv = (gu + W(gu)) / 6 * I, (gv + So(gv)) / 6 * I
        cx, cy, cz = tn + E(tn) + lu - E(lu), tn + N(tn) + lv - N(lv), interp4(G, tn)
    ax = (0.5 * un * cx - fx) * I
    ay = (0.5 * vn * cy - fy) * I
    az = (wn * cz - fz) * G.wm * G.mid * G.inn
    if frozen is None:
        big = 1e40
        wet = G.tm > 0
        hi = torch.where(wet, torch.maximum(tb, aft), -big)
        lo = torch.where(wet, torch.minimum(tb, aft), big)
        up, do = hi, lo
        for f in (E, W, N, So):
            up, do = torch.maximum(up, f(hi)), torch.minimum(do, f(lo))
        above = lambda a: torch.where(G.lev == 0, a, U(a))  # noqa: E731
        up, do = torch.maximum(torch.maximum(up, above(hi)), D(hi)), torch.minimum(torch.minimum(do, above(lo)), D(lo))
        p, q = (lambda a: a.clamp(min=0)), (lambda a: a.clamp(max=0))
        pos = p(W(ax)) - q(ax) + p(So(ay)) - q(ay) + p(D(az)) - q(az)
        neg = p(ax) - q(W(ax)) + p(ay) - q(So(ay)) + p(az) - q(D(az))
        bt = G.e12t * e3["n"] / p2dt
        bu = (up - aft) / (pos + 1e-15) * bt * I
        bd = (aft - do) / (neg + 1e-15) * bt * I
        lim = lambda a, x, y: torch.where(a >= 0, torch.minimum(x[0], x[1]), torch.minimum(y[0], y[1])).clamp(max=1)  # noqa: E731
        frozen = (lim(ax, (bd, E(bu)), (bu, E(bd))) * I, lim(ay, (bd, N(bu)), (bu, N(bd))) * I,
                  lim(az, (bd, U(bu)), (bu, U(bd))) * G.inn * G.mid)
    ax, ay, az = ax * frozen[0], ay * frozen[1], az * frozen[2]
    return ta - (ax - W(ax) + ay - So(ay) + az - D(az)) / G.e12t / e3["n"] * I, frozen


def iso_coef(G, S, nam):
    E, W, So = lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, -1)
    U = lambda a: sh(a, dk=-1)  # noqa: E731
    au, av = nam["rn_aht_0"] * G.um * G.up, nam["rn_aht_0"] * G.vm * G.up
    ku = G.wm / (U(G.um) + W(G.um) + U(W(G.um)) + G.um).clamp(min=1)
    kv = G.wm / (U(G.vm) + So(G.vm) + U(So(G.vm)) + G.vm).clamp(min=1)
    hu, hv = (U(au) + W(au) + U(W(au)) + au) * ku, (U(av) + So(av) + U(So(av)) + av) * kv
    ah = (hu * S["wslpi"] ** 2 + hv * S["wslpj"] ** 2) * G.inn * G.mid
    return au, av, ku, kv, hu, hv, ah


def ex_iso(G, S, nam, e3, tb):
    """The iso-neutral trend (tra_ldf_iso, first pass, laplacian) of tracers (member, 2, ...)."""
    e3 = {k: (v[:, None] if v.dim() == 4 else v) for k, v in e3.items()}
    E, W, N, So = lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, 1), lambda a: sh(a, 0, -1)
    U, D = lambda a: sh(a, dk=-1), lambda a: sh(a, dk=1)
    au, av, ku, kv, hu, hv, _ = iso_coef(G, S, nam)
    us, vs, wi, wj = [S[n][:, None] for n in SLOPES]
    cut = torch.ones_like(G.inn)
    cut[-1], cut[:, -1] = 0, 0
    di, dj = (E(tb) - tb) * G.um * G.up, (N(tb) - tb) * G.vm * G.up
    if nam["ln_zps"]:
        di = torch.where((G.lev == G.mbku - 1) & (cut > 0), S["gtsu"][:, :, None], di)
        dj = torch.where((G.lev == G.mbkv - 1) & (cut > 0), S["gtsv"][:, :, None], dj)
    below = (tb - D(tb)) * D(G.wm)
    here = torch.where(G.lev == 0, below, (U(tb) - tb) * G.wm)
    mu = 1 / (E(G.wm) + D(G.wm) + D(E(G.wm)) + G.wm).clamp(min=1)
    mv = 1 / (N(G.wm) + D(G.wm) + D(N(G.wm)) + G.wm).clamp(min=1)
    fu = (au * G.e2u / G.e1u * e3["u"] * di - au * G.e2u * us * mu * (E(here) + below + E(below) + here)) * G.um * G.up
    fv = (av * G.e1v / G.e2v * e3["v"] * dj - av * G.e1v * vs * mv * (N(here) + below + N(below) + here)) * G.vm * G.up
    fw = (-hu * G.e2t * ku * wi * (U(di) + W(di) + U(W(di)) + di) - hv * G.e1t * kv * wj * (
        U(dj) + So(dj) + U(So(dj)) + dj)) * G.mid * G.inn
    return (fu - W(fu) + fv - So(fv) + fw - D(fw)) / G.e12t / e3["n"] * G.inn * G.up


def ex_zdf(G, S, nam, e3, ah, tb, ta):
    """The implicit vertical diffusion (tra_zdf_imp): the after tracers, zero on the frame."""
    p2dt = 2 * nam["rn_rdt"]
    k3 = lambda a, k: a[:, None, k] if a.dim() == 4 else a[k]  # noqa: E731
    kz = S["avt"] + ah
    kz = torch.where(G.lev == 0, torch.zeros_like(kz), kz)
    K = G.jpk
    piv, x, sup = [], [], []
    for k in range(K - 1):
        lo = -p2dt * k3(kz, k) / k3(e3["w"], k)
        su = -p2dt * k3(kz, k + 1) / k3(e3["w"], k + 1)
        d = k3(e3["a"], k) - lo - su
        rhs = k3(e3["b"], k) * tb[:, :, k] + p2dt * k3(e3["n"], k) * ta[:, :, k]
        if k:
            d = d - lo * sup[-1] / piv[-1]
            rhs = rhs - lo / piv[-1] * x[-1]
        piv.append(d)
        x.append(rhs)
        sup.append(su)
    x[-1] = x[-1] / piv[-1] * G.tm[K - 2]
    for k in range(K - 3, -1, -1):
        x[k] = (x[k] - sup[k] * x[k + 1]) / piv[k] * G.tm[k]
    return torch.where(G.inn * G.up > 0, torch.stack(x + [torch.zeros_like(x[0])], 2), ta)


def ex_tracers(G, S, nam, order):
    e3 = e3_of(G, S, nam)
    w2 = lambda a: a * G.up  # noqa: E731
    zun, zvn, zwn = w2(G.e2u * e3["u"] * S["un"]), w2(G.e1v * e3["v"] * S["vn"]), w2(G.e12t * S["wn"])
    ah = iso_coef(G, S, nam)[-1]
    ta, _ = ex_fct(G, S, nam, e3, zun, zvn, zwn, S["tsb"], S["tsn"], order)
    ta = ta + ex_iso(G, S, nam, e3, S["tsb"])
    ta = ex_zdf(G, S, nam, e3, ah, S["tsb"], ta)
    return dict(zun=zun, zvn=zvn, zwn=zwn, tsa=ta, ah_wslp2=ah, akz=ah)


def ex_lap(G, S, nam):
    e3 = {k: (v[:, None] if v.dim() == 4 else v) for k, v in e3_of(G, S, nam).items()}
    a, tb = nam["rn_aht_0"], S["tsb"]
    cut = torch.ones_like(G.inn)
    cut[-1], cut[:, -1] = 0, 0
    di, dj = sh(tb, 1) - tb, sh(tb, 0, 1) - tb
    if nam["ln_zps"]:
        di = torch.where((G.lev == G.mbku - 1) & (cut > 0), S["gtsu"][:, :, None], di)
        dj = torch.where((G.lev == G.mbkv - 1) & (cut > 0), S["gtsv"][:, :, None], dj)
    fu, fv = a * G.um * G.up * G.e2u / G.e1u * e3["u"] * di, a * G.vm * G.up * G.e1v / G.e2v * e3["v"] * dj
    ta = (fu - sh(fu, -1) + fv - sh(fv, 0, -1)) / (G.e12t * e3["n"]) * G.inn * G.up
    total = (tb * G.ssm).sum((1, 2, 3, 4))
    return dict(tsa=ta, sum=[float(x) for x in total])


def ex_momentum(G, S, nam):
    I = G.inn * G.up
    E, W, N, So = lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, 1), lambda a: sh(a, 0, -1)
    U, D = lambda a: sh(a, dk=-1), lambda a: sh(a, dk=1)
    un, vn, wn, ub, vb = S["un"], S["vn"], S["wn"], S["ub"], S["vb"]
    ke = 0.25 * (W(un) ** 2 + un ** 2 + So(vn) ** 2 + vn ** 2)
    ua, va = -(E(ke) - ke) / G.e1u, -(N(ke) - ke) / G.e2v
    w = 0.25 * G.e12t * wn
    au, av = (E(w) + w) * (U(un) - un) * G.mid, (N(w) + w) * (U(vn) - vn) * G.mid
    ua, va = ua - (au + D(au)) / G.e12u / G.e3u_0, va - (av + D(av)) / G.e12v / G.e3v_0
    cut = torch.ones_like(G.inn)
    cut[-1], cut[:, -1] = 0, 0
    curl = lambda u, v: (E(G.e2v * v) - G.e2v * v - N(G.e1u * u) + G.e1u * u) / (G.e1f * G.e2f) * cut  # noqa: E731
    z = G.ff_f * cut + curl(un, vn)
    fx, fy = G.e2u * un, G.e1v * vn
    ua = ua + 0.25 / G.e1u * (So(z) * (So(fy) + sh(fy, 1, -1)) + z * (fy + E(fy)))
    va = va - 0.25 / G.e2v * (W(z) * (W(fx) + sh(fx, -1, 1)) + z * (fx + N(fx)))
    ahmt, ahmf = 1e5 * G.tm * G.up, 1e5 * G.tm * sh(G.tm, 1) * sh(G.tm, 0, 1) * sh(G.tm, 1, 1) * G.up
    cu = ahmf * G.e3f_0 * curl(ub, vb)
    gx, gy = G.e2u * G.e3u_0 * ub, G.e1v * G.e3v_0 * vb
    dv = ahmt / G.e12t / G.e3t_0 * (gx - W(gx) + gy - So(gy))
    ua = ua - (cu - So(cu)) / G.e2u / G.e3u_0 + (E(dv) - dv) / G.e1u
    va = va + (cu - W(cu)) / G.e1v / G.e3v_0 + (N(dv) - dv) / G.e2v
    rhd = density(G, nam, S["tsn"])[0]
    rhd = rhd.float().to(F64) if rounded(S) else rhd
    c = -0.5 * nam["grav"] * G.e3w_0
    both = rhd + U(rhd)                                         # at the surface: the first level alone
    hx, hy = (c * (E(both) - both) / G.e1u).cumsum(1), (c * (N(both) - both) / G.e2v).cumsum(1)
    return dict(ua=(ua + hx) * I, va=(va + hy) * I)


def rounded(S):
    return S.get("_mixed", False)


def ex_density(G, S, nam):
    ab, an = expansion(G, nam, S["tsb"]), expansion(G, nam, S["tsn"])
    rhd, rhop = density(G, nam, S["tsn"])
    return dict(rab_b=ab, rab_n=an, rn2b=brunt(G, nam, S["tsb"], ab), rn2=brunt(G, nam, S["tsn"], an), rhd=rhd, rhop=rhop)


def ex_physics(G, S, nam):
    """zdf_mxl and ldf_slp. The closure's switches (the Langmuir depth, convection where N2 <= -1e-12, the limits
    of the mixing length) take other branches in 64 bits, so its fields have no 64-bit value here."""
    E, W, N, So = lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, 1), lambda a: sh(a, 0, -1)
    U, D = lambda a: sh(a, dk=-1), lambda a: sh(a, dk=1)
    rhd, n2, K = S["rhd"], S["rn2b"], G.jpk
    col = torch.nonzero(G.mbkt.flatten() == G.mbkt.max())[0, 0]
    e3t, e3w = [a.reshape(K, -1)[:, col].cpu() for a in (G.e3t_0, G.e3w_0)]
    dep, ref, nlb = 0.0, 10.0 - 0.1 * float(e3w.min()), K
    for k in range(K):
        if dep > ref:
            nlb = k + 1
            break
        dep += float(e3t[k])
    acc = torch.zeros_like(n2[:, 0])
    ml = torch.full_like(acc, float(nlb))
    for k in range(nlb, K):
        acc = acc + n2[:, k - 1].clamp(min=0) * G.e3w_0[k - 1]
        ml = torch.where(acc < nam["grav"] * 0.01 / nam["rau0"], torch.clamp(G.mbkt, max=k) + 1, ml)
    at = lambda a, k: a.expand(n2.shape).gather(1, (k.long() - 1).clamp(0, K - 1)[:, None])[:, 0]  # noqa: E731
    hmlp, hmlpt = at(G.gdepw32, ml) * G.ssm, at(G.gdept32, ml - 1) * G.ssm
    eps, g = 1e-20, nam["grav"]
    gu, gv = G.um * (E(rhd) - rhd), G.vm * (N(rhd) - rhd)
    dz = -(rhd + 1) / g * (n2 + D(n2)) * (1 - 0.5 * D(G.tm)) * G.mid
    cap = lambda b, a, e3, s: torch.minimum(torch.minimum(b, -s * a.abs()), -7e3 / e3 * a.abs())  # noqa: E731
    s1 = 1 / (nam["rn_slpmax"] or 0.01)
    au, av = gu / G.e1u, gv / G.e2v
    bu, bv = cap(0.5 * (dz + E(dz)), au, G.e3u_0, s1), cap(0.5 * (dz + N(dz)), av, G.e3v_0, s1)
    su, sv = au / (bu - eps), av / (bv - eps)
    ku, kv = torch.maximum(ml, E(ml)).clamp(1, K - 1), torch.maximum(ml, N(ml)).clamp(1, K - 1)
    uml, vml = at(su * G.um, ku) * G.inn, at(sv * G.vm, kv) * G.inn
    bw = -0.5 / g * n2 * (rhd + U(rhd) + 2)
    ci = (W(G.um) + G.um + U(W(G.um)) + U(G.um)).clamp(min=eps) * G.e1t
    cj = (So(G.vm) + G.vm + U(So(G.vm)) + U(G.vm)).clamp(min=eps) * G.e2t
    ai0, aj0 = (W(gu) + gu + U(W(gu)) + U(gu)) / ci, (So(gv) + gv + U(So(gv)) + U(gv)) / cj
    wi = lambda a, k: a * k / (cap(bw, a * k, G.e3w_0, 100.0) - eps)  # noqa: E731
    kk = (ml + 1).clamp(max=K)
    wiml, wjml = at(wi(ai0, G.tm) * G.tm, kk) * G.inn, at(wi(aj0, G.tm) * G.tm, kk) * G.inn
    hu = uml / torch.maximum(hmlpt, E(hmlpt)).clamp(min=5)
    hv = vml / torch.maximum(hmlpt, N(hmlpt)).clamp(min=5)
    om = (G.lev + 1 <= ml[:, None] - 1).to(F64)
    I = G.inn * G.mid
    fi, fj = torch.maximum(om, E(om)), torch.maximum(om, N(om))
    gd = G.gdept32
    du, dv = 0.5 * (gd + E(gd) - G.e3u_0[:1]), 0.5 * (gd + N(gd) - G.e3v_0[:1])
    zu = ((1 - fi) * su + fi * du * hu[:, None]) * G.um * I
    zv = ((1 - fj) * sv + fj * dv * hv[:, None]) * G.vm * I

    def shapiro(a):
        return (sh(a, -1, -1) + sh(a, 1, -1) + sh(a, -1, 1) + sh(a, 1, 1)
                + 2 * (So(a) + W(a) + E(a) + N(a)) + 4 * a) / 16 * I

    us = shapiro(zu) * (N(G.um) + So(G.um)) * 0.5 * (G.um + D(G.um)) * 0.5
    vs = shapiro(zv) * (E(G.vm) + W(G.vm)) * 0.5 * (G.vm + D(G.vm)) * 0.5
    fk = torch.maximum(om, U(om))
    ck = (G.gdepw32 - G.gdepw32[:1]) / (hmlp[:, None] - G.gdepw32[:1]).clamp(min=10)
    zi = (wi(ai0, G.wm) * (1 - fk) + ck * wiml[:, None] * fk) * G.wm * I
    zj = (wi(aj0, G.wm) * (1 - fk) + ck * wjml[:, None] * fk) * G.wm * I
    coast = (G.um + W(G.um)) * (G.vm + So(G.vm)) * 0.25 * G.wm
    return dict(en=None, dissl=None, avm_k=None, avt_k=None, avm=None, avt=None, avs=None, nmln=None, hmlp=hmlp,
                hmlpt=hmlpt, uslp=us, vslp=vs, wslpi=shapiro(zi) * coast, wslpj=shapiro(zj) * coast)


def ex_stepping(G, S, nam):
    E, W, N, So = lambda a: sh(a, 1), lambda a: sh(a, -1), lambda a: sh(a, 0, 1), lambda a: sh(a, 0, -1)
    r2dt, atfp, rau0, K = 2 * nam["rn_rdt"], nam["rn_atfp"], nam["rau0"], G.jpk
    un, vn = S["un"], S["vn"]
    fx, fy = G.e2u * G.e3u_0 * un, G.e1v * G.e3v_0 * vn
    div = (fx - W(fx) + fy - So(fy)) / G.e12t * G.inn * G.up * G.tm
    out = dict(wn=-torch.flip(torch.flip(div, (1,)).cumsum(1), (1,)) * G.up)

    def column(b, bt, mask, e3, mbk, shift, tau):
        a = (b * mask - bt[:, None]) * mask * G.up
        drag = 0.5 * (shift(S["rcdu_bot"]) + S["rcdu_bot"])
        last = (G.lev == mbk - 1).to(F64) * G.inn
        a = a + last * (r2dt * drag * bt)[:, None] / e3
        wmx = mask * torch.cat([torch.ones_like(mask[:1]), mask[:-1]])
        e3x = torch.minimum(G.e3w_0, torch.where(shift(G.e3w_0) > 0, shift(G.e3w_0), G.e3w_0))
        avm = 0.5 * r2dt * (shift(S["avm"]) + S["avm"]) / e3x * wmx
        lo = torch.where(G.lev == 0, 0.0, -avm / e3)
        su = -sh(avm, dk=1) / e3
        d = 1 - lo - su - last * (r2dt * drag)[:, None] / e3
        rhs = a + (G.lev == 0) * (r2dt * tau / rau0 * mask[0])[:, None] / e3
        piv, x = [d[:, 0]], [rhs[:, 0]]
        for k in range(1, K - 1):
            piv.append(d[:, k] - lo[:, k] * su[:, k - 1] / piv[-1])
            x.append(rhs[:, k] - lo[:, k] / piv[k - 1] * x[-1])
        x[-1] = x[-1] / piv[-1]
        for k in range(K - 3, -1, -1):
            x[k] = (x[k] - su[:, k] * x[k + 1]) / piv[k]
        return torch.where(G.inn * G.up > 0, torch.stack(x + [torch.zeros_like(x[0])], 1), a)

    for c, e3, m, mbk, shift, r1h in (("u", G.e3u_0, G.um, G.mbku, E, G.r1_hu_0), ("v", G.e3v_0, G.vm, G.mbkv, N, G.r1_hv_0)):
        a = column(S[c + "b"], S[c + "a_b"], m, e3, mbk, shift, S[c + "tau"])
        mean = lambda x: (e3 * x * m * G.up).sum(1) * r1h  # noqa: E731
        a = torch.where(G.up > 0, (a - mean(a)[:, None] + S[c + "a_b"][:, None]) * m, a) * G.inn
        b, n = S[c + "b"], S[c + "n"]
        nb = torch.where(G.up > 0, n + atfp * (b - 2 * n + a), b)
        nb = nb - (mean(nb) - S[c + "n_b"])[:, None] * m * G.up
        out[c + "a"], out[c + "b"], out[c + "n"] = a, nb, torch.where(G.up > 0, a, n)
        out[c + "n_b"], out[c + "b_b"] = mean(out[c + "n"]), mean(nb)
    tb, tn, ta = S["tsb"], S["tsn"], S["tsa"] * G.inn
    I = G.inn * G.up > 0
    out["tsb"] = torch.where(I, tn + atfp * (ta - 2 * tn + tb), tb) * G.inn
    out["tsn"], out["tsa"] = torch.where(I, ta, tn) * G.inn, ta
    out["sshb"] = S["sshn"] + atfp * (S["sshb"] - 2 * S["sshn"] + S["ssha"])
    out["sshn"] = S["ssha"]
    return out


def ex_adjoint(G, S, nam):
    """The gradient of <ab, tsb'> + <an, tsn'> through one linear tracer step (limiter and coefficients held)."""
    e3 = e3_of(G, S, nam)
    tr = (G.e2u * e3["u"] * S["un"] * G.up, G.e1v * e3["v"] * S["vn"] * G.up, G.e12t * S["wn"] * G.up)
    ah = iso_coef(G, S, nam)[-1]
    with torch.no_grad():
        _, frozen = ex_fct(G, S, nam, e3, *tr, S["tsb"], S["tsn"], 2)
    tb, tn = S["tsb"].clone().requires_grad_(), S["tsn"].clone().requires_grad_()
    ta = ex_fct(G, S, nam, e3, *tr, tb, tn, 2, frozen)[0] + ex_iso(G, S, nam, e3, tb)
    ta = ex_zdf(G, S, nam, e3, ah, tb, ta) * G.inn
    I = G.inn * G.up > 0
    nb = torch.where(I, tn + nam["rn_atfp"] * (ta - 2 * tn + tb), tb) * G.inn
    nn = torch.where(I, ta, tn) * G.inn
    ab, an = torch.autograd.grad((S["ab"] * nb + S["an"] * nn).sum(), (tb, tn))
    return dict(ab=ab, an=an)


def exact(case, seed):
    nam = namelist(case)
    G = grid_of(case)
    S = state(G, case, nam, seed)
    S["_mixed"] = case["prec"] == "mixed"
    kind = case["kind"]
    if kind == "adjoint":
        return ex_adjoint(G, S, nam)
    with torch.no_grad():
        if kind == "step":
            out = ex_spg(G, S, nam)
            tr = ex_tracers(G, {**S, "un": out["un"], "vn": out["vn"]}, nam, nam["nn_fct_h"])
            sal = tr["tsa"][:, 1]
            tr["tsa"] = torch.stack([tr["tsa"][:, 0], torch.where(sal < 0, 0.1, sal)], 1)
            out.update({n: tr[n] for n in ("tsa", "ah_wslp2", "akz")})
            return out
        if kind == "tracers":
            return ex_tracers(G, S, nam, case["fct"])
        return {"spg": ex_spg, "lap": ex_lap, "momentum": ex_momentum, "density": ex_density, "physics": ex_physics,
                "stepping": ex_stepping}[kind](G, S, nam)
