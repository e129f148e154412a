// k_adj.cuh -- adjoint kernels of the tracer routines (FP64), and tra_nxt.
//
// NEMO has no adjoint of these routines in its tree (its tangent-linear/adjoint,
// NEMOTAM, is a separate project); each kernel here is the transpose of the
// tangent-linear of the forward kernel with respect to the tracer arguments, with
// the coefficients (transports, diffusivities, slopes, scale factors, avt) held
// fixed and, for FCT, the limiter multipliers that the forward recorded.
//
// Gather form: one thread per (i,j,k) point computes the adjoint of the tracer at
// its own point by collecting the terms of every face flux that read it, so no two
// threads write one element and the result does not depend on scheduling. The
// face adjoints that several points share are recomputed by each of them.
// Conventions (those of the host mirror): an adjoint accumulates into the adjoints
// of the inputs (tb_ad += ...); a trend array that the forward only adds to keeps
// its adjoint unchanged.
#pragma once
#include "adj.h"

namespace nemo {

// 1-based point helpers of the gather kernels
struct Pt3 {
  int jpi, jpj, jpk;
  long n2;
  __device__ __forceinline__ long ij(int i, int j) const { return (long)(i - 1) + (long)(j - 1) * jpi; }
  __device__ __forceinline__ long q(int i, int j, int k) const { return ij(i, j) + (long)(k - 1) * n2; }
  // interior cell of a trend loop: 2..jpim1, 2..jpjm1, 1..jpkm1
  __device__ __forceinline__ bool cell(int i, int j, int k) const {
    return i >= 2 && i <= jpi - 1 && j >= 2 && j <= jpj - 1 && k >= 1 && k <= jpk - 1;
  }
  // an east (u) face of a flux loop: 1..jpim1, 1..jpjm1, 1..jpkm1
  __device__ __forceinline__ bool uface(int i, int j, int k) const {
    return i >= 1 && i <= jpi - 1 && j >= 1 && j <= jpj - 1 && k >= 1 && k <= jpk - 1;
  }
  __device__ __forceinline__ bool icol(int i, int j) const { return i >= 2 && i <= jpi - 1 && j >= 2 && j <= jpj - 1; }
};
template <class T>
__device__ __forceinline__ Pt3 pt3(const Dom<T>& d) { return Pt3{d.jpi, d.jpj, d.jpk, d.n2}; }

// x / e3t_n(k) and x / e3w_n(k): through the reciprocal profile (the correctly rounded
// quotient; divr for the first, whose x holds sensitivities that may be infinite) where the
// now scale factor is the rest-state profile
__device__ __forceinline__ double over_e3t(const Dom<double>& d, double x, long ij, int k, int m) {
  const double e = d.e3t_n(ij, k, m);
  return d.r1_e3t && d.e3t_n.s == 0 ? divr(x, e, d.r1_e3t[k - 1]) : x / e;
}
__device__ __forceinline__ double over_e3w(const Dom<double>& d, double x, long ij, int k, int m) {
  const double e = d.e3w_n(ij, k, m);
  return d.r1_e3w && d.e3w_n.s == 0 ? divq(x, e, d.r1_e3w[k - 1]) : x / e;
}
// x != 0 on the integer pipe (NaN counts as nonzero)
__device__ __forceinline__ bool nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }

// x times a zero, on the integer pipe: NaN where x is not finite
__device__ __forceinline__ double zero_of(double x) {
  return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000 ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
}

// ------------------------------------------------------------------ tra_adv_fct
// Adjoint of tra_adv_fct (traadv_fct.F90:54-327) with kn_fct_h = 4, the 4th-order centred
// horizontal fluxes (:191-227), at one point (2: k_fct_adj2 below); with kn_fct_v = 4 the
// compact vertical interpolation's part is k_fct_adj_v4's. With g = lam r1_e1e2t / e3t_n
// and h = g tmask on the interior cells (0 elsewhere), the limited antidiffusive flux of face f has the adjoint
// -(g(f) - g(f+1)); times the recorded multiplier (0 where the forward zeroed the
// flux) it is the adjoint of the flux before limiting, the centred flux of tn minus
// the upstream flux of tb (:182-190, :255-263). The upstream flux gets minus that,
// plus -(h(f) - h(f+1)) from its own trend (:158-170), and passes it to tb
// (:123-156).
__global__ void __launch_bounds__(128) k_fct_adj(Dom<double> d, FctAdj a) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const Pt3 P = pt3(d);
  const int i = c.i, j = c.j, k = c.k, jpi = d.jpi, jpk = d.jpk;
  const long q = c.q, n2 = d.n2, n3 = d.n3, mv = (long)c.m * n3;
  const RO<double> un = a.pun + mv;
  const RO<double> vn = a.pvn + mv;
  const RO<double> wn = a.pwn + mv;
  const bool ic = P.icol(i, j);
  const bool fe = P.uface(i, j, k), fw = P.uface(i - 1, j, k);
  const bool fn = P.uface(i, j, k), fs = P.uface(i, j - 1, k);  // v faces share the u ranges
  // vertical faces of the column: top (level k) and bottom (level k+1), antidiffusive
  // part on interior columns for levels 2..jpkm1, upstream part on every column
  const bool zt = ic && k >= 2 && k <= jpk - 1, zb = ic && k + 1 >= 2 && k + 1 <= jpk - 1;
  const bool ut = k >= 2 && k <= jpk - 1, ub = k + 1 <= jpk - 1;
  const ColInfo ci = d.ci[c.ij];
  const double wmt = wmsk<double>(ci, k), wmb = wmsk<double>(ci, k + 1);
  for (int n = 0; n < a.kjpt; ++n) {
    const long mo = ((long)c.m * a.kjpt + n) * n3;
    const RO<double> lam = a.lam + mo;
    const RO<double> tx = a.tape + ((long)c.m * a.kjpt + n) * 3 * n3;
    const RO<double> ty = tx + n3;
    const RO<double> tz = tx + 2 * n3;
    auto g = [&](int ii, int jj, int kk) -> double {
      if (!P.cell(ii, jj, kk)) return 0.0;
      const long o = P.ij(ii, jj);
      return over_e3t(d, lam[P.q(ii, jj, kk)] * d.r1_e1e2t[o], o, kk, c.m);
    };
    const double gc = g(i, j, k), ge = g(i + 1, j, k), gw = g(i - 1, j, k), gn = g(i, j + 1, k),
                 gs = g(i, j - 1, k), gu = g(i, j, k - 1), gd = g(i, j, k + 1);
    const double tmc = tmsk<double>(ci, k);
    const double hc = gc * tmc;
    const double he = fe ? ge * tmsk<double>(d.ci[c.ij + 1], k) : 0.0;
    const double hw = fw ? gw * tmsk<double>(d.ci[c.ij - 1], k) : 0.0;
    const double hn = fn ? gn * tmsk<double>(d.ci[c.ij + jpi], k) : 0.0;
    const double hs = fs ? gs * tmsk<double>(d.ci[c.ij - jpi], k) : 0.0;
    const double hu = k >= 2 ? gu * tmsk<double>(ci, k - 1) : 0.0;
    const double hd = k + 1 <= jpk ? gd * tmsk<double>(ci, k + 1) : 0.0;
    // limited antidiffusive fluxes -> their adjoints before limiting
    const double axe = fe ? tx[q] * (ge - gc) : 0.0;
    const double axw = fw ? tx[q - 1] * (gc - gw) : 0.0;
    const double ayn = fn ? ty[q] * (gn - gc) : 0.0;
    const double ays = fs ? ty[q - jpi] * (gc - gs) : 0.0;
    const double azt = zt ? tz[q] * (gu - gc) * wmt : 0.0;
    const double azb = zb ? tz[q + n2] * (gc - gd) * wmb : 0.0;
    double tnv = 0.0;
    if (fe) tnv += 0.5 * un[q] * axe;
    if (fw) tnv += 0.5 * un[q - 1] * axw;
    if (fn) tnv += 0.5 * vn[q] * ayn;
    if (fs) tnv += 0.5 * vn[q - jpi] * ays;
    if (a.kv == 2) {
      if (zt) tnv += wn[q] * 0.5 * azt;
      if (zb) tnv += wn[q + n2] * 0.5 * azb;
    }
    // zltu(m) = (ztu(m) + ztu(m-1)) / 6 enters the flux of u-face m with + and that
    // of face m-1 with -; ztu(m) = (tn(m+1) - tn(m)) umask(m). S: the adjoint of a
    // face's centred bracket; Z: of zltu (interior points only, lbc_lnk zeroes the
    // edges). Likewise in j.
    auto Su = [&](int fi) -> double {
      if (!P.uface(fi, j, k)) return 0.0;
      const long qf = P.q(fi, j, k);
      return 0.5 * un[qf] * (tx[qf] * (g(fi + 1, j, k) - g(fi, j, k)));
    };
    auto Sv = [&](int fj) -> double {
      if (!P.uface(i, fj, k)) return 0.0;
      const long qf = P.q(i, fj, k);
      return 0.5 * vn[qf] * (ty[qf] * (g(i, fj + 1, k) - g(i, fj, k)));
    };
    auto Zu = [&](int mi) -> double { return P.cell(mi, j, k) ? Su(mi) - Su(mi - 1) : 0.0; };
    auto Zv = [&](int mj) -> double { return P.cell(i, mj, k) ? Sv(mj) - Sv(mj - 1) : 0.0; };
    const double zu0 = Zu(i - 1), zu1 = Zu(i), zu2 = Zu(i + 1);
    const double zv0 = Zv(j - 1), zv1 = Zv(j), zv2 = Zv(j + 1);
    const double r1_6 = 1. / 6.;
    if (i >= 2) tnv += r1_6 * (zu0 + zu1) * umsk<double>(d.ci[c.ij - 1], k);
    tnv -= r1_6 * (zu1 + zu2) * umsk<double>(ci, k);
    if (j >= 2) tnv += r1_6 * (zv0 + zv1) * vmsk<double>(d.ci[c.ij - jpi], k);
    tnv -= r1_6 * (zv1 + zv2) * vmsk<double>(ci, k);
    // upstream fluxes: minus the antidiffusive adjoint plus their own trend's
    const double fxe = -axe + (he - hc), fxw = -axw + (hc - hw);
    const double fyn = -ayn + (hn - hc), fys = -ays + (hc - hs);
    const double fzt = -azt + (hu - hc), fzb = -azb + (hc - hd);
    double tbv = 0.0;
    if (fe) { const double u = un[q]; tbv += 0.5 * (u + fabs(u)) * fxe; }
    if (fw) { const double u = un[q - 1]; tbv += 0.5 * (u - fabs(u)) * fxw; }
    if (fn) { const double v = vn[q]; tbv += 0.5 * (v + fabs(v)) * fyn; }
    if (fs) { const double v = vn[q - jpi]; tbv += 0.5 * (v - fabs(v)) * fys; }
    if (ut) { const double w = wn[q]; tbv += (w + fabs(w)) * (0.5 * fzt * wmt); }
    if (ub) { const double w = wn[q + n2]; tbv += (w - fabs(w)) * (0.5 * fzb * wmb); }
    if (k == 1 && a.linssh) tbv += wn[q] * fzt;  // surface flux w tb (:146-156)
    a.tb_ad[mo + q] += tbv;
    a.tn_ad[mo + q] += tnv;
  }
}

// tra_adv_fct's adjoint with kn_fct_h = 2: a block marches down a chunk of kch levels over
// a tile of 32 x FADJ_Y points, one column a thread; each weight g and each face adjoint
// is formed once a tile, by the point that owns it, and passed to its neighbour by a
// shuffle (i) or through shared memory (j). The outer ring of the tile only feeds its
// inside (30 x (FADJ_Y - 2) points are written). Bound by the FP64 pipe: a point of
// k_fct_adj divides seven times a tracer and forms all six faces (1053 us at
// 302x202x31, T and S), 420 so. Values as k_fct_adj's: an upstream flux's adjoint f reaches the
// point upstream of its face as u f and the other as zero_of(u f) (0.5 (u + |u|) is u or 0).
constexpr int FADJ_Y = 16, FADJ_K = 8;  // the tile's rows, the most levels a chunk
__global__ void __launch_bounds__(32 * FADJ_Y) k_fct_adj2(Dom<double> d, FctAdj a, int kch) {
  constexpr int NT = 2;
  __shared__ double sg[NT][FADJ_Y][32], sp[NT][FADJ_Y][32], sr[NT][FADJ_Y][32];
  const int lane = threadIdx.x, row = threadIdx.y, jpi = d.jpi, jpk = d.jpk;
  const int i = blockIdx.x * 30 + lane, j = blockIdx.y * (FADJ_Y - 2) + row;  // 1-based, 0: outside
  const int nch = (jpk - 1 + kch - 1) / kch, m = blockIdx.z / nch;
  const int k0 = (int)(blockIdx.z - m * nch) * kch + 1, k1 = min(k0 + kch - 1, jpk - 1);
  const Pt3 P = pt3(d);
  const bool in = i >= 1 && i <= jpi && j >= 1 && j <= d.jpj;
  const bool own = in && lane >= 1 && lane <= 30 && row >= 1 && row <= FADJ_Y - 2;
  const bool ic = in && P.icol(i, j), face = in && i <= jpi - 1 && j <= d.jpj - 1;
  // the halo's weights are needed inside; its faces west and south of the tile's inside
  const long ij = in ? P.ij(i, j) : 0, n2 = d.n2, n3 = d.n3, mv = (long)m * n3;
  const bool last = lane == 31 || row == FADJ_Y - 1;  // no east / north neighbour in the tile
  const bool fx = face && !last;
  const ColInfo ci = d.ci[ij];
  ColInfo ce{}, cn{};
  if (fx) {
    ce = d.ci[ij + 1];
    cn = d.ci[ij + jpi];
  }
  const double r1 = d.r1_e1e2t[ij];
  const RO<double> un = a.pun + mv, vn = a.pvn + mv, wn = a.pwn + mv;
  for (int n0 = 0; n0 < a.kjpt; n0 += NT) {
    const int nt = a.kjpt - n0 < NT ? a.kjpt - n0 : NT;
    auto g = [&](int n, int k) -> double {  // lam r1_e1e2t / e3t_n of the own column
      return ic && k <= jpk - 1 ? over_e3t(d, a.lam[((long)m * a.kjpt + n) * n3 + ij + (long)(k - 1) * n2] * r1, ij, k, m)
                                : 0.0;
    };
    // carried: g(k); the parts of the top face of level k that its column gets below it
    double gc[NT] = {}, pz[NT] = {}, rz[NT] = {};
    // the vertical face between levels k-1 and k (weights gu, gk): its centred part on tn
    // and its upstream part, with w > 0 for the level below (k), w < 0 for that above
    auto zface = [&](int n, int k, double gu, double gk, double& p, double& r) {
      p = 0.0;
      r = 0.0;
      if (!in || k < 2 || k > jpk - 1) return;
      const long q = ij + (long)(k - 1) * n2;
      const double w = wn[q], wm = wmsk<double>(ci, k);
      double az = 0.0;
      if (ic) {
        az = msel(a.tape[(((long)m * a.kjpt + n) * 3 + 2) * n3 + q] * (gu - gk), wm);
        if (a.kv == 2) p = w * 0.5 * az;
      }
      const double fz = -az + (msel(gu, tmsk<double>(ci, k - 1)) - msel(gk, tmsk<double>(ci, k)));
      r = msel(w * fz, wm);
    };
    for (int nn = 0; nn < nt; ++nn) {
      gc[nn] = g(n0 + nn, k0);
      if (k0 > 1) zface(n0 + nn, k0, g(n0 + nn, k0 - 1), gc[nn], pz[nn], rz[nn]);
    }
    for (int k = k0; k <= k1; ++k) {
      const long q = ij + (long)(k - 1) * n2;
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) sg[nn][row][lane] = gc[nn];
      __syncthreads();
      const double u = fx ? un[q] : 0.0, v = fx ? vn[q] : 0.0;
      const double tm = tmsk<double>(ci, k);
      double px[NT], rx[NT], py[NT], ry[NT];
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) {
        const double ge = __shfl_down_sync(0xffffffffu, gc[nn], 1);
        px[nn] = rx[nn] = py[nn] = ry[nn] = 0.0;
        if (fx && nn < nt) {
          const RO<double> tx = a.tape + ((long)m * a.kjpt + n0 + nn) * 3 * n3;
          const double gn = sg[nn][row + 1][lane], hc = msel(gc[nn], tm);
          const double ax = tx[q] * (ge - gc[nn]), ay = tx[n3 + q] * (gn - gc[nn]);
          px[nn] = 0.5 * u * ax;
          py[nn] = 0.5 * v * ay;
          rx[nn] = u * (-ax + (msel(ge, tmsk<double>(ce, k)) - hc));
          ry[nn] = v * (-ay + (msel(gn, tmsk<double>(cn, k)) - hc));
        }
        sp[nn][row][lane] = py[nn];
        sr[nn][row][lane] = sgn_pos(v) ? zero_of(ry[nn]) : ry[nn];  // for the northern point
      }
      __syncthreads();
      const double wt = own && k >= 2 ? wn[q] : 0.0;
      const double wb = own && k + 1 <= jpk - 1 ? wn[q + n2] : 0.0;
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) {
        const double pw = __shfl_up_sync(0xffffffffu, px[nn], 1);
        const double rw = __shfl_up_sync(0xffffffffu, sgn_pos(u) ? zero_of(rx[nn]) : rx[nn], 1);
        if (nn >= nt) continue;
        const int n = n0 + nn;
        const double gd = g(n, k + 1);
        double pb, rb;
        zface(n, k + 1, gc[nn], gd, pb, rb);
        if (own) {
          const double tnv = px[nn] + pw + py[nn] + sp[nn][row - 1][lane] + pz[nn] + pb;
          double tbv = (sgn_pos(u) ? rx[nn] : zero_of(rx[nn])) + rw + (sgn_pos(v) ? ry[nn] : zero_of(ry[nn])) +
                       sr[nn][row - 1][lane];
          tbv += sgn_pos(wt) ? rz[nn] : zero_of(rz[nn]);
          tbv += sgn_pos(wb) ? zero_of(rb) : rb;
          if (k == 1 && a.linssh) tbv += wn[q] * -msel(gc[nn], tm);  // surface flux w tb (:146-156)
          const long o = ((long)m * a.kjpt + n) * n3 + q;
          a.tb_ad[o] += tbv;
          a.tn_ad[o] += tnv;
        }
        gc[nn] = gd;
        pz[nn] = pb;
        rz[nn] = rb;
      }
    }
  }
}

// With kn_fct_v = 4 (traadv_fct.F90:253-275): the vertical antidiffusive flux reads
// ztw = M^-1 R tn of interp_4th_cpt (:517-616). One interior column a thread: the
// adjoint V(k) = wn(k) az(k) of ztw(k), k = 2..jpk-1, then tn_ad += R^T M^-T V with
// the forward's rows (special top and bottom rows), pivots zwt, the back
// substitution undone forwards and the elimination backwards (as the oracle's
// ora_interp_4th_cpt_adj). Runs after k_fct_adj, which leaves this part out.
__global__ void k_fct_adj_v4(Dom<double> d, FctAdj a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i < 2 || i > d.jpi - 1 || j < 2 || j > d.jpj - 1) return;
  const int m = blockIdx.z, jpk = d.jpk;
  const Pt3 P = pt3(d);
  const long ij = P.ij(i, j), n2 = d.n2, n3 = d.n3, c3 = (long)m * n3 + ij;
  const ColInfo ci = d.ci[ij];
  const int ikt = 2, ikb = d.mbkt[ij];
  const RO<double> wn = a.pwn + (long)m * n3;
  const double r1 = d.r1_e1e2t[ij];
  auto row = [&](int k, double& dd, double& wi, double& ws, double& w) {
    const double wm = wmsk<double>(ci, k);
    if (k == ikt || k == ikb) { dd = 1.0; wi = 0.0; ws = 0.0; w = 0.5; }
    else { dd = 3.0 * wm + 1.0; wi = wm; ws = wm; w = 3.0 * wm; }
  };
  // the pivots (the same for every tracer)
  {
    double dd, wi, ws, w, wsp;
    row(2, dd, wi, wsp, w);
    a.zwt[c3 + n2] = dd;
    double tp = dd;
    for (int k = 3; k <= jpk - 1; ++k) {
      row(k, dd, wi, ws, w);
      tp = dd - wi * wsp / tp;
      a.zwt[c3 + (long)(k - 1) * n2] = tp;
      wsp = ws;
    }
  }
  for (int n = 0; n < a.kjpt; ++n) {
    const long mo = ((long)m * a.kjpt + n) * n3;
    const RO<double> lam = a.lam + mo;
    const RO<double> tz = a.tape + ((long)m * a.kjpt + n) * 3 * n3 + 2 * n3;
    auto g = [&](int k) -> double {
      return (k >= 1 && k <= jpk - 1) ? lam[ij + (long)(k - 1) * n2] * r1 / d.e3t_n(ij, k, m) : 0.0;
    };
    // V into za, then the back substitution undone (za: the adjoint of z)
    for (int k = 2; k <= jpk - 1; ++k) {
      const long q = ij + (long)(k - 1) * n2;
      const double az = tz[q] * (g(k - 1) - g(k)) * wmsk<double>(ci, k);
      a.za[c3 + (long)(k - 1) * n2] = wn[q] * az;
    }
    double carry = 0.0;
    for (int k = 2; k <= jpk - 2; ++k) {
      const long o = c3 + (long)(k - 1) * n2;
      double dd, wi, ws, w;
      row(k, dd, wi, ws, w);
      const double x = a.za[o] + carry;
      const double z = x / a.zwt[o];
      a.za[o] = z;
      carry = -ws * z;
    }
    {
      const long o = c3 + (long)(jpk - 2) * n2;
      a.za[o] = (a.za[o] + carry) / a.zwt[o];
    }
    // the elimination undone, then the right-hand side transposed
    double zk = a.za[c3 + (long)(jpk - 2) * n2];
    for (int k = jpk - 1; k >= 2; --k) {
      double dd, wi, ws, w;
      row(k, dd, wi, ws, w);
      const long o = c3 + (long)(k - 1) * n2;
      if (k >= 3) {
        const long om = o - n2;
        const double zm = a.za[om] - wi / a.zwt[om] * zk;
        a.za[om] = zm;
      }
      a.tn_ad[mo + ij + (long)(k - 1) * n2] += w * zk;
      a.tn_ad[mo + ij + (long)(k - 2) * n2] += w * zk;
      if (k >= 3) zk = a.za[o - n2];
    }
  }
}

// ------------------------------------------------------------------ tra_ldf_lap
// Adjoint of tra_ldf_lap (traldf_lap_blp.F90:95-145) at one point: the fluxes of
// the east and north faces of (i-1,j), (i,j), (i,j-1). A partial-step bottom face
// (k = mbku) takes the fixed pgu and passes nothing to tb.
__global__ void __launch_bounds__(128) k_lap_adj(Dom<double> d, LdfArgs<double> a, LdfAdj b) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const Pt3 P = pt3(d);
  const int i = c.i, j = c.j, k = c.k, jpi = d.jpi;
  const long q = c.q, n3 = d.n3;
  for (int n = 0; n < a.kjpt; ++n) {
    const long mo = ((long)c.m * a.kjpt + n) * n3;
    const RO<double> lam = b.lam + mo;
    auto g = [&](int ii, int jj) -> double {
      if (!P.cell(ii, jj, k)) return 0.0;
      const long o = P.ij(ii, jj);
      return lam[P.q(ii, jj, k)] / (d.e1e2t[o] * d.e3t_n(o, k, c.m));
    };
    // u face of column (ii,jj): zaheeu * (g(ii,jj) - g(ii+1,jj))
    auto fu = [&](int ii, int jj) -> double {
      if (!P.uface(ii, jj, k)) return 0.0;
      const long o = P.ij(ii, jj);
      const ColInfo cc = d.ci[o];
      if (a.zps && k == cc.mbku) return 0.0;
      const double z = a.zsign * ahu(d, a, cc, o, k, c.m) * d.e2_e1u[o] * d.e3u_n(o, k, c.m);
      return z * (g(ii, jj) - g(ii + 1, jj));
    };
    auto fv = [&](int ii, int jj) -> double {
      if (!P.uface(ii, jj, k)) return 0.0;
      const long o = P.ij(ii, jj);
      const ColInfo cc = d.ci[o];
      if (a.zps && k == cc.mbkv) return 0.0;
      const double z = a.zsign * ahv(d, a, cc, o, k, c.m) * d.e1_e2v[o] * d.e3v_n(o, k, c.m);
      return z * (g(ii, jj) - g(ii, jj + 1));
    };
    (void)jpi;
    b.tb_ad[mo + q] += fu(i - 1, j) - fu(i, j) + fv(i, j - 1) - fv(i, j);
  }
}

// ------------------------------------------------------------------ tra_ldf_iso
// The adjoint runs at the FP64 rate (1/58 of FP32: one FP64 operation per tracer cell
// costs as much time as 13 bytes of HBM traffic), so each coefficient and each product
// is formed once, by the point that owns its face, and kept in work arrays; as one
// gather kernel, in which every point formed the coefficients of its six w-points and
// eight faces for each tracer, the gradient stage alone took 2254 us at 302x202x31
// (T and S); the products take 172 and the gradient 245 us so.
//
// Stage 0: G = zsign lam r1_e1e2t / e3t_n on the interior cells, 0 elsewhere (the
// adjoint weight of a divergence, :278-284 and :359-366).
__global__ void __launch_bounds__(128) k_iso_adj_g(Dom<double> d, LdfArgs<double> a, LdfAdj b) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const Pt3 P = pt3(d);
  for (int n = 0; n < a.kjpt; ++n) {
    const long o = ((long)c.m * a.kjpt + n) * d.n3 + c.q;
    b.G[o] = P.cell(c.i, c.j, c.k) ? over_e3t(d, a.zsign * b.lam[o] * d.r1_e1e2t[c.ij], c.ij, c.k, c.m) : 0.0;
  }
}

// The vertical laplacian coefficients of the w-point (ij,k) on tb and on tbb, as the
// forward kernel forms them (traldf_iso.F90:337-357).
__device__ __forceinline__ void iso_adj_vlap(const Dom<double>& d, const LdfArgs<double>& a, long ij, int k, int m,
                                             double& ctb, double& ctbb) {
  const long qq = (long)m * d.n3 + ij + (long)(k - 1) * d.n2;
  const double f = msel(over_e3w(d, d.e1e2t[ij], ij, k, m), wmsk<double>(d.ci[ij], k));
  const double ahw = a.ah_wslp2[qq], akz = a.akz[qq];
  ctbb = 0.0;
  if (a.lap) ctb = f * (ahw - akz);
  else if (a.kpass == 1) ctb = ahw * f;
  else { ctb = ahw * f; ctbb = akz * f; }
}

// Stage 1: the products of the face and w-point coefficients (traldf_iso.F90:255-276
// horizontal, :297-332 vertical) with the differences of G their fluxes see. su, sv:
// cof1 (G - G(i+1)), cof2 (G - G(j+1)) at the u and v faces; t3, t4: zcoef3, zcoef4
// times the adjoint G(k) - G(k-1) of the vertical flux at the interior w-points.
__global__ void __launch_bounds__(128) k_iso_adj_prod(Dom<double> d, LdfArgs<double> a, LdfAdj b) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const Pt3 P = pt3(d);
  const int i = c.i, j = c.j, k = c.k, m = c.m, jpi = d.jpi;
  const long n3 = d.n3, q = c.q, qm = (long)m * n3 + q, ij = c.ij;
  const bool face = P.uface(i, j, k), wpt = P.icol(i, j) && k >= 2 && k <= d.jpk - 1;
  const ColInfo ci = d.ci[ij];
  double cof1 = 0.0, cof2 = 0.0, c3 = 0.0, c4 = 0.0;
  if (face) {
    const ColInfo ce = d.ci[ij + 1], cn = d.ci[ij + jpi];
    const double w0 = wmsk<double>(ci, k), w1 = wmsk<double>(ci, k + 1);
    const double zu = rcount4(wmsk<double>(ce, k), w1, wmsk<double>(ce, k + 1), w0);
    const double zv = rcount4(wmsk<double>(cn, k), w1, wmsk<double>(cn, k + 1), w0);
    cof1 = msel(-ahu(d, a, ci, ij, k, m) * d.e2u[ij] * a.uslp[qm] * zu, umsk<double>(ci, k));
    cof2 = msel(-ahv(d, a, ci, ij, k, m) * d.e1v[ij] * a.vslp[qm] * zv, vmsk<double>(ci, k));
  }
  if (wpt) {
    const IsoW<double> w = iso_w(d, a, ij, k, m, ci, d.ci[ij - 1], d.ci[ij - jpi]);
    c3 = -w.zahu_w * d.e2t[ij] * w.zmsku * a.wslpi[qm];
    c4 = -w.zahv_w * d.e1t[ij] * w.zmskv * a.wslpj[qm];
  }
  for (int n = 0; n < a.kjpt; ++n) {
    const long o = ((long)m * a.kjpt + n) * n3 + q;
    const RO<double> G = b.G;
    const double g = G[o];
    b.su[o] = face ? cof1 * (g - G[o + 1]) : 0.0;
    b.sv[o] = face ? cof2 * (g - G[o + jpi]) : 0.0;
    double t3 = 0.0, t4 = 0.0;
    if (wpt) {
      const double t = g - G[o - d.n2];
      if (nonzero(t)) {
        t3 = c3 * t;
        t4 = c4 * t;
      }
    }
    b.t3[o] = t3;
    b.t4[o] = t4;
  }
}

// Stage 2: adjoints of the masked gradients zdit(i,j,k), zdjt(i,j,k) (u and v faces)
// and of the vertical difference D(k) = (tb(k-1) - tb(k)) wmask(k) of column (i,j),
// k = 2..jpk (zdkt(k) = D(k), zdk1t(k) = D(k+1), zdkt(1) = D(2); :246-254). zdit(i,j,k)
// enters ztfw at (i,j) and (i+1,j), levels k and k+1, zdjt at (i,j) and (i,j+1); D(k)
// is zdkt of level k and zdk1t of level k-1 for the u faces of columns i-1 and i and
// the v faces of j-1 and j; at k = 2 also zdkt of level 1.
__global__ void __launch_bounds__(128) k_iso_adj_grad(Dom<double> d, LdfArgs<double> a, LdfAdj b) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const Pt3 P = pt3(d);
  const int i = c.i, j = c.j, k = c.k, m = c.m, jpi = d.jpi, jpk = d.jpk;
  const long n2 = d.n2, n3 = d.n3, ij = c.ij;
  const ColInfo ci = d.ci[ij];
  const bool face = P.uface(i, j, k), wpt = P.icol(i, j) && k >= 2 && k <= jpk - 1;
  double abe1 = 0.0, abe2 = 0.0, ctb = 0.0, ctbb = 0.0;
  if (face) {
    abe1 = msel(ahu(d, a, ci, ij, k, m) * d.e2_e1u[ij] * d.e3u_n(ij, k, m), umsk<double>(ci, k));
    abe2 = msel(ahv(d, a, ci, ij, k, m) * d.e1_e2v[ij] * d.e3v_n(ij, k, m), vmsk<double>(ci, k));
  }
  if (wpt) iso_adj_vlap(d, a, ij, k, m, ctb, ctbb);
  // the faces of columns i-1 and j-1 lie outside the flux loops where these are 0
  const bool hw = i > 1, hs = j > 1;
  for (int n = 0; n < a.kjpt; ++n) {
    const long o = ((long)m * a.kjpt + n) * n3 + c.q;
    const RO<double> G = b.G, su = b.su, sv = b.sv, t3 = b.t3, t4 = b.t4;
    double di = 0.0, dj = 0.0, dk = 0.0;
    if (face) {  // levels k, k+1 <= jpk
      const double g = G[o];
      di = abe1 * (g - G[o + 1]) + (t3[o + n2] + t3[o]) + (t3[o + 1] + t3[o + 1 + n2]);
      dj = abe2 * (g - G[o + jpi]) + (t4[o + n2] + t4[o]) + (t4[o + jpi] + t4[o + jpi + n2]);
      if (a.zps && k == ci.mbku) di = 0.0;
      if (a.zps && k == ci.mbkv) dj = 0.0;
    }
    if (k >= 2) {
      const double u0 = su[o], uw = hw ? su[o - 1] : 0.0, u1 = su[o - n2], uw1 = hw ? su[o - 1 - n2] : 0.0;
      const double v0 = sv[o], vs = hs ? sv[o - jpi] : 0.0, v1 = sv[o - n2], vs1 = hs ? sv[o - jpi - n2] : 0.0;
      double s = u0 + uw + u1 + uw1;
      s += v0 + vs + v1 + vs1;
      if (k == 2) s += u1 + uw1 + v1 + vs1;
      if (wpt) {
        const double t = G[o] - G[o - n2];
        if (nonzero(t)) s += ctb * t;
      }
      dk = s;
    }
    b.dit[o] = di;
    b.djt[o] = dj;
    b.dk[o] = dk;
  }
}

// Stage 3: tb_ad from the gradient adjoints (zdit = (tb(i+1)-tb(i)) umask, :218-227;
// D(k)), and tbb_ad from the second-pass vertical term (:343-356).
__global__ void __launch_bounds__(128) k_iso_adj_tb(Dom<double> d, LdfArgs<double> a, LdfAdj b) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const Pt3 P = pt3(d);
  const int i = c.i, j = c.j, k = c.k, jpi = d.jpi, jpk = d.jpk;
  const long q = c.q, n2 = d.n2, n3 = d.n3;
  const ColInfo ci = d.ci[c.ij];
  const bool tbb = !a.lap && a.kpass != 1;
  for (int n = 0; n < a.kjpt; ++n) {
    const long mo = ((long)c.m * a.kjpt + n) * n3;
    const RO<double> di = b.dit + mo;
    const RO<double> dj = b.djt + mo;
    const RO<double> dk = b.dk + mo;
    double v = 0.0;
    if (P.uface(i - 1, j, k)) v += msel(di[q - 1], umsk<double>(d.ci[c.ij - 1], k));
    if (P.uface(i, j, k)) v -= msel(di[q], umsk<double>(ci, k));
    if (P.uface(i, j - 1, k)) v += msel(dj[q - jpi], vmsk<double>(d.ci[c.ij - jpi], k));
    if (P.uface(i, j, k)) v -= msel(dj[q], vmsk<double>(ci, k));
    if (k + 1 <= jpk) v += msel(dk[q + n2], wmsk<double>(ci, k + 1));
    if (k >= 2) v -= msel(dk[q], wmsk<double>(ci, k));
    b.tb_ad[mo + q] += v;
    if (tbb && P.icol(i, j)) {
      const RO<double> G = b.G + mo;
      double u = 0.0, ctb, ctbb;
      if (k + 1 >= 2 && k + 1 <= jpk - 1) {
        iso_adj_vlap(d, a, c.ij, k + 1, c.m, ctb, ctbb);
        u += ctbb * (G[q + n2] - G[q]);
      }
      if (k >= 2 && k <= jpk - 1) {
        iso_adj_vlap(d, a, c.ij, k, c.m, ctb, ctbb);
        u -= ctbb * (G[q] - G[q - n2]);
      }
      b.tbb_ad[mo + q] += u;
    }
  }
}

// ------------------------------------------------------------------ tra_zdf_imp
// Adjoint of tra_zdf_imp (trazdf.F90:143-264) on one interior column: the
// back-substitution run forwards, then the elimination with its right-hand side
// e3t_b tb + p2dt e3t_n ta run backwards. The matrix is built as k_zdf_imp builds
// it in double precision: one division a level, 1 / zwt, and every quotient corrected
// from a reciprocal (divq; divr for the sensitivities); zwi(k+1) is zws(k).
__global__ void k_zdf_adj(Dom<double> d, ZdfArgs<double> a, ZdfAdj b) {
  ColIdx<double> c = col_index(d);
  if (!c.valid || !c.interior) return;
  const int jpk = d.jpk;
  const long n2 = d.n2, n3 = d.n3;
  const ColInfo ci = d.ci[c.ij];
  const long m3 = (long)c.m * n3;
  double rat[KMAX], zws[KMAX], zwt[KMAX], rz[KMAX];  // rz = 1 / zwt
  for (int n = 0; n < a.kjpt; ++n) {
    const bool build = (!a.is_trc && (n == 0 || (n == 1 && a.ddm))) || (a.is_trc && n == 0);
    if (build) {
      const RO<double> coef = (!a.is_trc && n == 0) ? a.avt : a.avs;
      auto wt = [&](int k) -> double {
        if (k == 1) return 0.0;
        const long q = m3 + c.ij + (long)(k - 1) * n2;
        double v = coef[q];
        if (a.add && k <= jpk - 1) v = v + a.add[q];
        return v;
      };
      double zwi = over_e3w(d, -a.p2dt * wt(1), c.ij, 1, c.m), tp = 0.0, rp = 0.0;
      for (int k = 1; k <= jpk - 1; ++k) {
        const double zs = over_e3w(d, -a.p2dt * wt(k + 1), c.ij, k + 1, c.m);
        double t = d.e3t_a(c.ij, k, c.m) - zwi - zs;
        if (k >= 2) {
          rat[k] = divq(zwi, tp, rp);
          t = t - divq(zwi * zwi, tp, rp);  // zws(k-1) = zwi(k)
        }
        zws[k] = zs;
        zwt[k] = tp = t;
        rz[k] = rp = 1.0 / t;
        zwi = zs;
      }
    }
    const long mo = ((long)c.m * a.kjpt + n) * n3;
    double* lam = b.lam + mo;
    double* tb = b.tb_ad + mo;
    // back-substitution (:252-264) run forwards
    double carry = 0.0;  // what level k receives from level k-1
    for (int k = 1; k <= jpk - 2; ++k) {
      const long q = c.ij + (long)(k - 1) * n2;
      const double x = divr(msel(lam[q] + carry, tmsk<double>(ci, k)), zwt[k], rz[k]);
      carry = -zws[k] * x;
      lam[q] = x;
    }
    {
      const long q = c.ij + (long)(jpk - 2) * n2;
      lam[q] = divr(msel(lam[q] + carry, tmsk<double>(ci, jpk - 1)), zwt[jpk - 1], rz[jpk - 1]);
    }
    // elimination (:238-250) run backwards
    double up = 0.0;  // what level k receives from level k+1
    for (int k = jpk - 1; k >= 1; --k) {
      const long q = c.ij + (long)(k - 1) * n2;
      const double y = lam[q] + up;
      up = k >= 2 ? -rat[k] * y : 0.0;
      tb[q] += d.e3t_b(c.ij, k, c.m) * y;
      lam[q] = a.p2dt * d.e3t_n(c.ij, k, c.m) * y;
    }
  }
}

// ---------------------------------------------------------------------- tra_nxt
// tra_nxt (tranxt.F90:66-188, tra_nxt_fix :191-237, linear free surface): lbc of tsa,
// then the Euler swap (first step of an Euler start) or the leapfrog with the Asselin
// filter on the interior, then lbc of tsb, tsn. Level march: memory bound (five fields a
// tracer, 470 MB at 752x502x31 in FP32, 69 us): 79 us, and 89 us as one point a thread.
template <class T>
__global__ void __launch_bounds__(32 * MARCH_Y) k_tra_nxt(Dom<T> d, T* tsb, T* tsn, T* tsa, T atfp, int euler, int kch) {
  const MarchIdx c = march_index(d, kch);
  if (c.i > d.jpi || c.j > d.jpj) return;
  const long o = 2 * (long)c.m * d.n3 + c.ij, n2 = d.n2, n3 = d.n3;
  if (!c.inner) {
    const int k1 = c.k1 == d.jpk - 1 ? d.jpk : c.k1;  // the last chunk's edge columns: jpk too
    for (int n = 0; n < 2; ++n)
      for (int k = c.k0; k <= k1; ++k) {
        const long q = o + n * n3 + (long)(k - 1) * n2;
        tsa[q] = T(0);
        if (!euler || k <= d.jpk - 1) tsn[q] = T(0);
        if (!euler) tsb[q] = T(0);
      }
    return;
  }
  if (euler) {
    for (int n = 0; n < 2; ++n)
      for (int k = c.k0; k <= c.k1; ++k) {
        const long q = o + n * n3 + (long)(k - 1) * n2;
        tsn[q] = tsa[q];
      }
    return;
  }
  march<T, 6>(
      c.k0, c.k1,
      [&](int k, T (&l)[6]) {
        const long q = o + (long)(k - 1) * n2;
        l[0] = tsb[q]; l[1] = tsn[q]; l[2] = tsa[q];
        l[3] = tsb[q + n3]; l[4] = tsn[q + n3]; l[5] = tsa[q + n3];
      },
      [&](int k, T (&l)[6]) {
        const long q = o + (long)(k - 1) * n2;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          // FP32: the time laplacian from the two differences, which round to small
          // values, instead of from the O(1) values (the same sum in exact arithmetic)
          const T b = l[3 * n], z = l[3 * n + 1], f = l[3 * n + 2];
          const T ztd = sizeof(T) == 4 ? (f - z) - (z - b) : f - T(2) * z + b;
          tsb[q + n * n3] = z + atfp * ztd;
          tsn[q + n * n3] = f;
        }
      });
}

// Adjoint of k_tra_nxt: on entry the adjoints of the swapped fields, on exit those
// of the fields before the swap.
__global__ void k_tra_nxt_adj(Dom<double> d, double* bb, double* nn, double* aa, double atfp, int euler) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const bool edge = !c.interior;
  for (int n = 0; n < 2; ++n) {
    const long o = ((long)c.m * 2 + n) * d.n3 + c.q;
    if (euler) {
      double v = aa[o];
      if (c.k <= d.jpk - 1) {
        v += nn[o];
        nn[o] = 0.0;
      }
      aa[o] = edge ? 0.0 : v;
    } else if (edge) {
      bb[o] = 0.0;
      nn[o] = 0.0;
      aa[o] = 0.0;
    } else if (c.k <= d.jpk - 1) {
      const double b = bb[o], v = nn[o];
      aa[o] = aa[o] + (v + atfp * b);
      nn[o] = b - 2.0 * atfp * b;
      bb[o] = atfp * b;
    }
  }
}

}  // namespace nemo
