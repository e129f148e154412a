// k_step.cuh -- the parts of the time step (step.F90:96-305) that close the path into
// a model step with the linear free surface: the vertical velocity from the
// horizontal divergence, the time step of dyn_zdf without vertical viscosity, the
// Asselin filter and swap of the momentum and of the sea surface height. The
// momentum trends outside the path (dyn_adv, dyn_vor, dyn_ldf, dyn_hpg) are held at
// 0 by the caller. T is the bulk type, A the type of the barotropic accumulators
// (ua_b, va_b, ssha: double in both forms).
#pragma once
#include "nemo_sin.h"
#include "step.h"

namespace nemo {

// levels that the column kernels below load before they use the first of them
template <class T>
constexpr int BATCH = sizeof(T) == 4 ? 8 : 4;

// div_hor (divhor.F90:76-106: the horizontal divergence of the interior, 0 on the
// closed edges) and wzv (sshwzv.F90:172-189: w integrated up from w(jpk) = 0), one
// column per thread, the next level loaded ahead of the running sum, which alone links
// the levels. FLAT: e3t, e3u, e3v are 1-D profiles, kept in shared memory with the
// reciprocals of e3t. 77 us before at 752x502x31 in FP32 (seven scale-factor loads and an
// IEEE division a level), 40 us now; 21 us by traffic.
template <class T, bool FLAT>
__global__ void __launch_bounds__(128) k_wzv(Dom<T> d, const T* __restrict__ un, const T* __restrict__ vn,
                                             T* __restrict__ wn, T z1_2dt) {
  __shared__ E3Prof<T> pt;
  __shared__ T pu[KMAX + 1], pv[KMAX + 1], pd[KMAX + 1];
  const ColIdx<T> c = col_index(d);
  const int jpi = d.jpi, jpk = d.jpk, m = c.m;
  if constexpr (FLAT) {
    pt.fill(d.e3t_n, m, jpk);
    const int k = threadIdx.y * 32 + threadIdx.x + 1;
    if (k <= jpk) {
      pu[k] = d.e3u_n(0, k, m);
      pv[k] = d.e3v_n(0, k, m);
      pd[k] = z1_2dt * (d.e3t_a(0, k, m) - d.e3t_b(0, k, m));
    }
    __syncthreads();
  }
  if (!c.valid) return;
  const long ij = c.ij, n2 = d.n2, c3 = (long)m * d.n3 + ij;
  const ColInfo ci = d.ci[ij];
  const int wst = c.interior ? 1 : 0, sst = wst * jpi;  // an edge column reads its own cells alone
  const T e2u = d.e2u[ij], e2uw = d.e2u[ij - wst], e1v = d.e1v[ij], e1vs = d.e1v[ij - sst], r1 = d.r1_e1e2t[ij];
  wn[c3 + (long)(jpk - 1) * n2] = T(0);
  T w = T(0);
  march<T, 4>(
      1, jpk - 1,
      [&](int x, T (&l)[4]) {
        const long q = c3 + (long)(jpk - 1 - x) * n2;
        l[0] = __ldg(un + q);
        l[1] = __ldg(un + q - wst);
        l[2] = __ldg(vn + q);
        l[3] = __ldg(vn + q - sst);
      },
      [&](int x, T (&l)[4]) {
        const int k = jpk - x;
        T hdiv, e3n, de;
        if constexpr (FLAT) {
          e3n = pt.e[k];
          de = pd[k];
          hdiv = divr((e2u * pu[k] * l[0] - e2uw * pu[k] * l[1] + e1v * pv[k] * l[2] - e1vs * pv[k] * l[3]) * r1, e3n,
                      pt.r[k]);
        } else {
          e3n = d.e3t_n(ij, k, m);
          de = z1_2dt * (d.e3t_a(ij, k, m) - d.e3t_b(ij, k, m));
          hdiv = (e2u * d.e3u_n(ij, k, m) * l[0] - e2uw * d.e3u_n(ij - wst, k, m) * l[1] +
                  e1v * d.e3v_n(ij, k, m) * l[2] - e1vs * d.e3v_n(ij - sst, k, m) * l[3]) * r1 / e3n;
        }
        if (!c.interior) hdiv = T(0);
        w = w - (e3n * hdiv + de) * tmsk<T>(ci, k);
        wn[c3 + (long)(k - 1) * n2] = w;
      });
}

// The time step of dyn_zdf (dynzdf.F90:112) with no vertical viscosity or drag.
template <class T>
__global__ void k_dyn_zdf_step(Dom<T> d, RO<T> ub, RO<T> vb, T* ua, T* va, T r2dt, RO<T> e3u_b, RO<T> e3v_b,
                               RO<T> e3u_a, RO<T> e3v_a) {
  const PtIdx c = pt_index(d);
  if (!c.valid || c.k > d.jpk - 1) return;
  const long q = (long)c.m * d.n3 + c.q;
  const ColInfo ci = d.ci[c.ij];
  if (e3u_b) {  // flux form with a variable volume: on the thickness-weighted velocity (:115-120)
    ua[q] = (e3u_b[q] * ub[q] + r2dt * d.e3u_n(c.ij, c.k, c.m) * ua[q]) / e3u_a[q] * umsk<T>(ci, c.k);
    va[q] = (e3v_b[q] * vb[q] + r2dt * d.e3v_n(c.ij, c.k, c.m) * va[q]) / e3v_a[q] * vmsk<T>(ci, c.k);
  } else {      // on the velocity (:109-114)
    ua[q] = (ub[q] + r2dt * ua[q]) * umsk<T>(ci, c.k);
    va[q] = (vb[q] + r2dt * va[q]) * vmsk<T>(ci, c.k);
  }
}

// One U- (V-) column of dyn_zdf (dynzdf.F90:47-499) with the implicit vertical
// viscosity: the time step and the removal of the barotropic after velocity ab (:112,
// :122-126), then, on the interior, the bottom stress of ab and the system of avm
// (:127-141, :205-302; iso-level lateral mixing, no adaptive-implicit advection) with
// the surface condition, the implicit drag on the bottom diagonal and the wind stress
// in the surface right-hand side, assembled and forward-eliminated in one downward
// sweep and back-substituted upwards. The W-point scale factor across the U- (V-) point
// is the MIN of the neighbouring e3w (the rest state of a linear free surface).
template <class T>
struct DynZdfProf {  // 1-D scale factors: e3, and the divisors e3(k) e3w(k+1), e3(k) e3w(k)
  T *e, *ds, *rs, *di, *ri;  // of jpk + 1 values each
  __device__ __forceinline__ DynZdfProf(T* p, int n) : e(p), ds(p + n), rs(p + 2 * n), di(p + 3 * n), ri(p + 4 * n) {}
};
inline int dyn_zdf_smem(int nt, int jpk, bool flat, int b) {
  return ((b == 4 ? 2 : 3) * nt * jpk + (flat ? 5 * (jpk + 1) : 0)) * b;
}
template <bool U, bool FLAT, class T>
__device__ __forceinline__ void dyn_zdf_column(const Dom<T>& d, const DynZdfArgs<T>& a, const ColIdx<T>& c, int nt, T* sx,
                                               T* ss, T* sd, const DynZdfProf<T>& pf) {
  constexpr int B = FLAT && sizeof(T) == 4 ? 5 : 4;  // levels loaded together
  const int jpk = d.jpk, K = jpk - 1, m = c.m, n2 = (int)d.n2;
  const long ij = c.ij, m3 = (long)m * d.n3 + ij, p2 = (long)m * d.n2 + ij;
  const int nb = U ? 1 : d.jpi;
  const ColInfo ci = d.ci[ij];
  const int kb = U ? ci.mbku : ci.mbkv, lo = U ? ci.ulo : ci.vlo, hi = U ? ci.uhi : ci.vhi;
  T* __restrict__ pa = (U ? a.ua : a.va) + m3;
  const T* __restrict__ pb = (U ? a.ub : a.vb) + m3;
  const T ab = (T)(U ? a.ua_b : a.va_b)[p2], r2dt = a.r2dt;
  auto mk = [&](int k) { return in_range(k, lo, hi) ? T(1) : T(0); };
  auto stepped = [&](T b, T x, T mu) { return ((b + r2dt * x) * mu - ab) * mu; };
  if (!c.interior) {
    for (int k = 1; k <= K; ++k) {
      const long o = (long)(k - 1) * n2;
      pa[o] = stepped(pb[o], pa[o], mk(k));
    }
    return;
  }
  const T* __restrict__ av = a.avm + m3 + n2;
  auto e3 = [&](int k) { return FLAT ? pf.e[k] : (U ? d.e3u_n : d.e3v_n)(ij, k, m); };
  auto e3xw = [&](int k) { return fmn(d.e3w_n(ij, k, m), d.e3w_n(ij + nb, k, m)); };
  const T rc = a.rcdu[p2 + nb] + a.rcdu[p2];
  // of the level above: the upper diagonal and the forward value (FP32: over the pivot),
  // the pivot and its reciprocal
  T ws_p = T(0), x_p = T(0), wd_p = T(1), rd_p = T(1);
  T mk0 = mk(1), s0 = T(0), w0 = T(0), wx0 = T(0);  // of level k: mask; of w-level k: avm sum, e3, mask
  auto load = [&](int kt, T (&l)[3 * B]) {
    const long b = (long)(kt - 1) * n2;
    const T *pbk = pb + b, *avk = av + b, *avn = avk + nb, *pak = pa + b;
#pragma unroll
    for (int y = 0; y < B; ++y) {
      const int o = min(y, K - kt) * n2;
      l[y] = __ldg(pbk + o);
      l[B + y] = pak[o];
      l[2 * B + y] = __ldg(avn + o) + __ldg(avk + o);
    }
  };
  auto sweep = [&](int kt, T (&l)[3 * B]) {
#pragma unroll
    for (int y = 0; y < B; ++y) {
      const int k = kt + y;
      if (k > K) break;
      const T ze3a = e3(k), mk1 = mk(k + 1), wx1 = mk1 * mk0, sv = l[2 * B + y];
      T x = stepped(l[y], l[B + y], mk0), w1 = T(0), zzws, wd;
      if constexpr (FLAT) {
        zzws = divr(-a.zdt * sv, pf.ds[k], pf.rs[k]) * wx1;
      } else {
        w1 = e3xw(k + 1);
        zzws = -a.zdt * sv / (ze3a * w1) * wx1;
      }
      if (k == kb) x = x + r2dt * T(0.5) * rc * ab / ze3a;
      T zzwi = T(0);
      if (k == 1) {
        wd = T(1) - zzws;
        x = x + r2dt * T(0.5) * ((U ? a.utau_b : a.vtau_b)[p2] + (U ? a.utau : a.vtau)[p2]) / (ze3a * a.rau0) * mk0;
      } else {
        zzwi = FLAT ? divr(-a.zdt * s0, pf.di[k], pf.ri[k]) * wx0 : -a.zdt * s0 / (ze3a * w0) * wx0;
        wd = T(1) - zzwi - zzws;
      }
      if (k == kb) wd = wd - r2dt * T(0.5) * rc / ze3a;
      const int o = (k - 1) * nt;
      if constexpr (sizeof(T) == 4) {
        if (k > 1) {
          wd = wd - zzwi * ws_p;
          x = x - zzwi * x_p;
        }
        rd_p = T(1) / wd;
        ws_p = divr(zzws, wd, rd_p);
        x_p = divr(x, wd, rd_p);
      } else {
        if (k > 1) {
          wd = wd - divr(zzwi * ws_p, wd_p, rd_p);
          x = x - divr(zzwi, wd_p, rd_p) * x_p;
        }
        sd[o] = wd;
        wd_p = wd; rd_p = T(1) / wd; ws_p = zzws; x_p = x;
      }
      ss[o] = ws_p;
      sx[o] = x_p;
      mk0 = mk1; s0 = sv; w0 = w1; wx0 = wx1;
    }
  };
  T la[3 * B], lb[3 * B];
  load(1, la);
  for (int kt = 1; kt <= K; kt += 2 * B) {  // a batch is loaded while the one before it is swept
    if (kt + B <= K) load(kt + B, lb);
    sweep(kt, la);
    if (kt + B > K) break;
    if (kt + 2 * B <= K) load(kt + 2 * B, la);
    sweep(kt + B, lb);
  }
  if (kb == jpk) pa[(long)(jpk - 1) * n2] = pa[(long)(jpk - 1) * n2] + r2dt * T(0.5) * rc * ab / e3(kb);
  T nxt = T(0);
#pragma unroll 4
  for (int k = K; k >= 1; --k) {
    const int o = (k - 1) * nt;
    nxt = (k == K) ? sx[o] : sx[o] - ss[o] * nxt;
    if constexpr (sizeof(T) == 8) nxt = nxt / sd[o];
    pa[(long)(k - 1) * n2] = nxt;
  }
}

// dyn_zdf, one U- or V-column per thread (grid z = 2 member + component). What the back
// substitution needs of the column stays in shared memory, so that ua, va and avm are read
// once and the result is written once, and a batch of levels is loaded while the one
// before it is swept; the quotients by scale factors (1-D with FLAT) and by the pivot are
// divr's. One thread for both components, with the time step as a pass of its own and the
// diagonals in global memory, took 340 us at 752x502x31 in FP32 (376 MB to move: 55 us).
// Bound by the loads in flight, so by the shared memory of a column: in FP32 the upper
// diagonal and the forward value are kept over the pivot (two values a level and no
// division on the way up, 24 warps an SM: 136 us) and not beside it (three: 200 us); it
// rounds less often (five times a level, not seven). FP64 keeps the reference's order.
template <class T>
constexpr int DZ_Y = sizeof(T) == 4 ? 4 : 2;
template <class T, bool FLAT>
__global__ void __launch_bounds__(32 * DZ_Y<T>, sizeof(T) == 8 ? 1 : FLAT ? 6 : 5) k_dyn_zdf_imp(Dom<T> d, DynZdfArgs<T> a) {
  extern __shared__ __align__(16) unsigned char col_smem[];
  constexpr int nt = 32 * DZ_Y<T>;
  const DynZdfProf<T> pf(reinterpret_cast<T*>(col_smem) + (sizeof(T) == 4 ? 2 : 3) * nt * d.jpk, d.jpk + 1);
  ColIdx<T> c = col_index(d);
  c.m = blockIdx.z >> 1;
  const bool isv = blockIdx.z & 1;
  if constexpr (FLAT) {
    const int k = threadIdx.y * 32 + threadIdx.x + 1;
    if (k <= d.jpk) {
      const T e = (isv ? d.e3v_n : d.e3u_n)(0, k, c.m);
      pf.e[k] = e;
      pf.ds[k] = e * d.e3w_n(0, min(k + 1, d.jpk), c.m);
      pf.rs[k] = T(1) / pf.ds[k];
      pf.di[k] = e * d.e3w_n(0, k, c.m);
      pf.ri[k] = T(1) / pf.di[k];
    }
    __syncthreads();
  }
  if (!c.valid) return;
  T* sx = reinterpret_cast<T*>(col_smem) + threadIdx.y * 32 + threadIdx.x;
  T *ss = sx + d.jpk * nt, *sd = ss + d.jpk * nt;  // sd: FP64
  if (isv) dyn_zdf_column<false, FLAT>(d, a, c, nt, sx, ss, sd, pf);
  else dyn_zdf_column<true, FLAT>(d, a, c, nt, sx, ss, sd, pf);
}

// dyn_nxt (dynnxt.F90:114-358; linear free surface, ln_dynspg_ts with ln_bt_fw), one
// U- or V-column per thread (grid z = 2 member + component): the barotropic part of the
// after velocity replaced by the sub-steps' ua_b; lbc of ua, va (the closed edges 0);
// the Euler swap or the Asselin filter and swap with the before velocity returned to
// the time-split barotropic estimate; the now and before barotropic velocities. The
// column waits for its sums in shared memory (the after velocity, copied there all levels
// at once, then the filtered before one), and a batch of the now and before velocities is
// loaded while the one before it is used: memory sees each field read once and written
// once, 564 MB at 752x502x31 in FP32, 83 us. With the column read back from memory by each
// of four passes it took 203 us; loaded four levels at a time, each batch waited for,
// 142 us; so 112 us (batches of 4: 138; of 15: 123).
constexpr int DN_Y = 4;
// one value of global memory into the thread's own place in shared memory
template <class T>
__device__ __forceinline__ void cp_async_val(T* smem, const T* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sa), "l"(gmem), "n"((int)sizeof(T)) : "memory");
}
// BPS: the blocks an SM it is compiled for.
template <class T, class A, int BPS>
__global__ void __launch_bounds__(32 * DN_Y, BPS) k_dyn_nxt(Dom<T> d, NxtArgs<T, A> a) {
  extern __shared__ __align__(16) unsigned char col_smem[];
  constexpr int nt = 32 * DN_Y, B = BATCH<T>;  // levels loaded together
  T* s = reinterpret_cast<T*>(col_smem) + threadIdx.y * 32 + threadIdx.x;
  const ColIdx<T> c = col_index(d);
  if (!c.valid) return;
  const int jpk = d.jpk, m = blockIdx.z >> 1, n2 = (int)d.n2;
  const bool isv = blockIdx.z & 1;
  const long ij = c.ij, m3 = (long)m * d.n3 + ij, p2 = (long)m * d.n2 + ij;
  const ColInfo ci = d.ci[ij];
  const int lo = isv ? ci.vlo : ci.ulo, hi = isv ? ci.vhi : ci.uhi;
  const T r1 = isv ? d.r1_hv_0[ij] : d.r1_hu_0[ij];
  const T ab = T((isv ? a.va_b : a.ua_b)[p2]);
  // three distinct arrays: restrict lets a batch's loads go ahead of its stores
  T* __restrict__ xa = (isv ? a.va : a.ua) + m3;
  T* __restrict__ xn = (isv ? a.vn : a.un) + m3;
  T* __restrict__ xb = (isv ? a.vb : a.ub) + m3;
  const E3Col<T> e3(isv ? d.e3v_n : d.e3u_n, ij, m);
  auto mk = [&](int k) { return in_range(k, lo, hi) ? T(1) : T(0); };
  // (:114-126)
  for (int k = 1; k <= jpk - 1; ++k) cp_async_val(s + (k - 1) * nt, xa + (long)(k - 1) * n2);
  auto load = [&](int kt, T (&l)[3 * B]) {
    const T *pn = xn + (long)(kt - 1) * n2, *pb = xb + (long)(kt - 1) * n2;
#pragma unroll
    for (int y = 0; y < B; ++y) {
      const int z = min(y, jpk - 1 - kt), o = z * n2;
      l[y] = pb[o];
      l[B + y] = pn[o];
      l[2 * B + y] = e3(kt + z);
    }
  };
  T la[3 * B], lb[3 * B];
  load(1, la);
  cp_async_wait_all();
  T ze = T(0);
#pragma unroll 4
  for (int k = 1; k <= jpk - 1; ++k) ze = ze + e3(k) * s[(k - 1) * nt] * mk(k);
  // the now and before barotropic velocities (:345-358) are summed where xn and xb
  // take their final values, level by level in the same order
  T sn = T(0), sb = T(0), sf = T(0);
  auto level = [&](int kt, const T (&l)[3 * B]) {
    T* pa = xa + (long)(kt - 1) * n2;
    T* pn = xn + (long)(kt - 1) * n2;
#pragma unroll
    for (int y = 0; y < B; ++y) {
      const int k = kt + y;
      if (k > jpk - 1) break;
      const T e = l[2 * B + y], mu = mk(k), vb = l[y], vn = l[B + y];
      // lbc_lnk of ua, va (:146): the closed edges
      const T u = c.interior ? (s[(k - 1) * nt] - ze * r1 + ab) * mu : T(0);
      pa[y * n2] = u;
      pn[y * n2] = u;
      if (a.euler) {  // (:168-171)
        sb = sb + e * vb * mu;
      } else {        // (:197-211); FP32: the time laplacian from differences (see k_tra_nxt)
        const T zf = vn + a.atfp * (sizeof(T) == 4 ? (u - vn) - (vn - vb) : vb - T(2) * vn + u);
        s[(k - 1) * nt] = zf;
        sf = sf + e * zf * mu;
      }
      sn = sn + e * u * mu;
    }
  };
  for (int kt = 1; kt <= jpk - 1; kt += 2 * B) {  // a batch is loaded while the one before it is used
    if (kt + B <= jpk - 1) load(kt + B, lb);
    level(kt, la);
    if (kt + B > jpk - 1) break;
    if (kt + 2 * B <= jpk - 1) load(kt + 2 * B, la);
    level(kt + B, lb);
  }
  if (!c.interior) xa[(long)(jpk - 1) * n2] = T(0);
  if (!a.euler) {  // (:312-324)
    const T nb = (isv ? a.vn_b : a.un_b)[p2];
    const T* ps = s;
    T* pb = xb;
#pragma unroll 4
    for (int k = 1; k <= jpk - 1; ++k, ps += nt, pb += n2) {
      const T e = e3(k), mu = mk(k);
      const T bk = *ps - (sf * r1 - nb) * mu;
      *pb = bk;
      sb = sb + e * bk * mu;
    }
  }
  (isv ? a.vn_b : a.un_b)[p2] = sn * r1;
  (isv ? a.vb_b : a.ub_b)[p2] = sb * r1;
}

// ssh_swp (sshwzv.F90:216-267), linear free surface, one point per thread.
template <class T, class A>
__global__ void k_ssh_swp(Dom<T> d, T* sshb, T* sshn, const A* __restrict__ ssha, T atfp, int euler) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const long p = (long)blockIdx.z * d.n2 + (long)(i - 1) + (long)(j - 1) * d.jpi;
  const T sa = T(ssha[p]);
  if (!euler)
    sshb[p] = sshn[p] + atfp * (sizeof(T) == 4 ? (sa - sshn[p]) - (sshn[p] - sshb[p]) : sshb[p] - T(2) * sshn[p] + sa);
  sshn[p] = sa;
}


// ----------------------------------------------------------------------- ldf_slp
// ldf_slp (ldfslp.F90:83-374) with ldf_slp_mxl (:620-729), z-coordinate with or
// without partial steps, without cavities, in three kernels: the slopes just below the mixed
// layer (one column per thread), the slopes before the Shapiro filter at u-, v- and
// w-points (a chunk of levels per thread), the filter with the coastal decrease and lbc
// (the same). The density gradients zgru, zgrv and zdzr of the reference's work arrays are
// formed where they are read, from the same operands in the same order.
template <class T, bool ZPS>
struct SlpPt {
  const Dom<T>& d;
  const SlpArgs<T>& a;
  long m3;
  int m;
  __device__ __forceinline__ long Q(int i, int j, int k) const {
    return (long)(i - 1) + (long)(j - 1) * d.jpi + (long)(k - 1) * d.n2;
  }
  __device__ __forceinline__ T um(int i, int j, int k) const { return umsk<T>(d.ci[Q(i, j, 1)], k); }
  __device__ __forceinline__ T vm(int i, int j, int k) const { return vmsk<T>(d.ci[Q(i, j, 1)], k); }
  __device__ __forceinline__ T tm(int i, int j, int k) const { return tmsk<T>(d.ci[Q(i, j, 1)], k); }
  __device__ __forceinline__ T prd(int i, int j, int k) const { return a.prd[m3 + Q(i, j, k)]; }
  // with partial steps (ZPS) the bottom level's gradients are zps_hde's
  // (ldfslp.F90:144-151); the z-coordinate form compiles without the test
  __device__ __forceinline__ T gru(int i, int j, int k) const {
    if constexpr (ZPS) {
      if (k == d.ci[Q(i, j, 1)].mbku) return a.gru_b[(long)m * d.n2 + Q(i, j, 1)];
    }
    return um(i, j, k) * (prd(i + 1, j, k) - prd(i, j, k));
  }
  __device__ __forceinline__ T grv(int i, int j, int k) const {
    if constexpr (ZPS) {
      if (k == d.ci[Q(i, j, 1)].mbkv) return a.grv_b[(long)m * d.n2 + Q(i, j, 1)];
    }
    return vm(i, j, k) * (prd(i, j + 1, k) - prd(i, j, k));
  }
  __device__ __forceinline__ T dzr(int i, int j, int k) const {
    if (k == 1) return T(0);
    const long q = m3 + Q(i, j, k);
    return a.zm1_g * (a.prd[q] + T(1)) * (a.pn2[q] + a.pn2[q + d.n2]) * (T(1) - T(0.5) * tm(i, j, k + 1));
  }
};

template <class T, bool ZPS>
__global__ void k_slp_mxl(Dom<T> d, SlpArgs<T> a) {
  ColIdx<T> c = col_index(d);
  if (!c.valid) return;
  const long p = (long)c.m * d.n2 + c.ij;
  if (!c.interior) {  // lbc_lnk of the four mixed-layer slopes: the closed edges 0
    a.uml[p] = T(0); a.vml[p] = T(0); a.wiml[p] = T(0); a.wjml[p] = T(0);
    a.hu[p] = T(0); a.hv[p] = T(0);
    return;
  }
  const SlpPt<T, ZPS> P{d, a, (long)c.m * d.n3, c.m};
  const int i = c.i, j = c.j, jpk = d.jpk, jpi = d.jpi;
  const long ij = c.ij, m2 = (long)c.m * d.n2;
  const int n0 = a.nmln[m2 + ij], ne = a.nmln[m2 + ij + 1], nn = a.nmln[m2 + ij + jpi];
  int iku = n0 > ne ? n0 : ne;
  iku = iku < 1 ? 1 : (iku > jpk - 1 ? jpk - 1 : iku);
  int ikv = n0 > nn ? n0 : nn;
  ikv = ikv < 1 ? 1 : (ikv > jpk - 1 ? jpk - 1 : ikv);
  T zbu = T(0.5) * (P.dzr(i, j, iku) + P.dzr(i + 1, j, iku));
  T zbv = T(0.5) * (P.dzr(i, j, ikv) + P.dzr(i, j + 1, ikv));
  const T zau = P.gru(i, j, iku) * d.r1_e1u[ij];
  const T zav = P.grv(i, j, ikv) * d.r1_e2v[ij];
  zbu = fmn(fmn(zbu, -a.z1_slpmax * fabs(zau)), T(-7.e+3) / d.e3u_n(ij, iku, c.m) * fabs(zau));
  zbv = fmn(fmn(zbv, -a.z1_slpmax * fabs(zav)), T(-7.e+3) / d.e3v_n(ij, ikv, c.m) * fabs(zav));
  const T uml = zau / (zbu - a.zeps) * P.um(i, j, iku);
  const T vml = zav / (zbv - a.zeps) * P.vm(i, j, ikv);
  const int ik = n0 + 1 < jpk ? n0 + 1 : jpk;
  const int ikm1 = ik - 1 > 1 ? ik - 1 : 1;
  const T zbw = a.zm1_2g * a.pn2[P.m3 + P.Q(i, j, ik)] * (P.prd(i, j, ik) + P.prd(i, j, ikm1) + T(2));
  const T zci = fmx(P.um(i - 1, j, ik) + P.um(i, j, ik) + P.um(i - 1, j, ikm1) + P.um(i, j, ikm1), a.zeps) * d.e1t[ij];
  const T zcj = fmx(P.vm(i, j - 1, ik) + P.vm(i, j, ik) + P.vm(i, j - 1, ikm1) + P.vm(i, j, ikm1), a.zeps) * d.e2t[ij];
  const T tmk = P.tm(i, j, ik);
  const T zai = (P.gru(i - 1, j, ik) + P.gru(i, j, ik) + P.gru(i - 1, j, ikm1) + P.gru(i, j, ikm1)) / zci * tmk;
  const T zaj = (P.grv(i, j - 1, ik) + P.grv(i, j, ik) + P.grv(i, j - 1, ikm1) + P.grv(i, j, ikm1)) / zcj * tmk;
  const T e3w = d.e3w_n(ij, ik, c.m);
  const T zbi = fmn(fmn(zbw, T(-100) * fabs(zai)), T(-7.e+3) / e3w * fabs(zai));
  const T zbj = fmn(fmn(zbw, T(-100) * fabs(zaj)), T(-7.e+3) / e3w * fabs(zaj));
  a.uml[p] = uml;
  a.vml[p] = vml;
  a.wiml[p] = zai / (zbi - a.zeps) * tmk;
  a.wjml[p] = zaj / (zbj - a.zeps) * tmk;
  // (:188-194) the mixed-layer slope over the depth of the last T-point in it
  const T h0 = a.hmlpt[p], he = a.hmlpt[p + 1], hn = a.hmlpt[p + jpi];
  a.hu[p] = uml / fmx(fmx(h0, he), T(5));
  a.hv[p] = vml / fmx(fmx(h0, hn), T(5));
}

// The slopes before the filter: u, v (:197-233) and w (:281-315) at levels 2..jpkm1;
// 0 on the closed edges (the lbc_lnk of :234 and :316). Level march: the masks' level
// ranges and the metrics of the column and its neighbours are loaded once a chunk, the
// densities of the level above and N^2 of the level are carried, and with 1-D scale
// factors (FLAT) the limits -7e3 / e3 come from a table. One point a thread, which looked
// up some twenty masks through memory, it took 154 us at 481x323x31 in FP32, 74 so (101
// registers; bounded to 80 or fewer it spills: 77 to 86 us).
template <class T, bool ZPS, bool FLAT>
__global__ void __launch_bounds__(32 * MARCH_Y) k_slp_pre(Dom<T> d, SlpArgs<T> a, int kch) {
  __shared__ T pu[KMAX + 1], pv[KMAX + 1], pw[KMAX + 1];  // -7e3 / e3u, e3v, e3w
  const MarchIdx c = march_index(d, kch);
  const int m = c.m, J = d.jpi;
  if constexpr (FLAT) {
    const int k = threadIdx.y * 32 + threadIdx.x + 1;
    if (k <= d.jpk) {
      pu[k] = T(-7.e+3) / d.e3u_n(0, k, m);
      pv[k] = T(-7.e+3) / d.e3v_n(0, k, m);
      pw[k] = T(-7.e+3) / d.e3w_n(0, k, m);
    }
    __syncthreads();
  }
  if (c.i > d.jpi || c.j > d.jpj) return;
  const int k0 = max(c.k0, 2);
  if (k0 > c.k1) return;
  const long n2 = d.n2, ij = c.ij, o = (long)m * d.n3 + ij, p = (long)m * n2 + ij;
  if (!c.inner) {
    for (int k = k0; k <= c.k1; ++k) {
      const long q = o + (long)(k - 1) * n2;
      a.zu[q] = T(0); a.zv[q] = T(0); a.zwi[q] = T(0); a.zwj[q] = T(0);
    }
    return;
  }
  const ColInfo ci = d.ci[ij], ce = d.ci[ij + 1], cn = d.ci[ij + J], cw = d.ci[ij - 1], cs = d.ci[ij - J];
  const T r1u = d.r1_e1u[ij], r1v = d.r1_e2v[ij], e1t = d.e1t[ij], e2t = d.e2t[ij];
  const T hu = a.hu[p], hv = a.hv[p], wiml = a.wiml[p], wjml = a.wjml[p];
  const int n0 = a.nmln[p], ne = a.nmln[p + 1], nn = a.nmln[p + J];
  const T gw1 = a.gdepw[o], zml = fmx(a.hmlp[p] - gw1, T(10));
  const T e3u1 = d.e3u_n(ij, 1, m), e3v1 = d.e3v_n(ij, 1, m);
  // with partial steps the bottom level's gradients are zps_hde's (ldfslp.F90:144-151)
  T gu0 = T(0), guw = T(0), gv0 = T(0), gvs = T(0);
  if constexpr (ZPS) {
    gu0 = a.gru_b[p]; guw = a.gru_b[p - 1]; gv0 = a.grv_b[p]; gvs = a.grv_b[p - J];
  }
  auto gru = [&](const ColInfo& x, int k, T lft, T rgt, T b) -> T {
    if constexpr (ZPS) {
      if (k == x.mbku) return b;
    }
    return umsk<T>(x, k) * (rgt - lft);
  };
  auto grv = [&](const ColInfo& x, int k, T lft, T rgt, T b) -> T {
    if constexpr (ZPS) {
      if (k == x.mbkv) return b;
    }
    return vmsk<T>(x, k) * (rgt - lft);
  };
  // carried: prd of the level above at the five points, the four gradients formed from
  // them, N^2 of the level at p, p+1, p+J
  const long qa = o + (long)(k0 - 2) * n2, qk = o + (long)(k0 - 1) * n2;
  T r0 = __ldg(a.prd + qa);
  T ui = gru(ci, k0 - 1, r0, __ldg(a.prd + qa + 1), gu0), uw = gru(cw, k0 - 1, __ldg(a.prd + qa - 1), r0, guw);
  T vi = grv(ci, k0 - 1, r0, __ldg(a.prd + qa + J), gv0), vs = grv(cs, k0 - 1, __ldg(a.prd + qa - J), r0, gvs);
  T b0 = __ldg(a.pn2 + qk), be = __ldg(a.pn2 + qk + 1), bn = __ldg(a.pn2 + qk + J);
  march<T, 12>(
      k0, c.k1,
      [&](int k, T (&l)[12]) {
        const long q = o + (long)(k - 1) * n2;
        const T *r = a.prd + q, *b = a.pn2 + q + n2, *g = a.gdept + q;
        l[0] = __ldg(r); l[1] = __ldg(r + 1); l[2] = __ldg(r - 1); l[3] = __ldg(r + J); l[4] = __ldg(r - J);
        l[5] = __ldg(b); l[6] = __ldg(b + 1); l[7] = __ldg(b + J);
        l[8] = __ldg(g); l[9] = __ldg(g + 1); l[10] = __ldg(g + J);
        l[11] = __ldg(a.gdepw + q);
      },
      [&](int k, T (&l)[12]) {
        const long q = o + (long)(k - 1) * n2;
        auto lim_u = [&](T z) { return FLAT ? pu[k] * z : T(-7.e+3) / d.e3u_n(ij, k, m) * z; };
        auto lim_v = [&](T z) { return FLAT ? pv[k] * z : T(-7.e+3) / d.e3v_n(ij, k, m) * z; };
        auto lim_w = [&](T z) { return FLAT ? pw[k] * z : T(-7.e+3) / d.e3w_n(ij, k, m) * z; };
        auto dzr = [&](T r, T n, T np, const ColInfo& x) -> T {
          return a.zm1_g * (r + T(1)) * (n + np) * (T(1) - T(0.5) * tmsk<T>(x, k + 1));
        };
        auto oml = [&](int n, int kk) -> T { return kk <= n - 1 ? T(1) : T(0); };
        const T u1 = gru(ci, k, l[0], l[1], gu0), uw1 = gru(cw, k, l[2], l[0], guw);
        const T v1 = grv(ci, k, l[0], l[3], gv0), vs1 = grv(cs, k, l[4], l[0], gvs);
        const T um0 = umsk<T>(ci, k), um0a = umsk<T>(ci, k - 1), umw = umsk<T>(cw, k), umwa = umsk<T>(cw, k - 1);
        const T vm0 = vmsk<T>(ci, k), vm0a = vmsk<T>(ci, k - 1), vms = vmsk<T>(cs, k), vmsa = vmsk<T>(cs, k - 1);
        // u- and v-points
        {
          const T zau = u1 * r1u, zav = v1 * r1v;
          const T dz0 = dzr(l[0], b0, l[5], ci);
          T zbu = T(0.5) * (dz0 + dzr(l[1], be, l[6], ce));
          T zbv = T(0.5) * (dz0 + dzr(l[3], bn, l[7], cn));
          zbu = fmn(fmn(zbu, -a.z1_slpmax * fabs(zau)), lim_u(fabs(zau)));
          zbv = fmn(fmn(zbv, -a.z1_slpmax * fabs(zav)), lim_v(fabs(zav)));
          const T o0 = oml(n0, k);
          const T zfi = fmx(o0, oml(ne, k));
          const T zfj = fmx(o0, oml(nn, k));
          const T zdepu = T(0.5) * ((l[8] + l[9]) - T(2) * T(0) - e3u1);
          const T zdepv = T(0.5) * ((l[8] + l[10]) - T(2) * T(0) - e3v1);
          a.zu[q] = ((T(1) - zfi) * zau / (zbu - a.zeps) + zfi * zdepu * hu) * um0;
          a.zv[q] = ((T(1) - zfj) * zav / (zbv - a.zeps) + zfj * zdepv * hv) * vm0;
        }
        // w-points
        {
          const T zbw = a.zm1_2g * b0 * (l[0] + r0 + T(2));
          const T zci = fmx(umw + um0 + umwa + um0a, a.zeps) * e1t;
          const T zcj = fmx(vms + vm0a + vmsa + vm0, a.zeps) * e2t;
          const T wmk = wmsk<T>(ci, k);
          const T zai = (uw1 + ui + uw + u1) / zci * wmk;
          const T zaj = (vs1 + vi + vs + v1) / zcj * wmk;
          const T zbi = fmn(fmn(zbw, T(-100) * fabs(zai)), lim_w(fabs(zai)));
          const T zbj = fmn(fmn(zbw, T(-100) * fabs(zaj)), lim_w(fabs(zaj)));
          const T zfk = fmx(oml(n0, k), oml(n0, k - 1));
          const T zck = (l[11] - gw1) / zml;
          a.zwi[q] = (zai / (zbi - a.zeps) * (T(1) - zfk) + zck * wiml * zfk) * wmk;
          a.zwj[q] = (zaj / (zbj - a.zeps) * (T(1) - zfk) + zck * wjml * zfk) * wmk;
        }
        r0 = l[0];
        ui = u1; uw = uw1; vi = v1; vs = vs1;
        b0 = l[5]; be = l[6]; bn = l[7];
      });
}

// The filtered slopes with the decrease near coasts and topography (:237-361) on
// the interior of levels 2..jpkm1; lbc_lnk (:365): 0 on the closed edges, every level.
// Level march; a warp covers 32 points of a row and writes the inner 30, so that of the
// nine neighbours of the 1-2-1 Shapiro filter (:237-275, :319-353) a point loads its own
// column's three and gets the others from the neighbour lanes. One point a thread with 36
// loads and 15 mask look-ups it took 58 us at 481x323x31 in FP32, 39 so (22 us by traffic).
template <class T>
__global__ void __launch_bounds__(32 * MARCH_Y) k_slp_filter(Dom<T> d, SlpArgs<T> a, int kch) {
  const MarchIdx c = march_index(d, kch, 30);
  const int J = d.jpi, j = c.j;
  if (j > d.jpj) return;  // whole warps
  const bool valid = c.i <= J, row = j >= 2 && j <= d.jpj - 1;
  const bool out = row && c.i >= 2 && c.i <= J - 1 && threadIdx.x >= 1 && threadIdx.x <= 30;
  const long n2 = d.n2, ij = (long)(min(c.i, J) - 1) + (long)(j - 1) * J, o = (long)c.m * d.n3 + ij;
  if (valid && (!row || c.i == 1 || c.i == J)) {
    const int k1 = c.k1 == d.jpk - 1 ? d.jpk : c.k1;  // the last chunk's edge columns: jpk too
    for (int k = c.k0; k <= k1; ++k) {
      const long q = o + (long)(k - 1) * n2;
      a.uslp[q] = T(0); a.vslp[q] = T(0); a.wslpi[q] = T(0); a.wslpj[q] = T(0);
    }
  }
  const int k0 = max(c.k0, 2);
  if (!row || k0 > c.k1) return;
  ColInfo ci{}, ce{}, cw{}, cn{}, cs{};
  if (out) {
    ci = d.ci[ij]; ce = d.ci[ij + 1]; cw = d.ci[ij - 1]; cn = d.ci[ij + J]; cs = d.ci[ij - J];
  }
  const T z1_16 = T(1) / T(16);
  march<T, 12>(
      k0, c.k1,
      [&](int k, T (&l)[12]) {
        const long q = o + (long)(k - 1) * n2;
        const T* z[4] = {a.zu + q, a.zv + q, a.zwi + q, a.zwj + q};
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          l[3 * f] = __ldg(z[f] - J);
          l[3 * f + 1] = __ldg(z[f]);
          l[3 * f + 2] = __ldg(z[f] + J);
        }
      },
      [&](int k, T (&l)[12]) {
        T z[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const T s = l[3 * f], m = l[3 * f + 1], n = l[3 * f + 2];
          const T sw = __shfl_up_sync(0xffffffffu, s, 1), se = __shfl_down_sync(0xffffffffu, s, 1);
          const T mw = __shfl_up_sync(0xffffffffu, m, 1), me = __shfl_down_sync(0xffffffffu, m, 1);
          const T nw = __shfl_up_sync(0xffffffffu, n, 1), ne = __shfl_down_sync(0xffffffffu, n, 1);
          z[f] = sw + se + nw + ne + T(2) * (s + mw + me + n) + T(4) * m;
        }
        if (out) {
          const long q = o + (long)(k - 1) * n2;
          const T um0 = umsk<T>(ci, k), vm0 = vmsk<T>(ci, k);
          T u = z1_16 * z[0];
          T v = z1_16 * z[1];
          u = u * (umsk<T>(cn, k) + umsk<T>(cs, k)) * T(0.5) * (um0 + umsk<T>(ci, k + 1)) * T(0.5);
          v = v * (vmsk<T>(ce, k) + vmsk<T>(cw, k)) * T(0.5) * (vm0 + vmsk<T>(ci, k + 1)) * T(0.5);
          const T zcofw = wmsk<T>(ci, k) * z1_16;
          const T wi = z[2] * zcofw;
          const T wj = z[3] * zcofw;
          const T zck = (um0 + umsk<T>(cw, k)) * (vm0 + vmsk<T>(cs, k)) * T(0.25);
          a.uslp[q] = u;
          a.vslp[q] = v;
          a.wslpi[q] = wi * zck;
          a.wslpj[q] = wj * zck;
        }
      });
}

// zps_hde (zpshde.F90:41-148): the horizontal gradients of the tracers at the last
// ocean level of the u- and v-points (the partial step), each tracer interpolated
// to the shallower bottom; the loop of the reference covers i <= jpim1, j <= jpjm1
// and lbc_lnk then zeroes the closed edges, so only the interior is nonzero.
template <class T>
__global__ void k_zps_hde(Dom<T> d, RO<T> pta, T* __restrict__ pgtu, T* __restrict__ pgtv, int kjpt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z, jpi = d.jpi;
  const long ij = (long)(i - 1) + (long)(j - 1) * jpi, n2 = d.n2, n3 = d.n3;
  const bool inner = i >= 2 && i <= jpi - 1 && j >= 2 && j <= d.jpj - 1;
  const ColInfo ci = d.ci[ij];
  const int iku = ci.mbku, ikum1 = iku - 1 > 1 ? iku - 1 : 1;
  const int ikv = ci.mbkv, ikvm1 = ikv - 1 > 1 ? ikv - 1 : 1;
  for (int n = 0; n < kjpt; ++n) {
    const long g = ((long)m * kjpt + n) * n2 + ij;
    if (!inner) {
      pgtu[g] = T(0);
      pgtv[g] = T(0);
      continue;
    }
    const RO<T> t = pta + ((long)m * kjpt + n) * n3;
    auto Q = [&](long o, int k) { return o + (long)(k - 1) * d.n2; };
    const T ze3wu = d.e3w_n(ij + 1, iku, m) - d.e3w_n(ij, iku, m);
    const T ze3wv = d.e3w_n(ij + jpi, ikv, m) - d.e3w_n(ij, ikv, m);
    T gu, gv;
    if (ze3wu >= T(0)) {
      const T zmaxu = ze3wu / d.e3w_n(ij + 1, iku, m);
      const T zti = t[Q(ij + 1, iku)] + zmaxu * (t[Q(ij + 1, ikum1)] - t[Q(ij + 1, iku)]);
      gu = umsk<T>(ci, 1) * (zti - t[Q(ij, iku)]);
    } else {
      const T zmaxu = -ze3wu / d.e3w_n(ij, iku, m);
      const T zti = t[Q(ij, iku)] + zmaxu * (t[Q(ij, ikum1)] - t[Q(ij, iku)]);
      gu = umsk<T>(ci, 1) * (t[Q(ij + 1, iku)] - zti);
    }
    if (ze3wv >= T(0)) {
      const T zmaxv = ze3wv / d.e3w_n(ij + jpi, ikv, m);
      const T ztj = t[Q(ij + jpi, ikv)] + zmaxv * (t[Q(ij + jpi, ikvm1)] - t[Q(ij + jpi, ikv)]);
      gv = vmsk<T>(ci, 1) * (ztj - t[Q(ij, ikv)]);
    } else {
      const T zmaxv = -ze3wv / d.e3w_n(ij, ikv, m);
      const T ztj = t[Q(ij, ikv)] + zmaxv * (t[Q(ij, ikvm1)] - t[Q(ij, ikv)]);
      gv = vmsk<T>(ci, 1) * (t[Q(ij + jpi, ikv)] - ztj);
    }
    pgtu[g] = gu;
    pgtv[g] = gv;
  }
}

// The unmasked in situ density anomaly of one (T, S, depth), eos_insitu_2d
// (eosbn2.F90:295-398): EOS-80 or the simplified equation of state
template <class T>
__device__ __forceinline__ T eos_rd_2d(const EosArgs<T>& a, T t, T sal, T dep);

// zps_hde's density part (zpshde.F90:150-184), one (i,j) a thread: T and S
// interpolated to the shallower bottom depth of the u- (v-) point as k_zps_hde does,
// their density there (eos_insitu_2d at gdept_n of the shallower bottom cell), its
// difference with prd on the deeper side; the closed edges 0 (lbc_lnk)
template <class T>
__global__ void k_zps_hde_rd(Dom<T> d, EosArgs<T> a, RO<T> prd, T* __restrict__ pgru, T* __restrict__ pgrv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z, jpi = d.jpi;
  const long ij = (long)(i - 1) + (long)(j - 1) * jpi, n2 = d.n2, n3 = d.n3;
  const long g = (long)m * n2 + ij;
  if (!(i >= 2 && i <= jpi - 1 && j >= 2 && j <= d.jpj - 1)) {
    pgru[g] = T(0);
    pgrv[g] = T(0);
    return;
  }
  const ColInfo ci = d.ci[ij];
  const int iku = ci.mbku, ikum1 = iku - 1 > 1 ? iku - 1 : 1;
  const int ikv = ci.mbkv, ikvm1 = ikv - 1 > 1 ? ikv - 1 : 1;
  auto Q = [&](long o, int k) { return o + (long)(k - 1) * n2; };
  const T ze3wu = d.e3w_n(ij + 1, iku, m) - d.e3w_n(ij, iku, m);
  const T ze3wv = d.e3w_n(ij + jpi, ikv, m) - d.e3w_n(ij, ikv, m);
  T zti[2], ztj[2];
  for (int n = 0; n < 2; ++n) {
    const RO<T> t = a.pts + ((long)m * 2 + n) * n3;
    if (ze3wu >= T(0)) {
      const T zmaxu = ze3wu / d.e3w_n(ij + 1, iku, m);
      zti[n] = t[Q(ij + 1, iku)] + zmaxu * (t[Q(ij + 1, ikum1)] - t[Q(ij + 1, iku)]);
    } else {
      const T zmaxu = -ze3wu / d.e3w_n(ij, iku, m);
      zti[n] = t[Q(ij, iku)] + zmaxu * (t[Q(ij, ikum1)] - t[Q(ij, iku)]);
    }
    if (ze3wv >= T(0)) {
      const T zmaxv = ze3wv / d.e3w_n(ij + jpi, ikv, m);
      ztj[n] = t[Q(ij + jpi, ikv)] + zmaxv * (t[Q(ij + jpi, ikvm1)] - t[Q(ij + jpi, ikv)]);
    } else {
      const T zmaxv = -ze3wv / d.e3w_n(ij, ikv, m);
      ztj[n] = t[Q(ij, ikv)] + zmaxv * (t[Q(ij, ikvm1)] - t[Q(ij, ikv)]);
    }
  }
  const long m3 = (long)m * n3;
  const T zhi = ze3wu >= T(0) ? a.gdept[m3 + Q(ij, iku)] : a.gdept[m3 + Q(ij + 1, iku)];
  const T zhj = ze3wv >= T(0) ? a.gdept[m3 + Q(ij, ikv)] : a.gdept[m3 + Q(ij + jpi, ikv)];
  const T zri = eos_rd_2d(a, zti[0], zti[1], zhi), zrj = eos_rd_2d(a, ztj[0], ztj[1], zhj);
  const T um1 = umsk<T>(ci, 1), vm1 = vmsk<T>(ci, 1);
  pgru[g] = ze3wu >= T(0) ? um1 * (zri - prd[m3 + Q(ij, iku)]) : um1 * (prd[m3 + Q(ij + 1, iku)] - zri);
  pgrv[g] = ze3wv >= T(0) ? vm1 * (zrj - prd[m3 + Q(ij, ikv)]) : vm1 * (prd[m3 + Q(ij + jpi, ikv)] - zrj);
}

// ------------------------------------------------------------ surface forcing
// tra_sbc (trasbc.F90:53-206) without runoff and ice-shelf melt, one (i,j) point per
// thread: the move of qsr into qns without penetration (:76-79), the swap of the
// forcing trends (:81-100), the trends of the heat and salt fluxes with the
// concentration/dilution of the linear free surface (:104-118) and their addition to
// the first level of tsa (:123-129), on the reference's index ranges.
template <class T>
__global__ void k_tra_sbc(Dom<T> d, SbcArgs<T> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi;
  const long p = (long)m * d.n2 + ij, pt = 2 * (long)m * d.n2 + ij, ps = pt + d.n2;
  T qns = a.qns[p];
  if (!a.traqsr) {
    qns = qns + a.qsr[p];
    a.qns[p] = qns;
    a.qsr[p] = T(0);
  }
  T bt, bs;
  if (a.mode == 0) {
    bt = a.tsc[pt];
    bs = a.tsc[ps];
  } else if (a.mode == 1) {
    bt = T(0);
    bs = T(0);
  } else {
    bt = a.tsc_b[pt];
    bs = a.tsc_b[ps];
  }
  if (a.mode != 2) {
    a.tsc_b[pt] = bt;
    a.tsc_b[ps] = bs;
  }
  if (i < 2 || i > d.jpi - 1 || j < 2) {
    if (a.mode != 0) {  // first step: sbc_tsc = 0 everywhere
      a.tsc[pt] = T(0);
      a.tsc[ps] = T(0);
    }
    return;
  }
  T tt = a.r1_rau0_rcp * qns;
  T ts = a.r1_rau0 * a.sfx[p];
  if (a.linssh) {
    const long q = 2 * (long)m * d.n3 + ij;
    const T e = a.emp[p];
    tt = tt + a.r1_rau0 * e * a.tsn[q];
    ts = ts + a.r1_rau0 * e * a.tsn[q + d.n3];
  }
  a.tsc[pt] = tt;
  a.tsc[ps] = ts;
  const long q = 2 * (long)m * d.n3 + ij;
  const T e3 = d.e3t_n(ij, 1, m);
  a.tsa[q] = a.tsa[q] + a.zfact * (bt + tt) / e3;
  a.tsa[q + d.n3] = a.tsa[q + d.n3] + a.zfact * (bs + ts) / e3;
}

// tra_qsr (traqsr.F90:77-302) with two bands (np_2BD, :243-256), one column per
// thread: the swap of the heat-content trend over the whole column (:134-147), the
// absorbed flux of levels 1..nksr, whose lower-interface attenuation is the next
// level's upper one (the same expression of the same depth, so computed once), the
// temperature trend (:260-267) and the first-level fraction with the closed lbc_lnk
// (:270-277: 0 on the domain edge).
template <class T>
__global__ void k_tra_qsr(Dom<T> d, QsrArgs<T> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi;
  const long c3 = (long)m * d.n3 + ij;
  const bool inner = i >= 2 && i <= d.jpi - 1 && j >= 2 && j <= d.jpj - 1;
  if (a.mode != 2) {
    const int k1 = inner ? a.nksr + 1 : 1;  // levels the solve below does not read
    for (int k = k1; k <= d.jpk; ++k) {
      const long q = c3 + (long)(k - 1) * d.n2;
      a.hc_b[q] = a.mode == 0 ? a.hc[q] : T(0);
    }
  }
  if (!inner) {
    a.fraq[(long)m * d.n2 + ij] = T(0);
    return;
  }
  const ColInfo ci = d.ci[ij];
  const T qsr = a.qsr[(long)m * d.n2 + ij];
  T* ta = a.tsa + 2 * (long)m * d.n3 + ij;  // temperature
  T g = a.gdepw[c3];
  T zc0 = a.zz0 * exp(-g * a.xsi0r) + a.zz1 * exp(-g * a.xsi1r);
  T h1 = T(0);
  for (int k = 1; k <= a.nksr; ++k) {
    const long q = c3 + (long)(k - 1) * d.n2;
    g = a.gdepw[q + d.n2];
    const T zc1 = a.zz0 * exp(-g * a.xsi0r) + a.zz1 * exp(-g * a.xsi1r);
    const T hb = a.mode == 0 ? a.hc[q] : (a.mode == 1 ? T(0) : a.hc_b[q]);
    if (a.mode != 2) a.hc_b[q] = hb;
    const T h = qsr * (zc0 * wmsk<T>(ci, k) - zc1 * wmsk<T>(ci, k + 1));
    a.hc[q] = h;
    const long qt = (long)(k - 1) * d.n2;
    ta[qt] = ta[qt] + a.z1_2 * (hb + h) / d.e3t_n(ij, k, m);
    if (k == 1) h1 = h;
    zc0 = zc1;
  }
  a.fraq[(long)m * d.n2 + ij] = qsr != T(0) ? h1 / (a.r1_rau0_rcp * qsr) : T(1);
}

// --------------------------------------------------------- equations of state
// eos_insitu, eos_insitu_pot, rab_3d and bn2, EOS-80 or the simplified one (np_seos),
// each FP64 expression in the reference's association.
// ---- EOS-80. FP64: one power k of the depth of a table in the reference's
// association (eosbn2.F90:242-265): acc = C(0,D); for j = D-1 .. 0,
// acc = (acc*zt + H_j*zs) + C(0,j), H_j = (..(C(n,j)*zs + C(n-1,j))*zs .. + C(1,j)),
// n = D - j.
template <int D>
__device__ __forceinline__ double e80_zn(const double* C, double zt, double zs) {
  double acc = C[e80_at(D, 0, D)];
#pragma unroll
  for (int j = D - 1; j >= 0; --j) {
    const int n = D - j;
    double h = C[e80_at(D, n, j)];
#pragma unroll
    for (int i = n - 1; i >= 1; --i) h = h * zs + C[e80_at(D, i, j)];
    acc = (acc * zt + h * zs) + C[e80_at(D, 0, j)];
  }
  return acc;
}
// all depth powers of a table; zn0: the surface part
template <int D0, int D1, int D2, int D3>
__device__ __forceinline__ double e80_poly(const double* C, double zt, double zs, double zh, double& zn0) {
  constexpr int o1 = e80_len(D0), o2 = o1 + e80_len(D1), o3 = o2 + e80_len(D2);
  const double z3 = e80_zn<D3>(C + o3, zt, zs), z2 = e80_zn<D2>(C + o2, zt, zs);
  const double z1 = e80_zn<D1>(C + o1, zt, zs);
  zn0 = e80_zn<D0>(C, zt, zs);
  return ((z3 * zh + z2) * zh + z1) * zh + zn0;
}
// FP32: Horner in s' = zs - s0, zt and zh with fused multiply-adds, two points to an
// instruction (fma.rn.f32x2), NP pairs of points a coefficient: the polynomials are
// issue-bound (70 multiply-adds a point in rab_3d, one coefficient load each).
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2_pack(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(F2 r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
template <int D, int NP>
__device__ __forceinline__ void e80_zn(const F2* C, const F2 (&zt)[NP], const F2 (&sp)[NP], F2 (&acc)[NP]) {
#pragma unroll
  for (int n = 0; n < NP; ++n) acc[n] = C[e80_at(D, 0, D)];
#pragma unroll
  for (int j = D - 1; j >= 0; --j) {
    F2 h[NP];
#pragma unroll
    for (int n = 0; n < NP; ++n) h[n] = C[e80_at(D, D - j, j)];
#pragma unroll
    for (int i = D - j - 1; i >= 0; --i) {
      const F2 c = C[e80_at(D, i, j)];
#pragma unroll
      for (int n = 0; n < NP; ++n) h[n] = f2_fma(h[n], sp[n], c);
    }
#pragma unroll
    for (int n = 0; n < NP; ++n) acc[n] = f2_fma(acc[n], zt[n], h[n]);
  }
}
template <int D0, int D1, int D2, int D3, int NP>
__device__ __forceinline__ void e80_poly(const F2* C, const F2 (&zt)[NP], const F2 (&sp)[NP], const F2 (&zh)[NP],
                                         F2 (&zn)[NP], F2 (&zn0)[NP]) {
  constexpr int o1 = e80_len(D0), o2 = o1 + e80_len(D1), o3 = o2 + e80_len(D2);
  F2 z[NP];
  e80_zn<D3>(C + o3, zt, sp, zn);
  e80_zn<D2>(C + o2, zt, sp, z);
#pragma unroll
  for (int n = 0; n < NP; ++n) zn[n] = f2_fma(zn[n], zh[n], z[n]);
  e80_zn<D1>(C + o1, zt, sp, z);
#pragma unroll
  for (int n = 0; n < NP; ++n) zn[n] = f2_fma(zn[n], zh[n], z[n]);
  e80_zn<D0>(C, zt, sp, zn0);
#pragma unroll
  for (int n = 0; n < NP; ++n) zn[n] = f2_fma(zn[n], zh[n], zn0[n]);
}

// The unmasked density anomaly and surface (potential) density (eos_insitu,
// eos_insitu_pot; eosbn2.F90:236-292, :400-462), or the expansion coefficients
// (rab_3d; :588-661), of U points: x = anomaly or alpha, y = rhop or beta.
template <bool RAB, bool E80, int U, class T>
__device__ __forceinline__ void eos_points(const EosArgs<T>& a, const T (&t)[U], const T (&s)[U], const T (&dep)[U],
                                           T (&x)[U], T (&y)[U]) {
  constexpr T r1_Z0 = T(1.e-4), r1_T0 = T(1.0 / 40.0), r1_S0 = T(1.0 / 40.0), rdeltaS = T(20.0);
  if constexpr (!E80) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const T zt = t[u] - T(10), zs = s[u] - T(35), zh = dep[u];
      if constexpr (RAB) {
        T zn = a.a0 * (T(1) + a.lambda1 * zt + a.mu1 * zh) + a.nu * zs;
        x[u] = zn * a.r1_rau0;
        zn = a.b0 * (T(1) - a.lambda2 * zs - a.mu2 * zh) - a.nu * zt;
        y[u] = zn * a.r1_rau0;
      } else {
        T zn = -a.a0 * (T(1) + T(0.5) * a.lambda1 * zt) * zt + a.b0 * (T(1) - T(0.5) * a.lambda2 * zs) * zs -
               a.nu * zt * zs;
        y[u] = a.rau0 + zn;
        zn = zn - (a.a0 * a.mu1 * zt + a.b0 * a.mu2 * zs) * zh;
        x[u] = zn * a.r1_rau0;
      }
    }
  } else if constexpr (sizeof(T) == 8) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const T zh = dep[u] * r1_Z0, zt = t[u] * r1_T0, zs = sqrt(fabs(s[u] + rdeltaS) * r1_S0);
      T zn0;
      if constexpr (RAB) {
        x[u] = e80_poly<5, 3, 1, 0>(a.e80.alp, zt, zs, zh, zn0) * a.r1_rau0;
        y[u] = e80_poly<5, 3, 1, 0>(a.e80.bet, zt, zs, zh, zn0) / zs * a.r1_rau0;
      } else {
        x[u] = e80_poly<6, 4, 2, 1>(a.e80.eos, zt, zs, zh, zn0) * a.r1_rau0 - T(1);
        y[u] = zn0;
      }
    }
  } else {
    constexpr int NP = (U + 1) / 2;
    float zs[2 * NP];
    F2 zt[NP], sp[NP], zh[NP], zn[NP], zn0[NP];
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      float w[2], h[2], v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int u = 2 * n + e < U ? 2 * n + e : U - 1;
        h[e] = dep[u] * r1_Z0;
        w[e] = t[u] * r1_T0;
        const float s2 = fabsf(s[u] + rdeltaS) * r1_S0;
        zs[2 * n + e] = sqrtf(s2);
        v[e] = (s2 - a.e80_s0 * a.e80_s0) / (zs[2 * n + e] + a.e80_s0);  // zs - s0 without cancellation
      }
      zt[n] = f2_pack(w[0], w[1]);
      zh[n] = f2_pack(h[0], h[1]);
      sp[n] = f2_pack(v[0], v[1]);
    }
    float p[2 * NP], q[2 * NP];
    if constexpr (RAB) {
      e80_poly<5, 3, 1, 0>(a.e80.alp, zt, sp, zh, zn, zn0);
#pragma unroll
      for (int n = 0; n < NP; ++n) f2_unpack(zn[n], p[2 * n], p[2 * n + 1]);
      e80_poly<5, 3, 1, 0>(a.e80.bet, zt, sp, zh, zn, zn0);
#pragma unroll
      for (int n = 0; n < NP; ++n) f2_unpack(zn[n], q[2 * n], q[2 * n + 1]);
    } else {  // the anomaly about the value at (35 psu, 0 degC, 0 m) first
      e80_poly<6, 4, 2, 1>(a.e80.eos, zt, sp, zh, zn, zn0);
#pragma unroll
      for (int n = 0; n < NP; ++n) {
        f2_unpack(zn[n], p[2 * n], p[2 * n + 1]);
        f2_unpack(zn0[n], q[2 * n], q[2 * n + 1]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = RAB ? p[u] * a.r1_rau0 : (p[u] + a.e80_anom) * a.r1_rau0;
      y[u] = RAB ? q[u] / zs[u] * a.r1_rau0 : q[u] + a.e80_rho0;
    }
  }
}

template <class T>
__device__ __forceinline__ T eos_rd_2d(const EosArgs<T>& a, T t, T sal, T dep) {
  if (a.eos80) {
    const T t1[1] = {t}, s1[1] = {sal}, h1[1] = {dep};
    T rd[1], rhop[1];
    eos_points<false, true>(a, t1, s1, h1, rd, rhop);
    return rd[0];
  }
  const T zt = t - T(10), zs = sal - T(35);
  const T zn = -a.a0 * (T(1) + T(0.5) * a.lambda1 * zt + a.mu1 * dep) * zt +
               a.b0 * (T(1) - T(0.5) * a.lambda2 * zs - a.mu2 * dep) * zs - a.nu * zt * zs;
  return zn * a.r1_rau0;
}

// eos_insitu (WHAT 0), eos_insitu_pot (1) and rab_3d (2) on levels 1..jpk-1: a thread
// owns one (i,j) of the flat 2-D plane (no stencil, so no ragged tiles) and a chunk of
// levels, EOS_U of them loaded before the first polynomial. The polynomials' operands
// come from the constant bank; the kernels are bound by instruction issue in FP32 (66 to
// 72 % of the slots: some 110 instructions a point of the polynomials; by traffic, 4 and 5
// fields, 28 and 35 us of 48 and 55) and by the FP64 pipe in FP64. As one point a thread, with
// the coefficients loaded from global memory, the six calls of a step's density (two
// rab_3d, two bn2, eos_insitu, eos_insitu_pot) took 679 us at 752x502x31 in FP32, 343 so.
// Blocks of 2 (FP64) and 4 warps: with 8, a small grid was a few blocks whose points shared an
// SM's FP64 pipe (rab_3d 20x17x10 16, 62x42x31 43 us, 9 and 32 so), and a large one had a
// longer last round (93x61x31x12 669, 648).
template <class T>
constexpr int EOS_BLOCK = sizeof(T) == 4 ? 128 : 64;
template <class T>
constexpr int EOS_LEV = sizeof(T) == 4 ? 4 : 1;  // FP64: four levels in a row left a small grid's FP64 pipes idle
template <class T, int WHAT, bool E80>
__global__ void __launch_bounds__(EOS_BLOCK<T>) k_eos(Dom<T> d, const __grid_constant__ EosArgs<T> a, int kch) {
  const long p = (long)blockIdx.x * EOS_BLOCK<T> + threadIdx.x;
  if (p >= d.n2) return;
  const int m = blockIdx.z, k0 = blockIdx.y * kch + 1, k1 = min(k0 + kch - 1, d.jpk - 1);
  const long c3 = (long)m * d.n3 + p, c4 = 2 * (long)m * d.n3 + p;
  const ColInfo ci = d.ci[p];
  const T* __restrict__ ts = a.pts + c4;
  const T* __restrict__ dep = (WHAT == 2 ? a.gdept : a.pdep) + c3;
  constexpr int EOS_U = EOS_LEV<T>;
  for (int k = k0; k <= k1; k += EOS_U) {
    T t[EOS_U], s[EOS_U], h[EOS_U];
#pragma unroll
    for (int u = 0; u < EOS_U; ++u) {
      const int ku = k + u <= k1 ? k + u : k1;
      const long o = (long)(ku - 1) * d.n2;
      t[u] = __ldg(ts + o);
      s[u] = __ldg(ts + d.n3 + o);
      h[u] = __ldg(dep + o);
    }
    T x[EOS_U], y[EOS_U];
    if constexpr (WHAT == 0 && !E80) {
#pragma unroll
      for (int u = 0; u < EOS_U; ++u) x[u] = eos_rd_2d(a, t[u], s[u], h[u]);
    } else {
      eos_points<WHAT == 2, E80>(a, t, s, h, x, y);
    }
#pragma unroll
    for (int u = 0; u < EOS_U; ++u) {
      if (k + u > k1) break;
      const long o = (long)(k + u - 1) * d.n2;
      const T tm = tmsk<T>(ci, k + u);
      if constexpr (WHAT == 2) {
        a.pab[c4 + o] = x[u] * tm;
        a.pab[c4 + d.n3 + o] = y[u] * tm;
      } else {
        if constexpr (WHAT == 1) a.prhop[c3 + o] = y[u] * tm;
        a.prd[c3 + o] = x[u] * tm;
      }
    }
  }
}

// bn2 (eosbn2.F90:889-933) on levels 2..jpk-1: a thread marches down a chunk of one
// flat (i,j)'s levels and carries T, S, the expansion coefficients and the depth of
// the level above, so that each of the 7 fields is read once; U of them are loaded together.
template <class T, int U>
__global__ void __launch_bounds__(EOS_BLOCK<T>) k_bn2(Dom<T> d, const __grid_constant__ EosArgs<T> a, int kch) {
  const long p = (long)blockIdx.x * EOS_BLOCK<T> + threadIdx.x;
  if (p >= d.n2) return;
  const int m = blockIdx.z, k0 = blockIdx.y * kch + 2, k1 = min(k0 + kch - 1, d.jpk - 1);
  if (k0 > k1) return;
  const long c3 = (long)m * d.n3 + p, c4 = 2 * (long)m * d.n3 + p, n3 = d.n3;
  const ColInfo ci = d.ci[p];
  const T* __restrict__ ts = a.pts + c4;
  const T* __restrict__ ab = a.pab_in + c4;
  const T* __restrict__ gt = a.gdept + c3;
  const T* __restrict__ gw = a.gdepw + c3;
  long o = (long)(k0 - 2) * d.n2;
  T tu = __ldg(ts + o), su = __ldg(ts + n3 + o), au = __ldg(ab + o), bu = __ldg(ab + n3 + o), hu = __ldg(gt + o);
  for (int k = k0; k <= k1; k += U) {
    T t[U], s[U], x[U], y[U], h[U], w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int ku = k + u <= k1 ? k + u : k1;
      o = (long)(ku - 1) * d.n2;
      t[u] = __ldg(ts + o);
      s[u] = __ldg(ts + n3 + o);
      x[u] = __ldg(ab + o);
      y[u] = __ldg(ab + n3 + o);
      h[u] = __ldg(gt + o);
      w[u] = __ldg(gw + o);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k + u > k1) break;
      const T zrw = (w[u] - h[u]) / (hu - h[u]);
      const T zaw = x[u] * (T(1) - zrw) + au * zrw;
      const T zbw = y[u] * (T(1) - zrw) + bu * zrw;
      a.pn2[c3 + (long)(k + u - 1) * d.n2] =
          a.grav * (zaw * (tu - t[u]) - zbw * (su - s[u])) / d.e3w_n(p, k + u, m) * wmsk<T>(ci, k + u);
      tu = t[u]; su = s[u]; au = x[u]; bu = y[u]; hu = h[u];
    }
  }
}

// hpg_zco (dynhpg.F90:258-323), one interior column per thread: the pressure
// gradient integrated downwards from the surface in registers. The levels depend on one
// another through the running sums alone, so a batch of them is loaded together (the
// compiler cannot move the load of a trend over the store of the level above): 68 -> 41
// us at 752x502x31 in FP32 (35 us by traffic).
template <class T>
__global__ void __launch_bounds__(128) k_hpg_zco(Dom<T> d, const T* __restrict__ rhd, T* __restrict__ ua,
                                                 T* __restrict__ va, T zcoef0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i < 2 || i > d.jpi - 1 || j < 2 || j > d.jpj - 1) return;
  const int m = blockIdx.z;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi;
  const long c3 = (long)m * d.n3 + ij;
  const T r1u = d.r1_e1u[ij], r1v = d.r1_e2v[ij];
  const int n2 = (int)d.n2;
  const E3Col<T> e3w(d.e3w_n, ij, m);
  T re = T(0), rn = T(0), r0 = T(0), zhpi = T(0), zhpj = T(0);
  constexpr int U = BATCH<T>;
  for (int kt = 1; kt <= d.jpk - 1; kt += U) {
    const long b = c3 + (long)(kt - 1) * n2;
    const T *pr = rhd + b, *prn = pr + d.jpi;
    T* __restrict__ pu = ua + b;
    T* __restrict__ pv = va + b;
    T s0[U], se[U], sn[U], a0[U], a1[U], ew[U];
#pragma unroll
    for (int x = 0; x < U; ++x) {
      const int z = min(x, d.jpk - 1 - kt), q = z * n2;
      s0[x] = __ldg(pr + q);
      se[x] = __ldg(pr + q + 1);
      sn[x] = __ldg(prn + q);
      a0[x] = pu[q];
      a1[x] = pv[q];
      ew[x] = e3w(kt + z);
    }
#pragma unroll
    for (int x = 0; x < U; ++x) {
      const int k = kt + x;
      if (k > d.jpk - 1) break;
      const T zcoef1 = zcoef0 * ew[x];
      if (k == 1) {
        zhpi = zcoef1 * (se[x] - s0[x]) * r1u;
        zhpj = zcoef1 * (sn[x] - s0[x]) * r1v;
      } else {
        zhpi = zhpi + zcoef1 * ((se[x] + re) - (s0[x] + r0)) * r1u;
        zhpj = zhpj + zcoef1 * ((sn[x] + rn) - (s0[x] + r0)) * r1v;
      }
      pu[x * n2] = a0[x] + zhpi;
      pv[x * n2] = a1[x] + zhpj;
      r0 = s0[x];
      re = se[x];
      rn = sn[x];
    }
  }
}

// zdf_mxl (zdfmxl.F90:59-141), one (i,j) column per thread: N^2 integrated
// downwards from nlb10 against the density criterion, the turbocline searched upwards
// from the bottom, then the depths of the two levels.
template <class T>
__global__ void k_zdf_mxl(Dom<T> d, MxlArgs<T> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi;
  const long c3 = (long)m * d.n3 + ij, c2 = (long)m * d.n2 + ij;
  const int ikt = d.mbkt[ij];
  const ColInfo ci = d.ci[ij];
  int nmln = a.nlb10;
  T h = T(0);
  for (int k = a.nlb10; k <= d.jpk - 1; ++k) {
    const T n2 = a.rn2b[c3 + (long)(k - 1) * d.n2];
    h = h + (n2 > T(0) ? n2 : T(0)) * d.e3w_n(ij, k, m);
    if (h < a.zn2_c) nmln = (k < ikt ? k : ikt) + 1;
  }
  const T ssm = d.ssmask[ij];
  if (a.hmld) {
    int imld = ikt + 1;
    for (int k = d.jpk - 1; k >= a.nlb10; --k)
      if (a.avt[c3 + (long)(k - 1) * d.n2] < a.avt_c * wmsk<T>(ci, k)) imld = k;
    a.hmld[c2] = a.gdepw[c3 + (long)(imld - 1) * d.n2] * ssm;
  }
  a.nmln[c2] = nmln;
  a.hmlp[c2] = a.gdepw[c3 + (long)(nmln - 1) * d.n2] * ssm;
  a.hmlpt[c2] = a.gdept[c3 + (long)(nmln - 2) * d.n2] * ssm;
}

// ---------------------------------------------------------- momentum trends
// dyn_ldf_lap, vor_ene, dyn_keg and dyn_zad: a thread owns one (i,j) and marches down a
// chunk of levels. Each reads two or three 3-D fields at the point and its neighbours
// and updates ua and va, so memory bounds them once the instructions are few enough and
// a warp has its next level's loads in flight while it works on this one:
// * the 2-D metrics of the stencil (26 in vor_ene) are loaded once a chunk instead of
//   once a point;
// * level k + 1 is loaded before level k is computed and stored (the compiler cannot
//   move the load of a trend over the store of the level above);
// * quotients by what a chunk shares (the e1, e2 of the column; with 1-D scale factors,
//   FLAT, the e3 of the level, whose reciprocals the block forms once) are divr's.
// One point a thread, they took 248, 150 and 73 us and, one column a thread, dyn_zad
// 191 us at 752x502x31 in FP32; so they take 93, 65, 60 and 65 us (floors by traffic:
// 56, 42, 42 and 49 us; the rest is instruction issue and the latency left).
// dyn_ldf_lap (dynldf_lap_blp.F90:37-104), linear free surface (e3*_b = e3*_n):
// -curl(curl) + grad(div) of the before velocity, each relative vorticity zcur and
// divergence zdiv by the reference's expression, formed once a tile: a block covers 32 x
// LDF_Y points and writes the inner 30 x (LDF_Y - 2); zcur of the western and zdiv of the
// eastern point come from the neighbour lane, zcur of the southern and zdiv of the northern
// point from shared memory (two buffers, one barrier a level). A point that formed two of
// each took 96 registers, 16 loads a level and 107 us at 752x502x31 in FP32, 93 so (blocks
// of 10, 12, 16 rows: 94, 94, 97).
constexpr int LDF_Y = 8;
template <class T, bool FLAT>
__global__ void __launch_bounds__(32 * LDF_Y, FLAT && sizeof(T) == 4 ? 5 : 2) k_dyn_ldf_lap(Dom<T> d, const T* __restrict__ ahmt,
                                                            const T* __restrict__ ahmf, const T* __restrict__ pub,
                                                            const T* __restrict__ pvb, T* __restrict__ pua,
                                                            T* __restrict__ pva, T zsign, int kch) {
  __shared__ E3Prof<T> pt, pu, pv;
  __shared__ T pf[KMAX + 1], scur[2][LDF_Y][32], sdiv[2][LDF_Y][32];
  const MarchIdx c = march_index(d, kch, 30);
  const int J = d.jpi, x = threadIdx.x, y = threadIdx.y, j = blockIdx.y * (LDF_Y - 2) + y + 1;
  if constexpr (FLAT) {
    pt.fill(d.e3t_b, c.m, d.jpk);
    pu.fill(d.e3u_n, c.m, d.jpk);
    pv.fill(d.e3v_n, c.m, d.jpk);
    const int k = y * 32 + x + 1;
    if (k <= d.jpk) pf[k] = d.e3f_n(0, k, c.m);
    __syncthreads();
  }
  const int i0 = min(c.i, J), j0 = min(j, d.jpj);
  const bool out = c.i >= 2 && c.i <= J - 1 && x >= 1 && x <= 30 && j >= 2 && j <= d.jpj - 1 && y >= 1 && y <= LDF_Y - 2;
  // offsets that stay in the domain (a value formed with one of 0 is not used)
  const int e = i0 < J ? 1 : 0, w = i0 > 1 ? 1 : 0, n = j0 < d.jpj ? J : 0, s = j0 > 1 ? J : 0;
  const long p = (long)(i0 - 1) + (long)(j0 - 1) * J;
  const T rf0 = d.r1_e1e2f[p], rt0 = d.r1_e1e2t[p];
  const T v0 = d.e2v[p], ve = d.e2v[p + e], u0 = d.e1u[p], un = d.e1u[p + n];
  const T x0 = d.e2u[p], xw = d.e2u[p - w], y0 = d.e1v[p], ys = d.e1v[p - s];
  const T r2u = d.r1_e2u[p], r1u = d.r1_e1u[p], r1v = d.r1_e1v[p], r2v = d.r1_e2v[p];
  const long o = (long)c.m * d.n3 + p;
  march<T, 8>(
      c.k0, c.k1,
      [&](int k, T (&l)[8]) {
        const long q = o + (long)(k - 1) * d.n2;
        l[0] = __ldg(pub + q); l[1] = __ldg(pub + q + n); l[2] = __ldg(pvb + q); l[3] = __ldg(pvb + q - s);
        l[4] = __ldg(ahmf + q); l[5] = __ldg(ahmt + q);
        if (out) { l[6] = pua[q]; l[7] = pva[q]; }
      },
      [&](int k, T (&l)[8]) {
        T eu, ev, euw, evs, ef;
        if constexpr (FLAT) {
          eu = euw = pu.e[k];
          ev = evs = pv.e[k];
          ef = pf[k];
        } else {
          eu = d.e3u_n(p, k, c.m); euw = d.e3u_n(p - w, k, c.m);
          ev = d.e3v_n(p, k, c.m); evs = d.e3v_n(p - s, k, c.m);
          ef = d.e3f_n(p, k, c.m);
        }
        const T uw = __shfl_up_sync(0xffffffffu, l[0], 1), vr = __shfl_down_sync(0xffffffffu, l[2], 1);
        const T cur0 = l[4] * ef * rf0 * (ve * vr - v0 * l[2] - un * l[1] + u0 * l[0]);
        const T ht = l[5] * rt0;
        const T div0 = (FLAT ? divr(ht, pt.e[k], pt.r[k]) : ht / d.e3t_b(p, k, c.m)) *
                       (x0 * eu * l[0] - xw * euw * uw + y0 * ev * l[2] - ys * evs * l[3]);
        T (&bc)[LDF_Y][32] = scur[k & 1], (&bd)[LDF_Y][32] = sdiv[k & 1];
        bc[y][x] = cur0;
        bd[y][x] = div0;
        const T curw = __shfl_up_sync(0xffffffffu, cur0, 1), dive = __shfl_down_sync(0xffffffffu, div0, 1);
        __syncthreads();
        if (out) {
          const T curs = bc[y - 1][x], divn = bd[y + 1][x];
          auto over_u = [&](T a) { return FLAT ? divr(a, eu, pu.r[k]) : a / eu; };
          auto over_v = [&](T a) { return FLAT ? divr(a, ev, pv.r[k]) : a / ev; };
          const long q = o + (long)(k - 1) * d.n2;
          pua[q] = l[6] + zsign * (-over_u((cur0 - curs) * r2u) + (dive - div0) * r1u);
          pva[q] = l[7] + zsign * (over_v((cur0 - curw) * r1v) + (divn - div0) * r2v);
        }
      });
}

// vor_ene (dynvor.F90:324-429), z-coordinate without ln_dynvor_msk; KV: the vorticity
// (1 planetary, 2 relative, 4 total). The vorticities zwz and transports zwx, zwy of
// the four surrounding points are formed where read, each with the reference's
// expression.
template <class T, int KV>
__global__ void __launch_bounds__(32 * MARCH_Y) k_vor_ene(Dom<T> d, const T* __restrict__ pun, const T* __restrict__ pvn,
                                                          T* __restrict__ pua, T* __restrict__ pva, int kch) {
  const MarchIdx c = march_index(d, kch);
  if (!c.inner) return;
  const int J = d.jpi;
  const long p = c.ij;
  // metrics of the f-points p, s = p-J, w = p-1 (KV 1 reads ff_f alone)
  T f0 = T(0), fs = T(0), fw = T(0), rf0 = T(0), rfs = T(0), rfw = T(0);
  T v0 = T(0), ve = T(0), vs = T(0), vse = T(0), vw = T(0), u0 = T(0), un = T(0), us = T(0), uw = T(0), unw = T(0);
  if constexpr (KV != 2) {
    f0 = d.ff_f[p]; fs = d.ff_f[p - J]; fw = d.ff_f[p - 1];
  }
  if constexpr (KV != 1) {
    rf0 = d.r1_e1e2f[p]; rfs = d.r1_e1e2f[p - J]; rfw = d.r1_e1e2f[p - 1];
    v0 = d.e2v[p]; ve = d.e2v[p + 1]; vs = d.e2v[p - J]; vse = d.e2v[p - J + 1]; vw = d.e2v[p - 1];
    u0 = d.e1u[p]; un = d.e1u[p + J]; us = d.e1u[p - J]; uw = d.e1u[p - 1]; unw = d.e1u[p - 1 + J];
  }
  const T x0 = d.e2u[p], xw = d.e2u[p - 1], xn = d.e2u[p + J], xnw = d.e2u[p - 1 + J];
  const T y0 = d.e1v[p], ys = d.e1v[p - J], ye = d.e1v[p + 1], yse = d.e1v[p + 1 - J];
  const T ru = T(0.25) * d.r1_e1u[p], rv = T(0.25) * d.r1_e2v[p];
  auto zwz = [&](T ff, T rf, T rot) -> T { return KV == 1 ? ff : KV == 2 ? rot * rf : ff + rot * rf; };
  const long o = (long)c.m * d.n3 + p;
  march<T, 12>(
      c.k0, c.k1,
      [&](int k, T (&l)[12]) {
        const long q = o + (long)(k - 1) * d.n2;
        const T *u = pun + q, *v = pvn + q;
        l[0] = __ldg(u); l[1] = __ldg(u - 1); l[2] = __ldg(u + J); l[3] = __ldg(u - 1 + J);
        l[4] = KV == 1 ? T(0) : __ldg(u - J);
        l[5] = __ldg(v); l[6] = __ldg(v + 1); l[7] = __ldg(v - J); l[8] = __ldg(v + 1 - J);
        l[9] = KV == 1 ? T(0) : __ldg(v - 1);
        l[10] = pua[q]; l[11] = pva[q];
      },
      [&](int k, T (&l)[12]) {
        const T b0 = l[0], bw = l[1], bn = l[2], bnw = l[3], bs = l[4];
        const T c0 = l[5], ce = l[6], cs = l[7], cse = l[8], cw = l[9];
        const T zy1 = ys * cs + yse * cse;
        const T zy2 = y0 * c0 + ye * ce;
        const T zx1 = xw * bw + xnw * bnw;
        const T zx2 = x0 * b0 + xn * bn;
        const T zc = zwz(f0, rf0, ve * ce - v0 * c0 - un * bn + u0 * b0);
        const T zs = zwz(fs, rfs, vse * cse - vs * cs - u0 * b0 + us * bs);
        const T zw = zwz(fw, rfw, v0 * c0 - vw * cw - unw * bnw + uw * bw);
        const long q = o + (long)(k - 1) * d.n2;
        pua[q] = l[10] + ru * (zs * zy1 + zc * zy2);
        pva[q] = l[11] - rv * (zw * zx1 + zc * zx2);
      });
}

// dyn_keg (dynkeg.F90, nkeg_C2): the kinetic energy of the point and of its east /
// north neighbours formed where read.
template <class T>
__global__ void __launch_bounds__(32 * MARCH_Y) k_dyn_keg(Dom<T> d, const T* __restrict__ un, const T* __restrict__ vn,
                                                          T* __restrict__ ua, T* __restrict__ va, int kch) {
  const MarchIdx c = march_index(d, kch);
  if (!c.inner) return;
  const int J = d.jpi;
  const T e1u = d.e1u[c.ij], e2v = d.e2v[c.ij], re1u = T(1) / e1u, re2v = T(1) / e2v;
  auto hke = [](T u0, T u1, T v0, T v1) -> T {
    const T zu = u0 * u0 + u1 * u1;
    const T zv = v0 * v0 + v1 * v1;
    return T(0.25) * (zv + zu);
  };
  const long o = (long)c.m * d.n3 + c.ij;
  march<T, 12>(
      c.k0, c.k1,
      [&](int k, T (&l)[12]) {
        const long q = o + (long)(k - 1) * d.n2;
        const T *u = un + q, *v = vn + q;
        l[0] = __ldg(u); l[1] = __ldg(u - 1); l[2] = __ldg(u + 1); l[3] = __ldg(u + J); l[4] = __ldg(u - 1 + J);
        l[5] = __ldg(v); l[6] = __ldg(v - J); l[7] = __ldg(v + 1); l[8] = __ldg(v + 1 - J); l[9] = __ldg(v + J);
        l[10] = ua[q]; l[11] = va[q];
      },
      [&](int k, T (&l)[12]) {
        const T b0 = l[0], bw = l[1], be = l[2], bn = l[3], bnw = l[4];
        const T c0 = l[5], cs = l[6], ce = l[7], cse = l[8], cn = l[9];
        const T h = hke(bw, b0, cs, c0);
        const long q = o + (long)(k - 1) * d.n2;
        ua[q] = l[10] - divr(hke(b0, be, cse, ce) - h, e1u, re1u);
        va[q] = l[11] - divr(hke(bnw, bn, c0, cn) - h, e2v, re2v);
      });
}

// dyn_zad (dynzad.F90): the w-level momentum fluxes of the column carried down, each
// formed once (the one at the top of a chunk by both its chunks).
template <class T, bool FLAT>
__global__ void __launch_bounds__(32 * MARCH_Y) k_dyn_zad(Dom<T> d, const T* __restrict__ un, const T* __restrict__ vn,
                                                          const T* __restrict__ wn, T* __restrict__ ua,
                                                          T* __restrict__ va, int kch) {
  __shared__ E3Prof<T> pu, pv;
  const MarchIdx c = march_index(d, kch);
  const int m = c.m, J = d.jpi, K = d.jpk - 1;
  if constexpr (FLAT) {
    pu.fill(d.e3u_n, m, d.jpk);
    pv.fill(d.e3v_n, m, d.jpk);
    __syncthreads();
  }
  if (!c.inner) return;
  const long ij = c.ij, n2 = d.n2, c3 = (long)m * d.n3 + ij;
  const T e0 = T(0.25) * d.e1e2t[ij], e1 = T(0.25) * d.e1e2t[ij + 1], e2 = T(0.25) * d.e1e2t[ij + J];
  const T r1u = d.r1_e1e2u[ij], r1v = d.r1_e1e2v[ij];
  const long q0 = c3 + (long)(c.k0 - 1) * n2;
  T wu = T(0), wv = T(0);  // zwuw, zwvw at the top of level k
  T u0 = __ldg(un + q0), v0 = __ldg(vn + q0);
  if (c.k0 > 1) {
    const T z0 = e0 * __ldg(wn + q0), zi = e1 * __ldg(wn + q0 + 1), zj = e2 * __ldg(wn + q0 + J);
    wu = (zi + z0) * (__ldg(un + q0 - n2) - u0);
    wv = (zj + z0) * (__ldg(vn + q0 - n2) - v0);
  }
  march<T, 7>(
      c.k0, c.k1,
      [&](int k, T (&l)[7]) {  // wn, un, vn of the level below; ua, va
        const long q = c3 + (long)(k - 1) * n2, qb = k < K ? q + n2 : q;
        l[0] = __ldg(wn + qb); l[1] = __ldg(wn + qb + 1); l[2] = __ldg(wn + qb + J);
        l[3] = __ldg(un + qb); l[4] = __ldg(vn + qb);
        l[5] = ua[q]; l[6] = va[q];
      },
      [&](int k, T (&l)[7]) {
        T wu1 = T(0), wv1 = T(0);  // at its bottom (w-level k+1), 0 at jpk
        if (k < K) {
          const T z0 = e0 * l[0], zi = e1 * l[1], zj = e2 * l[2];
          wu1 = (zi + z0) * (u0 - l[3]);
          wv1 = (zj + z0) * (v0 - l[4]);
        }
        u0 = l[3];
        v0 = l[4];
        const T tu = (wu + wu1) * r1u, tv = (wv + wv1) * r1v;
        const long q = c3 + (long)(k - 1) * n2;
        if constexpr (FLAT) {
          ua[q] = l[5] - divr(tu, pu.e[k], pu.r[k]);
          va[q] = l[6] - divr(tv, pv.e[k], pv.r[k]);
        } else {
          ua[q] = l[5] - tu / d.e3u_n(ij, k, m);
          va[q] = l[6] - tv / d.e3v_n(ij, k, m);
        }
        wu = wu1;
        wv = wv1;
      });
}

// ---------------------------------------------------------------- usrdef_sbc (GYRE)
// SIN and COS of the analytic forcing: FP64 by the evaluations the test oracle shares
// (nemo_sin.h), FP32 by the library
template <class T> __device__ __forceinline__ T usr_sin(T x);
template <class T> __device__ __forceinline__ T usr_cos(T x);
template <> __device__ __forceinline__ double usr_sin<double>(double x) { return nemo_sin(x); }
template <> __device__ __forceinline__ double usr_cos<double>(double x) { return nemo_cos(x); }
template <> __device__ __forceinline__ float usr_sin<float>(float x) { return sinf(x); }
template <> __device__ __forceinline__ float usr_cos<float>(float x) { return cosf(x); }

// The point part of usrdef_sbc_oce (usrdef_sbc.F90:113-135, :160-172), one (i,j) a
// thread: sbc's swap of the before fields, qsr, the restoring qns from the before SST,
// the raw E-P, the wind stress
template <class T>
__global__ void k_usr_sbc_a(Dom<T> d, UsrSbcArgs<T> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi, p = (long)m * d.n2 + ij;
  const long q = (long)m * 2 * d.n3 + ij;  // surface temperature of the member
  if (a.s[6] != 0.0) {
    if (a.utau_b) a.utau_b[p] = a.utau[p];
    if (a.vtau_b) a.vtau_b[p] = a.vtau[p];
    if (a.emp_b) a.emp_b[p] = a.emp[p];
  }
  const T rpi = T(3.141592653589793);
  const T g = a.gphit[p];
  const T t_star = T(a.s[0]) * usr_cos<T>(rpi * (g - T(5.)) / T(a.s[1]));
  const T qsr = T(230) * usr_cos<T>(T(3.1415) * (g - T(a.s[2])) / T(0.9 * 180));
  a.qsr[p] = qsr;
  a.qns[p] = T(-40.e0) * (a.tsb[q] - t_star) - qsr;
  T emp;
  if (g >= T(14.845) && T(37.2) >= g)
    emp = T(0.7) * T(3.16e-5) * usr_sin<T>(rpi / T(2) * (g - T(37.2)) / T(24.6 - 37.2)) * T(a.s[3]);
  else
    emp = -T(0.8) * T(3.16e-5) * usr_sin<T>(rpi / T(2) * (g - T(37.2)) / T(46.8 - 37.2)) * T(a.s[4]);
  a.emp[p] = emp;
  const T ztaun = T(a.s[5]);
  a.utau[p] = -ztaun * usr_sin<T>(rpi * (a.gphiu[p] - T(15.)) / T(29. - 15.));
  a.vtau[p] = ztaun * usr_sin<T>(rpi * (a.gphiv[p] - T(15.)) / T(29. - 15.));
}

// The rest (usrdef_sbc.F90:137-144, :176-186): E-P less its domain mean, sfx = 0, the
// heat content of E-P at the now SST in qns, the wind-stress modulus (interior; the
// closed lbc_lnk zeroes the edges)
template <class T>
__global__ void k_usr_sbc_b(Dom<T> d, UsrSbcArgs<T> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (i > d.jpi || j > d.jpj) return;
  const int m = blockIdx.z;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi, p = (long)m * d.n2 + ij;
  const long q = (long)m * 2 * d.n3 + ij;
  const double zsumemp = a.gsum[m] / a.zsurf;
  const T tm = tmsk<T>(d.ci[ij], 1);
  const T emp = (T)((double)a.emp[p] - zsumemp * (double)tm);
  a.emp[p] = emp;
  a.sfx[p] = T(0);
  a.qns[p] = a.qns[p] - emp * a.tsn[q] * T(a.rcp);
  T tau = T(0);
  if (i >= 2 && i <= d.jpi - 1 && j >= 2 && j <= d.jpj - 1) {
    const T ztx = a.utau[p - 1] + a.utau[p];
    const T zty = a.vtau[p - d.jpi] + a.vtau[p];
    tau = T(0.5) * sqrt(ztx * ztx + zty * zty);
  }
  a.taum[p] = tau;
}

// the step's scalars of the forcing into device memory (a launch outside any
// captured graph, so a replay reads the values of its own step)
__global__ void k_usr_put(double* dst, double s0, double s1, double s2, double s3, double s4, double s5,
                          double s6) {
  dst[0] = s0; dst[1] = s1; dst[2] = s2; dst[3] = s3; dst[4] = s4; dst[5] = s5; dst[6] = s6;
}

// ---------------------------------------------------------------- zdf_phy (TKE)
// SIN of the Langmuir-cell source: FP64 by the evaluation the test oracle shares
// (nemo_sin.h), FP32 by the library
__device__ __forceinline__ double lc_sin(double x) { return nemo_sin_0pi(x); }
__device__ __forceinline__ float lc_sin(float x) { return sinf(x); }

// zdf_sh2 (zdfsh2.F90:57-74): the shear production at the interior w-points of levels
// 2..jpk-1, from 2 x that of the four uw- and vw-points around (with the closure's avm_k;
// with a linear free surface e3uw_n = e3uw_b = the rest-state MIN of the neighbouring
// e3w). Level march: the velocities of the level above are carried, the quotients by the
// squared e3 of the level are divr's with 1-D scale factors (FLAT). One point a thread
// it took 67 us at 481x323x31 in FP32, 34 so (17 us by traffic).
template <class T, bool FLAT>
__global__ void __launch_bounds__(32 * MARCH_Y) k_zdf_sh2(Dom<T> d, ZphyArgs<T> a, int kch) {
  __shared__ T pe[KMAX + 1], pr[KMAX + 1];  // e3w^2 and its reciprocal
  const MarchIdx c = march_index(d, kch);
  const int m = c.m, J = d.jpi;
  if constexpr (FLAT) {
    const int k = threadIdx.y * 32 + threadIdx.x + 1;
    if (k <= d.jpk) {
      const T e = d.e3w_n(0, k, m);
      pe[k] = e * e;
      pr[k] = T(1) / pe[k];
    }
    __syncthreads();
  }
  if (!c.inner) return;
  const int k0 = max(c.k0, 2);
  const long ij = c.ij, n2 = d.n2, o = (long)m * d.n3 + ij;
  const ColInfo ci = d.ci[ij], cw = d.ci[ij - 1], cs = d.ci[ij - J];
  const long qt = o + (long)(k0 - 2) * n2;  // the level above the first
  T u0 = a.un[qt], uw = a.un[qt - 1], v0 = a.vn[qt], vs = a.vn[qt - J];
  T x0 = a.ub[qt], xw = a.ub[qt - 1], y0 = a.vb[qt], ys = a.vb[qt - J];
  if (k0 > c.k1) return;
  march<T, 13>(
      k0, c.k1,
      [&](int k, T (&l)[13]) {
        const long q = o + (long)(k - 1) * n2;
        const T *un = a.un + q, *vn = a.vn + q, *ub = a.ub + q, *vb = a.vb + q, *av = a.avm_k + q;
        l[0] = __ldg(un); l[1] = __ldg(un - 1); l[2] = __ldg(vn); l[3] = __ldg(vn - J);
        l[4] = __ldg(ub); l[5] = __ldg(ub - 1); l[6] = __ldg(vb); l[7] = __ldg(vb - J);
        l[8] = __ldg(av); l[9] = __ldg(av + 1); l[10] = __ldg(av - 1); l[11] = __ldg(av + J); l[12] = __ldg(av - J);
      },
      [&](int k, T (&l)[13]) {
        auto over = [&](T x, long p, long nb) -> T {  // x / e^2, e = MIN(e3w(p), e3w(p + nb))
          if constexpr (FLAT) return divr(x, pe[k], pr[k]);
          const T e = fmn(d.e3w_n(p, k, m), d.e3w_n(p + nb, k, m));
          return x / (e * e);
        };
        const T um0 = umsk<T>(ci, k), umw = umsk<T>(cw, k), vm0 = vmsk<T>(ci, k), vms = vmsk<T>(cs, k);
        const T su1 = over((l[9] + l[8]) * (u0 - l[0]) * (x0 - l[4]), ij, 1) * (um0 * umsk<T>(ci, k - 1));
        const T su0 = over((l[8] + l[10]) * (uw - l[1]) * (xw - l[5]), ij - 1, 1) * (umw * umsk<T>(cw, k - 1));
        const T sv1 = over((l[11] + l[8]) * (v0 - l[2]) * (y0 - l[6]), ij, J) * (vm0 * vmsk<T>(ci, k - 1));
        const T sv0 = over((l[8] + l[12]) * (vs - l[3]) * (ys - l[7]), ij - J, J) * (vms * vmsk<T>(cs, k - 1));
        a.sh2[o + (long)(k - 1) * n2] =
            T(0.25) * ((su0 + su1) * (T(2) - umw * um0) + (sv0 + sv1) * (T(2) - vms * vm0));
        u0 = l[0]; uw = l[1]; v0 = l[2]; vs = l[3];
        x0 = l[4]; xw = l[5]; y0 = l[6]; ys = l[7];
      });
}

// The column part of zdf_phy, one water column per thread (its levels are coupled
// by the implicit TKE equation and the mixing-length limits):
//  tke_tke (zdftke.F90:168-440): surface value of en, Langmuir cells, the inverse
//    Prandtl number apdlr, the implicit system assembled and forward-eliminated in
//    one downward sweep, back-substituted upwards, the floor rn_emin;
//  tke_avn (:443-630): the buoyancy length sqrt(2 en / N^2), limited by nn_mxl in a
//    downward and an upward sweep, and on that upward sweep avm_k, avt_k, dissl, the
//    Prandtl correction of avt_k, then zdf_phy's avt, avm (zdfphy.F90:269-270),
//    zdf_evd (zdfevd.F90:76-109) and avs = avt (:284).
// Edge columns get the closed lbc_lnk of the five coefficients (zdfphy.F90:301-303).
// Each expression keeps the reference's association (the solve's in FP64). The column's
// system, lengths and Prandtl numbers stay in shared memory (the slots of the upper diagonal
// and the forward value take the limited and raw lengths), so that memory sees each field
// about once, and the next level is loaded ahead; with five work arrays in memory the column
// made some 30 passes over it, 269 us at 481x323x31 in FP32 (50 us by traffic). Bound by
// the loads in flight: three values a level (in FP32 the upper diagonal and the forward
// value over the pivot; en is read back) let 16 warps an SM run, 117 us; four values (the
// pivot, and en kept) 12 warps, 150 us. Blocks of 4 rows, not 2 (122) or 8 (156).
// SH: the values a level kept in shared memory, the others in work arrays (FP32 three; FP64,
// with the pivot, four, two or none: launch_zdf_phy).
// With 1-D scale factors (FLAT) the quotients by e3t e3w, and always those by the pivot,
// are divr's; where EVD acts is kept as a bit a level.
template <class T>
constexpr int TKE_Y = sizeof(T) == 4 ? 4 : 2;
template <class T, bool FLAT, int SH>
__global__ void __launch_bounds__(32 * TKE_Y<T>) k_zdf_tke(Dom<T> d, ZphyArgs<T> a) {
  extern __shared__ __align__(16) unsigned char col_smem[];
  __shared__ T pu[KMAX + 1], ru[KMAX + 1], pl[KMAX + 1], rl[KMAX + 1];  // e3t(k) e3w(k), e3t(k-1) e3w(k), reciprocals
  constexpr int nt = 32 * TKE_Y<T>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int m = blockIdx.z, jpk = d.jpk;
  if constexpr (FLAT) {
    static_assert(nt >= KMAX, "one thread a level");
    const int k = threadIdx.y * 32 + threadIdx.x + 1;
    if (k <= jpk) {
      const T e3w = d.e3w_n(0, k, m);
      pu[k] = d.e3t_n(0, k, m) * e3w;
      ru[k] = T(1) / pu[k];
      pl[k] = d.e3t_n(0, k > 1 ? k - 1 : 1, m) * e3w;
      rl[k] = T(1) / pl[k];
    }
    __syncthreads();
  }
  if (i > d.jpi || j > d.jpj) return;
  const long n2 = d.n2;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi;
  const long c3 = (long)m * d.n3 + ij, c2 = (long)m * d.n2 + ij;
  // the column's values, k = 1..jpk: su, sl at [k * n1], sp and (FP64) sd at [k * n1d]
  T *su = reinterpret_cast<T*>(col_smem) + threadIdx.y * 32 + threadIdx.x - nt, *sl = su + jpk * nt;
  T *sp = sl + jpk * nt, *sd = sp + jpk * nt;
  if constexpr (SH < 3) {
    sp = a.apdlr + c3 - n2;
    sd = a.zdiag + c3 - n2;
  }
  if constexpr (SH < 2) {
    su = a.zd_up + c3 - n2;
    sl = a.zd_lw + c3 - n2;
  }
  const auto n1 = [&] {
    if constexpr (SH >= 2) return nt;
    else return n2;
  }();
  const auto n1d = [&] {
    if constexpr (SH >= 3) return nt;
    else return n2;
  }();
  if (i == 1 || i == d.jpi || j == 1 || j == d.jpj) {
    for (int k = 1; k <= jpk; ++k) {
      const long q = c3 + (long)(k - 1) * n2;
      a.avm_k[q] = T(0); a.avt_k[q] = T(0); a.avm[q] = T(0); a.avt[q] = T(0);
      if (a.avs) a.avs[q] = T(0);
    }
    return;
  }
  const ColInfo ci = d.ci[ij];
  const T tm1 = tmsk<T>(ci, 1);
  const T taum = a.taum[c2];
  const T en1 = fmx(a.rn_emin0, a.zbbrau * taum) * tm1;  // surface boundary condition
  a.en[c3] = en1;
  // Langmuir cells: the depth zhlc of the first w-level whose cumulated potential
  // energy exceeds the Stokes-drift scale, and the source amplitude zfr
  T zhlc = T(1), zfr = T(0);
  if (a.ln_lc) {
    const T zus = a.lc_cof1 * taum;
    T zpelc = fmx(a.rn2b[c3], T(0)) * a.gdepw[c3] * d.e3w_n(ij, 1, m);
    int imlc = d.mbkt[ij] + 1;
    for (int k = 2; k <= jpk - 1; ++k) {
      const long q = c3 + (long)(k - 1) * n2;
      zpelc = zpelc + fmx(a.rn2b[q], T(0)) * a.gdepw[q] * d.e3w_n(ij, k, m);
      if (zpelc > zus) { imlc = k; break; }
    }
    zhlc = a.gdepw[c3 + (long)(imlc - 1) * n2];
    const T zs = a.lc_cof2 * sqrt(taum);
    zfr = (T(1) - T(4) * (a.fr_i ? a.fr_i[c2] : T(0))) * zs * zs * zs * tm1;
    if (zfr < T(0)) zfr = T(0);
  }
  // downward sweep: right-hand side, matrix, forward elimination
  // of the level above: the upper diagonal and the forward value (FP32: over the pivot),
  // the pivot and its reciprocal
  T up_p = T(0), lw_p = T(0), dg_p = T(1), rd_p = T(1);
  T avm_km1 = a.avm_k[c3], avm_k = a.avm_k[c3 + n2];
  unsigned long long evd_at = 0;  // levels (bit k - 1) where EVD acts
  march<T, 7>(
      2, jpk - 1,
      [&](int k, T (&l)[7]) {
        const long q = c3 + (long)(k - 1) * n2;
        l[0] = a.en[q]; l[1] = a.avm_k[q + n2]; l[2] = __ldg(a.sh2 + q); l[3] = a.dissl[q];
        l[4] = __ldg(a.rn2 + q); l[5] = __ldg(a.rn2b + q); l[6] = a.avt_k[q];
      },
      [&](int k, T (&l)[7]) {
        const T wm = wmsk<T>(ci, k), tm = tmsk<T>(ci, k);
        T en = l[0];
        if (zfr != T(0)) {
          const T dep = a.gdepw[c3 + (long)(k - 1) * n2];
          if (dep - zhlc < T(0) && wm != T(0)) {
            const T zwlc = a.rn_lc * lc_sin(a.rpi * dep / zhlc);
            en = en + a.rdt * zfr * (zwlc * zwlc * zwlc) / zhlc;
          }
        }
        const T avm_kp1 = l[1], sh2 = l[2], dissl = l[3];
        if (a.nn_pdl == 1) {
          const T zri = fmx(l[5], T(0)) * avm_k / (sh2 + a.rn_bshear);
          sp[k * n1d] = fmx(T(0.1), a.ri_cri / fmx(a.ri_cri, zri));
        }
        const T zcof = a.zfact1 * tm;
        if (a.ln_zdfevd && fmn(l[4], l[5]) <= T(-1.e-12)) evd_at |= 1ULL << (k - 1);
        T up = zcof * fmx(avm_kp1 + avm_k, T(2.e-5)), lw = zcof * fmx(avm_k + avm_km1, T(2.e-5));
        if constexpr (FLAT) {
          up = divr(up, pu[k], ru[k]);
          lw = divr(lw, pl[k], rl[k]);
        } else {
          const T e3w = d.e3w_n(ij, k, m);
          up = up / (d.e3t_n(ij, k, m) * e3w);
          lw = lw / (d.e3t_n(ij, k - 1, m) * e3w);
        }
        T dg = T(1) - lw - up + a.zfact2 * dissl * wm;
        const T rhs = en + a.rdt * (sh2 - l[6] * l[4] + a.zfact3 * dissl * en) * wm;
        T lf;
        if (k == 2) {
          lf = rhs - lw * en1;
        } else if constexpr (sizeof(T) == 4) {
          dg = dg - lw * up_p;
          lf = rhs - lw * lw_p;
        } else {
          dg = dg - divr(lw * up_p, dg_p, rd_p);
          lf = rhs - divr(lw, dg_p, rd_p) * lw_p;
        }
        rd_p = T(1) / dg;
        if constexpr (sizeof(T) == 4) {
          up_p = divr(up, dg, rd_p);
          lw_p = divr(lf, dg, rd_p);
        } else {
          sd[k * n1d] = dg;
          dg_p = dg; up_p = up; lw_p = lf;
        }
        su[k * n1] = up_p; sl[k * n1] = lw_p;
        avm_km1 = avm_k;
        avm_k = avm_kp1;
      });
  // upward sweep: back substitution, the floor, and the buoyancy length (into sl)
  T en_p = T(0);
  march<T, 1>(
      2, jpk - 1, [&](int x, T (&l)[1]) { l[0] = __ldg(a.rn2 + c3 + (long)(jpk - x) * n2); },
      [&](int x, T (&l)[1]) {
        const int k = jpk + 1 - x;
        T en = (k == jpk - 1) ? sl[k * n1] : sl[k * n1] - su[k * n1] * en_p;
        if constexpr (sizeof(T) == 8) en = en / sd[k * n1d];
        en_p = en;
        const T e = fmx(en, a.rn_emin) * wmsk<T>(ci, k);
        a.en[c3 + (long)(k - 1) * n2] = e;
        sl[k * n1] = fmx(a.rmxl_min, sqrt(T(2) * e / fmx(l[0], a.rsmall)));
      });
  const T mxl1 = a.ln_mxl0 ? fmx(a.rn_mxl0, a.zraug * taum * tm1) : a.rn_mxl0;
  // downward limits of nn_mxl = 2 (in place) and 3 (su, from the unlimited lengths)
  if (a.nn_mxl == 2 || a.nn_mxl == 3) {
    T* const out = a.nn_mxl == 2 ? sl : su;
    T p = mxl1;
    for (int k = 2; k <= jpk - 1; ++k) {
      p = fmn(p + d.e3t_n(ij, k - 1, m), sl[k * n1]);
      out[k * n1] = p;
    }
  }
  // upward sweep: the limited lengths, the coefficients, the ocean Kz
  const T evd = a.rn_evd;
  T nxt = a.rmxl_min;  // zmxlm(jpk)
  auto limit = [&](int x, T (&l)[1]) {
    const int k = jpk + 1 - x;
    const long q = c3 + (long)(k - 1) * n2;
    const T wm = wmsk<T>(ci, k), tm = tmsk<T>(ci, k);
    const T raw = sl[k * n1];
    T lm, ld;
    if (a.nn_mxl == 2) {
      lm = fmn(nxt + d.e3t_n(ij, k + 1, m), raw);
      ld = lm;
      nxt = lm;
    } else if (a.nn_mxl == 3) {
      const T dn = fmn(nxt + d.e3t_n(ij, k + 1, m), raw);
      nxt = dn;
      const T lu = su[k * n1];
      lm = fmn(lu, dn);
      ld = sqrt(lu * dn);
    } else if (a.nn_mxl == 1) {
      lm = fmn(d.e3w_n(ij, k, m), raw);
      ld = lm;
    } else {  // 0: bounded by the distances to the surface (mikt = 1) and the bottom
      const T dep = a.gdepw[q], e3w = d.e3w_n(ij, k, m);
      const T z = fmn(fmn(dep - a.gdepw[c3], raw), a.gdepw[c3 + (long)d.mbkt[ij] * n2] - dep);
      lm = z * wm + fmn(raw, e3w) * (T(1) - wm);
      ld = z * wm + fmn(lm, e3w) * (T(1) - wm);
    }
    const T zsqen = sqrt(l[0]);
    const T zav = a.rn_ediff * lm * zsqen;
    const T avmk = fmx(zav, a.rn_avm0) * wm;
    T avtk = fmx(zav, a.rn_avt0) * wm;
    a.dissl[q] = zsqen / ld;
    if (a.nn_pdl == 1) avtk = fmx(sp[k * n1d] * avtk, a.rn_avt0) * tm;
    a.avm_k[q] = avmk;
    a.avt_k[q] = avtk;
    T avt = avtk, avm = avmk;
    if (evd_at >> (k - 1) & 1) {
      avt = evd * wm;
      if (a.nn_evdm == 1) avm = evd * wm;
    }
    a.avt[q] = avt;
    a.avm[q] = avm;
    if (a.avs) a.avs[q] = avt;
  };
  march<T, 1>(2, jpk - 1, [&](int x, T (&l)[1]) { l[0] = a.en[c3 + (long)(jpk - x) * n2]; }, limit);
  // the surface level: coefficients from en(1) and the surface length; avt, avm
  // keep their values there unless zdf_evd acts
  {
    const T wm = tm1;
    const T zsqen = sqrt(en1);
    const T zav = a.rn_ediff * mxl1 * zsqen;
    a.avm_k[c3] = fmx(zav, a.rn_avm0) * wm;
    a.avt_k[c3] = fmx(zav, a.rn_avt0) * wm;
    a.dissl[c3] = zsqen / mxl1;
    T avt = a.avt[c3];
    if (a.ln_zdfevd && fmn(a.rn2[c3], a.rn2b[c3]) <= T(-1.e-12)) {
      avt = evd * wm;
      a.avt[c3] = avt;
      if (a.nn_evdm == 1) a.avm[c3] = evd * wm;
    }
    if (a.avs) a.avs[c3] = avt;
  }
}

}  // namespace nemo
