// k_tra.cuh -- tracer kernels: transports, FCT advection (upstream + antidiffusive
// fluxes, Zalesak limiter, final trend), compact 4th-order vertical interpolation,
// laplacian and rotated iso-neutral lateral diffusion, implicit vertical diffusion.
//
// Stencil kernels map one thread to one (i,j,k) point: the grid is x = i (32 per
// block, coalesced), y = j, z = (member, level). No state is carried along k, so
// every level of every column is independent and the GPU has ~jpi*jpj*jpk threads
// to hide memory latency with; neighbour values (i+-1, j+-1, k+-1) come from L1/L2.
// A value a reference loop computes once and its neighbours reuse (a face flux, a
// limiter coefficient at k+1) is recomputed by each thread that needs it, with the
// same operands in the same order. Only genuine column recurrences (the compact
// interpolation and the implicit vertical solve) keep one thread per column.
//
// Indices i, j, k are 1-based as in the Fortran they restate, and every expression
// keeps the reference's association (the FP64 instantiation is compiled without
// FMA contraction, so it reproduces the reference's FP64 arithmetic operation by
// operation).
#pragma once
#include "nemo_common.cuh"

namespace nemo {

constexpr int KMAX = 64;  // maximum jpk (checked at context creation)

template <class T>
struct ColIdx {
  int i, j, m;
  long ij;
  bool valid, interior;
};

// column kernels: grid x = i, y = j, z = member
template <class T>
__device__ __forceinline__ ColIdx<T> col_index(const Dom<T>& d) {
  ColIdx<T> c;
  c.i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  c.j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  c.m = blockIdx.z;
  c.valid = c.i <= d.jpi && c.j <= d.jpj;
  c.interior = c.i >= 2 && c.i <= d.jpi - 1 && c.j >= 2 && c.j <= d.jpj - 1;
  c.ij = (long)(c.i - 1) + (long)(c.j - 1) * d.jpi;
  return c;
}

struct PtIdx {
  int i, j, k, m;
  long ij, q;  // column offset, offset within one (jpi,jpj,jpk) field
  bool valid, interior;
};

// point kernels: grid x = i, y = j, z = member * jpk + (k - 1)
template <class T>
__device__ __forceinline__ PtIdx pt_index(const Dom<T>& d) {
  PtIdx c;
  c.i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  c.j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  c.k = (int)(blockIdx.z % (unsigned)d.jpk) + 1;
  c.m = (int)(blockIdx.z / (unsigned)d.jpk);
  c.valid = c.i <= d.jpi && c.j <= d.jpj;
  c.interior = c.i >= 2 && c.i <= d.jpi - 1 && c.j >= 2 && c.j <= d.jpj - 1;
  c.ij = (long)(c.i - 1) + (long)(c.j - 1) * d.jpi;
  c.q = c.ij + (long)(c.k - 1) * d.n2;
  return c;
}

// k-march kernels: grid x = i, y = j, z = member * nchunk + chunk. A thread walks
// the levels k0..k1 of one column (Dom::kch levels per chunk: KCH, fewer on a grid too
// small to fill the chip), keeping in registers what level k+1 shares with level k, so
// the vertical neighbours are loaded once.
constexpr int KCH = 16;
// Levels a chunk: the longest of 16, 8, 4, 2 with which the chunks of all columns still
// give each SM eight warps. A chunk reloads its first level's neighbours, so a large grid
// keeps 16 (8 costs 25 us of 1.35 ms a step at 752x502x31); at 32x22x31 a march of 16
// levels is 16 memory round trips in a row on 3 % of the SMs (78 us for the four kernels).
// In FP64 two warps already fill an SM's FP64 pipe, and what a chunk repeats costs more.
inline int tra_chunk(long n2, int nmem, int jpk, bool fp64) {
  const long want = SMS * 32L * (fp64 ? 2 : 8);
  int c = KCH;
  while (c > 2 && n2 * nmem * ((jpk + c - 1) / c) < want) c /= 2;
  return c;
}
struct KIdx {
  int i, j, m, k0, k1;
  long ij;
  bool valid, interior;
};
template <class T>
__device__ __forceinline__ KIdx k_index(const Dom<T>& d) {
  const int nch = (d.jpk + d.kch - 1) / d.kch;
  KIdx c;
  c.i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  c.j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  c.m = (int)(blockIdx.z / (unsigned)nch);
  const int ch = (int)blockIdx.z - c.m * nch;
  c.k0 = ch * d.kch + 1;
  c.k1 = c.k0 + d.kch - 1 < d.jpk ? c.k0 + d.kch - 1 : d.jpk;
  c.valid = c.i <= d.jpi && c.j <= d.jpj;
  c.interior = c.i >= 2 && c.i <= d.jpi - 1 && c.j >= 2 && c.j <= d.jpj - 1;
  c.ij = (long)(c.i - 1) + (long)(c.j - 1) * d.jpi;
  return c;
}

// Level-march kernels: grid x = i, y = j, z = member * nchunk + chunk; a thread walks the
// levels of a chunk of 1..jpk-1 and loads level k + 1 before it computes and stores
// level k (the compiler cannot move a load over a store that may alias it).
constexpr int MARCH_Y = 4;
struct MarchIdx {
  int i, j, m, k0, k1;
  long ij;
  bool inner;
};
template <class T>
__device__ __forceinline__ MarchIdx march_index(const Dom<T>& d, int kch, int width = 32) {
  const int nch = (d.jpk - 1 + kch - 1) / kch;
  MarchIdx c;
  c.i = blockIdx.x * width + threadIdx.x + 1;
  c.j = blockIdx.y * MARCH_Y + threadIdx.y + 1;
  c.m = (int)(blockIdx.z / (unsigned)nch);
  c.k0 = ((int)blockIdx.z - c.m * nch) * kch + 1;
  c.k1 = min(c.k0 + kch - 1, d.jpk - 1);
  c.ij = (long)(c.i - 1) + (long)(c.j - 1) * d.jpi;
  c.inner = c.i >= 2 && c.i <= d.jpi - 1 && c.j >= 2 && c.j <= d.jpj - 1;
  return c;
}
// Levels a thread walks: 32, 16, .. 1, the most that still gives every SM its resident
// warps (64 of 32 points); in FP32 up to 8 levels already at a quarter of them: a grid that
// small is in L2, and one or two levels a thread cost more than the warps gain (tra_nxt
// 152x102x31 8.4 us with 1 level, 6.6 with 4; 200x151x31 10.9 with 2, 9.9 with 4, 8.6 with 8;
// FP64 vor_ene 92x62x31 23 us with 1 level, 27 with 2).
template <class T>
inline int march_chunk(const Dom<T>& d) {
  const long full = SMS * 64L * 32;
  int f = 32;
  while (f > 1 && (long)d.n2 * d.nmem * ((d.jpk - 1 + f - 1) / f) < (sizeof(T) == 4 && f <= 8 ? full / 4 : full)) f /= 2;
  return f;
}
template <class T>
inline dim3 march_grid(const Dom<T>& d, int kch, int width = 32, int edge = 0) {
  return dim3((d.jpi - edge + width - 1) / width, (d.jpj + MARCH_Y - 1) / MARCH_Y, d.nmem * ((d.jpk - 1 + kch - 1) / kch));
}
// load(k, buffer) a level ahead of compute(k, buffer), for the levels k0..k1
template <class T, int N, class L, class C>
__device__ __forceinline__ void march(int k0, int k1, L load, C compute) {
  T a[N], b[N];
  load(k0, a);
  for (int k = k0; k <= k1; k += 2) {
    if (k + 1 <= k1) load(k + 1, b);
    compute(k, a);
    if (k + 1 > k1) break;
    if (k + 2 <= k1) load(k + 2, a);
    compute(k + 1, b);
  }
}
// The 1-D profile of a scale factor and its reciprocals, for the levels of a block (one
// thread a level; the caller synchronises).
template <class T>
struct E3Prof {
  T e[KMAX + 1], r[KMAX + 1];
  __device__ __forceinline__ void fill(const E3<T>& f, int m, int jpk) {
    const int k = threadIdx.y * 32 + threadIdx.x + 1;
    if (k <= jpk) {
      e[k] = f(0, k, m);
      r[k] = T(1) / e[k];
    }
  }
};

// one column of a scale-factor field, or the 1-D profile (stride 1)
template <class T>
struct E3Col {
  const T* p;
  int st;
  __device__ __forceinline__ E3Col(const E3<T>& e, long ij, int m) : p(e.p.p + m * e.sm + ij * (long)e.s), st((int)e.sk) {}
  __device__ __forceinline__ T operator()(int k) const { return __ldg(p + (long)(k - 1) * st); }
};
// --------------------------------------------------------------------------------
// traadv.F90:99-124: zun = e2u*e3u_n*un, zvn = e1v*e3v_n*vn, zwn = e1e2t*wn, 0 at jpk.
template <class T>
__global__ void k_adv_trp(Dom<T> d, const T* __restrict__ un, const T* __restrict__ vn,
                          const T* __restrict__ wn, T* __restrict__ zun, T* __restrict__ zvn,
                          T* __restrict__ zwn) {
  const PtIdx c = pt_index(d);
  if (!c.valid) return;
  const long q = (long)c.m * d.n3 + c.q;
  if (c.k == d.jpk) {
    zun[q] = T(0); zvn[q] = T(0); zwn[q] = T(0);
    return;
  }
  zun[q] = d.e2u[c.ij] * d.e3u_n(c.ij, c.k, c.m) * un[q];
  zvn[q] = d.e1v[c.ij] * d.e3v_n(c.ij, c.k, c.m) * vn[q];
  zwn[q] = d.e1e2t[c.ij] * wn[q];
}

// Lateral diffusion arguments (also carried by the FCT kernels for the fused
// advection + iso-neutral trend of the hot path).
template <class T>
struct LdfArgs {
  RO<T> pahu, pahv;          // NULL: aht_c * umask/vmask above jpk (ldftra.F90:292-372)
  T aht_c;
  RO<T> pgu, pgv;            // partial-step gradients (jpi,jpj,kjpt) when zps
  int zps;
  RO<T> ptb, ptbb;
  T* pta;
  int kjpt, kpass;
  T zsign;
  // iso-neutral
  RO<T> uslp, vslp, wslpi, wslpj;
  T *ah_wslp2, *akz;
  int lap, blp, msc;
  T z2dt, z1_2dt;
  T *zftu, *zftv, *ztfw;     // work: iso-neutral fluxes (jpi,jpj,jpk,kjpt)
  int tma;                   // FP32 hot configuration: stage the tracer planes by TMA
  int* err;                  // device error flag (a timed-out wait of the TMA kernel)
  int polls;                 // bound of each wait on a tensor copy (polls of <= ~1 us)
};

// Arguments shared by the three FCT kernels.
template <class T>
struct FctArgs {
  T p2dt;
  T r1_p2dt;                 // 1 / p2dt, correctly rounded
  RO<T> pun, pvn, pwn;       // transports, or velocities when trp != 0
  int trp;                   // 1: scale velocities to transports on the fly (traadv.F90:110-114)
  RO<T> ptb, ptn;            // (jpi,jpj,jpk,kjpt)
  const T* pta_in;           // NULL: the trend starts from tsa = 0 (step.F90:234)
  T* pta;                    // (jpi,jpj,jpk,kjpt)
  T *zwi, *ax, *ay, *az;     // work: monotone guess and antidiffusive fluxes (jpi,jpj,jpk,kjpt)
  T *betup, *betdo;          // work: limiter coefficients (jpi,jpj,jpk,kjpt)
  RO<T> ztw;                 // compact 4th-order tn at w-points (kn_fct_v = 4), or NULL
  int kjpt, kn_fct_h, kn_fct_v, linssh;
  int with_iso;              // stage c also adds the iso-neutral trend (kpass 1) of `iso`
  LdfArgs<T> iso;
  int tma;                   // FP32 hot configuration: stage the planes by TMA
  int fused;                 // with tma: the three stages as one kernel (k_fct_fused_tma)
  int* err;                  // device error flag (a timed-out wait of a TMA kernel)
  int polls;                 // bound of each wait on a tensor copy (polls of <= ~1 us)
  T* lim;                    // NULL, or where k_fct_c records the limiter multipliers
                             // ((member*kjpt + n)*3 + face)*n3, for the adjoint
};

// ---- value-exact helpers of the FCT and iso-neutral kernels. FP64 runs at 1/58 of
// the FP32 rate on this GPU, and compares, min/max and products by 0/1 masks all
// occupy that pipe; these forms move them to the integer pipe or drop them while
// giving the reference's values (at most the sign of a zero differs, which no later
// operation of these routines can see: zeros are added, multiplied or compared
// with SIGN of key_nosignedzero).

// the sign bit of x is clear (x > 0 or x = +0; -0 counts as negative)
template <class T>
__device__ __forceinline__ bool sgn_pos(T x) {
  if constexpr (sizeof(T) == 8) return __double2hiint(x) >= 0;
  else return __float_as_int(x) >= 0;
}
// integer with the order of the FP64 values (-0 just below +0)
__device__ __forceinline__ long long ord_key(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
// MAX / MIN of two values: FP64 through the integer order of the values, FP32 by
// the min/max instruction
template <class T>
__device__ __forceinline__ T vmax(T a, T b) {
  if constexpr (sizeof(T) == 8) return ord_key(a) > ord_key(b) ? a : b;
  else return fmaxf(a, b);
}
template <class T>
__device__ __forceinline__ T vmin(T a, T b) {
  if constexpr (sizeof(T) == 8) return ord_key(a) < ord_key(b) ? a : b;
  else return fminf(a, b);
}
// MAX(0, x) and MIN(0, x)
template <class T>
__device__ __forceinline__ T pos_part(T x) { return sgn_pos(x) ? x : T(0); }
template <class T>
__device__ __forceinline__ T neg_part(T x) { return sgn_pos(x) ? T(0) : x; }
// x * m for a 0/1 mask m: FP64 selects (no product), FP32 keeps the product
template <class T>
__device__ __forceinline__ T msel(T x, T m) {
  if constexpr (sizeof(T) == 8) return __double2hiint(m) != 0 ? x : T(0);
  else return x * m;
}
// x / y given ry = 1 / y correctly rounded. FP64: Markstein's final correction
// (P. Markstein, IBM J. Res. Dev. 34, 1990): with q0 = x * ry the remainder
// e = x - q0 * y is exact as one fused multiply-add and q0 + e * ry rounds to the
// correctly rounded quotient, i.e. the reference's x / y, in three FP64 operations
// instead of a division. FP32: the division itself.
template <class T>
__device__ __forceinline__ T divq(T x, T y, T ry) {
  if constexpr (sizeof(T) == 8) {
    const double q0 = __dmul_rn(x, ry);
    return __fma_rn(__fma_rn(-q0, y, x), ry, q0);
  } else {
    (void)ry;
    return x / y;
  }
}

// x / y given ry = 1 / y correctly rounded: divq's correction, in both precisions and
// without a branch (three multiply-adds instead of the division's dozen instructions);
// a quotient that is not finite is that of x ry (FP64 tests it on the integer pipe), where
// divq's correction would turn an infinite one into NaN. Exact for |x| > 2^-100 (2^-960).
template <class T>
__device__ __forceinline__ T divr(T x, T y, T ry) {
  if constexpr (sizeof(T) == 8) {
    const T q = __dmul_rn(x, ry);
    const T r = __fma_rn(__fma_rn(-q, y, x), ry, q);
    const int h = __double2hiint(q);
    const bool finite = (h & 0x7ff00000) != 0x7ff00000;
    return __hiloint2double(finite ? __double2hiint(r) : h, finite ? __double2loint(r) : __double2loint(q));
  } else {
    const T q = __fmul_rn(x, ry);
    return isfinite(q) ? __fmaf_rn(__fmaf_rn(-q, y, x), ry, q) : q;
  }
}
// x / e3t_n(k): FP64 through the reciprocal profile where e3t_n is the rest-state profile
template <class T>
__device__ __forceinline__ T over_e3t_n(const Dom<T>& d, T x, T e3n, int k) {
  if constexpr (sizeof(T) == 8) {
    if (d.r1_e3t && d.e3t_n.s == 0) return divr(x, e3n, d.r1_e3t[k - 1]);
  }
  return x / e3n;
}
// z * x for z = 1 or -1, off the FP64 pipe
template <class T>
__device__ __forceinline__ T signed_by(T z, T x) {
  if constexpr (sizeof(T) == 8) return z < T(0) ? -x : x;
  else return z * x;
}

// Upstream flux 0.5 * ((u + |u|) * tl + (u - |u|) * tr) (traadv_fct.F90:126-136):
// exactly u * tl for u > 0 and u * tr for u < 0 (the doubled product scales exactly
// and the other term is an exact 0), formed as one product of the selected value.
// The product is rounded on its own (no contraction into the sum that follows), so
// every kernel that forms this flux gets the same value.
template <class T>
__device__ __forceinline__ T rmul(T a, T b) {
  if constexpr (sizeof(T) == 8) return __dmul_rn(a, b);
  else return __fmul_rn(a, b);
}
template <class T>
__device__ __forceinline__ T ups(T u, T tl, T tr) {
  return rmul(u, sgn_pos(u) ? tl : tr);
}

// FCT stage a: upstream trend into pta, monotone guess zwi, antidiffusive fluxes
// (traadv_fct.F90:119-278) with the lbc_lnk of :280 folded in (edge values 0).
// k-march: the upstream flux through the w-face between levels k and k+1 is
// computed once (the bottom flux of k is the top flux of k+1), and tb, tn of
// level k, the transport through that face and the T masks are carried to level k+1.
// H4, V4: the orders (4) of the horizontal and vertical antidiffusive fluxes; TRP: pun,
// pvn, pwn are velocities to be scaled; I: the index type within a member's tracers (int
// where they fit, half the address arithmetic). With all of that decided at run time a
// point took 690 instructions (T and S, FCT 4/4, FP32): 359 us at 500x400x56, 335 so (a
// form with its planes staged by TMA 347: the seven other fields of a level bound it).
template <class T, class I, bool H4, bool V4, bool TRP, int BPS = (sizeof(T) == 4 ? 8 : 3)>
__global__ void __launch_bounds__(128, BPS) k_fct_a(Dom<T> d, FctArgs<T> a) {
  const KIdx c = k_index(d);
  if (!c.valid) return;
  const int jpi = d.jpi, jpk = d.jpk;
  const I n2 = (I)d.n2, n3 = (I)d.n3;
  const long ij = c.ij, mb = (long)c.m * a.kjpt * d.n3 + ij, mv = (long)c.m * d.n3 + ij;
  T *zwi = a.zwi + mb, *ax = a.ax + mb, *ay = a.ay + mb, *az = a.az + mb, *ta = a.pta + mb;
  const T* tai = a.pta_in ? a.pta_in + mb : nullptr;
  auto edge = [&](I q) {  // no work: 0 (pta: its input)
    zwi[q] = T(0); ax[q] = T(0); ay[q] = T(0); az[q] = T(0);
    if (!tai) ta[q] = T(0);
    else if (tai != ta) ta[q] = tai[q];
  };
  if (!c.interior) {
    for (int k = c.k0; k <= c.k1; ++k)
      for (int n = 0; n < a.kjpt; ++n) edge((I)(k - 1) * n2 + n * n3);
    return;
  }
  const ColInfo ci = d.ci[ij];
  ColInfo ciw{}, cie{}, cis{}, cin{};
  if constexpr (H4) {
    ciw = d.ci[ij - 1]; cie = d.ci[ij + 1]; cis = d.ci[ij - jpi]; cin = d.ci[ij + jpi];
  }
  const bool e_in = c.i + 1 <= jpi - 1, n_in = c.j + 1 <= d.jpj - 1;
  const T r1_e1e2t = d.r1_e1e2t[ij];
  const T r1_6 = T(1) / T(6);
  const T su0 = TRP ? d.e2u[ij] : T(1), suw = TRP ? d.e2u[ij - 1] : T(1);
  const T sv0 = TRP ? d.e1v[ij] : T(1), svs = TRP ? d.e1v[ij - jpi] : T(1), sw = TRP ? d.e1e2t[ij] : T(1);
  const E3Col<T> e3tn(d.e3t_n, ij, c.m), e3tb(d.e3t_b, ij, c.m), e3ta(d.e3t_a, ij, c.m);
  const E3Col<T> e3u0(d.e3u_n, ij, c.m), e3uw(d.e3u_n, ij - 1, c.m), e3v0(d.e3v_n, ij, c.m), e3vs(d.e3v_n, ij - jpi, c.m);
  const T *un = a.pun.p + mv, *vn = a.pvn.p + mv, *wn = a.pwn.p + mv;
  const T *ptb = a.ptb.p + mb, *ptn = a.ptn.p + mb, *ztw = V4 ? a.ztw.p + mb : nullptr;
  const T p2dt = a.p2dt;
  constexpr int NT = 2;  // tracers per pass over the levels
  for (int n0 = 0; n0 < a.kjpt; n0 += NT) {
    const int nt = a.kjpt - n0 < NT ? a.kjpt - n0 : NT;
    // carried from level k-1: tb(k-1), tn(k-1), the bottom upstream flux of k-1
    T tbp[NT] = {}, tnp[NT] = {}, zwzb[NT] = {};
    T wt = T(0);  // transport through the top face of level k
    T tkm = c.k0 > 1 ? tmsk<T>(ci, c.k0 - 1) : T(1), tk = tmsk<T>(ci, c.k0);
    for (int k = c.k0; k <= c.k1; ++k) {
      const I q = (I)(k - 1) * n2;
      if (k == jpk) {
        for (int nn = 0; nn < nt; ++nn) edge(q + (n0 + nn) * n3);
        continue;
      }
      const bool first = k == c.k0;
      T ue = __ldg(un + q), uw = __ldg(un + q - 1), vn_ = __ldg(vn + q), vs = __ldg(vn + q - jpi);
      if (first) wt = TRP ? sw * __ldg(wn + q) : __ldg(wn + q);
      T wb = (k + 1 <= jpk - 1) ? __ldg(wn + q + n2) : T(0);
      if constexpr (TRP) {
        ue = su0 * e3u0(k) * ue;
        uw = suw * e3uw(k) * uw;
        vn_ = sv0 * e3v0(k) * vn_;
        vs = svs * e3vs(k) * vs;
        wb = sw * wb;
      }
      const T e3n = e3tn(k), e3b = e3tb(k), e3a = e3ta(k);
      const T tkp = tmsk<T>(ci, k + 1);
      const T tm = tk, wk = msel(tk, tkm), wk1 = msel(tkp, tk);
      T um0 = T(0), umw = T(0), ume = T(0), vm0 = T(0), vms = T(0), vmn = T(0);
      if constexpr (H4) {
        um0 = umsk<T>(ci, k); umw = umsk<T>(ciw, k); ume = umsk<T>(cie, k);
        vm0 = vmsk<T>(ci, k); vms = vmsk<T>(cis, k); vmn = vmsk<T>(cin, k);
      }
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) {
        if (nn >= nt) break;
        const I o = q + (n0 + nn) * n3;
        const T *tb = ptb + o, *tn = ptn + o;
        const T tb0 = __ldg(tb);
        if (first && k > 1) {  // the carried values of level k-1
          tbp[nn] = __ldg(tb - n2);
          tnp[nn] = __ldg(tn - n2);
          zwzb[nn] = ups(wt, tb0, tbp[nn]) * wk;
        }
        const T tin = tai ? tai[o] : T(0);
        const T zwx_e = ups(ue, tb0, __ldg(tb + 1)), zwx_w = ups(uw, __ldg(tb - 1), tb0);
        const T zwy_n = ups(vn_, tb0, __ldg(tb + jpi)), zwy_s = ups(vs, __ldg(tb - jpi), tb0);
        // upstream vertical fluxes at the top (k) and bottom (k+1) faces (:137-156)
        const T zwz_t = (k == 1) ? (a.linssh ? wt * tb0 : T(0)) : zwzb[nn];
        const T zwz_b = (k + 1 <= jpk - 1) ? ups(wb, __ldg(tb + n2), tb0) * wk1 : T(0);
        const T ztra = -(zwx_e - zwx_w + zwy_n - zwy_s + zwz_t - zwz_b) * r1_e1e2t;
        // horizontal antidiffusive fluxes (:180-251)
        const T tn0 = __ldg(tn), tne = __ldg(tn + 1), tnn = __ldg(tn + jpi);
        T axv, ayv;
        if constexpr (!H4) {
          axv = T(0.5) * ue * (tn0 + tne) - zwx_e;
          ayv = T(0.5) * vn_ * (tn0 + tnn) - zwy_n;
        } else {
          const T ztu_w = (tn0 - __ldg(tn - 1)) * umw;
          const T ztu_0 = (tne - tn0) * um0;
          const T zltu0 = (ztu_0 + ztu_w) * r1_6;
          T zltue = T(0);
          if (e_in) zltue = ((__ldg(tn + 2) - tne) * ume + ztu_0) * r1_6;
          const T ztv_s = (tn0 - __ldg(tn - jpi)) * vms;
          const T ztv_0 = (tnn - tn0) * vm0;
          const T zltv0 = (ztv_0 + ztv_s) * r1_6;
          T zltvn = T(0);
          if (n_in) zltvn = ((__ldg(tn + 2 * jpi) - tnn) * vmn + ztv_0) * r1_6;
          const T zC2t_u = tn0 + tne;
          const T zC2t_v = tn0 + tnn;
          axv = T(0.5) * ue * (zC2t_u + zltu0 - zltue) - zwx_e;
          ayv = T(0.5) * vn_ * (zC2t_v + zltv0 - zltvn) - zwy_n;
        }
        // vertical antidiffusive flux at the top face of level k (:253-278)
        T azv = T(0);
        if (k >= 2) {
          if constexpr (!V4) azv = (wt * T(0.5) * (tn0 + tnp[nn]) - zwz_t) * wk;
          else azv = (wt * __ldg(ztw + o) - zwz_t) * wk;
        }
        ta[o] = tin + over_e3t_n(d, ztra, e3n, k) * tm;
        zwi[o] = (e3b * tb0 + p2dt * ztra) / e3a * tm;
        ax[o] = axv;
        ay[o] = ayv;
        az[o] = azv;
        tbp[nn] = tb0;
        tnp[nn] = tn0;
        zwzb[nn] = zwz_b;
      }
      wt = wb;
      tkm = tk;
      tk = tkp;
    }
  }
}

// zbup / zbdo of nonosc (traadv_fct.F90:361-364) at one point.
// With tm = 1 the reference's pbef*tm - zbig*(1-tm) is pbef exactly, with tm = 0 it is
// -zbig (pbef, paft finite), so the masked extrema reduce to a select.
template <class T>
__device__ __forceinline__ void bupdo(T pbef, T paft, T tm, T& up, T& dn) {
  const T zbig = Big<T>::v;
  bool wet;
  if constexpr (sizeof(T) == 8) wet = __double2hiint(tm) != 0;  // tm is 0 or 1
  else wet = tm != T(0);
  up = wet ? vmax(pbef, paft) : -zbig;
  dn = wet ? vmin(pbef, paft) : zbig;
}
// FCT stage b: nonosc extrema and limiter coefficients zbetup / zbetdo
// (traadv_fct.F90:366-400), edge values 0 (lbc_lnk of :400). k-march: tb, zwi and
// their masked extrema of levels k and k+1 and az(k+1) are carried down.
template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 4) k_fct_b(Dom<T> d, FctArgs<T> a) {
  const KIdx c = k_index(d);
  if (!c.valid) return;
  const int jpi = d.jpi, jpk = d.jpk;
  const long n2 = d.n2, n3 = d.n3, ij = c.ij;
  const T zrtrn = T(1.e-15);
  auto zero = [&](int k) {
    const long q = ij + (long)(k - 1) * n2;
    for (int n = 0; n < a.kjpt; ++n) {
      const long mo = ((long)c.m * a.kjpt + n) * n3;
      a.betup[mo + q] = T(0);
      a.betdo[mo + q] = T(0);
    }
  };
  if (!c.interior) {
    for (int k = c.k0; k <= c.k1; ++k) zero(k);
    return;
  }
  const ColInfo ci = d.ci[ij], ciw = d.ci[ij - 1], cie = d.ci[ij + 1], cis = d.ci[ij - jpi], cin = d.ci[ij + jpi];
  const T e1e2t = d.e1e2t[ij];
  constexpr int NT = 2;
  for (int n0 = 0; n0 < a.kjpt; n0 += NT) {
    const int nt = a.kjpt - n0 < NT ? a.kjpt - n0 : NT;
    // carried: masked extrema (up, dn) of the column at level k-1 and k, az(k)
    T upm[NT] = {}, dnm[NT] = {}, up0[NT] = {}, dn0[NT] = {}, azk[NT] = {}, zwik[NT] = {};
    for (int k = c.k0; k <= c.k1; ++k) {
      if (k == jpk) {
        const long q = ij + (long)(k - 1) * n2;
        for (int nn = 0; nn < nt; ++nn) {
          const long mo = ((long)c.m * a.kjpt + n0 + nn) * n3;
          a.betup[mo + q] = T(0);
          a.betdo[mo + q] = T(0);
        }
        continue;
      }
      const bool first = k == c.k0;
      const long q = ij + (long)(k - 1) * n2, qp = q + n2;
      const T zbt = e1e2t * d.e3t_n(ij, k, c.m) / a.p2dt;
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) {
        if (nn >= nt) break;
        const long mo = ((long)c.m * a.kjpt + n0 + nn) * n3;
        const RO<T> tb = a.ptb + mo;
        const RO<T> zwi = a.zwi + mo;
        const RO<T> ax = a.ax + mo;
        const RO<T> ay = a.ay + mo;
        const RO<T> az = a.az + mo;
        if (first) {  // extrema of the column at levels k and k-1, az(k)
          zwik[nn] = zwi[q];
          bupdo(tb[q], zwik[nn], tmsk<T>(ci, k), up0[nn], dn0[nn]);
          if (k > 1) bupdo(tb[q - n2], zwi[q - n2], tmsk<T>(ci, k - 1), upm[nn], dnm[nn]);
          else { upm[nn] = up0[nn]; dnm[nn] = dn0[nn]; }
          azk[nn] = az[q];
        }
        T upp, dnp;  // level k+1 of the column
        bupdo(tb[qp], zwi[qp], tmsk<T>(ci, k + 1), upp, dnp);
        // the reference's order: centre, west, east, south, north, above, below
        T up = up0[nn], dn = dn0[nn], u2, d2;
        bupdo(tb[q - 1], zwi[q - 1], tmsk<T>(ciw, k), u2, d2); up = vmax(up, u2); dn = vmin(dn, d2);
        bupdo(tb[q + 1], zwi[q + 1], tmsk<T>(cie, k), u2, d2); up = vmax(up, u2); dn = vmin(dn, d2);
        bupdo(tb[q - jpi], zwi[q - jpi], tmsk<T>(cis, k), u2, d2); up = vmax(up, u2); dn = vmin(dn, d2);
        bupdo(tb[q + jpi], zwi[q + jpi], tmsk<T>(cin, k), u2, d2); up = vmax(up, u2); dn = vmin(dn, d2);
        up = vmax(up, upm[nn]); dn = vmin(dn, dnm[nn]);
        up = vmax(up, upp); dn = vmin(dn, dnp);
        const T axw = ax[q - 1], ax0 = ax[q], ays = ay[q - jpi], ay0 = ay[q], az0 = azk[nn], azb = az[qp];
        const T zpos = pos_part(axw) - neg_part(ax0) + pos_part(ays) - neg_part(ay0) + pos_part(azb) - neg_part(az0);
        const T zneg = pos_part(ax0) - neg_part(axw) + pos_part(ay0) - neg_part(ays) + pos_part(az0) - neg_part(azb);
        const T zw = zwik[nn];
        a.betup[mo + q] = (up - zw) / (zpos + zrtrn) * zbt;
        a.betdo[mo + q] = (zw - dn) / (zneg + zrtrn) * zbt;
        upm[nn] = up0[nn]; dnm[nn] = dn0[nn];
        up0[nn] = upp; dn0[nn] = dnp;
        azk[nn] = azb;
        zwik[nn] = zwi[qp];
      }
    }
  }
}

// Limiter multiplier of an antidiffusive flux f (traadv_fct.F90:407-422): c*a + (1-c)*b.
// With zc = 0.5 + SIGN(0.5, f) in {0, 1} the sum is exactly a where f >= 0 and b
// where f < 0 (products by 1 and 0 are exact), so the operands are selected first.
template <class T>
__device__ __forceinline__ T limit_mult(T f, T bdo0, T bup1, T bup0, T bdo1) {
  const bool p = sgn_pos(f);
  return vmin(T(1), vmin(p ? bdo0 : bup0, p ? bup1 : bdo1));
}
// Limited antidiffusive flux: f * ( c*a + (1-c)*b ).
template <class T>
__device__ __forceinline__ T limit(T f, T bdo0, T bup1, T bup0, T bdo1) {
  return rmul(f, limit_mult(f, bdo0, bup1, bup0, bdo1));
}

// interp_4th_cpt (traadv_fct.F90:517-616): compact 4th-order tn at w-points for the
// interior columns, levels 2..jpkm1, one tridiagonal solve per column and tracer (grid z =
// kjpt member + tracer). Rows: identity with the centred average at ikt = 2 (mikt + 1
// without ice-shelf cavities) and ikb = mbkt, diagonal 4 with off-diagonals 1 between them
// (wmask 1), identity with 0 elsewhere; so the pivots of a column's run of wet rows are
// one sequence, 4, 4 - 1/4, ..., which the block forms once. The forward values stay in
// shared memory, and four levels are loaded while the four before them are used. With
// pivots and forward values in local memory and both tracers in a thread it took 156 us
// at 500x400x56 in FP32, 66 so (27 us by traffic).
constexpr int I4_Y = 4;
template <class T>
__global__ void __launch_bounds__(32 * I4_Y) k_interp4(Dom<T> d, RO<T> ptn, T* __restrict__ ztw, int kjpt) {
  extern __shared__ __align__(16) unsigned char i4_smem[];
  __shared__ T piv[KMAX + 1], rp[KMAX + 1];  // pivots of a run of wet rows, their reciprocals
  constexpr int nt = 32 * I4_Y, B = 4;
  T* const out = reinterpret_cast<T*>(i4_smem) + threadIdx.y * 32 + threadIdx.x;  // [k * nt]
  const int jpk = d.jpk, K = jpk - 1, n2 = (int)d.n2;
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    T p = T(4);
    for (int n = 0; n <= K; ++n) {
      piv[n] = p;
      rp[n] = T(1) / p;
      p = T(4) - rp[n];
    }
  }
  __syncthreads();
  const int i = blockIdx.x * 32 + threadIdx.x + 1, j = blockIdx.y * I4_Y + threadIdx.y + 1;
  if (i < 2 || i > d.jpi - 1 || j < 2 || j > d.jpj - 1) return;
  const long ij = (long)(i - 1) + (long)(j - 1) * d.jpi, mo = (long)blockIdx.z * d.n3 + ij;
  const ColInfo ci = d.ci[ij];
  const int ikb = d.mbkt[ij];
  const int ks = max(3, ci.tlo + 1), ke = ikb < 3 ? 2 : min(min((int)ci.thi, ikb - 1), K);  // the run of wet rows
  const T* __restrict__ t = ptn.p + mo;
  auto load = [&](int k0, T (&l)[B]) {
    const T* p = t + (long)(k0 - 1) * n2;
#pragma unroll
    for (int y = 0; y < B; ++y) l[y] = __ldg(p + min(y, K - k0) * n2);
  };
  T tm = __ldg(t), prev = T(0);
  auto sweep = [&](int k0, T (&l)[B]) {
#pragma unroll
    for (int y = 0; y < B; ++y) {
      const int k = k0 + y;
      if (k > K) break;
      const bool run = k >= ks && k <= ke;
      const T sum = l[y] + tm;
      T x = run ? T(3) * sum : (k == 2 || k == ikb) ? T(0.5) * sum : T(0);
      if (run) x = x - (k == ks ? prev : rp[k - ks - 1] * prev);
      out[k * nt] = x;
      prev = x;
      tm = l[y];
    }
  };
  T la[B], lb[B];
  load(2, la);
  for (int k0 = 2; k0 <= K; k0 += 2 * B) {
    if (k0 + B <= K) load(k0 + B, lb);
    sweep(k0, la);
    if (k0 + B > K) break;
    if (k0 + 2 * B <= K) load(k0 + 2 * B, la);
    sweep(k0 + B, lb);
  }
  T nxt = T(0);
  T* __restrict__ w = ztw + mo;
#pragma unroll 4
  for (int k = K; k >= 2; --k) {
    T x = out[k * nt];
    if (k >= ks && k <= ke) {
      if (k < K) x = x - nxt;
      x = sizeof(T) == 8 ? divr(x, piv[k - ks], rp[k - ks]) : x / piv[k - ks];
    }
    nxt = x;
    w[(long)(k - 1) * n2] = x;
  }
}


// --------------------------------------------------------------------------------
// Eddy diffusivity at a u (v) point: the bound array, else aht_c * umask (vmask)
// above level jpk. W: the caller guarantees k < jpk and a wet point.
template <bool W = false, class T>
__device__ __forceinline__ T ahu(const Dom<T>& d, const LdfArgs<T>& a, const ColInfo& c, long ij, int k, int m) {
  if (a.pahu) return a.pahu[(long)m * d.n3 + ij + (long)(k - 1) * d.n2];
  if constexpr (W) return a.aht_c * T(1);
  else return k < d.jpk ? a.aht_c * umsk<T>(c, k) : T(0);
}
template <bool W = false, class T>
__device__ __forceinline__ T ahv(const Dom<T>& d, const LdfArgs<T>& a, const ColInfo& c, long ij, int k, int m) {
  if (a.pahv) return a.pahv[(long)m * d.n3 + ij + (long)(k - 1) * d.n2];
  if constexpr (W) return a.aht_c * T(1);
  else return k < d.jpk ? a.aht_c * vmsk<T>(c, k) : T(0);
}

// tra_ldf_lap (traldf_lap_blp.F90:95-145) at one interior point.
template <class T>
__global__ void k_ldf_lap(Dom<T> d, LdfArgs<T> a) {
  const PtIdx c = pt_index(d);
  if (!c.valid || !c.interior || c.k > d.jpk - 1) return;
  const int jpi = d.jpi, k = c.k;
  const long n3 = d.n3, n2 = d.n2, q = c.q;
  const ColInfo ci = d.ci[c.ij], ciw = d.ci[c.ij - 1], cis = d.ci[c.ij - jpi];
  const long ijw = c.ij - 1, ijs = c.ij - jpi;
  const T zu0 = a.zsign * ahu(d, a, ci, c.ij, k, c.m) * d.e2_e1u[c.ij] * d.e3u_n(c.ij, k, c.m);
  const T zuw = a.zsign * ahu(d, a, ciw, ijw, k, c.m) * d.e2_e1u[ijw] * d.e3u_n(ijw, k, c.m);
  const T zv0 = a.zsign * ahv(d, a, ci, c.ij, k, c.m) * d.e1_e2v[c.ij] * d.e3v_n(c.ij, k, c.m);
  const T zvs = a.zsign * ahv(d, a, cis, ijs, k, c.m) * d.e1_e2v[ijs] * d.e3v_n(ijs, k, c.m);
  const T den = d.e1e2t[c.ij] * d.e3t_n(c.ij, k, c.m);
  for (int n = 0; n < a.kjpt; ++n) {
    const long mo = ((long)c.m * a.kjpt + n) * n3;
    const long go = ((long)c.m * a.kjpt + n) * n2;
    const RO<T> tb = a.ptb + mo;
    T* ta = a.pta + mo;
    const T tb0 = tb[q];
    T ztu0 = zu0 * (tb[q + 1] - tb0);
    T ztuw = zuw * (tb0 - tb[q - 1]);
    T ztv0 = zv0 * (tb[q + jpi] - tb0);
    T ztvs = zvs * (tb0 - tb[q - jpi]);
    if (a.zps) {
      if (k == ci.mbku) ztu0 = zu0 * a.pgu[go + c.ij];
      if (k == ciw.mbku) ztuw = zuw * a.pgu[go + ijw];
      if (k == ci.mbkv) ztv0 = zv0 * a.pgv[go + c.ij];
      if (k == cis.mbkv) ztvs = zvs * a.pgv[go + ijs];
    }
    ta[q] = ta[q] + (ztu0 - ztuw + ztv0 - ztvs) / den;
  }
}

// Masked horizontal gradient zdit / zdjt of tra_ldf_iso (traldf_iso.F90:218-241).
template <bool W = false, class T>
__device__ __forceinline__ T dit(const LdfArgs<T>& a, const ColInfo& c, const RO<T>& tb, long q, int k, long g) {
  if (a.zps && k == c.mbku) return a.pgu[g];
  return (tb[q + 1] - tb[q]) * umk<W, T>(c, k);
}
template <bool W = false, class T>
__device__ __forceinline__ T djt(const LdfArgs<T>& a, const ColInfo& c, const RO<T>& tb, long q, int k, long g, int jpi) {
  if (a.zps && k == c.mbkv) return a.pgv[g];
  return (tb[q + jpi] - tb[q]) * vmk<W, T>(c, k);
}

// w-point mask weights and averaged eddy diffusivities of an interior point, level
// 2 <= k <= jpkm1 (traldf_iso.F90:150-157 and :297-304: the same expressions)
template <class T>
struct IsoW {
  T zmsku, zmskv, zahu_w, zahv_w;
};
template <bool W = false, class T>
__device__ __forceinline__ IsoW<T> iso_w(const Dom<T>& d, const LdfArgs<T>& a, long ij, int k, int m,
                                         const ColInfo& ci, const ColInfo& ciw, const ColInfo& cis) {
  const int jpi = d.jpi;
  const T wm = wmk<W, T>(ci, k);
  IsoW<T> w;
  w.zmsku = msel(rcount4(umk<W, T>(ci, k - 1), umk<W, T>(ciw, k), umk<W, T>(ciw, k - 1), umk<W, T>(ci, k)), wm);
  w.zmskv = msel(rcount4(vmk<W, T>(ci, k - 1), vmk<W, T>(cis, k), vmk<W, T>(cis, k - 1), vmk<W, T>(ci, k)), wm);
  w.zahu_w = (ahu<W>(d, a, ci, ij, k - 1, m) + ahu<W>(d, a, ciw, ij - 1, k, m) + ahu<W>(d, a, ciw, ij - 1, k - 1, m) +
              ahu<W>(d, a, ci, ij, k, m)) * w.zmsku;
  w.zahv_w = (ahv<W>(d, a, ci, ij, k - 1, m) + ahv<W>(d, a, cis, ij - jpi, k, m) + ahv<W>(d, a, cis, ij - jpi, k - 1, m) +
              ahv<W>(d, a, ci, ij, k, m)) * w.zmskv;
  return w;
}

// ah_wslp2 (traldf_iso.F90:146-164) and akz (:166-202) at one interior point, level
// 2 <= k <= jpkm1: computed on the first pass, read back on the second.
template <bool W = false, class T>
__device__ __forceinline__ void iso_coefs_at(const Dom<T>& d, const LdfArgs<T>& a, long ij, int k, int m,
                                             const ColInfo& ci, const ColInfo& ciw, const ColInfo& cis,
                                             const IsoW<T>& w, T& ahw, T& akz) {
  const long q = (long)m * d.n3 + ij + (long)(k - 1) * d.n2;
  if (a.kpass != 1) {
    ahw = a.ah_wslp2[q];
    akz = a.akz[q];
    return;
  }
  const int jpi = d.jpi;
  const T wi = a.wslpi[q], wj = a.wslpj[q];
  ahw = w.zahu_w * wi * wi + w.zahv_w * wj * wj;
  if (a.msc) {
    const T e1u0 = d.e1u[ij], e1uw = d.e1u[ij - 1], e2v0 = d.e2v[ij], e2vs = d.e2v[ij - jpi];
    T akzv = T(0.25) * ((ahu<W>(d, a, ci, ij, k, m) + ahu<W>(d, a, ci, ij, k - 1, m)) / (e1u0 * e1u0) +
                        (ahu<W>(d, a, ciw, ij - 1, k, m) + ahu<W>(d, a, ciw, ij - 1, k - 1, m)) / (e1uw * e1uw) +
                        (ahv<W>(d, a, ci, ij, k, m) + ahv<W>(d, a, ci, ij, k - 1, m)) / (e2v0 * e2v0) +
                        (ahv<W>(d, a, cis, ij - jpi, k, m) + ahv<W>(d, a, cis, ij - jpi, k - 1, m)) / (e2vs * e2vs));
    const T e3w = d.e3w_n(ij, k, m);
    if (a.blp) {
      akzv = T(16) * ahw * (akzv + ahw / (e3w * e3w));
    } else if (a.lap) {
      const T ze3w_2 = e3w * e3w;
      const T zcoef0 = a.z2dt * (akzv + ahw / ze3w_2);
      akzv = fmx(zcoef0 - T(0.5), T(0)) * ze3w_2 * a.z1_2dt;
    }
    akz = akzv;
  } else {
    akz = ahw;
  }
}

// Iso-neutral fluxes (traldf_iso.F90:146-357) of one column, k-march: on the first
// pass the coefficients ah_wslp2 / akz (levels 2..jpkm1, interior); the horizontal
// fluxes zftu / zftv of the east and north faces (i <= jpim1, j <= jpjm1,
// k <= jpkm1, :255-276); the vertical flux ztfw of the top face of each level
// (interior; 0 at levels 1 and jpk, :291-357). Each flux is computed once, by the
// column that owns its face. Carried from level k to k+1: tb of the three columns
// whose differences the fluxes take, the vertical gradients zdk1t(k) (= zdkt(k+1))
// and the four horizontal gradients zdit / zdjt that the w-face flux averages.
template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 3) k_iso_flux(Dom<T> d, LdfArgs<T> a) {
  const KIdx c = k_index(d);
  if (!c.valid) return;
  const int jpi = d.jpi, jpj = d.jpj, jpk = d.jpk;
  const long n2 = d.n2, n3 = d.n3, ij = c.ij, ijw = ij - 1, ijs = ij - jpi;
  const long m3 = (long)c.m * n3;
  if (!(c.i <= jpi - 1 && c.j <= jpj - 1)) return;  // no face owned (interior columns are inside)
  const bool icol = c.interior;
  const ColInfo ci = d.ci[ij], cie = d.ci[ij + 1], cin = d.ci[ij + jpi];
  ColInfo ciw{}, cis{};
  if (icol) {
    ciw = d.ci[ijw];
    cis = d.ci[ijs];
  }
  constexpr int NT = 2;
  for (int n0 = 0; n0 < a.kjpt; n0 += NT) {
    const int nt = a.kjpt - n0 < NT ? a.kjpt - n0 : NT;
    // carried, per tracer: tb(k) at (i,j), (i+1,j), (i,j+1); zdk1t(k-1) there; zdit at
    // (i,j) and (i-1,j) and zdjt at (i,j) and (i,j-1) of level k-1; tb(k-1) at (i,j)
    T t0c[NT] = {}, tec[NT] = {}, tnc[NT] = {}, k10[NT] = {}, k1e[NT] = {}, k1n[NT] = {};
    T di0[NT] = {}, diw[NT] = {}, dj0[NT] = {}, djs[NT] = {}, tup[NT] = {};
    for (int k = c.k0; k <= c.k1; ++k) {
      const long q = ij + (long)(k - 1) * n2;
      if (k == jpk) {  // interior: ztfw = 0 at jpk
        if (icol)
          for (int nn = 0; nn < nt; ++nn) a.ztfw[((long)c.m * a.kjpt + n0 + nn) * n3 + q] = T(0);
        continue;
      }
      const bool first = k == c.k0;
      const bool vface = icol && k >= 2;
      // tracer-independent coefficients of the faces of (i,j,k)
      T pah = ahu(d, a, ci, ij, k, c.m);
      const T zabe1 = pah * d.e2_e1u[ij] * d.e3u_n(ij, k, c.m);
      const T zmsku_h = rcount(wmsk<T>(cie, k) + wmsk<T>(ci, k + 1) + wmsk<T>(cie, k + 1) + wmsk<T>(ci, k));
      const T zcof1 = -pah * d.e2u[ij] * a.uslp[m3 + q] * zmsku_h;
      pah = ahv(d, a, ci, ij, k, c.m);
      const T zabe2 = pah * d.e1_e2v[ij] * d.e3v_n(ij, k, c.m);
      const T zmskv_h = rcount(wmsk<T>(cin, k) + wmsk<T>(ci, k + 1) + wmsk<T>(cin, k + 1) + wmsk<T>(ci, k));
      const T zcof2 = -pah * d.e1v[ij] * a.vslp[m3 + q] * zmskv_h;
      const T um = umsk<T>(ci, k), vm = vmsk<T>(ci, k);
      const T wk = wmsk<T>(ci, k), wk1 = wmsk<T>(ci, k + 1), wke = wmsk<T>(cie, k), wk1e = wmsk<T>(cie, k + 1);
      const T wkn = wmsk<T>(cin, k), wk1n = wmsk<T>(cin, k + 1);
      T zcoef3 = T(0), zcoef4 = T(0), zvert = T(0), ahw = T(0), akz = T(0);
      if (vface) {
        const IsoW<T> w = iso_w(d, a, ij, k, c.m, ci, ciw, cis);
        iso_coefs_at(d, a, ij, k, c.m, ci, ciw, cis, w, ahw, akz);
        if (a.kpass == 1) {
          a.ah_wslp2[m3 + q] = ahw;
          a.akz[m3 + q] = akz;
        }
        zcoef3 = -w.zahu_w * d.e2t[ij] * w.zmsku * a.wslpi[m3 + q];
        zcoef4 = -w.zahv_w * d.e1t[ij] * w.zmskv * a.wslpj[m3 + q];
        // the laplacian diagonal term of :359-366 without its tracer difference
        if (a.lap) zvert = d.e1e2t[ij] / d.e3w_n(ij, k, c.m) * wk * (ahw - akz);
      }
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) {
        if (nn >= nt) break;
        const int n = n0 + nn;
        const long mo = ((long)c.m * a.kjpt + n) * n3;
        const long go = ((long)c.m * a.kjpt + n) * n2;
        const RO<T> tb = a.ptb + mo;
        // masked horizontal gradients zdit / zdjt (:218-241) at column offset o, level kk
        auto zdit = [&](const ColInfo& cc, long o, int kk, T tl, T tr) -> T {
          if (a.zps && kk == cc.mbku) return a.pgu[go + ij + o];
          return (tr - tl) * umsk<T>(cc, kk);
        };
        auto zdjt = [&](const ColInfo& cc, long o, int kk, T tl, T tr) -> T {
          if (a.zps && kk == cc.mbkv) return a.pgv[go + ij + o];
          return (tr - tl) * vmsk<T>(cc, kk);
        };
        if (first) {
          t0c[nn] = tb[q]; tec[nn] = tb[q + 1]; tnc[nn] = tb[q + jpi];
          if (k > 1) {
            const long qm = q - n2;
            const T u0 = tb[qm], ue = tb[qm + 1], un = tb[qm + jpi];
            k10[nn] = (u0 - t0c[nn]) * wk;
            k1e[nn] = (ue - tec[nn]) * wke;
            k1n[nn] = (un - tnc[nn]) * wkn;
            tup[nn] = u0;
            if (icol) {
              const T uw = tb[qm - 1], us = tb[qm - jpi];
              di0[nn] = zdit(ci, 0, k - 1, u0, ue);
              diw[nn] = zdit(ciw, -1, k - 1, uw, u0);
              dj0[nn] = zdjt(ci, 0, k - 1, u0, un);
              djs[nn] = zdjt(cis, -jpi, k - 1, us, u0);
            }
          }
        }
        const T t0 = t0c[nn], te = tec[nn], tn = tnc[nn];
        const T t1 = tb[q + n2], te1 = tb[q + 1 + n2], tn1 = tb[q + jpi + n2];
        // vertical gradients (:250-254): zdk1t(k) = (tb(k)-tb(k+1))*wmask(k+1),
        // zdkt(k) = zdk1t(k-1), zdkt(1) = zdk1t(1)
        const T dk1_0 = (t0 - t1) * wk1, dk1_e = (te - te1) * wk1e, dk1_n = (tn - tn1) * wk1n;
        const T dk0_0 = k == 1 ? dk1_0 : k10[nn];
        const T dk0_e = k == 1 ? dk1_e : k1e[nn];
        const T dk0_n = k == 1 ? dk1_n : k1n[nn];
        const T zdi = zdit(ci, 0, k, t0, te);
        const T zdj = zdjt(ci, 0, k, t0, tn);
        a.zftu[mo + q] = (zabe1 * zdi + zcof1 * (dk0_e + dk1_0 + dk1_e + dk0_0)) * um;
        a.zftv[mo + q] = (zabe2 * zdj + zcof2 * (dk0_n + dk1_0 + dk1_n + dk0_0)) * vm;
        if (icol) {
          const T tw = tb[q - 1], ts = tb[q - jpi];
          const T zdiw = zdit(ciw, -1, k, tw, t0);
          const T zdjs = zdjt(cis, -jpi, k, ts, t0);
          T z = T(0);
          if (vface) {
            const T sdi = di0[nn] + zdiw + diw[nn] + zdi;
            const T sdj = dj0[nn] + zdjs + djs[nn] + zdj;
            z = zcoef3 * sdi + zcoef4 * sdj;
            if (a.lap) {
              z = z + zvert * (tup[nn] - t0);
            } else {
              const RO<T> tbb = a.ptbb + mo;
              const T e1e2t = d.e1e2t[ij];
              const T e3w = d.e3w_n(ij, k, c.m);
              if (a.kpass == 1) z = z + ahw * e1e2t * (tup[nn] - t0) / e3w * wk;
              else z = z + e1e2t / e3w * wk * (ahw * (tup[nn] - t0) + akz * (tbb[q - n2] - tbb[q]));
            }
          }
          a.ztfw[mo + q] = z;
          di0[nn] = zdi; diw[nn] = zdiw; dj0[nn] = zdj; djs[nn] = zdjs;
        }
        k10[nn] = dk1_0; k1e[nn] = dk1_e; k1n[nn] = dk1_n;
        tup[nn] = t0;
        t0c[nn] = t1; tec[nn] = te1; tnc[nn] = tn1;
      }
    }
  }
}

// Divergence of the iso-neutral fluxes of tracer n at interior point (i,j,k), added
// to tav in the reference's order: horizontal (:278-284), then vertical (:359-366).
template <class T>
__device__ __forceinline__ T iso_div(const Dom<T>& d, const LdfArgs<T>& a, const PtIdx& c, int n, T tav) {
  const long mo = ((long)c.m * a.kjpt + n) * d.n3, q = c.q;
  const T r1 = d.r1_e1e2t[c.ij], e3tn = d.e3t_n(c.ij, c.k, c.m);
  const RO<T> fu = a.zftu + mo;
  const RO<T> fv = a.zftv + mo;
  const RO<T> fw = a.ztfw + mo;
  tav = tav + over_e3t_n(d, signed_by(a.zsign, fu[q] - fu[q - 1] + fv[q] - fv[q - d.jpi]) * r1, e3tn, c.k);
  tav = tav + over_e3t_n(d, signed_by(a.zsign, fw[q] - fw[q + d.n2]) * r1, e3tn, c.k);
  return tav;
}

// tra_ldf_iso divergence step at one interior point (k <= jpkm1).
template <class T>
__global__ void k_iso_div(Dom<T> d, LdfArgs<T> a) {
  const PtIdx c = pt_index(d);
  if (!c.valid || !c.interior || c.k > d.jpk - 1) return;
  for (int n = 0; n < a.kjpt; ++n) {
    T* ta = a.pta + ((long)c.m * a.kjpt + n) * d.n3;
    ta[c.q] = iso_div(d, a, c, n, ta[c.q]);
  }
}

// FCT stage c: limit the fluxes (traadv_fct.F90:404-426) and add the divergence of
// the corrected fluxes to pta (:288-297); with_iso also adds the iso-neutral trend
// divergence of the same point from the fluxes k_iso_flux computed (the tra_ldf
// call that follows tra_adv in step.F90:248-252). k-march: the limited flux through
// the w-face between k and k+1, the coefficients of level k+1 and the iso-neutral
// vertical flux of that face are carried down.
template <class T>
__global__ void __launch_bounds__(128) k_fct_c(Dom<T> d, FctArgs<T> a) {
  const KIdx c = k_index(d);
  if (!c.valid || !c.interior) return;
  const int jpi = d.jpi, jpk = d.jpk;
  const long n2 = d.n2, n3 = d.n3, ij = c.ij;
  const T r1_e1e2t = d.r1_e1e2t[ij];
  const bool w_lim = c.i - 1 >= 2;  // the face i-1 is limited only for i-1 >= 2 (then lbc: 0)
  const bool s_lim = c.j - 1 >= 2;
  const int k1 = c.k1 < jpk - 1 ? c.k1 : jpk - 1;
  constexpr int NT = 2;
  for (int n0 = 0; n0 < a.kjpt; n0 += NT) {
    const int nt = a.kjpt - n0 < NT ? a.kjpt - n0 : NT;
    // carried: limiter coefficients of the column at level k, the limited flux
    // through the top face of level k, the iso-neutral vertical flux of that face
    T bu0[NT] = {}, bd0[NT] = {}, azt[NT] = {}, fwt[NT] = {};
    for (int k = c.k0; k <= k1; ++k) {
      const bool first = k == c.k0;
      const long q = ij + (long)(k - 1) * n2, qp = q + n2;
      const T e3n = d.e3t_n(ij, k, c.m);
#pragma unroll
      for (int nn = 0; nn < NT; ++nn) {
        if (nn >= nt) break;
        const int n = n0 + nn;
        const long mo = ((long)c.m * a.kjpt + n) * n3;
        const RO<T> ax = a.ax + mo;
        const RO<T> ay = a.ay + mo;
        const RO<T> az = a.az + mo;
        const RO<T> bu = a.betup + mo;
        const RO<T> bd = a.betdo + mo;
        T* ta = a.pta + mo;
        if (first) {
          bu0[nn] = bu[q];
          bd0[nn] = bd[q];
          // pcc(k), not limited at k = 1
          azt[nn] = k >= 2 ? limit(az[q], bd0[nn], bu[q - n2], bu0[nn], bd[q - n2]) : az[q];
          if (a.with_iso) fwt[nn] = RO<T>(a.iso.ztfw + mo)[q];
        }
        const T b_u = bu0[nn], b_d = bd0[nn];
        const T bup = bu[qp], bdp = bd[qp];
        const T axl = limit(ax[q], b_d, bu[q + 1], b_u, bd[q + 1]);
        const T axlw = w_lim ? limit(ax[q - 1], bd[q - 1], b_u, bu[q - 1], b_d) : T(0);
        const T ayl = limit(ay[q], b_d, bu[q + jpi], b_u, bd[q + jpi]);
        const T ayls = s_lim ? limit(ay[q - jpi], bd[q - jpi], b_u, bu[q - jpi], b_d) : T(0);
        // pcc(k+1): the limited flux through the bottom face
        const T azl_b = limit(az[qp], bdp, b_u, bup, b_d);
        if (a.lim) {  // the multipliers of the faces this point owns
          T* L = a.lim + ((long)c.m * a.kjpt + n) * 3 * n3;
          L[q] = limit_mult(ax[q], b_d, bu[q + 1], b_u, bd[q + 1]);
          L[n3 + q] = limit_mult(ay[q], b_d, bu[q + jpi], b_u, bd[q + jpi]);
          L[2 * n3 + qp] = limit_mult(az[qp], bdp, b_u, bup, b_d);
        }
        T tav = ta[q] - over_e3t_n(d, (axl - axlw + ayl - ayls + azt[nn] - azl_b) * r1_e1e2t, e3n, k);
        if (a.with_iso) {
          // iso-neutral divergence: horizontal (traldf_iso.F90:278-284), then
          // vertical (:359-366)
          const RO<T> fu = a.iso.zftu + mo;
          const RO<T> fv = a.iso.zftv + mo;
          const RO<T> fw = a.iso.ztfw + mo;
          const T fwb = fw[qp];
          tav = tav + over_e3t_n(d, signed_by(a.iso.zsign, fu[q] - fu[q - 1] + fv[q] - fv[q - jpi]) * r1_e1e2t, e3n, k);
          tav = tav + over_e3t_n(d, signed_by(a.iso.zsign, fwt[nn] - fwb) * r1_e1e2t, e3n, k);
          fwt[nn] = fwb;
        }
        ta[q] = tav;
        bu0[nn] = bup;
        bd0[nn] = bdp;
        azt[nn] = azl_b;
      }
    }
  }
}

// Edge points of the second MSC loop (traldf_iso.F90:179-197), which runs over
// ji = 1..jpim1, jj = 1..jpjm1 and therefore also updates row 1 and column 1.
template <class T>
__global__ void k_iso_msc_edges(Dom<T> d, LdfArgs<T> a) {
  ColIdx<T> c = col_index(d);
  if (!c.valid || c.interior) return;
  if (c.i > d.jpi - 1 || c.j > d.jpj - 1) return;
  for (int k = 2; k <= d.jpk - 1; ++k) {
    const long q = (long)c.m * d.n3 + c.ij + (long)(k - 1) * d.n2;
    const T e3w = d.e3w_n(c.ij, k, c.m);
    const T ahw = a.ah_wslp2[q];
    T akzv = a.akz[q];
    if (a.blp) {
      akzv = T(16) * ahw * (akzv + ahw / (e3w * e3w));
    } else if (a.lap) {
      const T ze3w_2 = e3w * e3w;
      const T zcoef0 = a.z2dt * (akzv + ahw / ze3w_2);
      akzv = fmx(zcoef0 - T(0.5), T(0)) * ze3w_2 * a.z1_2dt;
    }
    a.akz[q] = akzv;
  }
}

// akz = ah_wslp2 on the whole array (traldf_iso.F90:200-201) for the points the
// interior sweep does not write: levels 1 and jpk of interior columns, every level
// of the edge columns. Blocks z = 2 member + 0: the two levels, one (i,j) a thread; + 1: the
// edge columns, one point a thread (a thread that copied a whole edge column waited for
// jpk memory round trips in a row: 27 us at 500x400x56).
template <class T>
__global__ void __launch_bounds__(256) k_iso_akz_copy_edges(Dom<T> d, LdfArgs<T> a) {
  const long t = (long)blockIdx.x * 256 + threadIdx.x, step = (long)gridDim.x * 256;
  const long base = (long)(blockIdx.z >> 1) * d.n3;
  if (blockIdx.z & 1) {
    const int jpi = d.jpi, per = 2 * jpi + 2 * d.jpj;
    for (long e = t; e < (long)per * d.jpk; e += step) {
      const int k = (int)(e / per), x = (int)(e - (long)k * per);
      const int i = x < 2 * jpi ? x % jpi : (x - 2 * jpi) & 1 ? jpi - 1 : 0;
      const int j = x < 2 * jpi ? (x < jpi ? 0 : d.jpj - 1) : (x - 2 * jpi) >> 1;
      const long q = base + (long)k * d.n2 + (long)j * jpi + i;
      a.akz[q] = a.ah_wslp2[q];
    }
  } else {
    const long bot = base + (long)(d.jpk - 1) * d.n2;
    for (long p = t; p < d.n2; p += step) {
      const T x = a.ah_wslp2[base + p], y = a.ah_wslp2[bot + p];
      a.akz[base + p] = x;
      a.akz[bot + p] = y;
    }
  }
}

// --------------------------------------------------------------------------------
// tra_zdf_imp (trazdf.F90:143-264) for the interior columns; pta becomes the after
// tracer. With clamp_sal the salinity WHERE( tsa < 0 ) tsa = 0.1 of trazdf.F90:83 is
// applied on the values this kernel writes.
template <class T>
struct ZdfArgs {
  T p2dt;
  RO<T> ptb;
  T* pta;
  int kjpt;
  RO<T> avt, avs, add;       // add: ah_wslp2 (standard iso), akz (msc) or NULL
  int ddm, is_trc, clamp_sal;
};

// tra_zdf_imp in FP64, one column a thread with the pivots in local memory: the operations
// of trazdf.F90:218-264 in order, with every quotient correctly rounded as the reference's
// division gives it, but formed from a reciprocal (divq): one division per level
// (1 / zwt(k)) where the reference divides six times (zwi, zws, the two pivot quotients of
// the 1st recurrence and the 3rd recurrence of each of T and S); zwi(k+1) is zws(k), the
// same expression, formed once; the divisions by e3w use the rest-state reciprocal profile
// where e3w is it.
template <class T>
__global__ void k_zdf_imp(Dom<T> d, ZdfArgs<T> a) {
  static_assert(sizeof(T) == 8, "FP32: k_zdf_imp32");
  ColIdx<T> c = col_index(d);
  if (!c.valid || !c.interior) return;
  const int jpk = d.jpk;
  const long n2 = d.n2, n3 = d.n3;
  const ColInfo ci = d.ci[c.ij];
  const long m3 = (long)c.m * n3;
  // rat(k) = zwi(k) / zwt(k-1): the tracer-independent factor of the 2nd recurrence
  T rat[KMAX], zws[KMAX], zwt[KMAX], aux[KMAX];  // aux = 1 / zwt
  for (int n = 0; n < a.kjpt; ++n) {
    const bool build = (!a.is_trc && (n == 0 || (n == 1 && a.ddm))) || (a.is_trc && n == 0);
    if (build) {
      const RO<T> coef = (!a.is_trc && n == 0) ? a.avt : a.avs;
      // zwt(k) = avt(k) (+ iso-neutral coefficient), zwt(1) = 0 (:153-176)
      auto wt = [&](int k) -> T {
        if (k == 1) return T(0);
        const long q = m3 + c.ij + (long)(k - 1) * n2;
        T v = coef[q];
        if (a.add && k <= jpk - 1) v = v + a.add[q];
        return v;
      };
      // 1st recurrence as written in the reference (trazdf.F90:218-234)
      const bool r3w = d.r1_e3w && d.e3w_n.s == 0;  // e3w is the rest-state profile
      auto over_e3w = [&](T x, int k) {
        const T e = d.e3w_n(c.ij, k, c.m);
        return r3w ? divq(x, e, d.r1_e3w[k - 1]) : x / e;
      };
      T zwi = over_e3w(-a.p2dt * wt(1), 1);
      for (int k = 1; k <= jpk - 1; ++k) {
        zws[k] = over_e3w(-a.p2dt * wt(k + 1), k + 1);
        const T zwd = d.e3t_a(c.ij, k, c.m) - zwi - zws[k];
        if (k == 1) {
          zwt[k] = zwd;
        } else {
          rat[k] = divq(zwi, zwt[k - 1], aux[k - 1]);
          zwt[k] = zwd - divq(zwi * zws[k - 1], zwt[k - 1], aux[k - 1]);
        }
        aux[k] = T(1) / zwt[k];
        zwi = zws[k];
      }
    }
    const long mo = ((long)c.m * a.kjpt + n) * n3;
    const RO<T> tb = a.ptb + mo;
    T* ta = a.pta + mo;
    const bool clamp = a.clamp_sal && !a.is_trc && n == 1;
    // 2nd recurrence (:238-250), the forward values kept in pta as in the reference
    T prev = T(0);
    for (int k = 1; k <= jpk - 1; ++k) {
      const long q = c.ij + (long)(k - 1) * n2;
      const T zrhs = d.e3t_b(c.ij, k, c.m) * tb[q] + a.p2dt * d.e3t_n(c.ij, k, c.m) * ta[q];
      prev = (k == 1) ? zrhs : zrhs - rat[k] * prev;
      ta[q] = prev;
    }
    // 3rd recurrence (:252-264)
    T nxt;
    {
      const int k = jpk - 1;
      const long q = c.ij + (long)(k - 1) * n2;
      nxt = divq(ta[q], zwt[k], aux[k]) * tmsk<T>(ci, k);
      ta[q] = (clamp && nxt < T(0)) ? T(0.1) : nxt;
    }
    for (int k = jpk - 2; k >= 1; --k) {
      const long q = c.ij + (long)(k - 1) * n2;
      nxt = divq(ta[q] - zws[k] * nxt, zwt[k], aux[k]) * tmsk<T>(ci, k);
      ta[q] = (clamp && nxt < T(0)) ? T(0.1) : nxt;
    }
  }
}

// Asynchronous 4-byte copy global -> shared (the thread waits for its own copies).
__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// FP32, jpk = NK known at compile time: the elimination of k_zdf_imp with two
// arrays, zw(k) = zwi(k) (zws(k) is zwi(k+1): both are -p2dt zwt(k+1) / e3w(k+1))
// and the reciprocal pivots 1 / zwt(k), and everything per column in shared memory: each thread copies the levels of its own column
// (diffusivities, then ta and tb of each tracer) with asynchronous copies, all in
// flight together and without registers, then solves from shared memory (pivots zw
// and 1/zwt there too; the forward values overwrite ta). No block synchronisation:
// a thread reads only what it wrote or copied. Dynamic shared memory:
// 4 * NK * (threads per block) floats.
template <int NK>
__global__ void __launch_bounds__(128, 3) k_zdf_imp_async(Dom<float> d, ZdfArgs<float> a) {
  extern __shared__ float zsm[];
  const int nt = blockDim.x * blockDim.y, t = threadIdx.y * blockDim.x + threadIdx.x;
  float* sx = zsm + t;                // sx[(k-1) * nt]: ta, then the forward values
  float* sb = zsm + NK * nt + t;      // sb[(k-1) * nt]: tb (first: the added coefficient)
  float* zw = zsm + 2 * NK * nt + t;  // zw[(k-1) * nt] = zwi(k), k = 1..NK
  float* rz = zsm + 3 * NK * nt + t;  // rz[(k-1) * nt] = 1 / zwt(k), k = 1..NK-1
  ColIdx<float> c = col_index(d);
  if (!c.valid || !c.interior) return;
  constexpr int K1 = NK - 1;
  const long n2 = d.n2, n3 = d.n3;
  const ColInfo ci = d.ci[c.ij];
  const long m3 = (long)c.m * n3;
  const float p2dt = a.p2dt;
  bool built = false, built_avt = false;
  for (int n = 0; n < a.kjpt; ++n) {
    // zwt = avt (T; S without double diffusion) or avs (S with it, passive tracers)
    const bool use_avt = !a.is_trc && (n == 0 || !a.ddm);
    if (!built || use_avt != built_avt) {
      const float* coef = (use_avt ? a.avt : a.avs).p + m3 + c.ij;
      const float* add = a.add ? a.add.p + m3 + c.ij : nullptr;
      for (int k = 2; k <= NK; ++k) {
        cp_async4(sx + (k - 1) * nt, coef + (long)(k - 1) * n2);
        if (add && k <= NK - 1) cp_async4(sb + (k - 1) * nt, add + (long)(k - 1) * n2);
      }
      cp_async_wait_all();
      zw[0] = -p2dt * 0.0f / d.e3w_n(c.ij, 1, c.m);
#pragma unroll 4
      for (int k = 2; k <= NK; ++k) {
        float wt = sx[(k - 1) * nt];
        if (add && k <= NK - 1) wt = wt + sb[(k - 1) * nt];
        zw[(k - 1) * nt] = -p2dt * wt / d.e3w_n(c.ij, k, c.m);
      }
      float g = 0.0f, rprev = 0.0f;
#pragma unroll 4
      for (int k = 1; k <= K1; ++k) {
        const float e3a = d.e3t_a(c.ij, k, c.m);
        const float zk = zw[(k - 1) * nt];
        g = (k == 1) ? e3a - zk : e3a - zk * (g * rprev);
        rprev = 1.0f / (g - zw[k * nt]);
        rz[(k - 1) * nt] = rprev;
      }
      built = true;
      built_avt = use_avt;
    }
    const long mo = ((long)c.m * a.kjpt + n) * n3 + c.ij;
    const float* tb = a.ptb.p + mo;
    float* ta = a.pta + mo;
    const bool clamp = a.clamp_sal && !a.is_trc && n == 1;
    for (int k = 1; k <= K1; ++k) {
      cp_async4(sx + (k - 1) * nt, ta + (long)(k - 1) * n2);
      cp_async4(sb + (k - 1) * nt, tb + (long)(k - 1) * n2);
    }
    cp_async_wait_all();
    // Increment form: the system is solved for d = x - tb, M d = rhs - M tb, whose
    // right-hand side holds only the trend and differences of tb, so the O(1)
    // tracer values are rounded once, in x = tb + d (the reference's form rounds
    // the full values in both recurrences: ~10 ulps of salinity per step).
    float prev = 0.0f, tbm = 0.0f;
#pragma unroll 4
    for (int k = 1; k <= K1; ++k) {
      const float tbk = sb[(k - 1) * nt];
      float r = p2dt * d.e3t_n(c.ij, k, c.m) * sx[(k - 1) * nt] +
                (d.e3t_b(c.ij, k, c.m) - d.e3t_a(c.ij, k, c.m)) * tbk;
      if (k > 1) r = r - zw[(k - 1) * nt] * (tbm - tbk);    // zwi(k) (tb(k-1) - tb(k))
      if (k < K1) r = r - zw[k * nt] * (sb[k * nt] - tbk);  // zws(k) (tb(k+1) - tb(k))
      else r = r + zw[k * nt] * tbk;                        // last row: no x(k+1)
      prev = (k == 1) ? r : r - zw[(k - 1) * nt] * rz[(k - 2) * nt] * prev;
      sx[(k - 1) * nt] = prev;
      tbm = tbk;
    }
    float dnx = 0.0f;  // x(k+1) - tb(k+1) of the stored (masked) x(k+1)
#pragma unroll 4
    for (int k = K1; k >= 1; --k) {
      const float yk = sx[(k - 1) * nt], tbk = sb[(k - 1) * nt];
      const float dk = (k == K1 ? yk : yk - zw[k * nt] * dnx) * rz[(k - 1) * nt];
      const float x = (tbk + dk) * tmsk<float>(ci, k);
      dnx = x - tbk;
      ta[(long)(k - 1) * n2] = (clamp && x < 0.0f) ? 0.1f : x;
    }
  }
}

// tra_zdf_imp in FP32: a block owns 32 columns of a row and ZW warps share their levels.
// Everything a level does by itself -- the loads, the off-diagonal zw(k) = zwi(k) (zws(k)
// is zwi(k+1): both are -p2dt zwt(k+1) / e3w(k+1)), the right-hand side -- runs on all
// warps; only the recurrences are serial, in shared memory: the pivots by one warp, each
// tracer's elimination and back substitution by a warp of its own. A column is 6 to 8
// planes deep in every field, so on a grid beyond L2 each access opens another DRAM row:
// one level in flight a thread beats eight (189 against 274 us at 500x400x56), where one
// thread a column with the pivots in local memory took 429 us (80 us by traffic).
//
// The pivots are formed without cancellation: with g(k) = zwt(k) + zws(k),
// zwt(k) = zwd(k) - zwi(k) zws(k-1)/zwt(k-1) is g(k) - zws(k) where
// g(k) = e3t_a(k) - zwi(k) g(k-1)/zwt(k-1): a sum of non-negative terms (zwi, zws <= 0),
// whereas zwd - zwi zws/zwt cancels to O(e3t) from O(p2dt avt/e3w) when the vertical
// diffusivity is large. The system is solved in increment form, for d = x - tb,
// M d = rhs - M tb, whose right-hand side holds only the trend and differences of tb, so
// the O(1) tracer values are rounded once, in x = tb + d (the reference's form rounds
// the full values in both recurrences: ~10 ulps of salinity per step).
constexpr int ZW = 6;
inline int zdf32_smem(int jpk) { return 6 * (jpk + 1) * 32 * (int)sizeof(float); }
template <int W>
__global__ void __launch_bounds__(32 * W) k_zdf_imp32(Dom<float> d, ZdfArgs<float> a) {
  extern __shared__ float zsm[];
  constexpr int NC = 32;
  const int lane = threadIdx.x, w = threadIdx.y, jpk = d.jpk, K = jpk - 1, A = (jpk + 1) * NC;
  float* zw = zsm + lane;  // [k * NC]: zwi(k), k = 1..jpk
  float* rz = zw + A;      // e3t_a(k), then 1 / zwt(k), k = 1..K
  float* sy = rz + A;      // two tracers: ta, then the right-hand side, then the forward values
  float* sb = sy + 2 * A;  // two tracers: tb
  const int nx = (d.jpi + NC - 1) / NC, j = (int)(blockIdx.x / nx) + 2, i0 = (int)(blockIdx.x % nx) * NC + lane + 1;
  const int i = min(i0, d.jpi), m = blockIdx.y;
  const bool ok = i0 >= 2 && i0 <= d.jpi - 1;
  const long n2 = d.n2, n3 = d.n3, ij = (long)(i - 1) + (long)(j - 1) * d.jpi, c3 = (long)m * n3 + ij;
  const float p2dt = a.p2dt;
  bool built = false, built_avt = false;
  for (int n0 = 0; n0 < a.kjpt;) {
    // zwt = avt (T; S without double diffusion) or avs (S with it, passive tracers); two
    // tracers of one matrix go together
    auto from_avt = [&](int n) { return !a.is_trc && (n == 0 || !a.ddm); };
    const bool use_avt = from_avt(n0);
    const int nn = n0 + 1 < a.kjpt && from_avt(n0 + 1) == use_avt ? 2 : 1;
    const bool build = !built || use_avt != built_avt;
    const long mo = ((long)m * a.kjpt + n0) * n3 + ij;
    const float *tb = a.ptb.p + mo, *coef = (use_avt ? a.avt : a.avs).p + c3, *add = a.add ? a.add.p + c3 : coef;
    float* ta = a.pta + mo;
    for (int k = w + 1; k <= jpk; k += W) {  // one level in flight a thread
      const long o = (long)(k - 1) * n2;
      float t[2], b[2];
      for (int n = 0; n < 2; ++n) {
        t[n] = n < nn ? ta[o + n * n3] : 0.0f;
        b[n] = n < nn ? __ldg(tb + o + n * n3) : 0.0f;
      }
      const float v = __ldg(coef + o), x = __ldg(add + o);
      const float ew = d.e3w_n(ij, k, m), ea = d.e3t_a(ij, k, m), en = d.e3t_n(ij, k, m), eb = d.e3t_b(ij, k, m);
      if (build) {
        const float wt = k == 1 ? 0.0f : a.add && k <= K ? v + x : v;
        zw[k * NC] = -p2dt * wt / ew;
        rz[k * NC] = ea;
      }
      for (int n = 0; n < nn; ++n) {
        sb[n * A + k * NC] = b[n];
        sy[n * A + k * NC] = p2dt * en * t[n] + (eb - ea) * b[n];
      }
    }
    __syncthreads();
    constexpr int C = 4;  // levels whose operands a serial warp reads together
    if (w > 0) {          // right-hand sides
      for (int k = w; k <= K; k += W - 1) {
        const float zi = zw[k * NC], zs = zw[(k + 1) * NC];
        for (int n = 0; n < nn; ++n) {
          const float* b = sb + n * A + k * NC;
          const float tbk = b[0];
          float r = sy[n * A + k * NC];
          if (k > 1) r = r - zi * (b[-NC] - tbk);  // zwi(k) (tb(k-1) - tb(k))
          if (k < K) r = r - zs * (b[NC] - tbk);   // zws(k) (tb(k+1) - tb(k))
          else r = r + zs * tbk;                   // last row: no x(k+1)
          sy[n * A + k * NC] = r;
        }
      }
    } else if (build) {  // pivots
      float g = 0.0f, rprev = 0.0f, zk = zw[NC];
      for (int k0 = 1; k0 <= K; k0 += C) {
        float e[C], z[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
          const int k = min(k0 + u, K);
          e[u] = rz[k * NC];
          z[u] = zw[(k + 1) * NC];
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
          if (k0 + u > K) break;
          g = e[u] - (k0 + u == 1 ? zk : zk * (g * rprev));
          rprev = 1.0f / (g - z[u]);
          rz[(k0 + u) * NC] = rprev;
          zk = z[u];
        }
      }
    }
    __syncthreads();
    if (w < nn) {
      float *y = sy + w * A, *b = sb + w * A, *to = ta + w * n3;
      float prev = 0.0f, rp = 0.0f;
      for (int k0 = 1; k0 <= K; k0 += C) {
        float r[C], f[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
          const int k = min(k0 + u, K);
          r[u] = y[k * NC];
          f[u] = zw[k * NC] * rp;
          rp = rz[k * NC];
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
          if (k0 + u > K) break;
          prev = k0 + u == 1 ? r[u] : r[u] - f[u] * prev;
          y[(k0 + u) * NC] = prev;
        }
      }
      const ColInfo ci = d.ci[ij];
      const bool clamp = a.clamp_sal && !a.is_trc && n0 + w == 1;
      float dnx = 0.0f;  // x(k+1) - tb(k+1) of the stored (masked) x(k+1)
      for (int k0 = K; k0 >= 1; k0 -= C) {
        float r[C], q[C], z[C], h[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
          const int k = max(k0 - u, 1);
          r[u] = y[k * NC];
          q[u] = rz[k * NC];
          z[u] = k == K ? 0.0f : zw[(k + 1) * NC];
          h[u] = b[k * NC];
        }
#pragma unroll
        for (int u = 0; u < C; ++u) {
          const int k = k0 - u;
          if (k < 1) break;
          const float x = (h[u] + (r[u] - z[u] * dnx) * q[u]) * tmsk<float>(ci, k);
          dnx = x - h[u];
          if (ok) to[(long)(k - 1) * n2] = (clamp && x < 0.0f) ? 0.1f : x;
        }
      }
    }
    built = true;
    built_avt = use_avt;
    n0 += nn;
    if (n0 < a.kjpt) __syncthreads();
  }
}

// WHERE( x < 0 ) x = 0.1 (trazdf.F90:83) on n values.
template <class T>
__global__ void k_clamp_neg(T* x, long n) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long s = (long)gridDim.x * blockDim.x;
  for (; i < n; i += s)
    if (x[i] < T(0)) x[i] = T(0.1);
}

}  // namespace nemo
