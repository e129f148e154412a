// inst_impl.cuh -- definitions of the launchers declared in launch.h; included by
// inst_fp64.cu and inst_fp32.cu, each of which instantiates one precision.
#pragma once
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>

#include "launch.h"
#include "k_hot.cuh"
#include "k_tma.cuh"

namespace nemo {

constexpr int BX = 32, BY = 4;

// one thread per water column (recurrences along k); ty: block height
template <class T>
static dim3 col_grid(const Dom<T>& d, int ty = BY) {
  return dim3((d.jpi + BX - 1) / BX, (d.jpj + ty - 1) / ty, d.nmem);
}

// one thread per kch-level chunk of a column: z = member * nchunk + chunk
template <class T>
static dim3 kc_grid(const Dom<T>& d, int ty = BY) {
  return dim3((d.jpi + BX - 1) / BX, (d.jpj + ty - 1) / ty, d.nmem * ((d.jpk + d.kch - 1) / d.kch));
}

// the rounds of blocks that such a grid takes with bps of them an SM (a last chunk of few
// levels is left out: its blocks are short)
template <class T>
static long kc_rounds(const Dom<T>& d, int bps) {
  const long tiles = (long)((d.jpi + BX - 1) / BX) * ((d.jpj + BY - 1) / BY) * d.nmem;
  const long blocks = tiles * (d.jpk / d.kch + (d.jpk % d.kch > d.kch / 2 ? 1 : 0));
  return (blocks + bps * SMS - 1) / (bps * SMS);
}

// one thread per (i,j,k) point: z = member * jpk + (k - 1)
template <class T>
static dim3 pt_grid(const Dom<T>& d) {
  return dim3((d.jpi + BX - 1) / BX, (d.jpj + BY - 1) / BY, d.nmem * d.jpk);
}

template <class T>
cudaError_t launch_adv_trp(const Dom<T>& d, const T* un, const T* vn, const T* wn, T* zun, T* zvn, T* zwn,
                           cudaStream_t s) {
  k_adv_trp<T><<<pt_grid(d), dim3(BX, BY), 0, s>>>(d, un, vn, wn, zun, zvn, zwn);
  ktick(NEMO_K_ADV_TRP, s);
  return cudaGetLastError();
}

// cuTensorMapEncodeTiled from the driver, through the runtime (no libcuda link)
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)p;
  }();
  return fn;
}

// Tensor map of nf 3-D fields of floats stored one after the other per member, as a
// 3-D tensor (jpi, jpj, jpk * nf * nmem), with a box of bx x by points of one level.
// False (no TMA) when the rows are not a multiple of 16 bytes (jpi % 4 != 0) or the
// base is not 16-byte aligned.
template <class T>
static bool field_tensor_map(const Dom<T>& d, const T* base, int nf, unsigned bx, unsigned by, CUtensorMap* map) {
  const auto fn = tensor_map_encoder();
  if (!fn || sizeof(T) != 4 || d.jpi % 4 != 0 || ((uintptr_t)base & 15) != 0) return false;
  cuuint64_t dims[3] = {(cuuint64_t)d.jpi, (cuuint64_t)d.jpj, (cuuint64_t)d.jpk * nf * d.nmem};
  cuuint64_t strides[2] = {(cuuint64_t)d.jpi * sizeof(T), (cuuint64_t)d.n2 * sizeof(T)};
  cuuint32_t box[3] = {bx, by, 1}, es[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)base, dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the tensor maps of stage b's planes (two tracers each); false: no TMA
template <class T>
static bool fct_b_maps(const Dom<T>& d, const FctArgs<T>& a, PlaneMaps<FB_NF>& mb) {
  const T* fb[5] = {a.ptb.p, a.zwi, a.ax, a.ay, a.az};
  for (int f = 0; f < 5; ++f) {
    if (!field_tensor_map(d, fb[f], 2, TM_W, TM_H, &mb.m[2 * f])) return false;
    mb.m[2 * f + 1] = mb.m[2 * f];
  }
  return true;
}
// The instance of the general stage a for a call's orders and transports. FP32: eight blocks
// an SM spill, and 4th-order horizontal with 2nd-order vertical fluxes the most (100 bytes);
// there the fewest of six, seven and eight blocks with the same rounds (us a call with 3-D e3:
// 200x151x31 100, 103, 111; 302x202x31 187, 159, 169; 480x320x31 352, 347, 330).
template <class T, class I>
static auto fct_a_of(const Dom<T>& d, const FctArgs<T>& a) {
  const bool h = a.kn_fct_h == 4, v = a.kn_fct_v == 4;
  if constexpr (sizeof(T) == 4 && sizeof(I) == 4) {
    if (h && !v) {
      const long r = kc_rounds(d, 8);
      if (kc_rounds(d, 6) == r) return a.trp ? k_fct_a<T, I, true, false, true, 6> : k_fct_a<T, I, true, false, false, 6>;
      if (kc_rounds(d, 7) == r) return a.trp ? k_fct_a<T, I, true, false, true, 7> : k_fct_a<T, I, true, false, false, 7>;
    }
  }
  if (a.trp)
    return h ? (v ? k_fct_a<T, I, true, true, true> : k_fct_a<T, I, true, false, true>)
             : (v ? k_fct_a<T, I, false, true, true> : k_fct_a<T, I, false, false, true>);
  return h ? (v ? k_fct_a<T, I, true, true, false> : k_fct_a<T, I, true, false, false>)
           : (v ? k_fct_a<T, I, false, true, false> : k_fct_a<T, I, false, false, false>);
}
template <class T>
cudaError_t launch_fct(const Dom<T>& d, const FctArgs<T>& a, cudaStream_t s) {
  if (hot_fct_ok(d, a) && !a.lim) {  // the limiter is recorded by k_fct_c only
    if constexpr (sizeof(T) == 4) {
      if (a.tma && a.err && a.kjpt == 2) {  // planes staged by TMA
        if (a.fused && a.trp && !a.pta_in) {  // the three stages in one kernel
          PlaneMaps<FF_NIN> maps;
          const bool ok = field_tensor_map(d, a.pun.p, 1, FF_BW, FF_BH, &maps.m[0]) &&
                          field_tensor_map(d, a.pvn.p, 1, FF_BW, FF_BH, &maps.m[1]) &&
                          field_tensor_map(d, a.pwn.p, 1, FF_BW, FF_BH, &maps.m[2]) &&
                          field_tensor_map(d, a.ptb.p, a.kjpt, FF_BW, FF_BH, &maps.m[3]) &&
                          field_tensor_map(d, a.ptn.p, a.kjpt, FF_BW, FF_BH, &maps.m[4]);
          if (ok) {
            if (cudaError_t e = smem_opt_in(k_fct_fused_tma<T>, FF_SMEM)) return e;
            const dim3 grid((d.jpi + TM_X - 1) / TM_X, (d.jpj + TM_Y - 1) / TM_Y, d.nmem);
            k_fct_fused_tma<T><<<grid, dim3(TM_X, TM_Y), FF_SMEM, s>>>(d, a, maps, a.err, a.polls);
            ktick(NEMO_K_FCT_FUSED, s);
            return cudaGetLastError();
          }
        } else {  // stages a and b with TMA-staged planes, then stage c
          PlaneMaps<FA_NF> ma;
          PlaneMaps<FB_NF> mb;
          bool ok = field_tensor_map(d, a.pun.p, 1, TM_W, TM_H, &ma.m[0]) &&
                    field_tensor_map(d, a.pvn.p, 1, TM_W, TM_H, &ma.m[1]) &&
                    field_tensor_map(d, a.pwn.p, 1, TM_W, TM_H, &ma.m[2]) &&
                    field_tensor_map(d, a.ptb.p, 2, TM_W, TM_H, &ma.m[3]) &&
                    field_tensor_map(d, a.ptn.p, 2, TM_W, TM_H, &ma.m[5]);
          ma.m[4] = ma.m[3];  // tb, tn: one map each, read at the two tracers' levels
          ma.m[6] = ma.m[5];
          ok = ok && fct_b_maps(d, a, mb);
          if (ok) {
            const auto stage_a = a.trp && !a.pta_in ? k_fct_a_tma<T, true> : k_fct_a_tma<T, false>;
            if (cudaError_t e = smem_opt_in(stage_a, FA_SMEM)) return e;
            if (cudaError_t e = smem_opt_in(k_fct_b_tma<T>, FB_SMEM)) return e;
            const dim3 grid((d.jpi + TM_X - 1) / TM_X, (d.jpj + TM_Y - 1) / TM_Y, d.nmem * ((d.jpk + d.kch - 1) / d.kch));
            stage_a<<<grid, dim3(TM_X, TM_Y), FA_SMEM, s>>>(d, a, ma, a.err, a.polls);
            ktick(NEMO_K_FCT_A_TMA, s);
            k_fct_b_tma<T><<<grid, dim3(TM_X, TM_Y), FB_SMEM, s>>>(d, a, mb, a.err, a.polls);
            ktick(NEMO_K_FCT_B_TMA, s);
            const int tc = kty(NEMO_K_FCT_C);
            k_fct_c_hot<T, false><<<kc_grid(d, tc), dim3(BX, tc), 0, s>>>(d, a);
            ktick(NEMO_K_FCT_C, s);
            return cudaGetLastError();
          }
        }
      }
    }
    const int ta = kty(NEMO_K_FCT_A);
    auto kern = !a.trp ? k_fct_a_hot<T, false, true> : a.pta_in ? k_fct_a_hot<T, true, true> : k_fct_a_hot<T, true, false>;
    if constexpr (sizeof(T) == 4) {
      if (!a.trp && kc_rounds(d, 8) < kc_rounds(d, 6)) kern = k_fct_a_hot<T, false, true, 8>;
    }
    kern<<<kc_grid(d, ta), dim3(BX, ta), 0, s>>>(d, a);
    ktick(NEMO_K_FCT_A, s);
  } else {
    if (a.kn_fct_v == 4) {
      const int level = 32 * I4_Y * (int)sizeof(T), smem = level * (d.jpk + 1);
      if (cudaError_t e = smem_opt_in(k_interp4<T>, level * (KMAX + 1))) return e;
      k_interp4<T><<<dim3((d.jpi + 31) / 32, (d.jpj + I4_Y - 1) / I4_Y, d.nmem * a.kjpt), dim3(32, I4_Y), smem, s>>>(
          d, a.ptn, const_cast<T*>(a.ztw.p), a.kjpt);
      ktick(NEMO_K_INTERP4, s);
    }
    const bool small = (long)a.kjpt * d.n3 < (1L << 31);
    const auto kern = small ? fct_a_of<T, int>(d, a) : fct_a_of<T, long>(d, a);
    kern<<<kc_grid(d), dim3(BX, BY), 0, s>>>(d, a);
    ktick(NEMO_K_FCT_A, s);
  }
  bool b_done = false;
  if constexpr (sizeof(T) == 4) {  // stage b takes any e3t_n (its planes staged by TMA: any orders of stage a)
    // ... unless the plain kernel's grid is one round of blocks and this one's more: tra_adv_fct
    // 4/2 with 3-D e3 at 320x220x31 181 against 192 us; 352x260x31, two rounds of both, 245 and 229
    PlaneMaps<FB_NF> mb;
    const long tiles = (long)((d.jpi + TM_X - 1) / TM_X) * ((d.jpj + TM_Y - 1) / TM_Y) * d.nmem * ((d.jpk + d.kch - 1) / d.kch);
    const bool plain = kc_rounds(d, 8) == 1 && tiles > 3 * SMS;
    if (a.tma && a.err && a.kjpt == 2 && !a.lim && !plain && d.n3 < (1L << 30) && fct_b_maps(d, a, mb)) {
      if (cudaError_t e = smem_opt_in(k_fct_b_tma<T>, FB_SMEM)) return e;
      const dim3 grid((d.jpi + TM_X - 1) / TM_X, (d.jpj + TM_Y - 1) / TM_Y, d.nmem * ((d.jpk + d.kch - 1) / d.kch));
      k_fct_b_tma<T><<<grid, dim3(TM_X, TM_Y), FB_SMEM, s>>>(d, a, mb, a.err, a.polls);
      ktick(NEMO_K_FCT_B_TMA, s);
      b_done = true;
    }
  }
  if (!b_done) {
    const int tb = kty(NEMO_K_FCT_B);
    if (hot_fct_ok(d, a) && !a.lim) k_fct_b_hot<T><<<kc_grid(d, tb), dim3(BX, tb), 0, s>>>(d, a);
    else k_fct_b<T><<<kc_grid(d), dim3(BX, BY), 0, s>>>(d, a);
    ktick(NEMO_K_FCT_B, s);
  }
  const int tc = kty(NEMO_K_FCT_C);
  // FP64 without the iso-neutral trend: the general kernel, two tracers a pass, is the
  // faster (210 against 346 us at 362x242x31); with it (more loads a level) the other is
  if (!hot_fct_c_ok(d, a) || (sizeof(T) == 8 && !a.with_iso)) k_fct_c<T><<<kc_grid(d, tc), dim3(BX, tc), 0, s>>>(d, a);
  else if (d.e3t_n.s == 0) k_fct_c_hot<T, false><<<kc_grid(d, tc), dim3(BX, tc), 0, s>>>(d, a);
  else k_fct_c_hot<T, true><<<kc_grid(d, tc), dim3(BX, tc), 0, s>>>(d, a);
  ktick(NEMO_K_FCT_C, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_ldf_lap(const Dom<T>& d, const LdfArgs<T>& a, cudaStream_t s) {
  k_ldf_lap<T><<<pt_grid(d), dim3(BX, BY), 0, s>>>(d, a);
  ktick(NEMO_K_LDF_LAP, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_ldf_iso(const Dom<T>& d, const LdfArgs<T>& a, int copy_akz_edges, int msc_edges, cudaStream_t s) {
  launch_iso_flux<T>(d, a, s);
  k_iso_div<T><<<pt_grid(d), dim3(BX, BY), 0, s>>>(d, a);
  ktick(NEMO_K_ISO_DIV, s);
  return launch_iso_edges<T>(d, a, copy_akz_edges, msc_edges, s);
}

template <class T>
cudaError_t launch_iso_flux(const Dom<T>& d, const LdfArgs<T>& a, cudaStream_t s) {
  if (hot_iso_ok(d, a)) {
    if constexpr (sizeof(T) == 4) {
      IsoMaps maps;
      if (a.tma && a.err && field_tensor_map(d, a.ptb.p, a.kjpt, TM_W, TM_H, &maps.tb) &&
          field_tensor_map(d, a.uslp.p, 1, TM_X, TM_Y, &maps.uslp) &&
          field_tensor_map(d, a.vslp.p, 1, TM_X, TM_Y, &maps.vslp) &&
          field_tensor_map(d, a.wslpi.p, 1, TM_X, TM_Y, &maps.wslpi) &&
          field_tensor_map(d, a.wslpj.p, 1, TM_X, TM_Y, &maps.wslpj)) {
        const dim3 grid((d.jpi + TM_X - 1) / TM_X, (d.jpj + TM_Y - 1) / TM_Y, d.nmem * ((d.jpk + d.kch - 1) / d.kch));
        (iso_3d(d, a) ? k_iso_flux_tma<T, true, true> : k_iso_flux_tma<T, false, true>)<<<grid, dim3(TM_X, TM_Y), 0, s>>>(
            d, a, maps, a.err, a.polls);
        ktick(NEMO_K_ISO_FLUX_TMA, s);
        return cudaGetLastError();
      }
      // rows not 16 bytes apart: the planes copied by the threads. 281 against 342 us of
      // k_iso_flux_hot at 749x502x31, 101 against 138 at 310x367, 18.3 against 19.0 at
      // 121x152; on smaller grids (7.0 against 6.2 us at 62x42) a march is too short for it.
      // At 230 to 270 points a row, with the data in L2, the other is the faster by itself
      // (242x162x31 50 against 62 us), but its blocks leave no room for the sub-steps that a
      // step runs beside it: 418 us a step against 348
      if (a.tma && a.err && d.n2 * d.nmem >= 16384) {
        const dim3 grid((d.jpi + TM_X - 1) / TM_X, (d.jpj + TM_Y - 1) / TM_Y, d.nmem * ((d.jpk + d.kch - 1) / d.kch));
        (iso_3d(d, a) ? k_iso_flux_tma<T, true, false> : k_iso_flux_tma<T, false, false>)<<<grid, dim3(TM_X, TM_Y), 0, s>>>(
            d, a, maps, a.err, a.polls);
        ktick(NEMO_K_ISO_FLUX, s);
        return cudaGetLastError();
      }
    }
    const int ti = kty(NEMO_K_ISO_FLUX);
    (iso_3d(d, a) ? k_iso_flux_hot<T, true> : k_iso_flux_hot<T, false>)<<<kc_grid(d, ti), dim3(BX, ti), 0, s>>>(d, a);
  } else {
    k_iso_flux<T><<<kc_grid(d), dim3(BX, BY), 0, s>>>(d, a);
  }
  ktick(NEMO_K_ISO_FLUX, s);
  return cudaGetLastError();
}

// the points of ah_wslp2 / akz the interior sweep does not write (edge columns,
// levels 1 and jpk; row and column 1 of the MSC correction)
template <class T>
cudaError_t launch_iso_edges(const Dom<T>& d, const LdfArgs<T>& a, int copy_akz_edges, int msc_edges, cudaStream_t s) {
  if (copy_akz_edges && !hot_iso_ok(d, a)) {  // the specialised flux kernel copies them itself
    k_iso_akz_copy_edges<T><<<dim3((unsigned)((d.n2 + 255) / 256), 1, 2 * d.nmem), 256, 0, s>>>(d, a);
    ktick(NEMO_K_ISO_AKZ_EDGES, s);
  }
  if (msc_edges) {
    k_iso_msc_edges<T><<<col_grid(d), dim3(BX, BY), 0, s>>>(d, a);
    ktick(NEMO_K_ISO_MSC_EDGES, s);
  }
  return cudaGetLastError();
}

// FP32 with the GYRE's 31 levels: one thread a column (k_zdf_imp_async, columns of 32 x 4 in
// shared memory, three blocks an SM) or a block a row of 32 columns (k_zdf_imp32)? The former
// takes 20 to 23 us a round of blocks up to the second, and on a grid of more rounds its march
// of all columns down the same planes is kinder to DRAM; the latter some 15 us and 13 more per
// thousand blocks: 182x122 20 against 15, 212x142 20 and 21, 272x182 23 and 26, 302x202 35 and
// 32, 400x260 40 and 47, 752x502 118 and 150, 60 members of 33x23 22 and 34.
template <class T>
static bool zdf31_by_column(const Dom<T>& d) {
  const long tiles = (long)((d.jpi + 30) / 32) * ((d.jpj + 2) / 4) * d.nmem;  // with an interior column
  const long rows = (long)((d.jpi + 31) / 32) * (d.jpj - 2) * d.nmem;         // blocks of k_zdf_imp32
  const long rounds = (tiles + 3 * SMS - 1) / (3 * SMS);
  return rows >= (rounds == 1 ? 900 : rounds == 2 ? 2500 : 0);
}
template <class T>
cudaError_t launch_zdf(const Dom<T>& d, const ZdfArgs<T>& a, cudaStream_t s) {
  if constexpr (sizeof(T) == 4) {
    if (d.jpi < 3 || d.jpj < 3) return cudaSuccess;  // no interior column
    if (d.jpk == 31 && zdf31_by_column(d)) {
      constexpr int smem_max = 4 * 31 * BX * BY * sizeof(float);
      if (cudaError_t e = smem_opt_in(k_zdf_imp_async<31>, smem_max)) return e;
      const int tz = kty(NEMO_K_ZDF_IMP);
      k_zdf_imp_async<31><<<col_grid(d, tz), dim3(BX, tz), 4 * 31 * BX * tz * sizeof(float), s>>>(d, a);
      ktick(NEMO_K_ZDF_IMP, s);
      return cudaGetLastError();
    }
    if (cudaError_t e = smem_opt_in(k_zdf_imp32<ZW>, zdf32_smem(KMAX))) return e;
    k_zdf_imp32<ZW><<<dim3((unsigned)((d.jpi + 31) / 32) * (d.jpj - 2), d.nmem), dim3(32, ZW), zdf32_smem(d.jpk), s>>>(d, a);
  } else {
    const int tz = kty(NEMO_K_ZDF_IMP);
    k_zdf_imp<T><<<col_grid(d, tz), dim3(BX, tz), 0, s>>>(d, a);
  }
  ktick(NEMO_K_ZDF_IMP, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_clamp(T* x, long n, cudaStream_t s) {
  long nb = (n + 255) / 256;
  if (nb > SMS * 16) nb = SMS * 16;
  if (nb < 1) nb = 1;
  k_clamp_neg<T><<<(unsigned)nb, 256, 0, s>>>(x, n);
  ktick(NEMO_K_CLAMP, s);
  return cudaGetLastError();
}

// the general sub-step kernel; five: compiled for five blocks an SM (FP32, variable volume)
template <class T>
static auto spg_p2_kernel(int vvl, int five) -> void (*)(Dom<T>, SpgArgs<T>, GridBar) {
  if constexpr (sizeof(T) == 4) {
    if (five) return k_spg_p2<T, true, 5>;
  }
  return vvl ? k_spg_p2<T, true> : k_spg_p2<T, false>;
}
// co-resident blocks per SM of the sub-step kernel, with or without the constant
// cache (dynamic shared memory beyond the 48 KB default needs the opt-in)
template <class T>
int spg_p2_blocks_per_sm(int cache, int vvl, int five) {
  const size_t dyn = cache ? P2_CACHE_BYTES : 0;
  auto kern = spg_p2_kernel<T>(vvl, five);
  if (cache && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) != cudaSuccess)
    return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 256, dyn) != cudaSuccess) return 0;
  return nb;
}

// co-resident blocks per SM of the specialised sub-step kernel (mixed form, linear
// free surface, ENE/MIX), with its constant cache
template <class T>
int spg_p2_ene_blocks_per_sm() {
  if constexpr (sizeof(T) != 4) {
    return 0;
  } else {
    if (cudaFuncSetAttribute(k_spg_p2_ene<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)P2H_CACHE_BYTES) != cudaSuccess)
      return 0;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_spg_p2_ene<T>, 256, P2H_CACHE_BYTES) != cudaSuccess)
      return 0;
    return nb;
  }
}

// the variants of k_spg_p2_res: threads, points a thread
struct SpgRes {
  void (*kern)(Dom<float>, SpgArgs<float>, int, int);
  int nt, ppt;
};
static SpgRes spg_res(int v, bool gen) {
  static const SpgRes t[2][P2R_NV] = {
      {{k_spg_p2_res<512, 1, false>, 512, 1}, {k_spg_p2_res<512, 2, false>, 512, 2}, {k_spg_p2_res<512, 4, false>, 512, 4}},
      {{k_spg_p2_res<512, 1, true>, 512, 1}, {k_spg_p2_res<512, 2, true>, 512, 2}, {k_spg_p2_res<512, 4, true>, 512, 4}}};
  return t[gen ? 1 : 0][v];
}
// its launch: csize blocks a member, as clusters
static cudaError_t spg_res_config(const SpgRes& v, bool gen, int csize, int rows, int jpi, int nmem,
                                  cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
  cfg = {};
  cfg.gridDim = dim3((unsigned)csize * nmem);
  cfg.blockDim = dim3(v.nt);
  cfg.dynamicSmemBytes = p2r_smem(v.nt * v.ppt, rows, jpi, gen);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (csize > 8) {  // more than the portable cluster size
    const cudaError_t e = cudaFuncSetAttribute(v.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  return cudaFuncSetAttribute(v.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P2R_SMEM_MAX);
}
template <class T>
cudaError_t launch_spg_res(const Dom<T>& d, const SpgArgs<T>& a, cudaStream_t s) {
  if constexpr (sizeof(T) == 4) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const SpgRes v = spg_res(a.res_v, a.res_gen);
    const cudaError_t e = spg_res_config(v, a.res_gen, a.res_c, a.res_rows, d.jpi, d.nmem, cfg, attr);
    cfg.stream = s;
    return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, v.kern, d, a, a.res_c, a.res_rows);
  } else {
    return cudaErrorInvalidValue;
  }
}
// clusters of k_spg_p2_res that the GPU holds at once (0: the shape does not fit)
template <class T>
int spg_res_clusters(int variant, int gen, int csize, int rows, int jpi) {
  if constexpr (sizeof(T) == 4) {
    const SpgRes v = spg_res(variant, gen);
    if ((long)rows * jpi > v.nt * v.ppt || p2r_smem(v.nt * v.ppt, rows, jpi, gen) > P2R_SMEM_MAX) return 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    int n = 0;
    if (spg_res_config(v, gen, csize, rows, jpi, 1, cfg, attr) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, v.kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  } else {
    return 0;
  }
}

template <class T>
cudaError_t launch_spg(const Dom<T>& d, const SpgArgs<T>& a, const GridBar& bar, int p2_blocks, cudaStream_t s) {
  if (a.vvl) {  // Coriolis factors from the now depths (:241-343)
    k_spg_cor<T><<<col_grid(d), dim3(BX, BY), 0, s>>>(d, a);
    ktick(NEMO_K_SPG_COR, s);
  }
  bool p1a_reg = false;
  if constexpr (sizeof(T) == 4) {
    if (d.jpk == 31) {  // the GYRE levels: columns in registers
      const int t1 = kty(NEMO_K_SPG_P1A);
      k_spg_p1a_reg<31><<<col_grid(d, t1), dim3(BX, t1), 0, s>>>(d, a);
      p1a_reg = true;
    }
  }
  if (!p1a_reg) {
    const int t1 = kty(NEMO_K_SPG_P1A);
    k_spg_p1a<T><<<col_grid(d, t1), dim3(BX, t1), 0, s>>>(d, a);
  }
  ktick(NEMO_K_SPG_P1A, s);
  const int t1b = kty(NEMO_K_SPG_P1B);
  k_spg_p1b<T><<<col_grid(d, t1b), dim3(BX, t1b), 0, s>>>(d, a);
  ktick(NEMO_K_SPG_P1B, s);
  cudaError_t e;
  if (a.res_c > 0) {
    e = launch_spg_res(d, a, s);
  } else {
    {  // the barrier's arrival counter starts at 0 in every launch
      cudaError_t ez = cudaMemsetAsync(bar.count, 0, sizeof(unsigned int), s);
      if (ez != cudaSuccess) return ez;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p2_blocks);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = a.cache ? P2_CACHE_BYTES : 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if constexpr (sizeof(T) == 4) {
      if (a.hot) {
        cfg.dynamicSmemBytes = P2H_CACHE_BYTES;
        e = cudaLaunchKernelEx(&cfg, k_spg_p2_ene<T>, d, a, bar);
      } else {
        e = cudaLaunchKernelEx(&cfg, spg_p2_kernel<T>(a.vvl, a.five), d, a, bar);
      }
    } else {
      e = cudaLaunchKernelEx(&cfg, spg_p2_kernel<T>(a.vvl, 0), d, a, bar);
    }
  }
  if (e != cudaSuccess) return e;
  ktick(NEMO_K_SPG_P2, s);
  const int t3 = kty(NEMO_K_SPG_P3);
  k_spg_p3<T><<<dim3((d.jpi + BX - 1) / BX, (d.jpj + t3 - 1) / t3, d.nmem * ((d.jpk + KCH3 - 1) / KCH3)),
                 dim3(BX, t3), 0, s>>>(d, a);
  ktick(NEMO_K_SPG_P3, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_lbc(T* p, int jpi, int jpj, long nslab, int is_f, T pval, cudaStream_t s) {
  long per = 2L * jpi + 2L * jpj;
  unsigned gx = (unsigned)((per + 255) / 256);
  unsigned gy = (unsigned)(nslab < 65535 ? nslab : 65535);
  k_lbc_closed<T><<<dim3(gx, gy), 256, 0, s>>>(p, jpi, jpj, nslab, is_f, pval);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_globsum(const T* x, const double* tmask_i, long n2, int nk, int nmem, double* part, int nblk,
                           unsigned* ticket, double* out, double* out_host, cudaStream_t s) {
  const long need = (n2 * nk + 256L * GS_PT<T> - 1) / (256L * GS_PT<T>);
  // FP64: the blocks of an ensemble's members share the chip (12 members of 93x61x62 158 us with
  // the most blocks each, 140 with 64)
  const long most = sizeof(T) == 8 ? std::min(nblk, std::max(nblk / nmem, 64)) : nblk;
  k_globsum<T><<<dim3((unsigned)std::min(need, most), nmem), 256, 0, s>>>(x, tmask_i, n2, nk, part, ticket, out, out_host);
  return cudaGetLastError();
}

#define NEMO_INSTANTIATE(T)                                                                                   \
  template cudaError_t launch_adv_trp<T>(const Dom<T>&, const T*, const T*, const T*, T*, T*, T*, cudaStream_t); \
  template cudaError_t launch_fct<T>(const Dom<T>&, const FctArgs<T>&, cudaStream_t);                        \
  template cudaError_t launch_ldf_lap<T>(const Dom<T>&, const LdfArgs<T>&, cudaStream_t);                    \
  template cudaError_t launch_ldf_iso<T>(const Dom<T>&, const LdfArgs<T>&, int, int, cudaStream_t);          \
  template cudaError_t launch_zdf<T>(const Dom<T>&, const ZdfArgs<T>&, cudaStream_t);                        \
  template cudaError_t launch_iso_edges<T>(const Dom<T>&, const LdfArgs<T>&, int, int, cudaStream_t);        \
  template cudaError_t launch_iso_flux<T>(const Dom<T>&, const LdfArgs<T>&, cudaStream_t);                   \
  template cudaError_t launch_clamp<T>(T*, long, cudaStream_t);                                              \
  template cudaError_t launch_spg<T>(const Dom<T>&, const SpgArgs<T>&, const GridBar&, int, cudaStream_t);   \
  template int spg_p2_blocks_per_sm<T>(int, int, int);                                                                 \
  template int spg_res_clusters<T>(int, int, int, int, int);                                                      \
  template int spg_p2_ene_blocks_per_sm<T>();                                                                 \
  template cudaError_t launch_lbc<T>(T*, int, int, long, int, T, cudaStream_t);                              \
  template cudaError_t launch_globsum<T>(const T*, const double*, long, int, int, double*, int, unsigned*, double*, \
                                         double*, cudaStream_t);

}  // namespace nemo
