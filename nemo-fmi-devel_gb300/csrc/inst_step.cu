// inst_step.cu -- launchers of the rest-of-step kernels, both precisions; compiled
// with --fmad=false so the FP64 form rounds as the reference's FP64 CPU build.
#include "k_diag.cuh"
#include "k_step.cuh"
#include "launch.h"

namespace nemo {

namespace {
constexpr int SX = 32, SY = 4;
template <class T>
dim3 s_col(const Dom<T>& d) { return dim3((d.jpi + SX - 1) / SX, (d.jpj + SY - 1) / SY, d.nmem); }
template <class T>
dim3 s_pt(const Dom<T>& d) { return dim3((d.jpi + SX - 1) / SX, (d.jpj + SY - 1) / SY, d.nmem * d.jpk); }
// Levels a thread of a level-march kernel walks: the longest of 4, 2, 1 times `step`
// that still gives every SM its resident warps twice over (64 warps of 32 points),
// so that a long march amortises its column's metrics on a large grid and a small one
// still fills the chip.
template <class T>
int level_chunk(const Dom<T>& d, int block, int step) {
  const long planes = (d.n2 + block - 1) / block * d.nmem;
  for (int f = 4; f > 1; f /= 2)
    if (planes * ((d.jpk + f * step - 1) / (f * step)) * block >= SMS * 64L * 32) return f * step;
  return step;
}
// the two components' columns: z = 2 member + component
template <class T>
dim3 s_cols2(const Dom<T>& d, int ty) { return dim3((d.jpi + SX - 1) / SX, (d.jpj + ty - 1) / ty, 2 * d.nmem); }
}  // namespace

template <class T>
cudaError_t launch_wzv(const Dom<T>& d, const T* un, const T* vn, T* wn, T z1_2dt, cudaStream_t s) {
  const bool flat = d.e3t_n.s == 0 && d.e3u_n.s == 0 && d.e3v_n.s == 0 && d.e3t_a.s == 0 && d.e3t_b.s == 0;
  (flat ? k_wzv<T, true> : k_wzv<T, false>)<<<s_col(d), dim3(SX, SY), 0, s>>>(d, un, vn, wn, z1_2dt);
  ktick(NEMO_K_WZV, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_dyn_zdf_step(const Dom<T>& d, const T* ub, const T* vb, T* ua, T* va, T r2dt, const T* e3u_b,
                                const T* e3v_b, const T* e3u_a, const T* e3v_a, cudaStream_t s) {
  k_dyn_zdf_step<T><<<s_pt(d), dim3(SX, SY), 0, s>>>(d, ub, vb, ua, va, r2dt, e3u_b, e3v_b, e3u_a, e3v_a);
  ktick(NEMO_K_DYN_ZDF_STEP, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_dyn_nxt(const Dom<T>& d, const NxtArgs<T, double>& a, cudaStream_t s) {
  const int level = 32 * DN_Y * (int)sizeof(T), smem = level * d.jpk;
  const dim3 g = s_cols2<T>(d, DN_Y);
  // FP64: 94 registers let five blocks an SM run, 72 (some spills) seven. More than one block an
  // SM takes the latter: 302x202x31 250 -> 183 us, 200x151x31 109 -> 105; 62x42x31 33 -> 39.
  constexpr int more = sizeof(T) == 8 ? 7 : 5;
  const auto kern = (long)g.x * g.y * g.z > SMS ? k_dyn_nxt<T, double, more> : k_dyn_nxt<T, double, 5>;
  if (cudaError_t e = smem_opt_in(kern, level * KMAX)) return e;
  kern<<<g, dim3(SX, DN_Y), smem, s>>>(d, a);
  ktick(NEMO_K_DYN_NXT, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_ssh_swp(const Dom<T>& d, T* sshb, T* sshn, const double* ssha, T atfp, int euler, cudaStream_t s) {
  k_ssh_swp<T, double><<<s_col(d), dim3(SX, SY), 0, s>>>(d, sshb, sshn, ssha, atfp, euler);
  ktick(NEMO_K_SSH_SWP, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_vvl_sf_nxt(const Dom<T>& d, const VvlArgs<T>& a, cudaStream_t s) {
  k_vvl_sf_nxt_t<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  k_vvl_sf_nxt_uv<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_VVL_SF, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_vvl_sf_swp(const Dom<T>& d, const VvlArgs<T>& a, cudaStream_t s) {
  k_vvl_sf_swp<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_VVL_SF, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_tra_nxt_vvl(const Dom<T>& d, const VvlArgs<T>& a, cudaStream_t s) {
  k_tra_nxt_vvl<T><<<s_pt(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_VVL_NXT, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_dyn_nxt_vvl(const Dom<T>& d, const VvlArgs<T>& a, cudaStream_t s) {
  k_dyn_nxt_vvl_a<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  k_dyn_nxt_vvl_b<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_VVL_NXT, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_ssh_swp_vvl(const Dom<T>& d, const VvlArgs<T>& a, T* sshb, T* sshn, cudaStream_t s) {
  k_ssh_swp_vvl<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a, sshb, sshn);
  ktick(NEMO_K_VVL_NXT, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_ldf_slp(const Dom<T>& d, const SlpArgs<T>& a, cudaStream_t s) {
  const int kch = march_chunk(d);
  const dim3 g = march_grid(d, kch);
  const bool flat = d.e3u_n.s == 0 && d.e3v_n.s == 0 && d.e3w_n.s == 0;
  if (a.gru_b) {  // partial steps: the bottom level's gradients from zps_hde
    k_slp_mxl<T, true><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
    (flat ? k_slp_pre<T, true, true> : k_slp_pre<T, true, false>)<<<g, dim3(SX, MARCH_Y), 0, s>>>(d, a, kch);
  } else {
    k_slp_mxl<T, false><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
    (flat ? k_slp_pre<T, false, true> : k_slp_pre<T, false, false>)<<<g, dim3(SX, MARCH_Y), 0, s>>>(d, a, kch);
  }
  k_slp_filter<T><<<march_grid(d, kch, 30, 2), dim3(SX, MARCH_Y), 0, s>>>(d, a, kch);  // a warp writes 30 interior points
  ktick(NEMO_K_LDF_SLP, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_zps_hde_rd(const Dom<T>& d, const EosArgs<T>& a, const T* prd, T* pgru, T* pgrv, cudaStream_t s) {
  k_zps_hde_rd<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a, prd, pgru, pgrv);
  ktick(NEMO_K_ZPS_HDE, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_zps_hde(const Dom<T>& d, const T* pta, T* pgtu, T* pgtv, int kjpt, cudaStream_t s) {
  k_zps_hde<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, pta, pgtu, pgtv, kjpt);
  ktick(NEMO_K_ZPS_HDE, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_tra_sbc(const Dom<T>& d, const SbcArgs<T>& a, cudaStream_t s) {
  k_tra_sbc<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_TRA_SBC, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_tra_qsr(const Dom<T>& d, const QsrArgs<T>& a, cudaStream_t s) {
  k_tra_qsr<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_TRA_QSR, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_eos(const Dom<T>& d, const EosArgs<T>& a, cudaStream_t s) {
  // bn2 of a grid too small to fill the chip: one level a thread, not a chunk of four (33x23x31
  // in FP32 4.4 against 5.2 us; even at 121x83)
  constexpr int B = EOS_BLOCK<T>, L = EOS_LEV<T>;
  const bool one = a.what == 3 && d.n2 * d.nmem < 8000;
  const int kch = one ? 1 : level_chunk(d, B, L);
  const dim3 g((unsigned)((d.n2 + B - 1) / B), (d.jpk - 1 + kch - 1) / kch, d.nmem);
  if (a.what == 3) (one ? k_bn2<T, 1> : k_bn2<T, L>)<<<g, B, 0, s>>>(d, a, kch);
  else if (a.what == 0) (a.eos80 ? k_eos<T, 0, true> : k_eos<T, 0, false>)<<<g, B, 0, s>>>(d, a, kch);
  else if (a.what == 1) (a.eos80 ? k_eos<T, 1, true> : k_eos<T, 1, false>)<<<g, B, 0, s>>>(d, a, kch);
  else (a.eos80 ? k_eos<T, 2, true> : k_eos<T, 2, false>)<<<g, B, 0, s>>>(d, a, kch);
  ktick(a.what == 3 ? NEMO_K_BN2 : NEMO_K_EOS, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dyn_hpg(const Dom<T>& d, const T* rhd, T* ua, T* va, T zcoef0, cudaStream_t s) {
  k_hpg_zco<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, rhd, ua, va, zcoef0);
  ktick(NEMO_K_DYN_HPG, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_zdf_mxl(const Dom<T>& d, const MxlArgs<T>& a, cudaStream_t s) {
  k_zdf_mxl<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_ZDF_MXL, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dyn_zdf_imp(const Dom<T>& d, const DynZdfArgs<T>& a, cudaStream_t s) {
  const bool flat = d.e3u_n.s == 0 && d.e3v_n.s == 0 && d.e3w_n.s == 0;
  const int smem = dyn_zdf_smem(32 * DZ_Y<T>, d.jpk, flat, (int)sizeof(T));
  const auto kern = flat ? k_dyn_zdf_imp<T, true> : k_dyn_zdf_imp<T, false>;
  if (cudaError_t e = smem_opt_in(kern, dyn_zdf_smem(32 * DZ_Y<T>, KMAX, flat, (int)sizeof(T)))) return e;
  kern<<<s_cols2<T>(d, DZ_Y<T>), dim3(SX, DZ_Y<T>), smem, s>>>(d, a);
  ktick(NEMO_K_DYN_ZDF_STEP, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_usr_sbc_a(const Dom<T>& d, const UsrSbcArgs<T>& a, cudaStream_t s) {
  k_usr_sbc_a<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_USR_SBC, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_usr_sbc_b(const Dom<T>& d, const UsrSbcArgs<T>& a, cudaStream_t s) {
  k_usr_sbc_b<T><<<s_col(d), dim3(SX, SY), 0, s>>>(d, a);
  ktick(NEMO_K_USR_SBC, s);
  return cudaGetLastError();
}
cudaError_t launch_usr_put(double* dst, const double* v, cudaStream_t s) {
  k_usr_put<<<1, 1, 0, s>>>(dst, v[0], v[1], v[2], v[3], v[4], v[5], v[6]);
  return cudaGetLastError();
}

// k_zdf_tke with SH values a level in shared memory, and the rounds of resident blocks that
// the grid takes (0: it cannot run)
template <class T>
struct TkeLaunch {
  void (*kern)(Dom<T>, ZphyArgs<T>);
  int smem, rounds;
};
template <class T, int SH>
static TkeLaunch<T> tke_launch(const Dom<T>& d, dim3 g, int nsm) {
  TkeLaunch<T> t{d.e3w_n.s == 0 && d.e3t_n.s == 0 ? k_zdf_tke<T, true, SH> : k_zdf_tke<T, false, SH>, 0, 0};
  const int level = SH * 32 * TKE_Y<T> * (int)sizeof(T);
  t.smem = level * d.jpk;
  int n = 0;
  if (smem_opt_in(t.kern, level * KMAX) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, t.kern, 32 * TKE_Y<T>, t.smem) != cudaSuccess || n < 1)
    return t;
  const long blocks = (long)g.x * g.y * g.z, wave = (long)n * nsm;
  t.rounds = (int)((blocks + wave - 1) / wave);
  return t;
}
template <class T>
cudaError_t launch_zdf_phy(const Dom<T>& d, const ZphyArgs<T>& a, int nsm, cudaStream_t s) {
  const int kch = march_chunk(d);
  const dim3 g((d.jpi + SX - 1) / SX, (d.jpj + TKE_Y<T> - 1) / TKE_Y<T>, d.nmem);
  TkeLaunch<T> t;
  if constexpr (sizeof(T) == 4) {
    t = tke_launch<T, 3>(d, g, nsm);
  } else {
    // FP64: a column's four values a level leave three blocks of two warps an SM at 31 levels
    // and one at 62. Of the forms with four, two and no values in shared memory (the rest in
    // work arrays) the one with the fewest rounds of blocks, then the most values: us a call
    // of zdf_phy 121x83x31 208, 216, 219; 200x151x31 512, 381, 383; 302x202x31 807, 968, 666;
    // 333x251x31 1039, 1051, 1303; 250x200x62 2499, 1237, 1163.
    t = tke_launch<T, 4>(d, g, nsm);
    for (const TkeLaunch<T>& x : {tke_launch<T, 2>(d, g, nsm), tke_launch<T, 0>(d, g, nsm)})
      if (x.rounds && (!t.rounds || x.rounds < t.rounds)) t = x;
  }
  if (!t.rounds) return cudaErrorLaunchOutOfResources;
  (d.e3w_n.s == 0 ? k_zdf_sh2<T, true> : k_zdf_sh2<T, false>)<<<march_grid(d, kch), dim3(SX, MARCH_Y), 0, s>>>(d, a, kch);
  ktick(NEMO_K_ZDF_PHY, s);
  t.kern<<<g, dim3(SX, TKE_Y<T>), t.smem, s>>>(d, a);
  ktick(NEMO_K_ZDF_PHY, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dyn_ldf_lap(const Dom<T>& d, const T* ahmt, const T* ahmf, const T* pub, const T* pvb, T* pua, T* pva,
                               T zsign, cudaStream_t s) {
  const int kch = march_chunk(d);
  const bool flat = d.e3f_n.s == 0 && d.e3t_b.s == 0 && d.e3u_n.s == 0 && d.e3v_n.s == 0;
  dim3 g = march_grid(d, kch, 30, 2);  // a block writes 30 x (LDF_Y - 2) interior points
  g.y = (max(d.jpj - 2, 1) + LDF_Y - 3) / (LDF_Y - 2);
  (flat ? k_dyn_ldf_lap<T, true> : k_dyn_ldf_lap<T, false>)<<<g, dim3(SX, LDF_Y), 0, s>>>(
      d, ahmt, ahmf, pub, pvb, pua, pva, zsign, kch);
  ktick(NEMO_K_DYN_LDF, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_vor_ene(const Dom<T>& d, int kvor, const T* pun, const T* pvn, T* pua, T* pva, cudaStream_t s) {
  const int kch = march_chunk(d);
  (kvor == 1 ? k_vor_ene<T, 1> : kvor == 2 ? k_vor_ene<T, 2> : k_vor_ene<T, 4>)<<<march_grid(d, kch), dim3(SX, MARCH_Y), 0, s>>>(
      d, pun, pvn, pua, pva, kch);
  ktick(NEMO_K_DYN_VOR, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dyn_keg(const Dom<T>& d, const T* un, const T* vn, T* ua, T* va, cudaStream_t s) {
  const int kch = march_chunk(d);
  k_dyn_keg<T><<<march_grid(d, kch), dim3(SX, MARCH_Y), 0, s>>>(d, un, vn, ua, va, kch);
  ktick(NEMO_K_DYN_KEG, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_dyn_zad(const Dom<T>& d, const T* un, const T* vn, const T* wn, T* ua, T* va, cudaStream_t s) {
  const int kch = march_chunk(d);
  const bool flat = d.e3u_n.s == 0 && d.e3v_n.s == 0;
  (flat ? k_dyn_zad<T, true> : k_dyn_zad<T, false>)<<<march_grid(d, kch), dim3(SX, MARCH_Y), 0, s>>>(d, un, vn, wn, ua, va,
                                                                                                 kch);
  ktick(NEMO_K_DYN_ZAD, s);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_stp_ctl(const Dom<T>& d, const T* sshn, const T* un, const T* ts, double* part, int nblk,
                           int someoce, double* out, unsigned long long* idx, int* flag, cudaStream_t s) {
  k_ctl_partial<T><<<dim3(nblk, d.nmem), DG_THREADS, 0, s>>>(d, sshn, un, ts, part);
  ktick(NEMO_K_STP_CTL, s);
  k_ctl_final<T><<<d.nmem, DG_THREADS, 0, s>>>(d, part, nblk, someoce, out, idx, flag);
  ktick(NEMO_K_STP_CTL, s);
  k_ctl_locate<T><<<dim3(nblk, d.nmem), DG_THREADS, 0, s>>>(d, sshn, un, ts, out, idx);
  ktick(NEMO_K_STP_CTL, s);
  k_ctl_pos<T><<<(d.nmem + 31) / 32, 32, 0, s>>>(d, out, idx);
  ktick(NEMO_K_STP_CTL, s);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_hsb_init(const Dom<T>& d, const HsbArgs<T>& a, int nblk, cudaStream_t s) {
  k_hsb_init<T><<<nblk, DG_THREADS, 0, s>>>(d, a);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_dia_hsb(const Dom<T>& d, const HsbArgs<T>& a, double* part, int nblk, cudaStream_t s) {
  k_hsb_partial<T><<<dim3(nblk, d.nmem), DG_THREADS, 0, s>>>(d, a, part);
  k_hsb_final<T><<<d.nmem, 32, 0, s>>>(d, a, part, nblk);
  ktick(NEMO_K_DIA_HSB, s);
  return cudaGetLastError();
}

#define NEMO_STEP_INST(T)                                                                                      \
  template cudaError_t launch_stp_ctl<T>(const Dom<T>&, const T*, const T*, const T*, double*, int, int,       \
                                         double*, unsigned long long*, int*, cudaStream_t);                    \
  template cudaError_t launch_hsb_init<T>(const Dom<T>&, const HsbArgs<T>&, int, cudaStream_t);                \
  template cudaError_t launch_dia_hsb<T>(const Dom<T>&, const HsbArgs<T>&, double*, int, cudaStream_t);         \
  template cudaError_t launch_wzv<T>(const Dom<T>&, const T*, const T*, T*, T, cudaStream_t);                  \
  template cudaError_t launch_dyn_zdf_step<T>(const Dom<T>&, const T*, const T*, T*, T*, T, const T*, const T*, \
                                              const T*, const T*, cudaStream_t);                            \
  template cudaError_t launch_dyn_nxt<T>(const Dom<T>&, const NxtArgs<T, double>&, cudaStream_t);              \
  template cudaError_t launch_ssh_swp<T>(const Dom<T>&, T*, T*, const double*, T, int, cudaStream_t);      \
  template cudaError_t launch_vvl_sf_nxt<T>(const Dom<T>&, const VvlArgs<T>&, cudaStream_t);                \
  template cudaError_t launch_vvl_sf_swp<T>(const Dom<T>&, const VvlArgs<T>&, cudaStream_t);                \
  template cudaError_t launch_tra_nxt_vvl<T>(const Dom<T>&, const VvlArgs<T>&, cudaStream_t);               \
  template cudaError_t launch_dyn_nxt_vvl<T>(const Dom<T>&, const VvlArgs<T>&, cudaStream_t);               \
  template cudaError_t launch_ssh_swp_vvl<T>(const Dom<T>&, const VvlArgs<T>&, T*, T*, cudaStream_t);       \
  template cudaError_t launch_ldf_slp<T>(const Dom<T>&, const SlpArgs<T>&, cudaStream_t);                  \
  template cudaError_t launch_zps_hde_rd<T>(const Dom<T>&, const EosArgs<T>&, const T*, T*, T*, cudaStream_t);  \
  template cudaError_t launch_zps_hde<T>(const Dom<T>&, const T*, T*, T*, int, cudaStream_t);             \
  template cudaError_t launch_tra_sbc<T>(const Dom<T>&, const SbcArgs<T>&, cudaStream_t);                  \
  template cudaError_t launch_tra_qsr<T>(const Dom<T>&, const QsrArgs<T>&, cudaStream_t);                  \
  template cudaError_t launch_eos<T>(const Dom<T>&, const EosArgs<T>&, cudaStream_t);                      \
  template cudaError_t launch_dyn_hpg<T>(const Dom<T>&, const T*, T*, T*, T, cudaStream_t);              \
  template cudaError_t launch_zdf_mxl<T>(const Dom<T>&, const MxlArgs<T>&, cudaStream_t);                  \
  template cudaError_t launch_dyn_zdf_imp<T>(const Dom<T>&, const DynZdfArgs<T>&, cudaStream_t);           \
  template cudaError_t launch_usr_sbc_a<T>(const Dom<T>&, const UsrSbcArgs<T>&, cudaStream_t);              \
  template cudaError_t launch_usr_sbc_b<T>(const Dom<T>&, const UsrSbcArgs<T>&, cudaStream_t);              \
  template cudaError_t launch_zdf_phy<T>(const Dom<T>&, const ZphyArgs<T>&, int, cudaStream_t);                 \
  template cudaError_t launch_dyn_ldf_lap<T>(const Dom<T>&, const T*, const T*, const T*, const T*, T*, T*, T,   \
                                             cudaStream_t);                                             \
  template cudaError_t launch_vor_ene<T>(const Dom<T>&, int, const T*, const T*, T*, T*, cudaStream_t);       \
  template cudaError_t launch_dyn_keg<T>(const Dom<T>&, const T*, const T*, T*, T*, cudaStream_t);             \
  template cudaError_t launch_dyn_zad<T>(const Dom<T>&, const T*, const T*, const T*, T*, T*, cudaStream_t);
NEMO_STEP_INST(double)
NEMO_STEP_INST(float)

}  // namespace nemo
