// CUDA kernels of the B200 chemistry engine (sm_100a) and their launchers.
//
// Two integration engines share one device implementation (ppb_bdf.cuh):
//  * plain: one thread per cell, FP64 everywhere, per-cell arrays in
//    thread-local memory, one launch over all cells -- the straightforward
//    GPU mapping of the reference's per-cell loop;
//  * tuned: one warp per cell, per-cell arrays in shared memory, a persistent
//    grid sized to the resident capacity of the GPU whose warps pull cells
//    from a device work queue, optional FP32 factorisation of I - gamma J
//    with FP64 iterative refinement.
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "ppb_work.cuh"
#include "ppb_engine.h"
#include "mech/mech_LiDryer.h"
#include "mech/mech_drm19.h"
#include "mech/mech_dodecane_lu.h"
#include "mech/mech_heptane_lu_88sk.h"
#include "mech/mech_CH4_lean_qss.h"
#include "mech/mech_C1-C2-NO_qss.h"
#include "mech/mech_LuEthylene_qss.h"
#include "mech/mech_grimech30.h"
#include "mech/mech_FFCM1_Red.h"
#include "mech/mech_chem-H.h"

namespace ppb {

const PPBMechTables* find_mechanism(const char* name)
{
  if (!strcmp(name, "LiDryer")) return &ppbm_LiDryer;
  if (!strcmp(name, "drm19")) return &ppbm_drm19;
  if (!strcmp(name, "dodecane_lu")) return &ppbm_dodecane_lu;
  if (!strcmp(name, "heptane_lu_88sk")) return &ppbm_heptane_lu_88sk;
  if (!strcmp(name, "CH4_lean_qss")) return &ppbm_CH4_lean_qss;
  if (!strcmp(name, "C1-C2-NO_qss")) return &ppbm_C1_C2_NO_qss;
  if (!strcmp(name, "LuEthylene_qss")) return &ppbm_LuEthylene_qss;
  if (!strcmp(name, "grimech30")) return &ppbm_grimech30;
  if (!strcmp(name, "FFCM1_Red")) return &ppbm_FFCM1_Red;
  if (!strcmp(name, "chem-H")) return &ppbm_chem_H;
  return nullptr;
}

// ------------------------------------------------------------ upload
namespace {
// Packs every table into one byte image with 16-byte aligned sections and
// records each section's offset in a DevMech whose pointers are offsets.
struct Packer {
  char* buf;     // destination image (nullptr: size only)
  size_t cap;    // capacity of buf
  size_t used = 0;
  bool overflow = false; // does not fit buf, or is beyond the limits of RxPack
  int wide = 0;          // DevMech::wide
  template <typename T>
  size_t add(const T* p, size_t n)
  {
    size_t off = (used + 15) & ~size_t(15);
    const size_t end = off + n * sizeof(T);
    if (buf && end <= cap) {
      if (n) memcpy(buf + off, p, n * sizeof(T));
    } else if (buf) {
      overflow = true;
    }
    used = end;
    return off;
  }
  // write n values at byte offset off (no alignment)
  template <typename T>
  void put(size_t off, const T* p, size_t n)
  {
    if (!buf) return;
    if (off + n * sizeof(T) > cap) {
      overflow = true;
      return;
    }
    memcpy(buf + off, p, n * sizeof(T));
  }
};

template <typename T>
void set_off(const T*& field, size_t off)
{
  field = reinterpret_cast<const T*>(off);
}
} // namespace

// A coefficient as a sum of doubles that are zero below their top 16 bits
// (whole numbers up to 31 are one, a full significand is eleven): returns the
// first, leaves the rest in c.
static unsigned coefficient_part(double& c)
{
  unsigned long long bits;
  memcpy(&bits, &c, 8);
  bits &= 0xffffull << 48;
  double top;
  memcpy(&top, &bits, 8);
  c -= top; // exact
  return (unsigned)(bits >> 48);
}

static int coefficient_parts(double c)
{
  int n = 0;
  do {
    coefficient_part(c);
    n++;
  } while (c != 0.0 && n < 11);
  return n;
}

// The entries (DevMech::wg, jh) of reaction r's coefficient c in species s's
// list, from its k-th on; returns their number.
static int put_coefficient(Packer& pk, size_t off, int N, int s, int k, int r, double c)
{
  int n = 0;
  do {
    const unsigned e = coefficient_part(c) << 16 | (unsigned)r;
    pk.put(off + ((size_t)(k + n) * N + s) * sizeof(unsigned), &e, 1);
    n++;
  } while (c != 0.0 && n < 11);
  return n;
}

// The rate records (RxRate) and the efficiency lists of the third-body and
// fall-off reactions, in the layouts of DevMech.
static void pack_rates(const PPBMechTables* t, Packer& pk, DevMech& dm)
{
  const int N = t->nsp, R = t->nrxn;
  auto third = [&](int r) {
    return t->rx_kind[r] == PPB_RX_THIRD || t->rx_kind[r] == PPB_RX_TROE || t->rx_kind[r] == PPB_RX_LINDEMANN;
  };
  int nal = 0, neff = 0;
  for (int r = 0; r < R; r++) {
    if (!third(r)) continue;
    nal++;
    int n = 0;
    for (int e = t->eff_off[r]; e < t->eff_off[r + 1]; e++) n += (t->eff_m1[e] != 0.0);
    neff = n > neff ? n : neff;
  }
  neff = (neff + EFF_UNROLL - 1) / EFF_UNROLL * EFF_UNROLL;
  if (R > 65535) pk.overflow = true;
  dm.nal = nal;
  dm.neff = neff;
  const size_t off_rr = (pk.used + 15) & ~size_t(15);
  const size_t off_m1 = off_rr + (size_t)R * sizeof(RxRate);
  const size_t off_sp = off_m1 + (size_t)neff * nal * sizeof(double);
  bool wide; // the reaction does not fit RxRate
  // the slots of a phase space: a repeated species first (see RxRate)
  auto slots = [&](const int* sp, const double* c, int n, unsigned char (&out)[3]) {
    int k = 0, runs = 0, repeats = 0;
    for (int pass = 0; pass < 2; pass++)
      for (int j = 0; j < n; j++) {
        const int o = (int)c[j];
        if ((double)o != c[j] || o < 1) wide = true;
        if ((o > 1) != (pass == 0)) continue;
        runs++;
        repeats += (o > 1);
        for (int q = 0; q < o; q++)
          if (k < 3) out[k++] = (unsigned char)sp[j];
          else wide = true;
      }
    // a single repeated run is a factor of its own only next to one other
    // run, or in front of them in species order
    if (repeats > 1 || (repeats == 1 && runs > 2 && (int)c[0] < 2)) wide = true;
    while (k < 3) out[k++] = (unsigned char)N;
  };
  int a = 0, fo = 0;
  for (int r = 0; r < R; r++) {
    RxRate p;
    memset(&p, 0, sizeof(p));
    wide = false;
    p.A = t->rx_A[r];
    p.beta = t->rx_beta[r];
    p.EaR = t->rx_EaR[r];
    slots(t->rx_fps_sp + r * PPB_MAXPS, t->rx_fps_c + r * PPB_MAXPS, t->rx_fps_n[r], p.fsp);
    for (int j = 0; j < 3; j++) p.rsp[j] = (unsigned char)N;
    for (int j = 0; j < 5; j++) p.kcs[j] = (unsigned char)N;
    if (t->rx_rev[r]) { // the reverse tables are read for a reversible reaction only
      slots(t->rx_rps_sp + r * PPB_MAXPS, t->rx_rps_c + r * PPB_MAXPS, t->rx_rps_n[r], p.rsp);
      if (t->rx_kc_n[r] > 5) wide = true;
      for (int j = 0; j < t->rx_kc_n[r] && j < 5; j++) {
        unsigned long long bits;
        memcpy(&bits, &t->rx_kc_c[r * PPB_MAXKC + j], 8);
        if (bits << 16) wide = true; // more than the top 16 bits of the double
        p.kcs[j] = (unsigned char)t->rx_kc_sp[r * PPB_MAXKC + j];
        p.kch[j] = (unsigned short)(bits >> 48);
      }
      if (t->rx_kcpow[r] < -1 || t->rx_kcpow[r] >= RR_WIDE - 1) wide = true;
    }
    if (third(r) && a > 255) wide = true;
    if (wide) pk.wide |= WIDE_RATES;
    p.flags = (unsigned char)((t->rx_rev[r] ? RR_REV : 0) | (third(r) ? RR_ALPHA : 0) |
                              (t->nqss > 0 && t->rx_rmfwd[r] ? RR_RMF : 0) |
                              ((wide ? RR_WIDE : t->rx_rev[r] ? t->rx_kcpow[r] + 1 : 1) << RR_KCPOW));
    p.fo = 255;
    if (t->rx_kind[r] == PPB_RX_TROE || t->rx_kind[r] == PPB_RX_LINDEMANN) p.fo = (unsigned char)fo++;
    if (third(r)) {
      int n = 0;
      for (int e = t->eff_off[r]; e < t->eff_off[r + 1]; e++) {
        if (t->eff_m1[e] == 0.0) continue;
        const unsigned char sp = (unsigned char)t->eff_sp[e];
        pk.put(off_m1 + ((size_t)n * nal + a) * sizeof(double), &t->eff_m1[e], 1);
        pk.put(off_sp + (size_t)n * nal + a, &sp, 1);
        n++;
      }
      for (; n < neff; n++) {
        const unsigned char sp = (unsigned char)N;
        const double z = 0.0;
        pk.put(off_m1 + ((size_t)n * nal + a) * sizeof(double), &z, 1);
        pk.put(off_sp + (size_t)n * nal + a, &sp, 1);
      }
      p.al = (unsigned char)a++;
    }
    for (int w = 0; w < 3; w++)
      pk.put(off_rr + ((size_t)w * R + r) * 16, reinterpret_cast<const char*>(&p) + 16 * w, 16);
  }
  pk.used = off_sp + (size_t)neff * nal;
  set_off(dm.rr, off_rr);
  set_off(dm.al_m1, off_m1);
  set_off(dm.al_sp, off_sp);
}

// Every table of a mechanism in the layouts of DevMech: the PPBMechTables
// arrays, then the lists and records derived from them.
static size_t pack_all(const PPBMechTables* t, Packer& pk, DevMech& dm)
{
  const int N = t->nsp, R = t->nrxn;
  dm = DevMech{};
  dm.nsp = N;
  dm.nrxn = R;
  dm.nqss = t->nqss;
  dm.nrq = t->nrq;
  // thermo entries: one per concentration slot for a QSS mechanism
  const int NT = t->nqss > 0 ? N + 1 + t->nqss : N;
#define PPB_ADD(field, ptr, count) set_off(dm.field, pk.add(ptr, count))
  PPB_ADD(mw, t->mw, N);
  PPB_ADD(imw, t->imw, N);
  PPB_ADD(tmid, t->tmid, NT);
  // thermo polynomials, coefficient-major (th_row, th_at)
  const int ld = thermo_ld(N);
  auto add_thermo = [&](const double* src, int nc) {
    const size_t off = (pk.used + 15) & ~size_t(15);
    for (int k = 0; k < nc; k++)
      for (int g = 0; g < 2; g++)
        for (int s = 0; s < ld; s++) {
          const double v = s < N ? src[(2 * s + g) * nc + k] : 0.0;
          pk.put(off + ((size_t)(2 * k + g) * ld + s) * sizeof(double), &v, 1);
        }
    pk.used = off + (size_t)2 * nc * ld * sizeof(double);
    return off;
  };
  set_off(dm.th_cv, add_thermo(t->th_cv, 5));
  set_off(dm.th_cp, add_thermo(t->th_cp, 5));
  set_off(dm.th_dcp, add_thermo(t->th_dcp, 4));
  set_off(dm.th_u, add_thermo(t->th_u, 6));
  set_off(dm.th_h, add_thermo(t->th_h, 6));
  set_off(dm.th_g, add_thermo(t->th_g, 7));
  {
    const int Q = t->nqss;
    const size_t off = (pk.used + 15) & ~size_t(15);
    for (int k = 0; k < 7; k++)
      for (int g = 0; g < 2; g++)
        for (int q = 0; q < Q; q++)
          pk.put(off + ((size_t)(2 * k + g) * Q + q) * sizeof(double), &t->th_g[(2 * (N + 1 + q) + g) * 7 + k], 1);
    pk.used = off + (size_t)14 * Q * sizeof(double);
    set_off(dm.th_gq, off);
  }
  {
    // e/(RT W) and h/(RT W) at the T solve's bounds
    const size_t off = (pk.used + 15) & ~size_t(15);
    const double lim[2] = {90.0, 4000.0};
    for (int eh = 0; eh < 2; eh++)
      for (int b = 0; b < 2; b++)
        for (int s = 0; s < ld; s++) {
          double v = 0.0;
          if (s < N) {
            const double T = lim[b], tm = t->tmid[s];
            const double* c = (eh ? t->th_h : t->th_u) + (2 * s + ((tm >= 0.0 && T < tm) ? 0 : 1)) * 6;
            const double T2 = T * T, T3 = T * T * T, T4 = T * T * T * T;
            v = (c[0] + c[1] * T + c[2] * T2 + c[3] * T3 + c[4] * T4 + c[5] * (1.0 / T)) * t->imw[s];
          }
          pk.put(off + ((size_t)(2 * eh + b) * ld + s) * sizeof(double), &v, 1);
        }
    pk.used = off + (size_t)4 * ld * sizeof(double);
    set_off(dm.th_lim, off);
  }
  PPB_ADD(rx_kind, t->rx_kind, R);
  PPB_ADD(rx_rev, t->rx_rev, R);
  PPB_ADD(rx_kcpow, t->rx_kcpow, R);
  PPB_ADD(rx_A, t->rx_A, R);
  PPB_ADD(rx_beta, t->rx_beta, R);
  PPB_ADD(rx_EaR, t->rx_EaR, R);
  PPB_ADD(rx_sum_nuk, t->rx_sum_nuk, R);
  PPB_ADD(fps_n, t->rx_fps_n, R);
  PPB_ADD(fps_sp, t->rx_fps_sp, R * PPB_MAXPS);
  PPB_ADD(fps_c, t->rx_fps_c, R * PPB_MAXPS);
  PPB_ADD(rps_n, t->rx_rps_n, R);
  PPB_ADD(rps_sp, t->rx_rps_sp, R * PPB_MAXPS);
  PPB_ADD(rps_c, t->rx_rps_c, R * PPB_MAXPS);
  PPB_ADD(kc_n, t->rx_kc_n, R);
  PPB_ADD(kc_sp, t->rx_kc_sp, R * PPB_MAXKC);
  PPB_ADD(kc_c, t->rx_kc_c, R * PPB_MAXKC);
  PPB_ADD(wup_n, t->rx_wup_n, R);
  PPB_ADD(wup_sp, t->rx_wup_sp, R * PPB_MAXW);
  PPB_ADD(wup_c, t->rx_wup_c, R * PPB_MAXW);
  PPB_ADD(jn_n, t->rx_jn_n, R);
  PPB_ADD(jn_sp, t->rx_jn_sp, R * PPB_MAXJN);
  PPB_ADD(jn_c, t->rx_jn_c, R * PPB_MAXJN);
  PPB_ADD(hr_n, t->rx_hr_n, R);
  PPB_ADD(hr_sp, t->rx_hr_sp, R * PPB_MAXPS);
  PPB_ADD(hr_c, t->rx_hr_c, R * PPB_MAXPS);
  PPB_ADD(hp_n, t->rx_hp_n, R);
  PPB_ADD(hp_sp, t->rx_hp_sp, R * PPB_MAXPS);
  PPB_ADD(hp_c, t->rx_hp_c, R * PPB_MAXPS);
  PPB_ADD(eff_off, t->eff_off, R + 1);
  PPB_ADD(eff_sp, t->eff_sp, t->eff_off[R]);
  PPB_ADD(eff_e, t->eff_e, t->eff_off[R]);
  PPB_ADD(eff_m1, t->eff_m1, t->eff_off[R]);
  PPB_ADD(fo_d, t->fo_d, R * PPB_NFOD);
  PPB_ADD(fo_i, t->fo_i, R * PPB_NFOI);
  if (t->nqss > 0) {
    PPB_ADD(q_rx, t->q_rx, t->nrq);
    PPB_ADD(q_off, t->q_off, t->nqss + 1);
    PPB_ADD(q_term, t->q_term, t->q_off[t->nqss]);
    PPB_ADD(q_role, t->q_role, t->q_off[t->nqss]);
    PPB_ADD(q_coef, t->q_coef, t->q_off[t->nqss]);
    PPB_ADD(rx_rmfwd, t->rx_rmfwd, R);
    // the balance solve keeps a 32-bit coupling mask; slots are bytes
    if (t->nqss > 32 || N + 1 + t->nqss > 255) pk.overflow = true;
  } else {
    PPB_ADD(q_rx, t->rx_kind, 0);
    PPB_ADD(q_off, t->rx_kind, 0);
    PPB_ADD(q_term, t->rx_kind, 0);
    PPB_ADD(q_role, t->rx_kind, 0);
    PPB_ADD(q_coef, t->rx_A, 0);
    PPB_ADD(rx_rmfwd, t->rx_kind, 0);
  }
#undef PPB_ADD
  // gather lists, written entry by entry at exact offsets (no temporary
  // containers, so packing itself allocates nothing)
  int longest = 0;
  for (int s = 0; s < N; s++) {
    int cnt = 0;
    for (int r = 0; r < R; r++)
      for (int j = 0; j < t->rx_wup_n[r]; j++)
        if (t->rx_wup_sp[r * PPB_MAXW + j] == s) cnt += coefficient_parts(t->rx_wup_c[r * PPB_MAXW + j]);
    longest = cnt > longest ? cnt : longest;
  }
  const int wgl = (longest + WG_UNROLL - 1) / WG_UNROLL * WG_UNROLL + WG_UNROLL;
  const size_t off_gn = (pk.used + 15) & ~size_t(15);
  const size_t off_g = (off_gn + N * sizeof(int) + 15) & ~size_t(15);
  int k = 0;
  for (int s = 0; s < N; s++) {
    k = 0;
    for (int r = 0; r < R; r++) {
      for (int j = 0; j < t->rx_wup_n[r]; j++) {
        if (t->rx_wup_sp[r * PPB_MAXW + j] != s) continue;
        k += put_coefficient(pk, off_g, N, s, k, r, t->rx_wup_c[r * PPB_MAXW + j]);
      }
    }
    pk.put(off_gn + s * sizeof(int), &k, 1);
    for (; k < wgl; k++) {
      const unsigned e = 0;
      pk.put(off_g + ((size_t)k * N + s) * sizeof(unsigned), &e, 1);
    }
  }
  pk.used = off_g + (size_t)wgl * N * sizeof(unsigned);
  set_off(dm.wg_n, off_gn);
  set_off(dm.wg, off_g);
  // aJacobian net-stoichiometry gather (species -> (reaction, nu)), reaction order
  int jtotal = 0;
  for (int r = 0; r < R; r++)
    for (int j = 0; j < t->rx_jn_n[r]; j++) jtotal += (t->rx_jn_c[r * PPB_MAXJN + j] != 0.0);
  const size_t off_joff = (pk.used + 15) & ~size_t(15);
  const size_t off_jrx = (off_joff + (N + 1) * sizeof(int) + 15) & ~size_t(15);
  const size_t off_jc = (off_jrx + jtotal * sizeof(int) + 15) & ~size_t(15);
  k = 0;
  for (int sp = 0; sp < N; sp++) {
    pk.put(off_joff + sp * sizeof(int), &k, 1);
    for (int r = 0; r < R; r++) {
      for (int j = 0; j < t->rx_jn_n[r]; j++) {
        if (t->rx_jn_sp[r * PPB_MAXJN + j] != sp || t->rx_jn_c[r * PPB_MAXJN + j] == 0.0) continue;
        pk.put(off_jrx + k * sizeof(int), &r, 1);
        pk.put(off_jc + k * sizeof(double), &t->rx_jn_c[r * PPB_MAXJN + j], 1);
        k++;
      }
    }
  }
  pk.put(off_joff + N * sizeof(int), &k, 1);
  pk.used = off_jc + jtotal * sizeof(double);
  {
    int jl = 0;
    for (int sp = 0; sp < N; sp++) {
      int c = 0;
      for (int r = 0; r < R; r++)
        for (int j = 0; j < t->rx_jn_n[r]; j++)
          if (t->rx_jn_sp[r * PPB_MAXJN + j] == sp && t->rx_jn_c[r * PPB_MAXJN + j] != 0.0)
            c += coefficient_parts(t->rx_jn_c[r * PPB_MAXJN + j]);
      jl = c > jl ? c : jl;
    }
    const size_t off_n = (pk.used + 15) & ~size_t(15);
    const size_t off_e = (off_n + N * sizeof(int) + 15) & ~size_t(15);
    for (int sp = 0; sp < N; sp++) {
      int c = 0;
      for (int r = 0; r < R; r++)
        for (int j = 0; j < t->rx_jn_n[r]; j++) {
          const double nu = t->rx_jn_c[r * PPB_MAXJN + j];
          if (t->rx_jn_sp[r * PPB_MAXJN + j] != sp || nu == 0.0) continue;
          c += put_coefficient(pk, off_e, N, sp, c, r, nu);
        }
      pk.put(off_n + sp * sizeof(int), &c, 1);
      for (; c < jl; c++) {
        const unsigned e = 0;
        pk.put(off_e + ((size_t)c * N + sp) * sizeof(unsigned), &e, 1);
      }
    }
    pk.used = off_e + (size_t)jl * N * sizeof(unsigned);
    set_off(dm.jh_n, off_n);
    set_off(dm.jh, off_e);
  }
  set_off(dm.jg_off, off_joff);
  set_off(dm.jg_rx, off_jrx);
  set_off(dm.jg_c, off_jc);
  // packed reaction records and fall-off records
  const size_t off_rxp = (pk.used + 15) & ~size_t(15);
  int nfo = 0;
  for (int r = 0; r < R; r++)
    if (t->rx_kind[r] == PPB_RX_TROE || t->rx_kind[r] == PPB_RX_LINDEMANN) nfo++;
  int nalpha = 0;
  for (int r = 0; r < R; r++)
    if (t->rx_kind[r] == PPB_RX_THIRD || t->rx_kind[r] == PPB_RX_TROE || t->rx_kind[r] == PPB_RX_LINDEMANN)
      nalpha++;
  const size_t off_fop = off_rxp + (size_t)R * sizeof(RxPack);
  const size_t off_fow = off_fop + (size_t)nfo * sizeof(FoPack);
  const size_t off_effd = off_fow + (size_t)nfo * sizeof(FoPack);
  int fo = 0, aslot = 0;
  for (int r = 0; r < R; r++) {
    RxPack p;
    memset(&p, 0, sizeof(p));
    p.A = t->rx_A[r];
    p.beta = t->rx_beta[r];
    p.EaR = t->rx_EaR[r];
    for (int j = 0; j < 4; j++) p.fsp[j] = (unsigned char)N;
    for (int j = 0; j < 8; j++) p.rsp[j] = (unsigned char)N;
    for (int j = 0; j < 6; j++) {
      p.kcs[j] = (unsigned char)N;
      p.jns[j] = (unsigned char)N;
    }
    int nf = 0, nr = 0;
    for (int j = 0; j < t->rx_fps_n[r]; j++)
      for (int q = 0; q < (int)t->rx_fps_c[r * PPB_MAXPS + j]; q++)
        if (nf < 4) p.fsp[nf++] = (unsigned char)t->rx_fps_sp[r * PPB_MAXPS + j];
        else pk.overflow = true;
    for (int j = 0; j < t->rx_rps_n[r]; j++)
      for (int q = 0; q < (int)t->rx_rps_c[r * PPB_MAXPS + j]; q++)
        if (nr < 8) p.rsp[nr++] = (unsigned char)t->rx_rps_sp[r * PPB_MAXPS + j];
        else pk.overflow = true;
    p.nf = (unsigned char)nf;
    p.nr = (unsigned char)nr;
    // the enthalpy-sum lists of the Jacobian must be the phase-space lists
    // (true without non-stoichiometric orders): the packed Jacobian reads
    // both from the slots
    {
      int cnt = 0;
      for (int j = 0; j < t->rx_hr_n[r]; j++) {
        const int sp = t->rx_hr_sp[r * PPB_MAXPS + j];
        int o = 0;
        for (int q = 0; q < nf; q++) o += (p.fsp[q] == sp);
        if ((double)o != t->rx_hr_c[r * PPB_MAXPS + j]) pk.overflow = true;
        cnt += o;
      }
      if (cnt != nf) pk.overflow = true;
      if (t->rx_rev[r]) {
        cnt = 0;
        for (int j = 0; j < t->rx_hp_n[r]; j++) {
          const int sp = t->rx_hp_sp[r * PPB_MAXPS + j];
          int o = 0;
          for (int q = 0; q < nr; q++) o += (p.rsp[q] == sp);
          if ((double)o != t->rx_hp_c[r * PPB_MAXPS + j]) pk.overflow = true;
          cnt += o;
        }
        if (cnt != nr) pk.overflow = true;
      }
    }
    if (t->rx_kc_n[r] > 6 || t->rx_jn_n[r] > 6) pk.overflow = true;
    for (int j = 0; j < t->rx_kc_n[r]; j++)
      if ((double)(signed char)t->rx_kc_c[r * PPB_MAXKC + j] != t->rx_kc_c[r * PPB_MAXKC + j]) pk.overflow = true;
    for (int j = 0; j < t->rx_jn_n[r]; j++)
      if ((double)(signed char)t->rx_jn_c[r * PPB_MAXJN + j] != t->rx_jn_c[r * PPB_MAXJN + j]) pk.overflow = true;
    for (int j = 0; j < t->rx_kc_n[r] && j < 6; j++) {
      p.kcs[j] = (unsigned char)t->rx_kc_sp[r * PPB_MAXKC + j];
      p.kcc[j] = (signed char)t->rx_kc_c[r * PPB_MAXKC + j];
    }
    for (int j = 0; j < t->rx_jn_n[r] && j < 6; j++) {
      p.jns[j] = (unsigned char)t->rx_jn_sp[r * PPB_MAXJN + j];
      p.jnc[j] = (signed char)t->rx_jn_c[r * PPB_MAXJN + j];
    }
    p.njn = (unsigned char)t->rx_jn_n[r];
    p.kind = (unsigned char)t->rx_kind[r];
    p.rev = (unsigned char)t->rx_rev[r];
    p.kcpow = (signed char)t->rx_kcpow[r];
    p.sum_nuk = (signed char)t->rx_sum_nuk[r];
    p.eff0 = (unsigned short)t->eff_off[r];
    p.effn = (unsigned short)(t->eff_off[r + 1] - t->eff_off[r]);
    p.fo = 255;
    p.rmf = (unsigned char)(t->nqss > 0 && t->rx_rmfwd[r] ? 1 : 0);
    if (t->rx_kind[r] == PPB_RX_TROE || t->rx_kind[r] == PPB_RX_LINDEMANN) {
      const double* d = t->fo_d + r * PPB_NFOD;
      const int* fi = t->fo_i + r * PPB_NFOI;
      FoPack f;
      memset(&f, 0, sizeof(f));
      f.P0 = d[PPB_FO_P0];
      f.k0 = d[PPB_FO_K0];
      f.beta0 = d[PPB_FO_BETA0];
      f.EaR0 = d[PPB_FO_EAR0];
      f.prdim = d[PPB_FO_PRDIM];
      f.a = d[PPB_FO_A];
      f.T3 = d[PPB_FO_T3];
      f.T1 = d[PPB_FO_T1];
      f.T2 = d[PPB_FO_T2];
      f.oma = d[PPB_FO_OMA];
      f.iT3 = d[PPB_FO_IT3];
      f.iT1 = d[PPB_FO_IT1];
      f.ntroe = (unsigned char)fi[PPB_FOI_NTROE];
      f.p1 = (unsigned char)fi[PPB_FOI_P1];
      f.p2 = (unsigned char)fi[PPB_FOI_P2];
      f.j1 = (unsigned char)fi[PPB_FOI_J1];
      f.j2 = (unsigned char)fi[PPB_FOI_J2];
      f.j3 = (unsigned char)fi[PPB_FOI_J3];
      f.lindemann = (unsigned char)(t->rx_kind[r] == PPB_RX_LINDEMANN);
      pk.put(off_fop + fo * sizeof(FoPack), &f, 1);
      for (int w = 0; w < 7; w++)
        pk.put(off_fow + ((size_t)w * nfo + fo) * 16, reinterpret_cast<const char*>(&f) + 16 * w, 16);
      p.fo = (unsigned char)fo++;
    }
    if (t->rx_kind[r] == PPB_RX_THIRD || t->rx_kind[r] == PPB_RX_TROE || t->rx_kind[r] == PPB_RX_LINDEMANN) {
      const double one = 1.0;
      for (int q = 0; q < N; q++) pk.put(off_effd + ((size_t)aslot * N + q) * sizeof(double), &one, 1);
      for (int e = t->eff_off[r]; e < t->eff_off[r + 1]; e++)
        pk.put(off_effd + ((size_t)aslot * N + t->eff_sp[e]) * sizeof(double), &t->eff_e[e], 1);
      p.aslot = (unsigned short)aslot++;
    }
    pk.put(off_rxp + r * sizeof(RxPack), &p, 1);
  }
  if (N > 127 || nfo > 254) pk.overflow = true;
  pk.used = off_effd + (size_t)nalpha * N * sizeof(double);
  set_off(dm.effd, off_effd);
  // Jacobian column lists (species -> reactions reaching its column)
  {
    auto reaches = [&](int r, int k) {
      const int kind = t->rx_kind[r];
      if (kind == PPB_RX_THIRD || kind == PPB_RX_TROE || kind == PPB_RX_LINDEMANN) return true;
      for (int j = 0; j < t->rx_fps_n[r]; j++)
        if (t->rx_fps_sp[r * PPB_MAXPS + j] == k) return true;
      if (t->rx_rev[r])
        for (int j = 0; j < t->rx_rps_n[r]; j++)
          if (t->rx_rps_sp[r * PPB_MAXPS + j] == k) return true;
      return false;
    };
    int jcl = 0;
    for (int k = 0; k < N; k++) {
      int c = 0;
      for (int r = 0; r < R; r++) c += reaches(r, k);
      jcl = c > jcl ? c : jcl;
    }
    jcl++; // an entry of padding ends every list
    const size_t off_jcn = (pk.used + 15) & ~size_t(15);
    const size_t off_jc = (off_jcn + N * sizeof(int) + 15) & ~size_t(15);
    // derivative of a phase space by species k: its multiplicity and the other
    // factors in species order
    auto deriv = [&](const int* sp, const double* c, int ns, int k, unsigned char (&f)[2]) {
      int mult = 0, q = 0;
      for (int j = 0; j < ns; j++) {
        int o = (int)c[j];
        if (sp[j] == k) {
          mult = o;
          o--;
        }
        for (; o > 0; o--)
          if (q < 2) f[q++] = (unsigned char)sp[j];
          else pk.wide |= WIDE_JAC;
      }
      if (mult > 15) pk.wide |= WIDE_JAC;
      return mult;
    };
    int e = 0;
    for (int k = 0; k < N; k++) {
      e = 0;
      for (int r = 0; r < R; r++) {
        if (!reaches(r, k)) continue;
        JcEntry je;
        memset(&je, 0, sizeof(je));
        je.r = (unsigned short)r;
        for (int q = 0; q < 2; q++) je.fs[q] = je.rs[q] = (unsigned char)N;
        const int kind = t->rx_kind[r];
        int mf = 0, mr = 0;
        for (int j = 0; j < t->rx_fps_n[r]; j++)
          if (t->rx_fps_sp[r * PPB_MAXPS + j] == k) mf = 1;
        if (t->rx_rev[r])
          for (int j = 0; j < t->rx_rps_n[r]; j++)
            if (t->rx_rps_sp[r * PPB_MAXPS + j] == k) mr = 1;
        if (mf) mf = deriv(t->rx_fps_sp + r * PPB_MAXPS, t->rx_fps_c + r * PPB_MAXPS, t->rx_fps_n[r], k, je.fs);
        if (mr) mr = deriv(t->rx_rps_sp + r * PPB_MAXPS, t->rx_rps_c + r * PPB_MAXPS, t->rx_rps_n[r], k, je.rs);
        je.c = (unsigned char)(mf | (mr << 4));
        je.flags = (unsigned char)((mf ? JC_INR : 0) | (mr ? JC_INP : 0));
        je.e = 1.0;
        if (kind == PPB_RX_THIRD || kind == PPB_RX_TROE || kind == PPB_RX_LINDEMANN) {
          je.flags |= JC_ALPHA;
          for (int q = t->eff_off[r]; q < t->eff_off[r + 1]; q++)
            if (t->eff_sp[q] == k) {
              je.e = t->eff_e[q];
              je.flags |= JC_LISTED;
            }
        }
        int m = 0;
        for (int j = 0; j < t->rx_jn_n[r]; j++) {
          if (t->rx_jn_c[r * PPB_MAXJN + j] == 0.0) continue;
          unsigned long long bits;
          memcpy(&bits, &t->rx_jn_c[r * PPB_MAXJN + j], 8);
          if (m >= 5 || (bits << 16)) {
            pk.wide |= WIDE_JAC;
            break;
          }
          je.nu[m] = (unsigned short)(bits >> 48);
          je.sp[m++] = (unsigned char)t->rx_jn_sp[r * PPB_MAXJN + j];
        }
        for (int w = 0; w < 2; w++)
          pk.put(off_jc + ((size_t)(2 * e + w) * N + k) * 16, reinterpret_cast<const char*>(&je) + 16 * w, 16);
        e++;
      }
      pk.put(off_jcn + k * sizeof(int), &e, 1);
      for (; e < jcl; e++) {
        const char z[16] = {};
        for (int w = 0; w < 2; w++) pk.put(off_jc + ((size_t)(2 * e + w) * N + k) * 16, z, 16);
      }
    }
    if (R > 65535) pk.overflow = true;
    pk.used = off_jc + (size_t)2 * jcl * N * 16;
    set_off(dm.jc_n, off_jcn);
    set_off(dm.jc, off_jc);
    // member lists (phase-space species only) and the third-body list
    auto member = [&](int r, int k) {
      for (int j = 0; j < t->rx_fps_n[r]; j++)
        if (t->rx_fps_sp[r * PPB_MAXPS + j] == k) return true;
      if (t->rx_rev[r])
        for (int j = 0; j < t->rx_rps_n[r]; j++)
          if (t->rx_rps_sp[r * PPB_MAXPS + j] == k) return true;
      return false;
    };
    int mtot = 0;
    for (int k = 0; k < N; k++)
      for (int r = 0; r < R; r++) mtot += member(r, k);
    const size_t off_jmoff = (pk.used + 15) & ~size_t(15);
    const size_t off_jmrx = (off_jmoff + (N + 1) * sizeof(int) + 15) & ~size_t(15);
    e = 0;
    for (int k = 0; k < N; k++) {
      pk.put(off_jmoff + k * sizeof(int), &e, 1);
      for (int r = 0; r < R; r++) {
        if (!member(r, k)) continue;
        const unsigned short rr = (unsigned short)r;
        pk.put(off_jmrx + e * sizeof(unsigned short), &rr, 1);
        e++;
      }
    }
    pk.put(off_jmoff + N * sizeof(int), &e, 1);
    pk.used = off_jmrx + (size_t)mtot * sizeof(unsigned short);
    const size_t off_aloff = (pk.used + 15) & ~size_t(15);
    const size_t off_alrx = off_aloff + 16;
    int na = 0;
    for (int r = 0; r < R; r++) {
      const int kind = t->rx_kind[r];
      if (kind != PPB_RX_THIRD && kind != PPB_RX_TROE && kind != PPB_RX_LINDEMANN) continue;
      const unsigned short rr = (unsigned short)r;
      pk.put(off_alrx + na * sizeof(unsigned short), &rr, 1);
      na++;
    }
    const int al[2] = {0, na};
    pk.put(off_aloff, al, 2);
    pk.used = off_alrx + (size_t)na * sizeof(unsigned short);
    set_off(dm.jm_off, off_jmoff);
    set_off(dm.jm_rx, off_jmrx);
    set_off(dm.al_off, off_aloff);
    set_off(dm.al_rx, off_alrx);
  }
  dm.nfo = nfo;
  set_off(dm.fow, off_fow);
  set_off(dm.rxp, off_rxp);
  set_off(dm.fop, off_fop);
  pack_rates(t, pk, dm);
  dm.wide = pk.wide;
  // SRK parameters (zeros for a mechanism without them)
  const double* srk = find_srk(t->name);
  std::vector<double> nosrk;
  if (!srk) {
    nosrk.assign((size_t)4 * N, 0.0);
    srk = nosrk.data();
  }
  set_off(dm.srk, pk.add(srk, (size_t)4 * N));
  return pk.used;
}

size_t packed_mechanism_bytes(const PPBMechTables* t)
{
  Packer pk{nullptr, 0};
  DevMech dm;
  return pack_all(t, pk, dm);
}

// Image of the tables in host memory `buf` (capacity cap) and the device
// pointer struct for the image placed at device address `dev_base`.
int pack_mechanism(const PPBMechTables* t, char* buf, size_t cap, const void* dev_base, DevMech* out)
{
  Packer pk{buf, cap};
  DevMech dm;
  pack_all(t, pk, dm);
  if (pk.overflow) return -1;
  const char* b = (const char*)dev_base;
  // every pointer member of DevMech follows the ints
  const size_t first = offsetof(DevMech, mw);
  const size_t count = (sizeof(DevMech) - first) / sizeof(void*);
  for (size_t i = 0; i < count; i++) {
    const void** slot = (const void**)((char*)&dm + first + i * sizeof(void*));
    *slot = b + (size_t)(*slot);
  }
  *out = dm;
  return 0;
}

int upload_mechanism(const PPBMechTables* t, DeviceMechanism* out)
{
  const size_t bytes = packed_mechanism_bytes(t);
  std::vector<char> img(bytes);
  void* d = nullptr;
  cudaError_t e = cudaMalloc(&d, bytes);
  if (e != cudaSuccess) return (int)e;
  DevMech dm;
  if (pack_mechanism(t, img.data(), bytes, d, &dm)) {
    cudaFree(d);
    return (int)cudaErrorInvalidValue;
  }
  e = cudaMemcpy(d, img.data(), bytes, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    return (int)e;
  }
  out->host = t;
  cudaGetDevice(&out->device);
  out->blob = d;
  out->dm = new DevMech(dm);
  return 0;
}

void free_mechanism(DeviceMechanism* m)
{
  if (m->blob) cudaFree(m->blob);
  delete m->dm;
  m->blob = nullptr;
  m->dm = nullptr;
}

size_t team_cell_bytes(const PPBMechTables* t, int lu_fp32)
{
  return lu_fp32 ? team_bytes<float>(t->nsp, t->nrxn, t->nqss, t->nrq)
                 : team_bytes<double>(t->nsp, t->nrxn, t->nqss, t->nrq);
}

#define PPB_DECL(NS)                                                                                              \
  int launch_react_##NS(const DeviceMechanism&, const Options&, int, const LaunchConfig&, Batch, double, int*,      \
                        cudaStream_t);                                                                             \
  int launch_ajacobian_##NS(const DevMech&, const double*, const double*, int, double*, int, int, cudaStream_t);      \
  int react_occupancy_##NS(const DevMech&, int, const LaunchConfig&);
PPB_DECL(9)
PPB_DECL(13)
PPB_DECL(22)
PPB_DECL(39)
PPB_DECL(21)
PPB_DECL(53)
PPB_DECL(88)

#define PPB_DECL_ARK(NS) int launch_ark_##NS(const DeviceMechanism&, const ArkParams&, const ArkBuffers&, int*, cudaStream_t);
PPB_DECL_ARK(9)
PPB_DECL_ARK(21)
PPB_DECL_ARK(53)
PPB_DECL_ARK(88)

int launch_ark(const DeviceMechanism& m, const ArkParams& P, const ArkBuffers& B, int* grid, cudaStream_t st)
{
  switch (m.host->nsp) {
  case 9: return launch_ark_9(m, P, B, grid, st);
  case 21: return launch_ark_21(m, P, B, grid, st);
  case 53: return launch_ark_53(m, P, B, grid, st);
  case 88: return launch_ark_88(m, P, B, grid, st);
  default: return (int)cudaErrorNotSupported;
  }
}

int launch_react(const DeviceMechanism& m, const Options& o, int method, const LaunchConfig& lc, Batch b,
                 double dt, int* queue, cudaStream_t st)
{
  switch (m.host->nsp) {
  case 9:
    return launch_react_9(m, o, method, lc, b, dt, queue, st);
  case 13:
    return launch_react_13(m, o, method, lc, b, dt, queue, st);
  case 22:
    return launch_react_22(m, o, method, lc, b, dt, queue, st);
  case 39:
    return launch_react_39(m, o, method, lc, b, dt, queue, st);
  case 21:
    return launch_react_21(m, o, method, lc, b, dt, queue, st);
  case 53:
    return launch_react_53(m, o, method, lc, b, dt, queue, st);
  case 88:
    return launch_react_88(m, o, method, lc, b, dt, queue, st);
  default:
    return (int)cudaErrorNotSupported;
  }
}

int react_occupancy(const DeviceMechanism& m, int method, const LaunchConfig& lc)
{
  const DevMech& M = *m.dm;
  switch (M.nsp) {
  case 9: return react_occupancy_9(M, method, lc);
  case 13: return react_occupancy_13(M, method, lc);
  case 22: return react_occupancy_22(M, method, lc);
  case 39: return react_occupancy_39(M, method, lc);
  case 21: return react_occupancy_21(M, method, lc);
  case 53: return react_occupancy_53(M, method, lc);
  case 88: return react_occupancy_88(M, method, lc);
  default: return 0;
  }
}

// ------------------------------------------------------------ layout
// Tiled transpose through shared memory: AoS rows of nc_aos doubles per cell
// (first ncomp used) <-> species-major planes of leading dimension ld.
__global__ void k_aos_to_soa(const double* __restrict__ aos, int nc_aos, double* __restrict__ soa, int ld,
                             int ncomp, int ncells)
{
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int c = c0 + r, i = i0 + threadIdx.x;
    if (c < ncells && i < ncomp) tile[r][threadIdx.x] = aos[(size_t)c * nc_aos + i];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r, c = c0 + threadIdx.x;
    if (c < ncells && i < ncomp) soa[(size_t)i * ld + c] = tile[threadIdx.x][r];
  }
}

__global__ void k_soa_to_aos(const double* __restrict__ soa, int ld, int ncomp, double* __restrict__ aos, int nc_aos,
                             int ncells)
{
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r, c = c0 + threadIdx.x;
    if (c < ncells && i < ncomp) tile[threadIdx.x][r] = soa[(size_t)i * ld + c];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int c = c0 + r, i = i0 + threadIdx.x;
    if (c < ncells && i < ncomp) aos[(size_t)c * nc_aos + i] = tile[r][threadIdx.x];
  }
}

int launch_aos_to_soa(const double* aos, int nc_aos, double* soa, int ld, int ncomp, int ncells, cudaStream_t st)
{
  if (ncells <= 0 || ncomp <= 0) return 0;
  dim3 grid((ncells + 31) / 32, (ncomp + 31) / 32), block(32, 8);
  k_aos_to_soa<<<grid, block, 0, st>>>(aos, nc_aos, soa, ld, ncomp, ncells);
  return (int)cudaGetLastError();
}

int launch_soa_to_aos(const double* soa, int ld, int ncomp, double* aos, int nc_aos, int ncells, cudaStream_t st)
{
  if (ncells <= 0 || ncomp <= 0) return 0;
  dim3 grid((ncells + 31) / 32, (ncomp + 31) / 32), block(32, 8);
  k_soa_to_aos<<<grid, block, 0, st>>>(soa, ld, ncomp, aos, nc_aos, ncells);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------ pointwise

// One thread per cell touches only sc, g and wdot of the point layout (the
// net-rate scratch serves the teams): the extent of its local buffer.
__host__ __device__ inline size_t point1_doubles(int N) { return 3 * ((size_t)N + 1); }

template <int TEAM>
__global__ void k_production_rate(DevMech M, const double* sc, const double* T, double* wdot, int ncells)
{
  extern __shared__ __align__(16) double psm[];
  Team<TEAM> tm;
  const int N = M.nsp;
  const int per_block = blockDim.x / TEAM;
  const int slot = threadIdx.x / TEAM;
  const int c = blockIdx.x * per_block + slot;
  double local[8 * 96];
  const size_t pd = point_doubles(N, M.nrxn, false);
  double* base = (TEAM == 1) ? local : psm + (size_t)slot * (pd + point_qss_doubles(N, M.nqss, M.nrq));
  if (TEAM == 1 && c >= ncells) return;
  const int cc = c < ncells ? c : ncells - 1;
  double* s_sc = base;
  double* s_g = base + (N + 1);
  double* s_w = base + 2 * (N + 1);
  double* s_qd = base + 8 * (N + 1);
  double* qco = nullptr;
  if (M.nqss > 0) { // the QSS tail: sc and g over all slots, the solve's scratch
    s_sc = base + (TEAM == 1 ? point1_doubles(N) : pd);
    s_g = s_sc + (N + 1 + M.nqss);
    qco = s_g + (N + 1 + M.nqss);
  }
  for (int s = tm.lane; s < N; s += TEAM) s_sc[s] = sc[(size_t)cc * N + s];
  if (tm.lane == 0) s_sc[N] = 1.0; // padding slot of the packed reaction records
  tm.sync();
  RateScratch rs{s_sc, s_g, s_qd, nullptr, qco};
  production_rate<TEAM>(tm, M, s_w, s_sc, T[cc], rs);
  if (c < ncells)
    for (int s = tm.lane; s < N; s += TEAM) wdot[(size_t)c * N + s] = s_w[s];
}

template <int TEAM>
__global__ void k_t_from_energy(DevMech M, int eh, const double* e, const double* Y, double* T, int ncells)
{
  Team<TEAM> tm;
  const int per_block = blockDim.x / TEAM;
  const int c = blockIdx.x * per_block + threadIdx.x / TEAM;
  if (TEAM == 1 && c >= ncells) return;
  const int cc = c < ncells ? c : ncells - 1;
  double t = T[cc];
  t_from_energy<TEAM>(tm, M, eh, e[cc], Y + (size_t)cc * M.nsp, t);
  if (c < ncells && tm.lane == 0) T[c] = t;
}

// doubles of one cell of k_reactor_rhs (with the QSS tail of a QSS
// mechanism); one thread per cell uses the first 8 (N + 1) and the tail
// (its rates need no net-rate scratch), placed there
__host__ __device__ inline size_t rhs_point_doubles(const DevMech& M, bool one_thread)
{
  const size_t n = M.nsp + 1;
  return (one_thread ? 8 * n : 10 * n + M.nrxn) + point_qss_doubles(M.nsp, M.nqss, M.nrq);
}

template <int TEAM, bool QSS>
__global__ void k_reactor_rhs(DevMech M, int rtype, double t, const double* y, const double* rhoe,
                              const double* rhoesrc, const double* src, double* ydot, int ncells)
{
  extern __shared__ __align__(16) double psm[];
  Team<TEAM> tm;
  const int N = M.nsp, n = N + 1;
  const int per_block = blockDim.x / TEAM;
  const int slot = threadIdx.x / TEAM;
  const int c = blockIdx.x * per_block + slot;
  double local[10 * 96];
  if (TEAM == 1 && c >= ncells) return;
  const int cc = c < ncells ? c : ncells - 1;
  double* base = (TEAM == 1) ? local : psm + (size_t)slot * rhs_point_doubles(M, false);
  double* s_y = base;
  double* s_f = base + n;
  double* s_src = base + 2 * n;
  double* Yb = base + 3 * n;
  double* scb = base + 4 * n;
  double* gb = base + 5 * n;
  double* wb = base + 6 * n;
  double* eb = base + 7 * n;
  double* qd = base + 10 * n;
  double* qco = nullptr;
  if (M.nqss > 0) { // the QSS tail: sc and g over all slots, the solve's scratch
    scb = base + (TEAM == 1 ? 8 * n : 10 * n + M.nrxn);
    gb = scb + (n + M.nqss);
    qco = gb + (n + M.nqss);
  }
  for (int i = tm.lane; i < n; i += TEAM) {
    s_y[i] = y[(size_t)cc * n + i];
    s_src[i] = (i < N) ? src[(size_t)cc * N + i] : 0.0;
  }
  tm.sync();
  reactor_rhs<TEAM, QSS>(tm, M, rtype, t, s_y, s_f, rhoe[cc], rhoesrc[cc], s_src, Yb, scb, gb, qd, wb, eb, qco);
  if (c < ncells)
    for (int i = tm.lane; i < n; i += TEAM) ydot[(size_t)c * n + i] = s_f[i];
}

int launch_production_rate(const DeviceMechanism& m, const double* sc, const double* T, double* wdot, int ncells,
                           int team, cudaStream_t st)
{
  const DevMech& M = *m.dm;
  if (ncells <= 0) return 0;
  if (team == 1) {
    // one thread per cell: the cell's arrays in an 8 x 96-double local buffer
    if (point1_doubles(M.nsp) + point_qss_doubles(M.nsp, M.nqss, M.nrq) > 8 * 96) return (int)cudaErrorNotSupported;
    k_production_rate<1><<<(ncells + 63) / 64, 64, 0, st>>>(M, sc, T, wdot, ncells);
  } else {
    const int cells_per_block = 4;
    const size_t shm =
      (point_doubles(M.nsp, M.nrxn, false) + point_qss_doubles(M.nsp, M.nqss, M.nrq)) * 8 * cells_per_block;
    cudaFuncSetAttribute((const void*)k_production_rate<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
    k_production_rate<32><<<(ncells + cells_per_block - 1) / cells_per_block, 32 * cells_per_block, shm, st>>>(
      M, sc, T, wdot, ncells);
  }
  return (int)cudaGetLastError();
}

#define PPB_ADJ_DECL(NS)                                                                                          \
  int plan_adjoint_##NS(const DevMech& M, int mode, int lu_fp32, AdjPlan* p);                                      \
  int launch_adjoint_##NS(const DevMech& M, const Options& o, int mode, int lu_fp32, const AdjPlan& p,             \
                          const AdjBatch& b, const AdjLayout& L, double dt, int* queue, double* grad,              \
                          int accumulate, cudaStream_t st);                                                        \
  int launch_rhs_exact_##NS(const DevMech& M, int rtype, double t, const double* y, const double* rhoe,            \
                            const double* rhoesrc, const double* src, const double* v, double* f_out,              \
                            double* J_out, double* fE_out, double* vy_out, double* vE_out, double* vp_out,         \
                            int ncells, cudaStream_t st);
PPB_ADJ_DECL(9)
PPB_ADJ_DECL(21)
PPB_ADJ_DECL(53)
PPB_ADJ_DECL(88)
#undef PPB_ADJ_DECL
#define PPB_ADJB_DECL(NS)                                                                                         \
  int launch_adjoint_batched_##NS(const DevMech& M, const Options& o, int lu_fp32, const AdjBatch& b, AdjCells& C, \
                                  double dt, int* queue, double* grad, int accumulate, AdjGrow grow, void* ctx,    \
                                  cudaStream_t st);                                                               \
  size_t adj_cp_bytes_##NS(int lu_fp32);
PPB_ADJB_DECL(9)
PPB_ADJB_DECL(21)
PPB_ADJB_DECL(53)
PPB_ADJB_DECL(88)
#undef PPB_ADJB_DECL

int launch_adjoint_batched(const DeviceMechanism& m, const Options& o, int lu_fp32, const AdjBatch& b, AdjCells& C,
                           double dt, int* queue, double* grad, int accumulate, AdjGrow grow, void* grow_ctx,
                           cudaStream_t st)
{
  const DevMech& M = *m.dm;
#define PPB_B(NS) return launch_adjoint_batched_##NS(M, o, lu_fp32, b, C, dt, queue, grad, accumulate, grow, grow_ctx, st)
  switch (M.nsp) {
  case 9: PPB_B(9);
  case 21: PPB_B(21);
  case 53: PPB_B(53);
  case 88: PPB_B(88);
  default: return (int)cudaErrorNotSupported;
  }
#undef PPB_B
}

size_t adj_cp_bytes(int N, int lu_fp32)
{
  switch (N) {
  case 9: return adj_cp_bytes_9(lu_fp32);
  case 21: return adj_cp_bytes_21(lu_fp32);
  case 53: return adj_cp_bytes_53(lu_fp32);
  case 88: return adj_cp_bytes_88(lu_fp32);
  default: return 0;
  }
}

size_t adj_item_bytes(int N, int R)
{
  // [Jc n*n][AT n*n][fE n][ek n][dq R][4 scalars][n pivots], 16-byte aligned
  const size_t n = N + 1;
  size_t stride = 2 * n * n + 2 * n + (size_t)R + 4 + (n + 1) / 2;
  stride = (stride + 1) & ~size_t(1);
  return stride * 8;
}

int plan_adjoint(const DeviceMechanism& m, int mode, int lu_fp32, AdjPlan* p)
{
  const DevMech& M = *m.dm;
  switch (M.nsp) {
  case 9: return plan_adjoint_9(M, mode, lu_fp32, p);
  case 21: return plan_adjoint_21(M, mode, lu_fp32, p);
  case 53: return plan_adjoint_53(M, mode, lu_fp32, p);
  case 88: return plan_adjoint_88(M, mode, lu_fp32, p);
  default: return (int)cudaErrorNotSupported;
  }
}

int launch_adjoint(const DeviceMechanism& m, const Options& o, int mode, int lu_fp32, const AdjPlan& p,
                   const AdjBatch& b, const AdjLayout& L, double dt, int* queue, double* grad, int accumulate,
                   cudaStream_t st)
{
  const DevMech& M = *m.dm;
  switch (M.nsp) {
  case 9: return launch_adjoint_9(M, o, mode, lu_fp32, p, b, L, dt, queue, grad, accumulate, st);
  case 21: return launch_adjoint_21(M, o, mode, lu_fp32, p, b, L, dt, queue, grad, accumulate, st);
  case 53: return launch_adjoint_53(M, o, mode, lu_fp32, p, b, L, dt, queue, grad, accumulate, st);
  case 88: return launch_adjoint_88(M, o, mode, lu_fp32, p, b, L, dt, queue, grad, accumulate, st);
  default: return (int)cudaErrorNotSupported;
  }
}

int launch_rhs_exact(const DeviceMechanism& m, int rtype, double t, const double* y, const double* rhoe,
                     const double* rhoesrc, const double* src, const double* v, double* f_out, double* J_out,
                     double* fE_out, double* vy_out, double* vE_out, double* vp_out, int ncells, cudaStream_t st)
{
  const DevMech& M = *m.dm;
#define PPB_RX(NS)                                                                                                 \
  return launch_rhs_exact_##NS(M, rtype, t, y, rhoe, rhoesrc, src, v, f_out, J_out, fE_out, vy_out, vE_out, vp_out, \
                               ncells, st)
  switch (M.nsp) {
  case 9: PPB_RX(9);
  case 21: PPB_RX(21);
  case 53: PPB_RX(53);
  case 88: PPB_RX(88);
  default: return (int)cudaErrorNotSupported;
  }
#undef PPB_RX
}

int launch_ajacobian(const DeviceMechanism& m, const double* sc, const double* T, int consP, double* J, int ncells,
                     int team, cudaStream_t st)
{
  if (ncells <= 0) return 0;
  const DevMech& M = *m.dm;
  switch (M.nsp) {
  case 9:
    return launch_ajacobian_9(M, sc, T, consP, J, ncells, team, st);
  case 13:
    return launch_ajacobian_13(M, sc, T, consP, J, ncells, team, st);
  case 22:
    return launch_ajacobian_22(M, sc, T, consP, J, ncells, team, st);
  case 39:
    return launch_ajacobian_39(M, sc, T, consP, J, ncells, team, st);
  case 21:
    return launch_ajacobian_21(M, sc, T, consP, J, ncells, team, st);
  case 53:
    return launch_ajacobian_53(M, sc, T, consP, J, ncells, team, st);
  case 88:
    return launch_ajacobian_88(M, sc, T, consP, J, ncells, team, st);
  default:
    return (int)cudaErrorNotSupported;
  }
}

int launch_t_from_energy(const DeviceMechanism& m, int eh, const double* e, const double* Y, double* T, int ncells,
                         int team, cudaStream_t st)
{
  if (ncells <= 0) return 0;
  const DevMech& M = *m.dm;
  if (team == 1) {
    k_t_from_energy<1><<<(ncells + 63) / 64, 64, 0, st>>>(M, eh, e, Y, T, ncells);
  } else {
    k_t_from_energy<32><<<(ncells + 3) / 4, 128, 0, st>>>(M, eh, e, Y, T, ncells);
  }
  return (int)cudaGetLastError();
}

int launch_reactor_rhs(const DeviceMechanism& m, int reactor_type, double t, const double* y, const double* rhoe,
                       const double* rhoesrc, const double* src, double* ydot, int ncells, int team,
                       cudaStream_t st)
{
  if (ncells <= 0) return 0;
  const DevMech& M = *m.dm;
  if (team == 1) {
    // one thread per cell: the cell's arrays in a 10 x 96-double local buffer
    if (rhs_point_doubles(M, true) > 10 * 96) return (int)cudaErrorNotSupported;
    k_reactor_rhs<1, false><<<(ncells + 63) / 64, 64, 0, st>>>(M, reactor_type, t, y, rhoe, rhoesrc, src, ydot,
                                                                 ncells);
  } else {
    const int cells_per_block = 4;
    const size_t shm = rhs_point_doubles(M, false) * 8 * cells_per_block;
    auto k = M.nqss > 0 ? k_reactor_rhs<32, true> : k_reactor_rhs<32, false>;
    cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
    k<<<(ncells + cells_per_block - 1) / cells_per_block, 32 * cells_per_block, shm, st>>>(
      M, reactor_type, t, y, rhoe, rhoesrc, src, ydot, ncells);
  }
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------ box path
// ReactorUtils.H:160-220 (box_flatten) for one cell per thread: Array4 views
// -> species-major batch, T recomputed from the energy with the stored T as
// the Newton start.
__device__ inline long a4(const BoxView& v, int i, int j, int k, int n)
{
  return (long)(i - v.lo[0]) + (long)(j - v.lo[1]) * v.jstride + (long)(k - v.lo[2]) * v.kstride + (long)n * v.nstride;
}

__device__ inline long a4i(const BoxViewI& v, int i, int j, int k, int n)
{
  return (long)(i - v.lo[0]) + (long)(j - v.lo[1]) * v.jstride + (long)(k - v.lo[2]) * v.kstride + (long)n * v.nstride;
}

__global__ void k_box_flatten(DevMech M, int rtype, int clean, BoxArgs a, Batch b)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= b.ncells) return;
  const int lx = a.hi[0] - a.lo[0] + 1, ly = a.hi[1] - a.lo[1] + 1;
  const int i = a.lo[0] + c % lx, j = a.lo[1] + (c / lx) % ly, k = a.lo[2] + c / (lx * ly);
  const int N = M.nsp;
  int* mk = const_cast<int*>(b.mask);
  if (mk) mk[c] = a.mask.p ? a.mask.p[a4i(a.mask, i, j, k, 0)] : 1;
  double Y[96];
  double rho_old = 0.0, rho = 0.0;
  if (clean)
    for (int n = 0; n < N; n++) rho_old += a.rY.p[a4(a.rY, i, j, k, n)];
  for (int n = 0; n < N; n++) {
    const double v = a.rY.p[a4(a.rY, i, j, k, n)];
    const double rYn = clean ? fmin(fmax(0.0, v), rho_old) : v;
    b.y[(size_t)n * b.ld + c] = rYn;
    b.src[(size_t)n * b.ld + c] = a.rYsrc.p[a4(a.rYsrc, i, j, k, n)];
    rho += rYn;
    Y[n] = rYn;
  }
  const double rinv = 1.0 / rho;
  for (int n = 0; n < N; n++) Y[n] *= rinv;
  double T = a.T.p[a4(a.T, i, j, k, 0)];
  const double rE = a.rE.p[a4(a.rE, i, j, k, 0)];
  const_cast<double*>(b.rhoe)[c] = rE;
  const_cast<double*>(b.rhoesrc)[c] = a.rEs.p[a4(a.rEs, i, j, k, 0)];
  Team<1> tm;
  t_from_energy<1>(tm, M, rtype == 2, rE * rinv, Y, T);
  b.y[(size_t)N * b.ld + c] = T;
}

// ReactorUtils.H:222-291 (box_unflatten): batch -> Array4 views, energy
// advanced by dt * source, T from the new energy, FC = cost (0 if masked).
__global__ void k_box_unflatten(DevMech M, int rtype, int clean, BoxArgs a, Batch b, double dt)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= b.ncells) return;
  const int lx = a.hi[0] - a.lo[0] + 1, ly = a.hi[1] - a.lo[1] + 1;
  const int i = a.lo[0] + c % lx, j = a.lo[1] + (c / lx) % ly, k = a.lo[2] + c / (lx * ly);
  const int N = M.nsp;
  if (b.mask && b.mask[c] == -1) {
    a.FC.p[a4(a.FC, i, j, k, 0)] = 0.0;
    return;
  }
  double Y[96];
  double rho_old = 0.0, rho_oc = 0.0, rho = 0.0;
  if (clean) {
    for (int n = 0; n < N; n++) rho_old += a.rY.p[a4(a.rY, i, j, k, n)];
    for (int n = 0; n < N; n++) {
      Y[n] = fmin(fmax(0.0, a.rY.p[a4(a.rY, i, j, k, n)]), rho_old);
      rho_oc += Y[n];
    }
  }
  for (int n = 0; n < N; n++) {
    const long idx = a4(a.rY, i, j, k, n);
    const double yv = b.y[(size_t)n * b.ld + c];
    const double rYn = clean ? a.rY.p[idx] + (yv - Y[n]) * rho_old / rho_oc : yv;
    a.rY.p[idx] = rYn;
    rho += rYn;
    Y[n] = rYn;
  }
  const double rinv = 1.0 / rho;
  for (int n = 0; n < N; n++) Y[n] *= rinv;
  double T = b.y[(size_t)N * b.ld + c];
  const long ie = a4(a.rE, i, j, k, 0);
  const double rE = b.rhoe[c] + dt * a.rEs.p[a4(a.rEs, i, j, k, 0)];
  a.rE.p[ie] = rE;
  Team<1> tm;
  t_from_energy<1>(tm, M, rtype == 2, rE * rinv, Y, T);
  a.T.p[a4(a.T, i, j, k, 0)] = T;
  a.FC.p[a4(a.FC, i, j, k, 0)] = a.fcunt ? (double)a.fcunt[c] : (double)(b.nfe ? b.nfe[c] : 0);
}

int launch_box_flatten(const DeviceMechanism& m, int rtype, int clean, const BoxArgs& a, Batch b, cudaStream_t st)
{
  if (b.ncells <= 0) return 0;
  k_box_flatten<<<(b.ncells + 127) / 128, 128, 0, st>>>(*m.dm, rtype, clean, a, b);
  return (int)cudaGetLastError();
}

int launch_box_unflatten(const DeviceMechanism& m, int rtype, int clean, const BoxArgs& a, Batch b, double dt,
                         cudaStream_t st)
{
  if (b.ncells <= 0) return 0;
  k_box_unflatten<<<(b.ncells + 127) / 128, 128, 0, st>>>(*m.dm, rtype, clean, a, b, dt);
  return (int)cudaGetLastError();
}

// rX += dt * rX_src on device arrays (the flat path's energy update,
// ReactorCvode.cpp:1652-1655)
__global__ void k_energy_update(double* rX, const double* rXs, double dt, int n)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) rX[c] = rX[c] + dt * rXs[c];
}

#ifdef PPB_PHASE_TIMERS
// the counters of every kernel object (one per species count and part)
#define PPB_PHASE_DECL(NS)                                                                                        \
  int phase_cycles_##NS##_p0(unsigned long long*, int);                                                           \
  int phase_cycles_##NS##_p1(unsigned long long*, int);                                                           \
  int phase_cycles_##NS##_p2(unsigned long long*, int);                                                           \
  int phase_cycles_##NS##_p3(unsigned long long*, int);                                                           \
  int phase_cycles_##NS##_p4(unsigned long long*, int);
#define PPB_PHASE_FNS(NS) phase_cycles_##NS##_p0, phase_cycles_##NS##_p1, phase_cycles_##NS##_p2, \
                          phase_cycles_##NS##_p3, phase_cycles_##NS##_p4
PPB_PHASE_DECL(9)
PPB_PHASE_DECL(13)
PPB_PHASE_DECL(21)
PPB_PHASE_DECL(22)
PPB_PHASE_DECL(39)
PPB_PHASE_DECL(53)
PPB_PHASE_DECL(88)

int phase_cycles(unsigned long long* out, int reset)
{
  for (int q = 0; q < PH_COUNT; q++) out[q] = 0;
  int (*fns[])(unsigned long long*, int) = {PPB_PHASE_FNS(9),  PPB_PHASE_FNS(13), PPB_PHASE_FNS(21),
                                            PPB_PHASE_FNS(22), PPB_PHASE_FNS(39), PPB_PHASE_FNS(53),
                                            PPB_PHASE_FNS(88)};
  for (auto fn : fns) {
    unsigned long long part[PH_COUNT];
    const int e = fn(part, reset);
    if (e) return e;
    for (int q = 0; q < PH_COUNT; q++) out[q] += part[q];
  }
  return 0;
}

#endif

int launch_energy_update(double* rX, const double* rX_src, double dt, int ncells, cudaStream_t st)
{
  if (ncells <= 0) return 0;
  k_energy_update<<<(ncells + 255) / 256, 256, 0, st>>>(rX, rX_src, dt, ncells);
  return (int)cudaGetLastError();
}

size_t cost_order_tmp_bytes(int n)
{
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, (const int*)nullptr, (int*)nullptr, (const int*)nullptr,
                                            (int*)nullptr, n);
  return bytes;
}

int launch_cost_order(const int* cost, int* keys_tmp, const int* iota, int* order, void* tmp, size_t tmp_bytes,
                      int n, cudaStream_t st)
{
  if (n <= 0) return 0;
  size_t bytes = tmp_bytes;
  return (int)cub::DeviceRadixSort::SortPairsDescending(tmp, bytes, cost, keys_tmp, iota, order, n, 0,
                                                        (int)(8 * sizeof(int)), st);
}

__global__ void k_iota(int* a, int n)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = i;
}

int launch_iota(int* a, int n, cudaStream_t st)
{
  if (n <= 0) return 0;
  k_iota<<<(n + 255) / 256, 256, 0, st>>>(a, n);
  return (int)cudaGetLastError();
}

// Fuego::PYT2RE / PYT2RH (Source/Eos/Fuego.H:313-327): density from P, T, Y
// (CKRHOY) and the mass-specific internal energy (eh = 0) or enthalpy
// (eh = 1) at T.
__global__ void k_pyt2re(DevMech M, int eh, const double* P, const double* T, const double* Y, double* rho, double* e,
                         int ncells)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const double* y = Y + (size_t)c * M.nsp;
  const double t = T[c];
  double yow = 0.0;
  for (int s = 0; s < M.nsp; s++) yow += y[s] * __ldg(M.imw + s);
  rho[c] = P[c] / (RU * t * yow);
  Team<1> tm;
  e[c] = mix_e<1>(tm, M, eh, t, y);
}

int launch_pyt2re(const DeviceMechanism& m, int eh, const double* P, const double* T, const double* Y, double* rho,
                  double* e, int ncells, cudaStream_t st)
{
  if (ncells <= 0) return 0;
  k_pyt2re<<<(ncells + 127) / 128, 128, 0, st>>>(*m.dm, eh, P, T, Y, rho, e, ncells);
  return (int)cudaGetLastError();
}

// Peak FP64 FMA throughput of the device: every thread runs 8 independent
// FMA chains; 2 flops per FMA.
__global__ void k_fp64_probe(double* out, int iters)
{
  double a[8];
#pragma unroll
  for (int j = 0; j < 8; j++) a[j] = threadIdx.x * 1e-9 + j;
  const double m = 0.999999999, c = 1e-9;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = fma(a[j], m, c);
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 8; j++) s += a[j];
  if (s == 12345.678) out[0] = s; // never true; keeps the chains live
}

int probe_fp64_peak(double* gflops, cudaStream_t st)
{
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  double* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 8);
  if (e != cudaSuccess) return (int)e;
  const int threads = 256, blocks = nsm * 8, iters = 4096;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  k_fp64_probe<<<blocks, threads, 0, st>>>(d, iters); // warm-up
  cudaEventRecord(a, st);
  const int reps = 5;
  for (int r = 0; r < reps; r++) k_fp64_probe<<<blocks, threads, 0, st>>>(d, iters);
  cudaEventRecord(b, st);
  e = cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(d);
  if (e != cudaSuccess) return (int)e;
  const double flops = 2.0 * 8.0 * iters * (double)threads * blocks * reps;
  *gflops = flops / (ms * 1e-3) / 1e9;
  return (int)cudaGetLastError();
}

} // namespace ppb
