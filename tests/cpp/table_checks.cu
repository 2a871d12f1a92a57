// Mechanism tables made at run time from a shipped mechanism with some of its
// reactions replaced, run through the engine's own packing, upload and
// launches (tests/test_table_limits.py).
#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <utility>
#include <vector>

#include "ppb_engine.h"
#include "ppb_work.cuh"

using namespace ppb;

namespace {
struct Mech {
  PPBMechTables t;
  DeviceMechanism d;
  std::vector<std::vector<int>> ints;
  std::vector<std::vector<double>> doubles;
  // a writable copy of n entries of a table
  int* own(const int*& p, size_t n)
  {
    ints.emplace_back(p, p + n);
    p = ints.back().data();
    return ints.back().data();
  }
  double* own(const double*& p, size_t n)
  {
    doubles.emplace_back(p, p + n);
    p = doubles.back().data();
    return doubles.back().data();
  }
};

void set_list(const int* n, const int* sp, const double* c, int width, int r, const std::map<int, int>& l, int sign = 1)
{
  int k = 0;
  for (auto& e : l) {
    if (!e.second) continue;
    const_cast<int*>(sp)[r * width + k] = e.first;
    const_cast<double*>(c)[r * width + k] = sign * e.second;
    k++;
  }
  const_cast<int*>(n)[r] = k;
}

// sum_r |nu| (|q_f| + |q_r|) per species, one thread per cell
__global__ void k_rate_scale(DevMech M, const double* sc, const double* T, double* out, int n)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double s[96], g[96];
  const int N = M.nsp;
  const double t = T[c], invT = 1.0 / t, logT = log(t), refC = 101325 / 8.31446 * invT;
  double mix = 0.0;
  for (int k = 0; k < N; k++) {
    s[k] = sc[(size_t)c * N + k];
    g[k] = g_RT(M, k, t, invT, logT);
    mix += s[k];
    out[(size_t)c * N + k] = 0.0;
  }
  s[N] = 1.0;
  g[N] = 0.0;
  for (int r = 0; r < M.nrxn; r++) {
    double qf, qr;
    rxn_qdot(M, r, t, invT, logT, refC, 1 / refC, mix, s, g, &qf, &qr);
    for (int j = 0; j < M.wup_n[r]; j++)
      out[(size_t)c * N + M.wup_sp[r * PPB_MAXW + j]] += fabs(M.wup_c[r * PPB_MAXW + j]) * (fabs(qf) + fabs(qr));
  }
}
} // namespace

extern "C" {
void* tc_new(const char* name)
{
  const PPBMechTables* b = find_mechanism(name);
  if (!b) return nullptr;
  Mech* m = new Mech;
  m->t = *b;
  PPBMechTables& t = m->t;
  const size_t R = t.nrxn;
  m->own(t.rx_kind, R), m->own(t.rx_rev, R), m->own(t.rx_kcpow, R), m->own(t.rx_sum_nuk, R);
  m->own(t.rx_A, R), m->own(t.rx_beta, R), m->own(t.rx_EaR, R);
  m->own(t.rx_fps_n, R), m->own(t.rx_fps_sp, R * PPB_MAXPS), m->own(t.rx_fps_c, R * PPB_MAXPS);
  m->own(t.rx_rps_n, R), m->own(t.rx_rps_sp, R * PPB_MAXPS), m->own(t.rx_rps_c, R * PPB_MAXPS);
  m->own(t.rx_kc_n, R), m->own(t.rx_kc_sp, R * PPB_MAXKC), m->own(t.rx_kc_c, R * PPB_MAXKC);
  m->own(t.rx_wup_n, R), m->own(t.rx_wup_sp, R * PPB_MAXW), m->own(t.rx_wup_c, R * PPB_MAXW);
  m->own(t.rx_jn_n, R), m->own(t.rx_jn_sp, R * PPB_MAXJN), m->own(t.rx_jn_c, R * PPB_MAXJN);
  m->own(t.rx_hr_n, R), m->own(t.rx_hr_sp, R * PPB_MAXPS), m->own(t.rx_hr_c, R * PPB_MAXPS);
  m->own(t.rx_hp_n, R), m->own(t.rx_hp_sp, R * PPB_MAXPS), m->own(t.rx_hp_c, R * PPB_MAXPS);
  return m;
}

void tc_free(void* h)
{
  Mech* m = (Mech*)h;
  if (m->d.blob) free_mechanism(&m->d);
  delete m;
}

// reaction r becomes sum nu_f sp_f <=> sum nu_p sp_p, A T^beta exp(-EaR / T)
void tc_reaction(void* h, int r, int nf, const int* sf, const int* of, int np, const int* sp, const int* op, double A,
                 double beta, double EaR)
{
  PPBMechTables& t = ((Mech*)h)->t;
  std::map<int, int> f, p, net;
  int order = 0;
  for (int j = 0; j < nf; j++) f[sf[j]] += of[j], net[sf[j]] -= of[j], order -= of[j];
  for (int j = 0; j < np; j++) p[sp[j]] += op[j], net[sp[j]] += op[j], order += op[j];
  const_cast<int*>(t.rx_kind)[r] = 0;
  const_cast<int*>(t.rx_rev)[r] = 1;
  const_cast<int*>(t.rx_kcpow)[r] = order;
  const_cast<double*>(t.rx_sum_nuk)[r] = order;
  const_cast<double*>(t.rx_A)[r] = A;
  const_cast<double*>(t.rx_beta)[r] = beta;
  const_cast<double*>(t.rx_EaR)[r] = EaR;
  set_list(t.rx_fps_n, t.rx_fps_sp, t.rx_fps_c, PPB_MAXPS, r, f);
  set_list(t.rx_rps_n, t.rx_rps_sp, t.rx_rps_c, PPB_MAXPS, r, p);
  set_list(t.rx_hr_n, t.rx_hr_sp, t.rx_hr_c, PPB_MAXPS, r, f);
  set_list(t.rx_hp_n, t.rx_hp_sp, t.rx_hp_c, PPB_MAXPS, r, p);
  set_list(t.rx_kc_n, t.rx_kc_sp, t.rx_kc_c, PPB_MAXKC, r, net, -1);
  set_list(t.rx_wup_n, t.rx_wup_sp, t.rx_wup_c, PPB_MAXW, r, net);
  set_list(t.rx_jn_n, t.rx_jn_sp, t.rx_jn_c, PPB_MAXJN, r, net);
}

// the first n plain reactions get a third body
void tc_third(void* h, int n)
{
  PPBMechTables& t = ((Mech*)h)->t;
  for (int r = 0; r < t.nrxn && n > 0; r++)
    if (t.rx_kind[r] == 0) const_cast<int*>(t.rx_kind)[r] = PPB_RX_THIRD, n--;
}

// the first net coefficient of reaction r in the production rates
void tc_coefficient(void* h, int r, double c) { const_cast<double*>(((Mech*)h)->t.rx_wup_c)[r * PPB_MAXW] = c; }

// n more QSS species with the first one's thermo and no reaction
void tc_more_qss(void* h, int n)
{
  Mech* m = (Mech*)h;
  PPBMechTables& t = m->t;
  const int slots = t.nsp + 1 + t.nqss, first = t.nsp + 1;
  auto more = [&](const double*& p, int nc) {
    std::vector<double> v(p, p + (size_t)slots * nc);
    for (int q = 0; q < n; q++) v.insert(v.end(), p + (size_t)first * nc, p + (size_t)(first + 1) * nc);
    m->doubles.push_back(v);
    p = m->doubles.back().data();
  };
  more(t.tmid, 1);
  more(t.th_cv, 10), more(t.th_cp, 10), more(t.th_dcp, 8), more(t.th_u, 12), more(t.th_h, 12), more(t.th_g, 14);
  std::vector<int> off(t.q_off, t.q_off + t.nqss + 1);
  off.insert(off.end(), n, off.back());
  m->ints.push_back(off);
  t.q_off = m->ints.back().data();
  t.nqss += n;
}

// packs the tables into host memory: 0 or -1 (refused)
int tc_pack(void* h)
{
  const PPBMechTables& t = ((Mech*)h)->t;
  std::vector<char> img(packed_mechanism_bytes(&t));
  DevMech dm;
  return pack_mechanism(&t, img.data(), img.size(), nullptr, &dm);
}

int tc_upload(void* h)
{
  Mech* m = (Mech*)h;
  return upload_mechanism(&m->t, &m->d);
}

int tc_rates(void* h, const double* sc, const double* T, double* wdot, int n, int team)
{
  return launch_production_rate(((Mech*)h)->d, sc, T, wdot, n, team, nullptr);
}

int tc_rate_scale(void* h, const double* sc, const double* T, double* out, int n)
{
  k_rate_scale<<<(n + 31) / 32, 32>>>(*((Mech*)h)->d.dm, sc, T, out, n);
  return (int)cudaGetLastError();
}

int tc_jacobian(void* h, const double* sc, const double* T, int consP, double* J, int n, int team)
{
  return launch_ajacobian(((Mech*)h)->d, sc, T, consP, J, n, team, nullptr);
}

// react, species-major; engine 0 plain, 1 tuned (4 warps a block); work: n + 1 ints
int tc_react(void* h, int engine, double* y, double* src, const double* rhoe, const double* rhoesrc, int* work, int n,
             double dt)
{
  Options o{};
  o.rtol = o.atol = 1e-10;
  o.max_order = 5, o.max_steps = 10000, o.max_nls_iters = 3, o.max_err_fails = 100, o.jac_eval_freq = 100;
  o.reactor_type = 1;
  Batch b{};
  b.y = y, b.src = src, b.rhoe = rhoe, b.rhoesrc = rhoesrc, b.status = work + 1, b.ncells = b.ld = n;
  LaunchConfig lc;
  lc.engine = engine ? ENGINE_TUNED : ENGINE_PLAIN;
  return launch_react(((Mech*)h)->d, o, METHOD_BDF, lc, b, dt, work, nullptr);
}
}
