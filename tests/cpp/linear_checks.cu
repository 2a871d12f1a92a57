// The team factorisation and solve of the integrator on given matrices, beside
// the one-thread factorisation and the solve that divides
// (tests/test_linear_algebra.py).  One block and one matrix a team.
#include "ppb_work.cuh"
#include "ppb_adjoint.cuh"

using namespace ppb;

namespace {
// A: [m][n n] column-major; b: [m][r][n].  Out: return codes, pivots and
// factors (one thread, team), dinv[0], solutions (dividing, register).
template <int TEAM, typename LT, int n>
__global__ void k_factor_solve(const double* A, const double* b, int r, int* ret, int* piv, double* lu, double* dinv0,
                               double* x)
{
  extern __shared__ __align__(16) char smem[];
  __shared__ double red[TEAM > 32 ? 4 * (TEAM / 32) : 1];
  if (threadIdx.x >= TEAM) return;
  const Team<TEAM> tm(red);
  double* v = (double*)smem;
  double *v2 = v + n, *dinv = v2 + n;
  LT* At = (LT*)(dinv + n);
  LT* As = At + n * (n + 1);
  int* pt = (int*)(As + n * n + (n & 1));
  int *ps = pt + n, *perm = ps + n, *rs = perm + n;
  const size_t c = blockIdx.x;
  for (int i = tm.lane; i < n * n; i += TEAM) At[i] = As[i] = (LT)A[c * n * n + i];
  tm.sync();
  if (tm.lane == 0) *rs = lu_factor<LT>(As, n, ps);
  tm.sync();
  const int rt = lu_factor_team<TEAM, LT, (n + Team<TEAM>::W - 1) / Team<TEAM>::W>(tm, At, n, pt);
  if (tm.lane == 0) {
    ret[2 * c] = *rs;
    ret[2 * c + 1] = rt;
  }
  if (rt) return;
  for (int i = tm.lane; i < n; i += TEAM) perm[i] = (int)At[n * n + i];
  diag_recip(tm, At, dinv, n);
  if (tm.lane == 0) dinv0[c] = dinv[0];
  for (int i = tm.lane; i < n; i += TEAM) {
    piv[(2 * c) * n + i] = ps[i];
    piv[(2 * c + 1) * n + i] = pt[i];
  }
  for (int i = tm.lane; i < n * n; i += TEAM) {
    lu[(2 * c) * n * n + i] = As[i];
    lu[(2 * c + 1) * n * n + i] = At[i];
  }
  for (int k = 0; k < r; k++) {
    for (int i = tm.lane; i < n; i += TEAM) v[i] = v2[i] = b[(c * r + k) * n + i];
    tm.sync();
    lu_solve<TEAM, LT>(tm, At, n, pt, v);
    lu_solve_reg<TEAM, LT, n>(tm, At, pt, perm, dinv, v2);
    for (int i = tm.lane; i < n; i += TEAM) {
      x[((2 * c) * r + k) * n + i] = v[i];
      x[((2 * c + 1) * r + k) * n + i] = v2[i];
    }
    tm.sync();
  }
}

// (I - gamma J)^-1 b (or of the transpose) by the adjoint's factorisation
template <int NS>
__global__ void k_adj(const double* J, double gamma, int transpose, const double* b, int* ret, double* x)
{
  extern __shared__ __align__(16) char smem[];
  constexpr int n = NS + 1;
  Team<32> tm;
  double* v = (double*)smem;
  double* Jc = v + n;
  double* A = Jc + n * n;
  int* piv = (int*)(A + n * (n + 1));
  const size_t c = blockIdx.x;
  for (int i = tm.lane; i < n * n; i += 32) Jc[i] = J[c * n * n + i];
  for (int i = tm.lane; i < n; i += 32) v[i] = b[c * n + i];
  tm.sync();
  const int rc = adj_factor<32, NS>(tm, n, Jc, gamma, transpose != 0, A, piv);
  if (tm.lane == 0) ret[c] = rc;
  if (rc) return;
  adj_solve<32>(tm, A, n, piv, v);
  for (int i = tm.lane; i < n; i += 32) x[c * n + i] = v[i];
}

template <int TEAM, typename LT, int n>
int factor_solve(const double* A, const double* b, int m, int r, int* ret, int* piv, double* lu, double* dinv0,
                 double* x)
{
  const size_t shm = 24 * n + sizeof(LT) * (n * (2 * n + 1) + 1) + 12 * n + 16;
  auto k = k_factor_solve<TEAM, LT, n>;
  cudaError_t e = cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
  if (e != cudaSuccess) return (int)e;
  k<<<m, TEAM < 32 ? 32 : TEAM, shm>>>(A, b, r, ret, piv, lu, dinv0, x);
  return (int)cudaGetLastError();
}
} // namespace

extern "C" int lc_factor_solve(int team, int fp32, int n, const double* A, const double* b, int m, int r, int* ret,
                               int* piv, double* lu, double* dinv0, double* x)
{
#define LC(T, N)                                                                                                      \
  if (team == T && n == N)                                                                                            \
    return fp32 ? factor_solve<T, float, N>(A, b, m, r, ret, piv, lu, dinv0, x)                                       \
                : factor_solve<T, double, N>(A, b, m, r, ret, piv, lu, dinv0, x);
  LC(16, 10) LC(16, 22) LC(32, 10) LC(32, 22) LC(32, 32) LC(32, 33) LC(32, 54) LC(32, 89)
  LC(64, 54) LC(128, 54) LC(128, 89) LC(256, 89)
  return -1;
}

extern "C" int lc_adjoint(int ns, const double* J, double gamma, int transpose, const double* b, int m, int* ret,
                          double* x)
{
#define LCA(NS)                                                                                                       \
  if (ns == NS) {                                                                                                     \
    const size_t shm = 8 * ((NS + 1) * (2 * NS + 4)) + 4 * (NS + 1);                                                  \
    cudaError_t e = cudaFuncSetAttribute((const void*)k_adj<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,          \
                                         (int)shm);                                                                   \
    if (e != cudaSuccess) return (int)e;                                                                              \
    k_adj<NS><<<m, 32, shm>>>(J, gamma, transpose, b, ret, x);                                                        \
    return (int)cudaGetLastError();                                                                                   \
  }
  LCA(9) LCA(31) LCA(32) LCA(53) LCA(64) LCA(88)
  return -1;
}
