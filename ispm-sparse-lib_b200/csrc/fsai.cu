// Factorized sparse approximate inverse built on the GPU.
//
// The reference builds its approximate inverse on the host, one factor row
// after another (right-looking AINV, fastainv/fastainv.cpp:395-566): every
// row update depends on the rows before it.  Here each row of a lower
// triangular factor G is independent -- the classic FSAI construction:
//
//     P_i = { j <= i : a_ij != 0 }            (the row's lower pattern of A)
//     A[P_i, P_i] y = e_i,   g_i = y / sqrt(y_i)
//
// so that diag(G A G^T) = 1 and M = G^T G ~ A^-1, with G's non-zeros on A's
// lower triangle.  On the 27-point GRF systems this preconditioner needs a
// few per cent more PCG iterations than the AINV factor with droptol 0.01
// while holding ~5% fewer non-zeros, and it is built in milliseconds instead
// of seconds.
//
// A group of lanes per row gathers the |P_i| x |P_i| local matrix (|P_i| <=
// 32), factors it (L D L^T) and back-substitutes.  FP64 throughout.  A local
// matrix that is not positive definite (indefinite A) falls back to the Jacobi row e_i / sqrt(a_ii) when a_ii > 0, else to e_i,
// and is counted.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "cuda_util.cuh"
#include "fsai.h"

namespace ispm {
namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kMaxPattern = 32;

// One factor row per group of G lanes (G = 4, 8, 16 or 32, the smallest that
// holds the longest pattern), 32 / G rows a warp; lane l owns row l of the
// local matrix in registers, KM columns of it (the longest pattern, rounded
// up).
//
// What bounds it: shared-memory and L1 wavefronts (81% of their rate on the
// 72^3 27-point matrix, issue slots 68%, DRAM 4%).  A row of that stencil (K =
// 14) needs about 110 FP64 multiply-adds a lane fed by shared-memory
// broadcasts, and its 14 x 14 local matrix comes from 14 rows of A that
// neighbouring factor rows share through L1; the bytes (12 per entry of A, 8
// per entry of G) are a fraction of that time.  373,248 rows take 0.44 ms;
// one warp a row with a walk per lane, a Cholesky factorization in shared
// memory and a serial back-substitution took 3.39 ms.  So:
//  * the group reads each row of A it needs as one coalesced run (the entries
//    from the diagonal on, the half the factorization uses) and finds their
//    places in the pattern by a binary search in shared memory, instead of a
//    lane walking a whole row entry by entry;
//  * L D L^T without square roots: column k goes once through shared memory
//    (unscaled), every lane updates its own row from broadcast reads, and one
//    reciprocal serves the column;
//  * the last row of L^-1, z = L^-T e, is all that the factor row needs
//    (g = z / sqrt(d_last)): one lane-parallel back-substitution, reading the
//    stored columns.
template <int G, int KM>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
    fsai_rows_kernel(int n, const int *__restrict__ a_rp, const int *__restrict__ a_ci,
                     const double *__restrict__ a_v, const int *__restrict__ g_rp,
                     double *__restrict__ g_v, unsigned *fallbacks)
{
  constexpr int R = 32 / G;   // rows a warp
  constexpr int LD = G + 2;   // row length: even (16-byte reads), rows on distinct banks
  constexpr int B = G < 8 ? G : 8;  // pattern rows whose loads are in flight together
  constexpr int kNone = 0x7fffffff;
  __shared__ __align__(16) double sm[kWarpsPerBlock * R][G][LD];
  __shared__ int pats[kWarpsPerBlock * R][G];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & (G - 1), grp = threadIdx.x / G;
  double(*S)[LD] = sm[grp];
  int *pat = pats[grp];
  const long long row = (long long)blockIdx.x * (kWarpsPerBlock * R) + grp;
  const bool live = row < n;  // a group past the end keeps its warp company with K = 0
  const int i = live ? (int)row : 0;
  const int g0 = live ? __ldg(g_rp + i) : 0;
  const int K = live ? __ldg(g_rp + i + 1) - g0 : 0;  // pattern = first K entries of row i
  const int kw = __reduce_max_sync(full, K);
  const int p = lane < K ? __ldg(a_ci + __ldg(a_rp + i) + lane) : kNone;
  pat[lane] = p;
  // row p of A from its diagonal on
  int start = 0, stop = 0;
  if (lane < K) {
    start = __ldg(a_rp + p) + (__ldg(g_rp + p + 1) - __ldg(g_rp + p)) - 1;
    stop = __ldg(a_rp + p + 1);
  }
#pragma unroll
  for (int k = 0; k < G; k += 2)
    *reinterpret_cast<double2 *>(&S[lane][k]) = make_double2(0.0, 0.0);
  __syncwarp();
  // S[r][c] = a(p_c, p_r), r >= c
  for (int c0 = 0; c0 < kw; c0 += B) {
    int col[B];
    double val[B];
#pragma unroll
    for (int q = 0; q < B; q++) {
      const int e = __shfl_sync(full, start, c0 + q, G) + lane;
      const bool in = e < __shfl_sync(full, stop, c0 + q, G);
      col[q] = in ? __ldg(a_ci + e) : kNone;
      val[q] = in ? __ldg(a_v + e) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < B; q++) {
      int e = 0, end = -1;  // (formed when a run goes on past the group)
      for (;;) {
        if (col[q] <= i) {
          int at = 0;
#pragma unroll
          for (int s = G / 2; s > 0; s >>= 1)
            at = pat[at + s] <= col[q] ? at + s : at;
          if (pat[at] == col[q])
            S[at][c0 + q] = val[q];
        }
        // a longer run: on while its last entry is still left of column i
        if (!__any_sync(full, lane == G - 1 && col[q] < i))
          break;
        if (end < 0) {
          e = __shfl_sync(full, start, c0 + q, G) + lane;
          end = __shfl_sync(full, stop, c0 + q, G);
        }
        e += G;
        const bool in = col[q] < i && e < end;
        col[q] = in ? __ldg(a_ci + e) : kNone;
        val[q] = in ? __ldg(a_v + e) : 0.0;
      }
    }
  }
  __syncwarp();
  double a[KM];
#pragma unroll
  for (int k = 0; k < KM; k += 2) {
    const double2 v = *reinterpret_cast<const double2 *>(&S[lane][k]);
    a[k] = v.x;
    a[k + 1] = v.y;
  }
  if (lane >= K) {  // identity past the pattern
#pragma unroll
    for (int k = 0; k < KM; k++)
      a[k] = k == lane ? 1.0 : 0.0;
  }
  __syncwarp();
  bool ok = true;
  double rd_own = 1.0, d_own = 1.0;
#pragma unroll
  for (int k = 0; k < KM; k++) {
    if (k < kw) {
      S[k][lane] = a[k];  // column k, unscaled (the lanes k .. are read)
      __syncwarp();
      const double d = S[k][k];
      ok = ok && d > 0.0;
      const double rd = 1.0 / d;
      if (lane == k) {
        rd_own = rd;
        d_own = d;
      }
      const double l = a[k] * rd;
#pragma unroll
      for (int j = (k + 1) & ~1; j < KM; j += 2) {
        const double2 u = *reinterpret_cast<const double2 *>(&S[k][j]);
        if (j > k)
          a[j] = fma(-l, u.x, a[j]);
        a[j + 1] = fma(-l, u.y, a[j + 1]);
      }
    }
  }
  __syncwarp();
  double s = 0.0, z = lane == K - 1 ? 1.0 : 0.0;
#pragma unroll
  for (int c = KM - 1; c > 0; c--) {
    if (c < kw) {
      const double zc = __shfl_sync(full, z, c, G);
      s = fma(S[lane][c], zc, s);  // used by the lanes left of c alone
      if (lane == c - 1 && c < K)
        z = -rd_own * s;
    }
  }
  const double dl = __shfl_sync(full, d_own, K > 0 ? K - 1 : 0, G);
  if (lane < K) {
    double g = z / sqrt(dl);
    if (!ok) {
      // Jacobi row on the diagonal entry (the last pattern slot is i)
      const double aii = __ldg(a_v + __ldg(a_rp + i) + K - 1);
      g = lane < K - 1 ? 0.0 : aii > 0.0 ? 1.0 / sqrt(aii) : 1.0;
      if (lane == 0)
        atomicAdd(fallbacks, 1u);
    }
    g_v[g0 + lane] = g;
  }
}

template <int G, int KM>
void launch_rows(int n, const int *a_rp, const int *a_ci, const double *a_v, const int *g_rp,
                 double *g_v, unsigned *fb, cudaStream_t s)
{
  const int rows = kWarpsPerBlock * (32 / G);
  fsai_rows_kernel<G, KM><<<(n + rows - 1) / rows, kWarpsPerBlock * 32, 0, s>>>(n, a_rp, a_ci, a_v,
                                                                            g_rp, g_v, fb);
}

}  // namespace

int fsai_lower_pattern(int n, const int *rp, const int *ci, std::vector<int> &g_rp,
                       std::vector<int> &g_ci)
{
  g_rp.assign(n + 1, 0);
  for (int i = 0; i < n; i++) {
    int cnt = 0, last = -1;
    for (int e = rp[i]; e < rp[i + 1]; e++) {
      if (ci[e] <= last || ci[e] < 0 || ci[e] >= n)
        return fail(ISPM_ERR_INVALID, "row %d columns not strictly increasing in [0, n)", i);
      last = ci[e];
      if (ci[e] <= i)
        cnt++;
    }
    if (cnt == 0 || ci[rp[i] + cnt - 1] != i)
      return fail(ISPM_ERR_INVALID, "row %d has no diagonal entry", i);
    if (cnt > kMaxPattern)
      return fail(ISPM_ERR_TOO_LARGE, "row %d has %d lower entries (at most %d)", i, cnt,
                  kMaxPattern);
    g_rp[i + 1] = g_rp[i] + cnt;
  }
  g_ci.resize(g_rp[n]);
  for (int i = 0; i < n; i++)
    std::copy(ci + rp[i], ci + rp[i] + (g_rp[i + 1] - g_rp[i]), g_ci.begin() + g_rp[i]);
  return ISPM_OK;
}

void fsai_transpose_pattern(int n, const std::vector<int> &g_rp, const std::vector<int> &g_ci,
                            std::vector<int> &t_rp, std::vector<int> &t_ci,
                            std::vector<unsigned> &t_of)
{
  // G^T in CSR; t_of[k] = position in G^T of G's entry k
  t_rp.assign(n + 1, 0);
  for (int c : g_ci)
    t_rp[c + 1]++;
  for (int i = 0; i < n; i++)
    t_rp[i + 1] += t_rp[i];
  t_ci.resize(g_ci.size());
  t_of.resize(g_ci.size());
  std::vector<int> fill(t_rp.begin(), t_rp.end() - 1);
  for (int i = 0; i < n; i++)
    for (int e = g_rp[i]; e < g_rp[i + 1]; e++) {
      const int at = fill[g_ci[e]]++;
      t_ci[at] = i;
      t_of[e] = (unsigned)at;
    }
}

int fsai_max_pattern(const std::vector<int> &g_rp)
{
  int k = 0;
  for (size_t i = 0; i + 1 < g_rp.size(); i++)
    k = std::max(k, g_rp[i + 1] - g_rp[i]);
  return k;
}

int fsai_build_values(int n, int max_pattern, const int *a_rp_d, const int *a_ci_d,
                      const double *a_v_d, const int *g_rp_d, double *g_v_d,
                      unsigned *fallbacks_d, cudaStream_t s)
{
  if (max_pattern > kMaxPattern)
    return fail(ISPM_ERR_INVALID, "FSAI pattern of %d entries (at most %d)", max_pattern,
                kMaxPattern);
  const auto rows = [](int k) {
    switch ((k + 1) / 2) {
    case 0:
    case 1:
    case 2: return launch_rows<4, 4>;
    case 3: return launch_rows<8, 6>;
    case 4: return launch_rows<8, 8>;
    case 5: return launch_rows<16, 10>;
    case 6: return launch_rows<16, 12>;
    case 7: return launch_rows<16, 14>;
    case 8: return launch_rows<16, 16>;
    case 9:
    case 10: return launch_rows<32, 20>;
    case 11:
    case 12: return launch_rows<32, 24>;
    case 13:
    case 14: return launch_rows<32, 28>;
    default: return launch_rows<32, 32>;
    }
  }(max_pattern);
  rows(n, a_rp_d, a_ci_d, a_v_d, g_rp_d, g_v_d, fallbacks_d, s);
  cudaError_t e = cudaPeekAtLastError();
  return e == cudaSuccess ? ISPM_OK : fail(ISPM_ERR_CUDA, "fsai rows: %s", cudaGetErrorString(e));
}

}  // namespace ispm

using namespace ispm;

namespace {

struct Scoped {
  std::vector<void *> p;
  ~Scoped()
  {
    for (void *q : p)
      cudaFree(q);
  }
  template <class T> int get(T **out, size_t count, const T *init = nullptr)
  {
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(ISPM_ERR_NOMEM, "cudaMalloc: %s", cudaGetErrorString(e));
    }
    p.push_back(q);
    *out = (T *)q;
    if (init && count)
      ISPM_CUDA_TRY(cudaMemcpy(q, init, count * sizeof(T), cudaMemcpyHostToDevice));
    return ISPM_OK;
  }
};

}  // namespace

extern "C" int ispm_fsai_sym_gpu(int out_dtype, int n, const int *row_ptr, const int *cols,
                                 const double *elms, ispm_csr **ainv1, ispm_csr **ainv2,
                                 unsigned *fallbacks)
{
  clear_error();
  if (!ainv1 || !ainv2)
    return fail(ISPM_ERR_INVALID, "output pointers are NULL");
  *ainv1 = *ainv2 = nullptr;
  if (n <= 0 || !row_ptr || (row_ptr[n] && (!cols || !elms)))
    return fail(ISPM_ERR_INVALID, "bad CSR");
  if (out_dtype != ISPM_F32 && out_dtype != ISPM_F64)
    return fail(ISPM_ERR_INVALID, "out_dtype %d", out_dtype);
  std::vector<int> g_rp, g_ci, t_rp, t_ci;
  std::vector<unsigned> t_of;
  if (int e = fsai_lower_pattern(n, row_ptr, cols, g_rp, g_ci))
    return e;
  fsai_transpose_pattern(n, g_rp, g_ci, t_rp, t_ci, t_of);
  const size_t nnz_a = (size_t)row_ptr[n], nnz_g = g_ci.size();
  Scoped mem;
  int *a_rp, *a_ci, *gr;
  double *a_v, *g_v;
  unsigned *fb;
  if (int e = mem.get(&a_rp, (size_t)n + 1, row_ptr))
    return e;
  if (int e = mem.get(&a_ci, nnz_a, cols))
    return e;
  if (int e = mem.get(&a_v, nnz_a, elms))
    return e;
  if (int e = mem.get(&gr, (size_t)n + 1, g_rp.data()))
    return e;
  if (int e = mem.get(&g_v, nnz_g))
    return e;
  if (int e = mem.get(&fb, 1))
    return e;
  ISPM_CUDA_TRY(cudaMemset(fb, 0, sizeof(unsigned)));
  if (int e = fsai_build_values(n, fsai_max_pattern(g_rp), a_rp, a_ci, a_v, gr, g_v, fb, 0))
    return e;
  std::vector<double> gv(nnz_g);
  ISPM_CUDA_TRY(cudaMemcpy(gv.data(), g_v, nnz_g * sizeof(double), cudaMemcpyDeviceToHost));
  unsigned nfb = 0;
  ISPM_CUDA_TRY(cudaMemcpy(&nfb, fb, sizeof(unsigned), cudaMemcpyDeviceToHost));
  if (fallbacks)
    *fallbacks = nfb;
  ispm_csr *g1 = new (std::nothrow) ispm_csr, *g2 = new (std::nothrow) ispm_csr;
  if (!g1 || !g2) {
    delete g1;
    delete g2;
    return fail(ISPM_ERR_NOMEM, "host allocation");
  }
  // Ainv1 = G (lower), Ainv2 = G^T, so Ainv2 Ainv1 = G^T G ~ A^-1 as for fastainv_sym
  for (ispm_csr *g : {g1, g2}) {
    g->m.n_rows = g->m.n_cols = n;
    g->m.n_nz = (int)nnz_g;
    g->m.dtype = out_dtype;
  }
  g1->m.row_ptr = g_rp;
  g1->m.cols = g_ci;
  g2->m.row_ptr = t_rp;
  g2->m.cols = t_ci;
  std::vector<double> tv(nnz_g);
  for (size_t k = 0; k < nnz_g; k++)
    tv[t_of[k]] = gv[k];
  if (out_dtype == ISPM_F64) {
    g1->m.elms_d = std::move(gv);
    g2->m.elms_d = std::move(tv);
  } else {
    g1->m.elms_f.assign(gv.begin(), gv.end());
    g2->m.elms_f.assign(tv.begin(), tv.end());
  }
  *ainv1 = g1;
  *ainv2 = g2;
  return ISPM_OK;
}
