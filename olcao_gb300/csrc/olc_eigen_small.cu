// Batched generalised Hermitian eigen-solver for small n, one CTA per k-point,
// everything in shared memory (FP64).
//
// Same mathematical steps as LAPACK zhegv (itype 1, 'V', 'U'), the routine the
// reference calls in solveZHEGV (src/olcao/interfaces.F90:73-120):
//   1. S = U^H U                      (zpotrf 'U'; info = n + j when the
//                                      leading minor j is not positive)
//   2. C = U^{-H} H U^{-1}            (zhegst itype 1)
//   3. C = V diag(w) V^H              here: cyclic Jacobi in FP32, refined to
//                                      FP64 rounding by residual products
//                                      (olc_jacobi.cuh)
//   4. X = U^{-1} V                   (back-transform, X^H S X = I)
// Eigenvalues are returned in ascending order with their vectors.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "olc_common.h"
#include "olc_jacobi.cuh"

namespace olc {

namespace {

constexpr int kSmallMaxN = jac::kMaxN;
using jac::cd;
using jac::cmul;
using jac::csub;

// Threads per pencil: about one per element of a column block of C V; fewer for
// the smallest, whose phases are bound by their barriers.
inline int threads_for(int n) { return n <= 16 ? 64 : n <= 24 ? 128 : 256; }

// One CTA per pencil.  Bound by the FP64 pipe (n = 32: about 0.9 million FP64
// operations per pencil, 4.6 million with FP64 sweeps throughout): 8192 pencils
// of n = 32 take 18.8 ms (73.0 before), 343 of n = 26 0.66 ms (2.29).
__global__ void __launch_bounds__(256) small_hegv_kernel(
    const double* __restrict__ hin, double* __restrict__ sin_, int n, int num_states,
    int s_factored, double* __restrict__ eig_out, double* __restrict__ vec_out,
    int32_t* __restrict__ info_out, double* __restrict__ trace_out) {
  extern __shared__ double smem[];
  const int k = blockIdx.x;
  const int tid = threadIdx.x;
  const int ld = jac::lead(n);
  const size_t nn = (size_t)n * n, ml = (size_t)n * ld;
  cd* U = reinterpret_cast<cd*>(smem);          // column-major, U[col * ld + row]
  cd* C = U + ml;
  cd* W = C + ml;
  cd* T = W + ml;
  __shared__ jac::Shared sh;

  const cd* Hg = reinterpret_cast<const cd*>(hin) + (size_t)k * nn;
  cd* Sg = reinterpret_cast<cd*>(sin_) + (size_t)k * nn;     // receives the factor
  for (int i = tid; i < (int)nn; i += blockDim.x) {
    const int at = (i / n) * ld + i % n;
    U[at] = Sg[i];
    C[at] = Hg[i];
  }
  jac::hegv_reduced(U, C, W, T, n, ld, s_factored != 0, Sg, sh, trace_out ? trace_out + (size_t)k * 82 : nullptr);
  if (sh.fail) {
    if (tid == 0 && info_out) info_out[k] = sh.fail;
    for (int i = tid; i < num_states; i += blockDim.x) eig_out[(size_t)k * num_states + i] = 0.0;
    return;
  }
  // ---- eigenvalues, sort, back-transform X = U^{-1} V ---------------------
  jac::sorted_order(n, sh);
  for (int i = tid; i < num_states; i += blockDim.x) eig_out[(size_t)k * num_states + i] = sh.w[sh.order[i]];
  if (vec_out) {
    for (int i = tid; i < (int)nn; i += blockDim.x) W[(i / n) * ld + i % n] = Sg[i];
    __syncthreads();
    // row r of every vector finished, then taken out of the rows above it
    for (int r = n - 1; r >= 0; --r) {
      const double inv = sh.dinv[r];
      for (int c = tid; c < n; c += blockDim.x) {
        cd& x = U[(size_t)c * ld + r];
        x.x *= inv;
        x.y *= inv;
      }
      __syncthreads();
      for (int e = tid; e < r * n; e += blockDim.x) {
        const int q = e % r, c = e / r;
        cd& x = U[(size_t)c * ld + q];
        x = csub(x, cmul(W[(size_t)r * ld + q], U[(size_t)c * ld + r]));
      }
      __syncthreads();
    }
    cd* X = reinterpret_cast<cd*>(vec_out) + (size_t)k * n * num_states;
    for (int i = tid; i < n * num_states; i += blockDim.x)
      X[i] = U[(size_t)sh.order[i / n] * ld + i % n];
  }
  if (tid == 0 && info_out) info_out[k] = 0;
}

}  // namespace

// Largest n sent to the batched in-shared-memory solver.  OLC_SMALL_SOLVER_MAX_N
// lowers it (0 routes every size to the library path; used to cross-check the
// two solvers on the same matrices).
int small_solver_max_n() {
  static int v = -1;
  if (v < 0) {
    v = kSmallMaxN;
    if (const char* e = std::getenv("OLC_SMALL_SOLVER_MAX_N")) v = std::min(kSmallMaxN, std::atoi(e));
  }
  return v;
}

// The shared memory of the largest pencil, for every launch: a limit set to the
// launch's own need could be lowered by another thread before it.
static int allow_smem() {
  return cuda_check(cudaFuncSetAttribute(small_hegv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)jac::smem_bytes(jac::kMaxN)),
                    "smem attribute");
}

// s_full is overwritten with its Cholesky factors.
int solve_small_batched(olc_context* ctx, const double* h_full, double* s_full, int n,
                        int num_states, double* eigenvalues, double* vectors, int32_t* info_host,
                        bool s_is_factored) {
  const int nk = ctx->dims.num_kpoints;
  const size_t smem = jac::smem_bytes(n);
  int st;
  if ((st = allow_smem())) return st;
  int32_t* dinfo = nullptr;
  if ((st = cuda_check(ctx_malloc(ctx, (void**)&dinfo, sizeof(int32_t) * nk, ctx->stream), "malloc info"))) return st;
  StageScope scope(ctx, OLC_STAGE_SOLVE);
  // OLC_SMALL_SOLVER_TRACE=1 prints each k-point's convergence history
  double* dtrace = nullptr;
  static const bool trace = std::getenv("OLC_SMALL_SOLVER_TRACE") != nullptr;
  if (trace) {
    const size_t tl = 82 * (size_t)nk;
    cudaMalloc(&dtrace, sizeof(double) * tl);
    cudaMemset(dtrace, 0, sizeof(double) * tl);
  }
  small_hegv_kernel<<<nk, threads_for(n), smem, ctx->stream>>>(h_full, s_full, n, num_states,
                                                         s_is_factored ? 1 : 0, eigenvalues,
                                                         vectors, dinfo, dtrace);
  if (dtrace) {
    std::vector<double> ht(82 * (size_t)nk);
    cudaMemcpy(ht.data(), dtrace, sizeof(double) * ht.size(), cudaMemcpyDeviceToHost);
    for (int k = 0; k < nk; ++k) {
      std::fprintf(stderr, "k=%d", k);
      for (int q = 0; q < 8 && ht[82 * k + 2 * q + 1] != 0.0; ++q)
        std::fprintf(stderr, " %.2e", ht[82 * k + 2 * q] / ht[82 * k + 2 * q + 1]);
      std::fprintf(stderr, "\n");
    }
    cudaFree(dtrace);
  }
  st = cuda_check(cudaGetLastError(), "small_hegv_kernel");
  std::vector<int32_t> hinfo(nk, 0);
  cudaMemcpyAsync(hinfo.data(), dinfo, sizeof(int32_t) * nk, cudaMemcpyDeviceToHost, ctx->stream);
  cudaFreeAsync(dinfo, ctx->stream);
  int s2 = cuda_check(cudaStreamSynchronize(ctx->stream), "small solve sync");
  if (st) return st;
  if (s2) return s2;
  int worst = 0;
  for (int k = 0; k < nk; ++k) {
    if (info_host) info_host[k] = hinfo[k];
    if (hinfo[k] && !worst) worst = hinfo[k];
  }
  if (worst > n) return fail(OLC_ERR_NOT_PD, "ZHEGV: overlap matrix not positive definite");
  if (worst) return fail(OLC_ERR_EIGEN, "eigen-solver did not converge");
  return OLC_OK;
}

// Launches the batched solver on full Hermitian h, s [nk][n][n] (s overwritten) with no
// allocation and no synchronisation (info is device memory).
int launch_small_hegv_raw(cudaStream_t stream, const double* h_full, double* s_full, int n,
                          int nk, int num_states, double* eigenvalues, double* vectors,
                          int32_t* info_dev) {
  const size_t smem = jac::smem_bytes(n);
  int st;
  if ((st = allow_smem())) return st;
  count_launch();
  small_hegv_kernel<<<nk, threads_for(n), smem, stream>>>(h_full, s_full, n, num_states, 0, eigenvalues,
                                                    vectors, info_dev, nullptr);
  return cuda_check(cudaGetLastError(), "small_hegv_kernel");
}

int small_solver_capacity_n() { return kSmallMaxN; }

}  // namespace olc
