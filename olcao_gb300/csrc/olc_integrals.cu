// Integral stages of the hot path on sm_103a.
//
// Stage 1 (primitive kernels, one thread per alpha-pair item, one launch per
//   angular class so a warp runs one straight-line recurrence):  the reference's
//   alpha loop body -- overlap2CIntg / kinetic2CIntg / massvel2CIntg
//   (integrals.F90:312-416, 1150-1236)
//   and the third-centre sums of nuclearPE / electronicPE (integrals.F90:
//   2275-2598) -- producing the harmonic block sh(lm1, lm2) of each item in
//   a scratch buffer.
// Stage 2 (contraction, one CTA per (pair, cell) task and column block): the
//   accumulation into pairXBasisFn2 and multWithBasisFn1 (integrals.F90:
//   402-410, intgSaving.F90:56-89), in the same two steps,
//   block(m1,m2) = sum c1(a1,m1) c2(a2,m2) sh(lm(m1), lm(m2)).
// Stage 3 (Bloch sum + scatter, one CTA per (pair, k range)):
//   applyPhaseFactors, kPointLatticeOriginShift and saveCurrentPair
//   (intgSaving.F90:95-505) -- out(m1,m2,k) = e^{ik.L} sum_R e^{ik.R} block_R
//   written straight into valeVale / coreVale / coreCore.
#include <algorithm>
#include <cstdio>

#include "olc_prim_kernel.cuh"

namespace olc {

// ---------------------------------------------------------------------------
// stage 1: primitive kernels
// ---------------------------------------------------------------------------
template <int OP, bool FAR32>
int launch_class(olc_context* ctx, cudaStream_t stream, int cls, const double* coeffs, int ep_type, int ep_alpha,
                 bool accumulate) {
  const ItemLists& it = ctx->items;
  PrimArgs a;
  a.task = it.task[cls];
  a.ab = it.ab[cls];
  a.n = it.count[cls];
  a.out = ctx->d_sh + it.sh_offset[cls];
  a.coeffs = coeffs;
  a.accumulate = accumulate ? 1 : 0;
  a.ep_type = ep_type;
  a.ep_alpha = ep_alpha;
  if (a.n == 0) return OLC_OK;
  a.log_split = 0;
  if (OP == OLC_OP_NUCLEAR || OP == OLC_OP_ELECPOT)
    while (a.log_split < 5 && ((long long)a.n << (a.log_split + 1)) <= kThirdWave) ++a.log_split;
  const dim3 block(kThirdThreads),
      grid((unsigned)((((long long)a.n << a.log_split) + kThirdThreads - 1) / kThirdThreads));
  StageScope scope(ctx, OLC_STAGE_PRIMITIVES);
  const int l1 = cls / (kMaxL + 1), l2 = cls % (kMaxL + 1);
  if (l1 == 3 || l2 == 3) {
    switch (OP) {
      case OLC_OP_OVERLAP: return launch_prim_f_overlap(stream, ctx->view, a, l1, l2, grid, block);
      case OLC_OP_KINETIC: return launch_prim_f_kinetic(stream, ctx->view, a, l1, l2, grid, block);
      case OLC_OP_MASSVEL: return launch_prim_f_massvel(stream, ctx->view, a, l1, l2, grid, block);
      case OLC_OP_NUCLEAR: return launch_prim_f_nuclear(stream, ctx->view, a, l1, l2, grid, block);
      default: return launch_prim_f_elecpot(stream, ctx->view, a, l1, l2, FAR32, grid, block);
    }
  }
  switch (l1 * 3 + l2) {
#define OLC_CASE(c, l1, l2)                                                                   \
  case c:                                                                                     \
    if constexpr (OP == OLC_OP_NUCLEAR || OP == OLC_OP_ELECPOT)                               \
      third_centre_kernel<OP, l1, l2, FAR32><<<grid, block, 0, stream>>>(ctx->view, a);  \
    else                                                                                      \
      prim_kernel<OP, l1, l2><<<grid, block, 0, stream>>>(ctx->view, a);                 \
    break;
    OLC_CASE(0, 0, 0) OLC_CASE(1, 0, 1) OLC_CASE(2, 0, 2)
    OLC_CASE(3, 1, 0) OLC_CASE(4, 1, 1) OLC_CASE(5, 1, 2)
    OLC_CASE(6, 2, 0) OLC_CASE(7, 2, 1) OLC_CASE(8, 2, 2)
#undef OLC_CASE
  }
  return cuda_check(cudaGetLastError(), "primitive kernel launch");
}

// Side streams of the third-centre classes (created at first use).  false: there are
// none, the classes run one after the other; the error that said so is cleared, so
// that it isn't taken for one of the launches that follow.
constexpr int kSideStreams = 3;
bool side_streams(olc_context* ctx) {
  if ((int)ctx->prim_streams.size() == kSideStreams) return true;
  if (!ctx->prim_fork && cudaEventCreateWithFlags(&ctx->prim_fork, cudaEventDisableTiming) != cudaSuccess) {
    ctx->prim_fork = nullptr;
    cudaGetLastError();
    return false;
  }
  while ((int)ctx->prim_streams.size() < kSideStreams) {
    cudaStream_t st = nullptr;
    cudaEvent_t ev = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
      if (st) cudaStreamDestroy(st);
      cudaGetLastError();
      return false;
    }
    ctx->prim_streams.push_back(st);
    ctx->prim_join.push_back(ev);
  }
  return true;
}

int run_primitives(olc_context* ctx, int op, int term, const double* coeffs, int precision,
                   bool accumulate) {
  int ep_type = -1, ep_alpha = 0;
  if (op == OLC_OP_ELECPOT && !coeffs) {
    ep_type = -2;
    for (size_t t = 0; t < ctx->hpots.size(); ++t)
      if (term >= ctx->hpots[t].cumul_alpha &&
          term < ctx->hpots[t].cumul_alpha + ctx->hpots[t].num_alphas) {
        ep_type = (int)t;
        ep_alpha = term - ctx->hpots[t].cumul_alpha;
      }
    if (ep_type < 0) return fail(OLC_ERR_ARG, "potential term index out of range");
  }
  // OLC_PREC_MIXED: far-shell electronic-potential images in FP32
  const bool far32 = precision == OLC_PREC_MIXED;
  // The third-centre classes write items of their own, and those of a small
  // system leave most of the chip idle one after the other (a transformation of
  // 50 to 350 us by a few blocks each), so they run beside each other: the
  // heaviest first, each on the stream with the least work so far.  Not while
  // stages are timed, whose events lie on the context's stream.  Set-up of a
  // two-atom oxide with f functions 42.0 -> 33.1 ms, of 64 silicon atoms 77.5 ->
  // 73.6 ms, band path of two-atom silicon 5.96 -> 5.48 ms.
  const bool third = op == OLC_OP_NUCLEAR || op == OLC_OP_ELECPOT;
  int order[kNumClasses];
  double cost[kNumClasses], load[kSideStreams + 1] = {};
  int busy = 0;
  for (int cls = 0; cls < kNumClasses; ++cls) {
    order[cls] = cls;
    cost[cls] = (double)ctx->items.count[cls] * ncart(cls / (kMaxL + 1)) * ncart(cls % (kMaxL + 1));
    busy += ctx->items.count[cls] > 0;
  }
  const bool fork = third && busy > 1 && !ctx->profiling && side_streams(ctx);
  int st = 0;
  if (fork) {
    std::stable_sort(order, order + kNumClasses, [&](int x, int y) { return cost[x] > cost[y]; });
    st = cuda_check(cudaEventRecord(ctx->prim_fork, ctx->stream), "fork primitives");
    for (int q = 0; q < kSideStreams && !st; ++q)
      st = cuda_check(cudaStreamWaitEvent(ctx->prim_streams[q], ctx->prim_fork, 0), "fork primitives");
  }
  for (int c = 0; c < kNumClasses && !st; ++c) {
    const int cls = order[c];
    cudaStream_t on = ctx->stream;
    if (fork) {
      const int q = (int)(std::min_element(load, load + kSideStreams + 1) - load);
      load[q] += cost[cls];
      if (q) on = ctx->prim_streams[q - 1];
    }
    switch (op) {
      case OLC_OP_OVERLAP: st = launch_class<OLC_OP_OVERLAP, false>(ctx, on, cls, nullptr, -1, 0, accumulate); break;
      case OLC_OP_KINETIC: st = launch_class<OLC_OP_KINETIC, false>(ctx, on, cls, nullptr, -1, 0, accumulate); break;
      case OLC_OP_MASSVEL: st = launch_class<OLC_OP_MASSVEL, false>(ctx, on, cls, nullptr, -1, 0, accumulate); break;
      case OLC_OP_NUCLEAR: st = launch_class<OLC_OP_NUCLEAR, false>(ctx, on, cls, nullptr, -1, 0, accumulate); break;
      case OLC_OP_ELECPOT:
        st = far32 ? launch_class<OLC_OP_ELECPOT, true>(ctx, on, cls, coeffs, ep_type, ep_alpha, accumulate)
                   : launch_class<OLC_OP_ELECPOT, false>(ctx, on, cls, coeffs, ep_type, ep_alpha, accumulate);
        break;
      default: st = fail(OLC_ERR_ARG, "unknown integral operator");
    }
  }
  if (fork)   // the context's stream goes on when every side stream is done, also after an error
    for (int q = 0; q < kSideStreams; ++q) {
      const int e1 = cuda_check(cudaEventRecord(ctx->prim_join[q], ctx->prim_streams[q]), "join primitives");
      const int e2 = cuda_check(cudaStreamWaitEvent(ctx->stream, ctx->prim_join[q], 0), "join primitives");
      if (!st) st = e1 ? e1 : e2;
    }
  return st;
}

// ---------------------------------------------------------------------------
// stage 2: contraction with the basis coefficients
// ---------------------------------------------------------------------------
struct ContractArgs {
  const int32_t* ab[kNumClasses];
  const int32_t* start[kNumClasses];
  const double* sh[kNumClasses];
  int ms;                   // block stride (max states)
  int rows;                 // rows of the half-contracted table (exponents x harmonics)
  double* block;            // [task][m2*ms + m1]
};

// One CTA per (task, kContractCols states of the second atom).  The FP64 pipe
// would bound one sum per element, so it runs in two steps, as pairXBasisFn2 and
// multWithBasisFn1 do (the pipe is then 39 % busy at 64 silicon atoms, and the loads
// of the primitive blocks bound it): T(a1, lm1; m2) = sum_a2 c2(a2, m2) sh(a1, a2; lm1, lm2)
// in shared memory, then block(m1, m2) = sum_a1 c1(a1, m1) T(a1, lm(m1); m2)
// -- about 9 n_a^2 M2 + n_a M1 M2 multiply-adds where one sum per element over
// all alpha pairs costs 3 n_a^2 M1 M2 operations.  Per operator: two-atom cell
// with f functions 1.32 -> 0.10 ms, 64-atom silicon cell 1.12 -> 0.7 ms, two-atom
// silicon cell 0.57 -> 0.07 ms.
constexpr int kContractCols = 8;
constexpr int kContractThreads = 128;

__global__ void __launch_bounds__(kContractThreads) contract_kernel(SysView v, ContractArgs a) {
  __shared__ const double* item[OLC_MAX_ALPHAS * OLC_MAX_ALPHAS];   // sh block of (a1, a2), null: none
  __shared__ double c2[kContractCols][OLC_MAX_ALPHAS];
  __shared__ int used[OLC_MAX_ALPHAS], w2[OLC_MAX_ALPHAS];        // a2 range of each a1; harmonics of each a2
  __shared__ int nrow;
  extern __shared__ double half[];                       // [column][a1 * ns1 + lm1]
  const int task = blockIdx.x, tid = threadIdx.x;
  const DevPair& p = v.pairs[v.tasks[task].pair];
  const DevType& t1 = v.types[v.site_type[p.i]];
  const DevType& t2 = v.types[v.site_type[p.j]];
  const int M1 = t1.nstates, M2 = t2.nstates, c0 = blockIdx.y * kContractCols;
  if (c0 >= M2) return;
  const int mc = min(kContractCols, M2 - c0);
  const int n1 = t1.nalpha, n2 = t2.nalpha;
  const int ns1 = (t1.lmax_alpha[0] + 1) * (t1.lmax_alpha[0] + 1);
  for (int e = tid; e < n1 * n2; e += kContractThreads) item[e] = nullptr;
  for (int e = tid; e < n2 * mc; e += kContractThreads)
    c2[e / n2][e % n2] = t2.basis[(e % n2) * OLC_MAX_STATES + c0 + e / n2];
  if (tid < OLC_MAX_ALPHAS) {
    used[tid] = 0;
    const int l2 = tid < n2 ? t2.lmax_alpha[tid] : -1;
    w2[tid] = (l2 + 1) * (l2 + 1);
  }
  if (tid == 0) nrow = 0;
  __syncthreads();
#pragma unroll
  for (int cls = 0; cls < kNumClasses; ++cls) {
    const int wi = (cls / (kMaxL + 1) + 1) * (cls / (kMaxL + 1) + 1), wj = (cls % (kMaxL + 1) + 1) * (cls % (kMaxL + 1) + 1);
    const int b = a.start[cls][task], en = a.start[cls][task + 1];
    for (int q = b + tid; q < en; q += kContractThreads) {
      const int ab = a.ab[cls][q], a1 = ab & 255, a2 = ab >> 8;
      item[a1 * n2 + a2] = a.sh[cls] + (size_t)q * (wi * wj);
      atomicMax(&used[a1], a2 + 1);
      atomicMax(&nrow, a1 + 1);
    }
  }
  __syncthreads();
  const int rows = nrow * ns1;
  for (int e = tid; e < rows * mc; e += kContractThreads) {
    const int row = e % rows, c = e / rows;
    const int a1 = row / ns1, lm1 = row % ns1;
    const int l1 = t1.lmax_alpha[a1], w1 = (l1 + 1) * (l1 + 1);
    double acc = 0.0;
    if (lm1 < w1) {
      const int lm2 = t2.lm_index[c0 + c] - 1, off = lm2 * w1 + lm1, na = used[a1];
      const double* const* it = item + a1 * n2;
      // the loads of six exponents in flight together
#pragma unroll 6
      for (int a2 = 0; a2 < na; ++a2) {
        const double* s = it[a2];
        if (s && lm2 < w2[a2]) acc = fma(c2[c][a2], s[off], acc);
      }
    }
    half[c * a.rows + row] = acc;
  }
  __syncthreads();
  double* out = a.block + (size_t)task * a.ms * a.ms;
  for (int e = tid; e < M1 * mc; e += kContractThreads) {
    const int m1 = e % M1, c = e / M1, lm1 = t1.lm_index[m1] - 1;
    double acc = 0.0;
#pragma unroll 4
    for (int a1 = 0; a1 < nrow; ++a1)
      acc = fma(t1.basis[a1 * OLC_MAX_STATES + m1], half[c * a.rows + a1 * ns1 + lm1], acc);
    out[(c0 + c) * a.ms + m1] = acc;
  }
}

// ---------------------------------------------------------------------------
// stage 3: Bloch sum, lattice-origin phase and scatter
// ---------------------------------------------------------------------------
__global__ void phase_table_kernel(SysView v, double* phase) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= v.nk * v.ncells) return;
  const int k = idx / v.ncells, n = idx % v.ncells;
  const double kr = v.kxyz[3 * k] * v.cells[4 * n] + v.kxyz[3 * k + 1] * v.cells[4 * n + 1] +
                    v.kxyz[3 * k + 2] * v.cells[4 * n + 2];
  double s, c;
  sincos(kr, &s, &c);
  phase[2 * idx] = c;
  phase[2 * idx + 1] = s;
}

struct BlochArgs {
  const double* block;
  int ms;
  int chunks;      // blocks a pair
  double* vv;
  double* cv;
  double* cc;
};

// Bound by the FP64 pipe, two multiply-adds per task, element and k, and where
// the pairs are few by the latency of their long task lists.  A thread sums one
// element at KU k-points, so that a task's block element and cell are loaded
// once for all of them; a block forms the pair's phases e^{i k.L} of its
// k-points once in shared memory (an FP64 sincos costs as much as dozens of
// tasks).  One thread an element and k with its own sincos, eight of them in
// a row, took 6.9 ms for 19 operators of 2080 pairs at 8 k-points and 3.3 ms for
// 36 operators of 3 pairs at 8, this form 3.8 and 1.5 ms.
constexpr int kBlochThreads = 256;

template <int KU>
__global__ void __launch_bounds__(kBlochThreads) bloch_scatter_kernel(SysView v, BlochArgs a) {
  __shared__ double2 shift[KU * (kBlochThreads + 1)];
  const DevPair p = v.pairs[blockIdx.x / a.chunks];
  const DevType& t1 = v.types[v.site_type[p.i]];
  const DevType& t2 = v.types[v.site_type[p.j]];
  const int M1 = t1.nstates, M2 = t2.nstates;
  const int per_k = M1 * M2;
  // sums e0 .. e0 + kBlochThreads of the pair's (group of KU k-points, element)
  const long long total = (long long)per_k * ((v.nk + KU - 1) / KU);
  const long long e0 = (long long)(blockIdx.x % a.chunks) * kBlochThreads;
  if (e0 >= total) return;
  const int g0 = (int)(e0 / per_k), k0 = g0 * KU;
  const int k1 = min(v.nk, ((int)(min(e0 + kBlochThreads, total) - 1) / per_k + 1) * KU);
  for (int q = threadIdx.x; q < k1 - k0; q += kBlochThreads) {
    const double* kv = v.kxyz + 3 * (size_t)(k0 + q);
    const double kl = kv[0] * p.L[0] + kv[1] * p.L[1] + kv[2] * p.L[2];
    double s = 0.0, c = 1.0;
    if (kl != 0.0) sincos(kl, &s, &c);
    shift[q] = make_double2(c, s);
  }
  __syncthreads();
  const long long e = e0 + threadIdx.x;
  if (e >= total) return;
  const size_t nv = v.vale_dim, nc = v.core_dim, ncells = v.ncells;
  const bool same = (p.i == p.j);
  const int vi1 = v.cum_vale[p.i], vi2 = v.cum_vale[p.j];
  const int ci1 = v.cum_core[p.i], ci2 = v.cum_core[p.j];
  const int vn1 = t1.nvale, vn2 = t2.nvale;
  const int kb = (int)(e / per_k) * KU, kn = min(KU, v.nk - kb);
  const int r = (int)(e % per_k);
  const int m1 = r % M1, m2 = r / M1;
  double sr[KU] = {}, si[KU] = {};
  const double2* ph = reinterpret_cast<const double2*>(v.phase) + kb * ncells;
  const double* bl = a.block + m2 * a.ms + m1;
  const size_t bs = (size_t)a.ms * a.ms;
#pragma unroll 4
  for (int t = p.task_begin; t < p.task_end; ++t) {
    const double2* pc = ph + v.tasks[t].cell;
    const double b = bl[t * bs];
#pragma unroll
    for (int q = 0; q < KU; ++q)
      if (q < kn) {
        const double2 z = pc[q * ncells];
        sr[q] += z.x * b;
        si[q] += z.y * b;
      }
  }
#pragma unroll
  for (int q = 0; q < KU; ++q) {
    if (q >= kn) break;
    const int k = kb + q;
    const double2 w = shift[k - k0];
    const double re = w.x * sr[q] - w.y * si[q], im = w.y * sr[q] + w.x * si[q];
    // saveCurrentPair (intgSaving.F90:201-505)
    if (m1 < vn1 && m2 < vn2) {
      const size_t row = vi1 + m1, col = vi2 + m2;
      double* d = a.vv + 2 * ((size_t)k * nv * nv + col * nv + row);
      if (same && m1 > m2) { d[0] = 0.0; d[1] = 0.0; }
      else { d[0] = re; d[1] = im; }
    } else if (m1 >= vn1 && m2 < vn2) {
      if (!same) {
        double* d = a.cv + 2 * ((size_t)k * nc * nv + (size_t)(vi2 + m2) * nc + ci1 + (m1 - vn1));
        d[0] = re;
        d[1] = im;
      }
    } else if (m1 < vn1 && m2 >= vn2) {
      double* d = a.cv + 2 * ((size_t)k * nc * nv + (size_t)(vi1 + m1) * nc + ci2 + (m2 - vn2));
      d[0] = re;
      d[1] = -im;
    } else {
      const int c1 = m1 - vn1, c2 = m2 - vn2;
      double* d = a.cc + 2 * ((size_t)k * nc * nc + (size_t)(ci2 + c2) * nc + ci1 + c1);
      d[0] = re;
      d[1] = im;
      if (!same) {
        double* e2 = a.cc + 2 * ((size_t)k * nc * nc + (size_t)(ci1 + c1) * nc + ci2 + c2);
        e2[0] = re;
        e2[1] = -im;
      }
    }
  }
}

int run_contract_bloch(olc_context* ctx, double* vv, double* cv, double* cc) {
  const SysView& v = ctx->view;
  const int ntasks = ctx->dims.num_pair_tasks;
  const size_t nv = v.vale_dim, nc = v.core_dim, nk = v.nk;
  int st;
  if ((st = cuda_check(cudaMemsetAsync(vv, 0, 16 * nv * nv * nk, ctx->stream), "memset vv"))) return st;
  if (nc) {
    if (!cv || !cc) return fail(OLC_ERR_ARG, "core outputs required when core_dim > 0");
    if ((st = cuda_check(cudaMemsetAsync(cv, 0, 16 * nc * nv * nk, ctx->stream), "memset cv"))) return st;
    if ((st = cuda_check(cudaMemsetAsync(cc, 0, 16 * nc * nc * nk, ctx->stream), "memset cc"))) return st;
  }
  if (ntasks == 0) return OLC_OK;
  ContractArgs ca;
  for (int c = 0; c < kNumClasses; ++c) {
    ca.ab[c] = ctx->items.ab[c];
    ca.start[c] = ctx->items.task_start[c];
    ca.sh[c] = ctx->d_sh + ctx->items.sh_offset[c];
  }
  ca.ms = ctx->max_states;
  ca.block = ctx->d_block;
  ca.rows = 0;
  for (const DevType& t : ctx->htypes)
    ca.rows = std::max(ca.rows, t.nalpha * (t.lmax_alpha[0] + 1) * (t.lmax_alpha[0] + 1));
  // at most 32 KB, with the static part below what every launch may have
  static_assert(kContractCols * sizeof(double) * OLC_MAX_ALPHAS * nharm(kMaxL) <= 32 * 1024, "contraction table");
  const size_t csmem = sizeof(double) * kContractCols * (size_t)ca.rows;
  {
    StageScope scope(ctx, OLC_STAGE_CONTRACT);
    const dim3 cgrid((unsigned)ntasks, (unsigned)((ctx->max_states + kContractCols - 1) / kContractCols));
    contract_kernel<<<cgrid, kContractThreads, csmem, ctx->stream>>>(v, ca);
  }
  if ((st = cuda_check(cudaGetLastError(), "contract_kernel"))) return st;
  BlochArgs ba;
  ba.block = ctx->d_block;
  ba.ms = ctx->max_states;
  const int per_k = ctx->max_states * ctx->max_states;
  ba.vv = vv;
  ba.cv = cv;
  ba.cc = cc;
  // Four k-points a thread, fewer where that leaves the chip short of threads:
  // blocks of a thousand such sums took 9.8 ms for the 36 operators of 3 pairs
  // that blocks of 256 single ones do in 1.5 ms.
  const size_t sums = ctx->hpairs.size() * (size_t)per_k * nk;
  int ku = 4;
  while (ku > 1 && sums / ku < 152 * 1024) ku /= 2;
  const auto kern = ku == 4 ? bloch_scatter_kernel<4> : ku == 2 ? bloch_scatter_kernel<2> : bloch_scatter_kernel<1>;
  ba.chunks = (int)(((size_t)per_k * ((nk + ku - 1) / ku) + kBlochThreads - 1) / kBlochThreads);
  const size_t blocks = ctx->hpairs.size() * (size_t)ba.chunks;
  if (blocks > 0x7fffffffu) return fail(OLC_ERR_UNSUPPORTED, "Bloch sums: too many pairs and k-points");
  StageScope scope(ctx, OLC_STAGE_BLOCH);
  kern<<<(unsigned)blocks, kBlochThreads, 0, ctx->stream>>>(v, ba);
  return cuda_check(cudaGetLastError(), "bloch_scatter_kernel");
}

int build_phase_table(olc_context* ctx) {
  const SysView& v = ctx->view;
  const int n = v.nk * v.ncells;
  count_launch();
  phase_table_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(v, const_cast<double*>(v.phase));
  return cuda_check(cudaGetLastError(), "phase_table_kernel");
}

// ---------------------------------------------------------------------------
// primitive batch (testing entry): explicit inputs, one thread per primitive
// ---------------------------------------------------------------------------
__global__ void prim_batch_kernel(int kind, int n, const double* in, const int32_t* lm,
                                  double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  auto lof = [](int lma) { return lma == 1 ? 0 : lma == 4 ? 1 : 2; };
  if (lm[2 * i] == 16 || lm[2 * i + 1] == 16) return;      // f classes: prim_batch_f_kernel
  const int c = lof(lm[2 * i]) * 3 + lof(lm[2 * i + 1]);
  const double* x = in + 12 * i;
  double* o = out + 256 * i;
  switch (c) {
    case 0: prim_one<0, 0>(kind, x, o); break;
    case 1: prim_one<0, 1>(kind, x, o); break;
    case 2: prim_one<0, 2>(kind, x, o); break;
    case 3: prim_one<1, 0>(kind, x, o); break;
    case 4: prim_one<1, 1>(kind, x, o); break;
    case 5: prim_one<1, 2>(kind, x, o); break;
    case 6: prim_one<2, 0>(kind, x, o); break;
    case 7: prim_one<2, 1>(kind, x, o); break;
    case 8: prim_one<2, 2>(kind, x, o); break;
  }
}

int primitive_batch_device(int kind, int n, const double* in, const int32_t* lmalpha,
                           double* out) {
  if (kind < 1 || kind > 8 || n < 0) return fail(OLC_ERR_ARG, "olc_primitive_batch: bad kind");
  for (int i = 0; i < n; ++i) {
    for (int s = 0; s < 2; ++s) {
      int l = lmalpha[2 * i + s];
      if (l != 1 && l != 4 && l != 9 && l != 16)
        return fail(OLC_ERR_ARG, "lmalpha must be 1, 4, 9 or 16");
    }
  }
  if (n == 0) return OLC_OK;
  double *din = nullptr, *dout = nullptr;
  int32_t* dlm = nullptr;
  int st = OLC_OK;
  if ((st = cuda_check(cudaMalloc(&din, sizeof(double) * 12 * n), "malloc"))) return st;
  if ((st = cuda_check(cudaMalloc(&dout, sizeof(double) * 256 * n), "malloc"))) { cudaFree(din); return st; }
  if ((st = cuda_check(cudaMalloc(&dlm, sizeof(int32_t) * 2 * n), "malloc"))) { cudaFree(din); cudaFree(dout); return st; }
  st = cuda_check(cudaMemcpy(din, in, sizeof(double) * 12 * n, cudaMemcpyHostToDevice), "copy");
  if (!st) st = cuda_check(cudaMemcpy(dlm, lmalpha, sizeof(int32_t) * 2 * n, cudaMemcpyHostToDevice), "copy");
  if (!st) st = cuda_check(cudaMemset(dout, 0, sizeof(double) * 256 * n), "memset");
  if (!st) {
    count_launch();
    prim_batch_kernel<<<(n + 63) / 64, 64>>>(kind, n, din, dlm, dout);
    switch (kind) {
      case 1: launch_prim_batch_f_overlap(n, din, dlm, dout); break;
      case 2: launch_prim_batch_f_kinetic(n, din, dlm, dout); break;
      case 3: launch_prim_batch_f_nuclear(n, din, dlm, dout); break;
      case 4: launch_prim_batch_f_elecpot(n, din, dlm, dout); break;
      case 5: launch_prim_batch_f_massvel(n, din, dlm, dout); break;
      default: launch_prim_batch_f_momentum(kind, n, din, dlm, dout); break;
    }
    count_launch(7);
    st = cuda_check(cudaGetLastError(), "prim_batch_kernel");
  }
  if (!st) st = cuda_check(cudaMemcpy(out, dout, sizeof(double) * 256 * n, cudaMemcpyDeviceToHost), "copy back");
  cudaFree(din);
  cudaFree(dout);
  cudaFree(dlm);
  return st;
}

}  // namespace olc
