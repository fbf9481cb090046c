// Primitive-stage device code shared by the translation units of the
// integral kernels (olc_integrals.cu: s, p, d classes; olc_integrals_f*.cu:
// the classes with an f function, compiled apart because their
// recurrences are large).
#pragma once

#include "olc_common.h"
#include "olc_primitives.cuh"

namespace olc {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ double elem_alpha(const SysView& v, int e, int a) {
  return v.elem_alpha[e * OLC_MAX_ALPHAS + a];
}

// alphaDist(a1, a2, e1, e2) of gaussRelations.f90:64-135 (same operation order)
__device__ __forceinline__ double alpha_dist(const SysView& v, int a1, int a2, int e1, int e2) {
  const double al = elem_alpha(v, e1, a1), ak = elem_alpha(v, e2, a2);
  return v.log_thresh / ak / (al / (al + ak));
}

struct ItemGeom {
  double A[3], B[3];
  double a1, a2, sep;
  int e1, e2, ia1, ia2;
};

// Returns the atom A of the item.
__device__ __forceinline__ int load_item(const SysView& v, int task, int ab, ItemGeom& g) {
  const DevTask tk = v.tasks[task];
  const DevPair p = v.pairs[tk.pair];
  const DevType& t1 = v.types[v.site_type[p.i]];
  const DevType& t2 = v.types[v.site_type[p.j]];
  g.ia1 = ab & 255;
  g.ia2 = ab >> 8;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    g.A[c] = v.site_pos[3 * p.i + c];
    g.B[c] = v.site_pos[3 * p.j + c] + p.L[c] + v.cells[4 * tk.cell + c];
  }
  g.a1 = t1.alphas[g.ia1];
  g.a2 = t2.alphas[g.ia2];
  g.e1 = t1.element;
  g.e2 = t2.element;
  g.sep = tk.sep;
  return p.i;
}

// ---------------------------------------------------------------------------
// stage 1: primitive kernels
// ---------------------------------------------------------------------------
struct PrimArgs {
  const int32_t* task;
  const int32_t* ab;
  int n;
  double* out;              // class block of the sh scratch
  const double* coeffs;     // device [pot_dim] (EP) or nullptr
  int accumulate;
  int ep_type;              // EP: potential type of a single term, -1 = all types
  int ep_alpha;             // EP: exponent index of a single term
  int log_split;            // third-centre operators: log2 of the lanes that share an item
};

// Two-centre operators, one thread per item.
template <int OP, int L1, int L2>
__global__ void __launch_bounds__(128) prim_kernel(SysView v, PrimArgs a) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= a.n) return;
  constexpr int N1 = ncart(L1), N2 = ncart(L2), NS = nharm(L1) * nharm(L2);
  ItemGeom g;
  load_item(v, a.task[idx], a.ab[idx], g);
  double cart[N1 * N2];
#pragma unroll
  for (int q = 0; q < N1 * N2; ++q) cart[q] = 0.0;
  if constexpr (OP == OLC_OP_OVERLAP) {
    add_overlap<L1, L2>(g.a1, g.a2, g.A, g.B, 1.0, cart);
  } else if constexpr (OP == OLC_OP_KINETIC) {
    add_kinetic<L1, L2>(g.a1, g.a2, g.A, g.B, 1.0, cart);
  } else {
    // gaussOverlapMV accumulates the primitive with a minus sign
    // (integrals.F90:1228-1236): the mass-velocity term lowers H
    add_massvel<L1, L2>(g.a1, g.a2, g.A, g.B, -1.0, cart);
  }
  store_harmonic<L1, L2, double>(cart, a.out + (size_t)idx * NS, a.accumulate != 0, 1.0);
}

// |S - C'|^2 <= radius^2 for the image D = C' - A and S = PS + A.
__device__ __forceinline__ bool within(const double4_16a& D, const double (&PS)[3], double tad) {
  const double y[3] = {PS[0] - D.x, PS[1] - D.y, PS[2] - D.z};
  return y[0] * y[0] + y[1] * y[1] + y[2] * y[2] <= tad;
}

// Third-centre operators (nuclear attraction, electronic potential), one
// thread per item: the moments about P summed over the images within the
// reference's radius (the image set of integrals.F90:2374-2418, 2533-2594),
// then one transformation into the item's Cartesian block.
//
// GB300's FP64 pipe issues a warp instruction every 64 cycles per scheduler,
// so the kernel is bound by the FP64 instructions of the lanes' images.  The
// images come from the atom's list (SysView::img_*) and are screened in FP32
// with a margin wider than its rounding; the survivors go to a queue of
// kQueue entries per thread in shared memory, so that a warp spends FP64
// instructions on rounds in which every lane has an image left, not on
// candidates that only one lane accepts; the exact test |P - C'|^2 <= radius^2
// is repeated in FP64 on them.  Measured on the 64-atom silicon cell's d-d
// class, one FP64 potential term: 2.0 ms (8.5 ms with a Cartesian block per
// image and the images found from the cell list); f-f on a two-atom cell:
// 0.52 ms (2.3 ms); nuclear d-d on the 64-atom cell: 6.0 ms (17.4 ms).  With
// the exponential from a table and, for one term, monomials of P - C' in
// place of the moments' recurrences (75 FP64 instructions a d-d image, not 94):
// 1.65 ms a d-d term of the 64-atom cell, f-f and nuclear as before.
//
// FAR32 (mixed precision): images whose suppression exp(-rho |P - C'|^2) about the
// pair's own centre is below exp(-kFarRho) are summed in FP32, in a queue and accumulators of their own, in the same
// pass (all 16 terms of the 64-atom cell's d-d class: 109 ms in two passes
// of Cartesian blocks before).
//
// Small systems have too few items for the chip (a two-atom cell's f-f class
// 40 to 60 blocks): 2^log_split threads then share an item, as many as keep all
// items in one wave of kThirdWave threads (two blocks an SM, the residency of
// the f classes).  For one operator they are warps of a block first, so that one
// full warp still transforms 32 items; where all potential terms are summed the
// images outweigh the transformation and lanes, which even out the items'
// image counts within a warp, are better (d-d class of a two-atom cell 4.4 ->
// 1.4 ms, by warps 1.9 ms).  With the f-f transformation as loops, the
// third-centre kernels of a two-atom oxide's set-up took 26 ms, 33 before.
constexpr int kThirdThreads = 128;
constexpr int kQueue = 16;
constexpr int kThirdWave = 152 * 2 * kThirdThreads;

template <int OP, int L1, int L2, bool FAR32>
__global__ void __launch_bounds__(kThirdThreads) third_centre_kernel(SysView v, PrimArgs a) {
  constexpr int N1 = ncart(L1), N2 = ncart(L2), NS = nharm(L1) * nharm(L2), LT = L1 + L2, NM = nmom(LT);
  __shared__ int queue[kQueue][kThirdThreads];
  __shared__ int farq[FAR32 ? kQueue : 1][FAR32 ? kThirdThreads : 1];
  __shared__ double exptab[64];
  if (threadIdx.x < 64) exptab[threadIdx.x] = kExp2Neg[threadIdx.x];
  __syncthreads();
  // split threads share an item and take its images in turn: the warps of a
  // block first (2^lw), then neighbouring lanes (2^ll); lanes alone where all
  // potential terms are summed
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lw = a.ep_type < 0 && OP != OLC_OP_NUCLEAR ? 0 : min(a.log_split, 2);
  const int ll = a.log_split - lw, split = 1 << a.log_split;
  const int sub = ((warp & ((1 << lw) - 1)) << ll) | (lane & ((1 << ll) - 1));
  const int idx = (int)((blockIdx.x * (kThirdThreads / 32) + warp) >> lw) * (32 >> ll) + (lane >> ll);
  const bool live = idx < a.n;
  ItemGeom g;
  const int atom = load_item(v, a.task[live ? idx : 0], a.ab[live ? idx : 0], g);
  const double z = g.a1 + g.a2, iz = 1.0 / z;
  double PA[3], PB[3], PS[3];
  // centre of the alpha-pair overlap (alphaCenter, gaussRelations.f90:122):
  // the screen's centre, the same point unless two types share an element
  // with different exponents
  const double al = elem_alpha(v, g.e1, g.ia1), ak = elem_alpha(v, g.e2, g.ia2);
  const bool same = al == g.a1 && ak == g.a2;
  const double izs = 1.0 / (al + ak), frac = 1.0 - g.sep / alpha_dist(v, g.ia1, g.ia2, g.e1, g.e2);
  double d2ab = 0.0, ps2 = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double ab = g.A[c] - g.B[c];
    PA[c] = -g.a2 * iz * ab;
    PB[c] = g.a1 * iz * ab;
    PS[c] = -ak * izs * ab;
    d2ab += ab * ab;
    ps2 += PS[c] * PS[c];
  }
  const double expAB = exp(-ratio(g.a1 * g.a2, z, iz) * d2ab);
  const float psf[3] = {(float)PS[0], (float)PS[1], (float)PS[2]};
  const float ap = (float)sqrt(ps2);
  float pah[3], pal[3];
  if (FAR32) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      pah[c] = (float)PA[c];
      pal[c] = (float)(PA[c] - (double)pah[c]);
    }
  }
  double E[NM];
  float Ef[FAR32 ? NM : 1];
#pragma unroll
  for (int q = 0; q < NM; ++q) {
    E[q] = 0.0;
    if (FAR32) Ef[q] = 0.f;
  }
  bool any = false;
  // one potential term: its images share an exponent and are summed as monomials
  const bool single = OP != OLC_OP_NUCLEAR && !FAR32 && a.ep_type >= 0;
  const double T = v.log_thresh;
  const int t0 = OP == OLC_OP_NUCLEAR || a.ep_type < 0 ? 0 : a.ep_type;
  const int t1 = OP == OLC_OP_NUCLEAR || a.ep_type < 0 ? v.num_pot_types : a.ep_type + 1;
  for (int t = t0; t < t1; ++t) {
    const DevPotType& pt = v.pot_types[t];
    if (OP == OLC_OP_NUCLEAR && pt.nuc_charge < 1.0e-8) continue;
    const int i0 = live ? v.img_start[atom * v.num_pot_types + t] : 0;
    const int i1 = live ? v.img_start[atom * v.num_pot_types + t + 1] : 0;
    const int j0 = OP == OLC_OP_NUCLEAR || a.ep_type < 0 ? 0 : a.ep_alpha;
    const int j1 = OP == OLC_OP_NUCLEAR ? 1 : a.ep_type < 0 ? pt.num_alphas : a.ep_alpha + 1;
    for (int j = j0; j < j1; ++j) {
      const double an = OP == OLC_OP_NUCLEAR ? v.elem_nuc_alpha[pt.element]
                                             : v.elem_pot_alpha[pt.element * OLC_MAX_POT_ALPHAS + j];
      const double tad = frac * (T * (al + ak + an) * izs / an);
      const double a3 = OP == OLC_OP_NUCLEAR ? pt.nuc_alpha : pt.alphas[j];
      const double z3 = z + a3, iz3 = 1.0 / z3, u = a3 * iz3, rho = ratio(z * a3, z3, iz3), h = 0.5 * iz3;
      double pref;      // of the moments, the image's exponential apart
      if (OP == OLC_OP_NUCLEAR) {
        pref = -pt.nuc_charge * 2.0 * (kPi * iz3) * expAB;
      } else {
        const double w = a.coeffs ? a.coeffs[pt.cumul_alpha + j] : 1.0, r = kPi * iz3;
        pref = w * r * sqrt(r) * expAB;
      }
      // FP32 screen: the largest distance from A, and the radius with a
      // margin of 1e-5 of that distance squared (FP32 differences of numbers
      // up to it are good to 1e-6 of it)
      const float reach = (ap + (float)sqrt(tad)) * 1.00001f;
      const float near2 = (float)tad + 1e-5f * reach * reach;
      // far images take the exact test here, where the margin leaves it open
      const float sure2 = (float)tad - 1e-5f * reach * reach;
      const float rhoh = (float)rho, rhol = (float)(rho - (double)rhoh);
      int c = i0 + sub;
      bool more = true;
      while (more) {
        int cnt = 0, cntf = 0;
        while (c < i1 && cnt < kQueue && (!FAR32 || cntf < kQueue)) {
          const float4 q = v.img_hi[c];
          if (q.w > reach) {
            c = i1;
            break;
          }
          const float x = psf[0] - q.x, y = psf[1] - q.y, w = psf[2] - q.z;
          const float d2 = x * x + y * y + w * w;
          if (d2 <= near2) {
            bool far = false;
            if (FAR32) {
              float p2 = d2;                               // |P - C'|^2, the suppression's
              if (!same) {
                const float px = pah[0] - q.x, py = pah[1] - q.y, pz = pah[2] - q.z;
                p2 = px * px + py * py + pz * pz;
              }
              far = rhoh * p2 > (float)kFarRho;
            }
            if (!far) {
              queue[cnt++][tid] = c;
            } else if (d2 <= sure2 || within(v.img_d[c], PS, tad)) {
              farq[FAR32 ? cntf++ : 0][FAR32 ? tid : 0] = c;
            }
          }
          c += split;
        }
        __syncwarp();
        for (int s = 0; s < cnt; ++s) {
          const double4_16a D = v.img_d[queue[s][tid]];
          const double x[3] = {PA[0] - D.x, PA[1] - D.y, PA[2] - D.z};       // P - C'
          const double d2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
          double ds = d2;
          if (!same) {
            const double y[3] = {PS[0] - D.x, PS[1] - D.y, PS[2] - D.z};
            ds = y[0] * y[0] + y[1] * y[1] + y[2] * y[2];
          }
          if (ds > tad) continue;
          any = true;
          const double p = pref * exp_neg(rho * d2, exptab);
          if (single) {
            add_monomials<LT>(x, p, E);
            continue;
          }
          const double gp[3] = {-u * x[0], -u * x[1], -u * x[2]};            // G - P
          if constexpr (OP == OLC_OP_NUCLEAR) {
            const double vz = z * iz3;
            const double gc[3] = {vz * x[0], vz * x[1], vz * x[2]};          // G - C'
            double F[LT + 1];
            boys_reference<LT>(z * vz * d2, F);
            add_nuclear_moments<LT>(gp, gc, h, p, F, E);
          } else {
            add_moments<LT, double>(gp, h, p, E);
          }
        }
        if constexpr (FAR32) {
          const float uf = (float)u, hf = (float)h, prf = (float)pref;
          for (int s = 0; s < cntf; ++s) {
            // |P - C'|^2 and rho |P - C'|^2 as FP32 pairs: the exponent keeps
            // its relative accuracy of about 1e-12 where FP32 alone would lose
            // 22..37 times 1e-7 of the exponential
            const int ci = farq[s][tid];
            const float4 qh = v.img_hi[ci], ql = v.img_lo[ci];
            float x[3], xl[3], g3[3];
            pair_sub(pah[0], pal[0], qh.x, ql.x, x[0], xl[0]);
            pair_sub(pah[1], pal[1], qh.y, ql.y, x[1], xl[1]);
            pair_sub(pah[2], pal[2], qh.z, ql.z, x[2], xl[2]);
            float sq[3], se = 0.f;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              sq[d] = __fmul_rn(x[d], x[d]);
              se += __fmaf_rn(x[d], x[d], -sq[d]) + 2.f * x[d] * xl[d];
              g3[d] = -uf * x[d];
            }
            float s1, e1, s2, e2;
            two_sum(sq[0], sq[1], s1, e1);
            two_sum(s1, sq[2], s2, e2);
            se += e1 + e2;
            const float eh = __fmul_rn(rhoh, s2);
            const float el = __fmaf_rn(rhoh, s2, -eh) + rhol * s2 + rhoh * se;
            add_moments<LT, float>(g3, hf, prf * expf(-eh) * (1.f - el), Ef);
            any = true;
          }
        }
        more = __any_sync(0xffffffffu, c < i1);
      }
    }
  }
  if (FAR32)
#pragma unroll
    for (int q = 0; q < NM; ++q) E[q] += (double)Ef[q];
  // two exponents past their element's table have no screen: no number, not 0
  if (ap != ap) {
    any = true;
#pragma unroll
    for (int q = 0; q < NM; ++q) E[q] = (double)ap;
  }
  for (int o = (1 << ll) >> 1; o; o >>= 1) {
    any |= __shfl_xor_sync(0xffffffffu, any ? 1 : 0, o) != 0;
#pragma unroll
    for (int q = 0; q < NM; ++q) E[q] += __shfl_xor_sync(0xffffffffu, E[q], o);
  }
  if (lw) {
    __shared__ double sums[NM][32];
    __shared__ bool anys[32];
    for (int w = 1; w < kThirdThreads / 32; ++w) {
      const int first = w & ~((1 << lw) - 1);           // the warp that keeps the item's sum
      if (first == w) continue;
      if (warp == w) {
        anys[lane] = any;
#pragma unroll
        for (int q = 0; q < NM; ++q) sums[q][lane] = E[q];
      }
      __syncthreads();
      if (warp == first) {
        any |= anys[lane];
#pragma unroll
        for (int q = 0; q < NM; ++q) E[q] += sums[q][lane];
      }
      __syncthreads();
    }
  }
  if (!live || sub) return;
  double* out = a.out + (size_t)idx * NS;
  if (!any) {
    if (!a.accumulate)
#pragma unroll
      for (int q = 0; q < NS; ++q) out[q] = 0.0;
    return;
  }
  if (single) {
    const double a3 = v.pot_types[a.ep_type].alphas[a.ep_alpha], iz3 = 1.0 / (z + a3);
    monomials_to_moments<LT>(a3 * iz3, 0.5 * iz3, E);
  }
  if constexpr (LT >= 6) {
    moments_to_harmonics<L1, L2>(E, PA, PB, out, a.accumulate != 0);
  } else {
    double cart[N1 * N2];
    moments_to_cart<L1, L2>(E, PA, PB, cart);
    store_harmonic<L1, L2, double>(cart, out, a.accumulate != 0, 1.0);
  }
}

// One primitive of explicit inputs (the testing entry olc_primitive_batch).
template <int L1, int L2>
__device__ __forceinline__ void prim_one(int kind, const double* in, double* out) {
  constexpr int N1 = ncart(L1), N2 = ncart(L2), NS1 = nharm(L1), NS2 = nharm(L2);
  double cart[N1 * N2];
#pragma unroll
  for (int q = 0; q < N1 * N2; ++q) cart[q] = 0.0;
  const double *A = in + 3, *B = in + 6, *C = in + 9;
  if (kind == 1) add_overlap<L1, L2>(in[0], in[1], A, B, 1.0, cart);
  else if (kind == 2) add_kinetic<L1, L2>(in[0], in[1], A, B, 1.0, cart);
  else if (kind == 3) add_nuclear<L1, L2>(in[0], in[1], in[2], A, B, C, 1.0, cart);
  else if (kind == 5) add_massvel<L1, L2>(in[0], in[1], A, B, 1.0, cart);
  else if (kind >= 6) add_momentum<L1, L2>(in[0], in[1], A, B, kind - 6, 1.0, cart);
  else {
    double d2 = 0.0;
    for (int c = 0; c < 3; ++c) d2 += (A[c] - B[c]) * (A[c] - B[c]);
    const double expAB = exp(-(in[0] * in[1] / (in[0] + in[1])) * d2);
    add_elec3c<L1, L2, double>(in[0], in[1], in[2], A, B, C, expAB, 1.0, cart);
  }
  double sh[NS1 * NS2];
  store_harmonic<L1, L2, double>(cart, sh, false, 1.0);
  for (int q = 0; q < NS2; ++q)
    for (int p2 = 0; p2 < NS1; ++p2) out[q * 16 + p2] = sh[q * NS1 + p2];
}


// f classes (olc_integrals_f*.cu): launches of the primitive kernels for the
// 7 classes with l1 = 3 or l2 = 3, one function per operator; far32 as in
// third_centre_kernel.
int launch_prim_f_overlap(cudaStream_t st, const SysView& v, const PrimArgs& a, int l1, int l2, dim3 g, dim3 b);
int launch_prim_f_kinetic(cudaStream_t st, const SysView& v, const PrimArgs& a, int l1, int l2, dim3 g, dim3 b);
int launch_prim_f_massvel(cudaStream_t st, const SysView& v, const PrimArgs& a, int l1, int l2, dim3 g, dim3 b);
int launch_prim_f_nuclear(cudaStream_t st, const SysView& v, const PrimArgs& a, int l1, int l2, dim3 g, dim3 b);
int launch_prim_f_elecpot(cudaStream_t st, const SysView& v, const PrimArgs& a, int l1, int l2, bool far32, dim3 g,
                          dim3 b);
// primitive batch entries of the f classes, one per kind (1 overlap,
// 2 kinetic, 3 nuclear, 4 three-centre, 5 mass velocity, 6-8 momentum x, y,
// z with the overlap), in the same translation units
void launch_prim_batch_f_overlap(int n, const double* in, const int32_t* lm, double* out);
void launch_prim_batch_f_kinetic(int n, const double* in, const int32_t* lm, double* out);
void launch_prim_batch_f_nuclear(int n, const double* in, const int32_t* lm, double* out);
void launch_prim_batch_f_elecpot(int n, const double* in, const int32_t* lm, double* out);
void launch_prim_batch_f_massvel(int n, const double* in, const int32_t* lm, double* out);
void launch_prim_batch_f_momentum(int kind, int n, const double* in, const int32_t* lm, double* out);

// Primitive batch kernel of one kind and one f class (a kernel per class
// keeps each recurrence's register allocation separate).
template <int KIND, int L1, int L2>
__global__ void prim_batch_f_kernel(int n, const double* in, const int32_t* lm, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  auto lof = [](int lma) { return lma == 1 ? 0 : lma == 4 ? 1 : lma == 9 ? 2 : 3; };
  if (lof(lm[2 * i]) != L1 || lof(lm[2 * i + 1]) != L2) return;
  prim_one<L1, L2>(KIND, in + 12 * i, out + 256 * i);
}

template <int KIND>
void launch_prim_batch_f_kind(int n, const double* in, const int32_t* lm, double* out) {
  const int g = (n + 63) / 64;
  prim_batch_f_kernel<KIND, 0, 3><<<g, 64>>>(n, in, lm, out);
  prim_batch_f_kernel<KIND, 1, 3><<<g, 64>>>(n, in, lm, out);
  prim_batch_f_kernel<KIND, 2, 3><<<g, 64>>>(n, in, lm, out);
  prim_batch_f_kernel<KIND, 3, 0><<<g, 64>>>(n, in, lm, out);
  prim_batch_f_kernel<KIND, 3, 1><<<g, 64>>>(n, in, lm, out);
  prim_batch_f_kernel<KIND, 3, 2><<<g, 64>>>(n, in, lm, out);
  prim_batch_f_kernel<KIND, 3, 3><<<g, 64>>>(n, in, lm, out);
}

}  // namespace olc
