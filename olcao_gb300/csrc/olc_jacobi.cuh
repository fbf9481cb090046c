// Generalised Hermitian eigen-solve of one small pencil by one CTA, all in
// shared memory, to FP64 accuracy: the steps of LAPACK zhegv (itype 1, upper)
// with the reduced problem solved in FP32 and refined in FP64.
//   1. B = U^H U (right-looking Cholesky; failure n + j + 1 as zpotrf/zhegv)
//   2. C = U^{-H} A U^{-1}
//   3. V ~ eigenvectors of C by parallel (round-robin) cyclic Jacobi in FP32
//   4. refinement passes in FP64 until V is orthonormal and V^H C V diagonal
//      to rounding (refine below)
// GB300's FP64 pipe runs at 1/64 of the FP32 rate, and a cyclic Jacobi solve
// is 8 to 10 sweeps of 36 n^2 (n - 1) / 2 FP64 operations.  A refinement pass
// is three products (V^H V, C V, V^H (C V)), 8 n^3, and squares the FP32
// error; two passes suffice.  8192 pencils of n = 32: see small_hegv_kernel.
// The caller loads U = B and C = A (column-major, leading dimension ld, full
// Hermitian), calls hegv_reduced, reads the eigenvalues from w and
// back-transforms V with U (x = U^{-1} v).
#pragma once

#include <cuda_runtime.h>

namespace olc {
namespace jac {

constexpr int kMaxN = 64;
constexpr int kChunk = 16;            // columns of C V formed at a time

struct cd { double x, y; };
__device__ __forceinline__ cd cmul(cd a, cd b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ cd cmulc(cd a, cd b) { return {a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x}; }  // conj(a)*b
__device__ __forceinline__ cd csub(cd a, cd b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ void fma_conj(cd& s, cd a, cd b) {       // s += conj(a) b
  s.x = fma(a.x, b.x, fma(a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(-a.y, b.x, s.y));
}
__device__ __forceinline__ void fma_plain(cd& s, cd a, cd b) {      // s += a b
  s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
}
__device__ __forceinline__ void fma_f(float2& s, float2 a, float2 b) {
  s.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, s.x));
  s.y = fmaf(a.x, b.y, fmaf(a.y, b.x, s.y));
}

// Odd leading dimension: lanes that walk rows or columns of a matrix of
// 16-byte elements then meet different banks.
__host__ __device__ inline int lead(int n) { return n | 1; }

struct Shared {
  int fail, flag;
  unsigned emax, rmax;
  double red[32];
  double sum;
  double dinv[kMaxN], w[kMaxN];
  int p[kMaxN / 2], q[kMaxN / 2];
  double c[kMaxN / 2], s[kMaxN / 2], phx[kMaxN / 2], phy[kMaxN / 2];
  int order[kMaxN];
};

// Bytes of dynamic shared memory: U / V, C, D and the chunk of C V.
__host__ __device__ inline size_t smem_bytes(int n) {
  return sizeof(cd) * ((size_t)3 * n * lead(n) + (size_t)kChunk * lead(n));
}

__device__ __forceinline__ double block_sum(double v, Shared& sh) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sh.red[q];
    sh.sum = t;
  }
  __syncthreads();
  return sh.sum;
}

// Element e of the upper triangle (i <= j) of an n x n matrix, e in
// [0, m (m + 1) / 2) with m = n rounded up to even; false for the padding.
__device__ __forceinline__ bool upper_element(int e, int m, int n, int& i, int& j) {
  const int x = e % (m + 1), y = e / (m + 1);
  if (x > y) { i = y; j = x - 1; }
  else { i = m - 1 - y; j = m - 1 - x; }
  return j < n;
}

// Pair `pi` of round `round` of the round-robin order over m (even) indices.
__device__ __forceinline__ void round_pair(int pi, int round, int m, int& p, int& q) {
  if (pi == 0) { p = round % (m - 1); q = m - 1; }
  else { p = (round + pi) % (m - 1); q = (round - pi + (m - 1)) % (m - 1); }
  if (p > q) { const int t = p; p = q; q = t; }
}

// Cyclic Jacobi sweep in FP64 over the pairs of D (full Hermitian, updated)
// whose entry exceeds `floor` and `ratio` times the distance of their diagonal
// values, accumulated into V.  ratio = 0: every pair, the plain method.
// Rotation: J = diag(1, e^{-i phi}) R(theta) on columns p, q.
static __device__ __noinline__ void sweep_f64(cd* D, cd* V, int n, int ld, double floor, double ratio, Shared& sh) {
  const int tid = threadIdx.x;
  const int m = (n + 1) & ~1, half = m / 2;
  for (int round = 0; round < m - 1; ++round) {
    if (tid == 0) sh.flag = 0;
    __syncthreads();
    if (tid < half) {
      const int pi = tid;
      int p, q;
      round_pair(pi, round, m, p, q);
      double c = 1.0, s = 0.0, phx = 1.0, phy = 0.0;
      if (q < n) {
        const cd cpq = D[(size_t)q * ld + p];
        const double app = D[(size_t)p * ld + p].x, aqq = D[(size_t)q * ld + q].x;
        const double b2 = cpq.x * cpq.x + cpq.y * cpq.y, g = ratio * (aqq - app);
        // hypot keeps |e^{-i phi}| = 1 when the entry is tiny (x*x + y*y
        // would drop into denormals and make the rotation non-unitary);
        // entries below 1e-18 of the diagonal scale are left alone
        const double b = ratio == 0.0 || (b2 > floor * floor && b2 > g * g) ? hypot(cpq.x, cpq.y) : 0.0;
        if (b > 1e-300 && b > 1e-18 * (fabs(app) + fabs(aqq))) {
          const double th = (aqq - app) / (2.0 * b);
          const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
          c = 1.0 / sqrt(t * t + 1.0);
          s = t * c;
          phx = cpq.x / b;
          phy = -cpq.y / b;
          sh.flag = 1;
        }
      }
      sh.p[pi] = p; sh.q[pi] = q; sh.c[pi] = c; sh.s[pi] = s; sh.phx[pi] = phx; sh.phy[pi] = phy;
    }
    __syncthreads();
    if (!sh.flag) {
      __syncthreads();
      continue;
    }
    // columns: D <- D J, V <- V J
    //   col_p' = c col_p - s e^{-i phi} col_q ; col_q' = s col_p + c e^{-i phi} col_q
    for (int e = tid; e < half * n; e += blockDim.x) {
      const int pi = e / n, r = e % n;
      const int p = sh.p[pi], q = sh.q[pi];
      if (q >= n || sh.s[pi] == 0.0) continue;
      const double c = sh.c[pi], s = sh.s[pi];
      const cd ph = {sh.phx[pi], sh.phy[pi]};
      {
        const cd xp = D[(size_t)p * ld + r], eq = cmul(ph, D[(size_t)q * ld + r]);
        D[(size_t)p * ld + r] = {c * xp.x - s * eq.x, c * xp.y - s * eq.y};
        D[(size_t)q * ld + r] = {s * xp.x + c * eq.x, s * xp.y + c * eq.y};
      }
      {
        const cd xp = V[(size_t)p * ld + r], eq = cmul(ph, V[(size_t)q * ld + r]);
        V[(size_t)p * ld + r] = {c * xp.x - s * eq.x, c * xp.y - s * eq.y};
        V[(size_t)q * ld + r] = {s * xp.x + c * eq.x, s * xp.y + c * eq.y};
      }
    }
    __syncthreads();
    // rows: D <- J^H D
    //   row_p' = c row_p - s e^{i phi} row_q ; row_q' = s row_p + c e^{i phi} row_q
    for (int e = tid; e < half * n; e += blockDim.x) {
      const int pi = e / n, col = e % n;
      const int p = sh.p[pi], q = sh.q[pi];
      if (q >= n || sh.s[pi] == 0.0) continue;
      const double c = sh.c[pi], s = sh.s[pi];
      const cd phc = {sh.phx[pi], -sh.phy[pi]};
      const cd xp = D[(size_t)col * ld + p], eq = cmul(phc, D[(size_t)col * ld + q]);
      D[(size_t)col * ld + p] = {c * xp.x - s * eq.x, c * xp.y - s * eq.y};
      D[(size_t)col * ld + q] = {s * xp.x + c * eq.x, s * xp.y + c * eq.y};
    }
    __syncthreads();
  }
}

// Cyclic Jacobi in FP32 of the Hermitian C (n x n, overwritten), vectors in V.
static __device__ __noinline__ void jacobi_f32(float2* C, float2* V, int n, int ld, Shared& sh) {
  const int tid = threadIdx.x;
  const int m = (n + 1) & ~1, half = m / 2;
  float f2 = 0.f;
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int r = e % n, c = e / n;
    V[c * ld + r] = make_float2(r == c ? 1.f : 0.f, 0.f);
    const float2 x = C[c * ld + r];
    f2 += x.x * x.x + x.y * x.y;
  }
  // entries below 2e-7 of the norm are FP32 noise; the refinement takes them
  const float tiny = 2e-7f * sqrtf((float)block_sum((double)f2, sh));
  float* rc = reinterpret_cast<float*>(sh.c);
  float* rs = reinterpret_cast<float*>(sh.s);
  float* rx = reinterpret_cast<float*>(sh.phx);
  float* ry = reinterpret_cast<float*>(sh.phy);
  for (int sweep = 0; sweep < 14; ++sweep) {
    if (tid == 0) sh.flag = 0;
    __syncthreads();
    for (int round = 0; round < m - 1; ++round) {
      if (tid < half) {
        int p, q;
        round_pair(tid, round, m, p, q);
        float c = 1.f, s = 0.f, phx = 1.f, phy = 0.f;
        if (q < n) {
          const float2 cpq = C[q * ld + p];
          const float b = sqrtf(cpq.x * cpq.x + cpq.y * cpq.y);
          if (b > tiny) {
            const float th = (C[q * ld + q].x - C[p * ld + p].x) / (2.f * b);
            const float t = (th >= 0.f ? 1.f : -1.f) / (fabsf(th) + sqrtf(th * th + 1.f));
            c = rsqrtf(t * t + 1.f);
            s = t * c;
            phx = cpq.x / b;
            phy = -cpq.y / b;
            sh.flag = 1;
          }
        }
        sh.p[tid] = p; sh.q[tid] = q; rc[tid] = c; rs[tid] = s; rx[tid] = phx; ry[tid] = phy;
      }
      __syncthreads();
      for (int e = tid; e < half * n; e += blockDim.x) {
        const int pi = e / n, r = e % n;
        const int p = sh.p[pi], q = sh.q[pi];
        const float c = rc[pi], s = rs[pi], hx = rx[pi], hy = ry[pi];
        if (q >= n || s == 0.f) continue;
        {
          const float2 xp = C[p * ld + r], xq = C[q * ld + r];
          const float ex = hx * xq.x - hy * xq.y, ey = hx * xq.y + hy * xq.x;
          C[p * ld + r] = make_float2(c * xp.x - s * ex, c * xp.y - s * ey);
          C[q * ld + r] = make_float2(s * xp.x + c * ex, s * xp.y + c * ey);
        }
        {
          const float2 xp = V[p * ld + r], xq = V[q * ld + r];
          const float ex = hx * xq.x - hy * xq.y, ey = hx * xq.y + hy * xq.x;
          V[p * ld + r] = make_float2(c * xp.x - s * ex, c * xp.y - s * ey);
          V[q * ld + r] = make_float2(s * xp.x + c * ex, s * xp.y + c * ey);
        }
      }
      __syncthreads();
      for (int e = tid; e < half * n; e += blockDim.x) {
        const int pi = e / n, col = e % n;
        const int p = sh.p[pi], q = sh.q[pi];
        const float c = rc[pi], s = rs[pi], hx = rx[pi], hy = -ry[pi];
        if (q >= n || s == 0.f) continue;
        const float2 xp = C[col * ld + p], xq = C[col * ld + q];
        const float ex = hx * xq.x - hy * xq.y, ey = hx * xq.y + hy * xq.x;
        C[col * ld + p] = make_float2(c * xp.x - s * ex, c * xp.y - s * ey);
        C[col * ld + q] = make_float2(s * xp.x + c * ex, s * xp.y + c * ey);
      }
      __syncthreads();
    }
    const int rotated = sh.flag;
    __syncthreads();
    if (!rotated) break;
  }
}

// V += V M for the n x n FP32 matrix M kept in the strictly lower slots of D
// (upper entry (i, j), i < j, in slot (j, i) as the first two floats; the
// entry (j, i) is sign * conj of it) with the real diagonal in diag(D).y when
// `diag`.  Row blocks of V are copied to FP32 first (buf, 2 kChunk rows).
static __device__ __noinline__ void apply_small(cd* V, const cd* D, int n, int ld, float sign, bool diag,
                                                float2* buf) {
  const int tid = threadIdx.x, rows = 2 * kChunk;
  for (int r0 = 0; r0 < n; r0 += rows) {
    const int nr = min(rows, n - r0);
    for (int e = tid; e < nr * n; e += blockDim.x) {
      const int r = e % nr, c = e / nr;
      const cd x = V[(size_t)c * ld + r0 + r];
      buf[r * ld + c] = make_float2((float)x.x, (float)x.y);
    }
    __syncthreads();
    for (int e = tid; e < nr * n; e += blockDim.x) {
      const int r = e % nr, j = e / nr;
      float2 s = make_float2(0.f, 0.f);
      for (int i = 0; i < j; ++i) fma_f(s, buf[r * ld + i], *reinterpret_cast<const float2*>(&D[(size_t)i * ld + j]));
      if (diag) {
        const float f = (float)D[(size_t)j * ld + j].y;
        const float2 b = buf[r * ld + j];
        s.x += f * b.x;
        s.y += f * b.y;
      }
      for (int i = j + 1; i < n; ++i) {
        const float2 u = *reinterpret_cast<const float2*>(&D[(size_t)j * ld + i]);
        fma_f(s, buf[r * ld + i], make_float2(sign * u.x, -sign * u.y));
      }
      cd& v = V[(size_t)j * ld + r0 + r];
      v.x += (double)s.x;
      v.y += (double)s.y;
    }
    __syncthreads();
  }
}

// Eigenpairs of C from approximate ones (V, any accuracy): returns with
// V^H C V diagonal and V orthonormal to FP64 rounding, eigenvalues in sh.w.
// One pass, with G = V^H V, D = V^H C V in FP64 and R = I - G:
//   Loewdin:  V <- V (I + R/2),  D'_ij = D_ij + R_ij (d_i + d_j) / 2
//   pairs whose entry is not small against the distance of their values (near
//   degeneracies) are rotated exactly (sweep_f64);
//   the rest to first order:  V <- V (I + E),  E_ij = D'_ij / (d_j - d_i).
// R and E are small, so they are kept and multiplied in FP32: their error is
// 6e-8 of a correction that the next pass measures in FP64 again.  A pass
// whose corrections are below 1e-8 leaves errors of their square and ends the
// iteration; the entries left alone are below 1e-14 / n of the diagonal's
// norm (together the 1e-14 bar of the plain method).  If the passes do not
// settle, the plain FP64 Jacobi iteration runs from V = I.
static __device__ __noinline__ void refine(cd* C, cd* V, cd* D, cd* T, int n, int ld, Shared& sh, double* trace) {
  constexpr double kRatio = 1e-4;
  const int tid = threadIdx.x;
  const int m = (n + 1) & ~1, upper = m * (m + 1) / 2;
  bool done = false;
  for (int pass = 0; pass < 8 && !done; ++pass) {
    if (tid == 0) { sh.emax = 0u; sh.rmax = 0u; }
    // ---- D = V^H C V (upper, FP64), R = I - V^H V (slots below, FP32) ----------
    double off = 0.0, dg = 0.0;
    for (int j0 = 0; j0 < n; j0 += kChunk) {
      const int nj = min(kChunk, n - j0);
      __syncthreads();
      for (int e = tid; e < nj * n; e += blockDim.x) {
        const int r = e % n, j = e / n;
        cd s = {0.0, 0.0};
        for (int q = 0; q < n; ++q) fma_plain(s, C[(size_t)q * ld + r], V[(size_t)(j0 + j) * ld + q]);
        T[j * ld + r] = s;
      }
      __syncthreads();
      for (int e = tid; e < nj * (j0 + nj); e += blockDim.x) {
        const int i = e % (j0 + nj), j = e / (j0 + nj);
        if (i > j0 + j) continue;
        cd s = {0.0, 0.0};
        for (int r = 0; r < n; ++r) fma_conj(s, V[(size_t)i * ld + r], T[j * ld + r]);
        if (i == j0 + j) {
          s.y = 0.0;
          sh.w[i] = s.x;
          dg += s.x * s.x;
        } else {
          off += 2.0 * (s.x * s.x + s.y * s.y);
        }
        D[(size_t)(j0 + j) * ld + i] = s;
      }
    }
    __syncthreads();
    float rm = 0.f;
    for (int e = tid; e < upper; e += blockDim.x) {
      int i, j;
      if (!upper_element(e, m, n, i, j)) continue;
      cd s = {i == j ? -1.0 : 0.0, 0.0};
      for (int r = 0; r < n; ++r) fma_conj(s, V[(size_t)i * ld + r], V[(size_t)j * ld + r]);
      const float2 h = make_float2(-0.5f * (float)s.x, -0.5f * (float)s.y);       // R / 2
      rm = fmaxf(rm, fmaxf(fabsf(h.x), fabsf(h.y)));
      if (!(h.x == h.x) || !(h.y == h.y)) rm = 1e30f;
      if (i == j) D[(size_t)i * ld + i].y = (double)h.x;
      else *reinterpret_cast<float2*>(&D[(size_t)i * ld + j]) = h;
    }
    atomicMax(&sh.rmax, __float_as_uint(rm));
    off = block_sum(off, sh);
    dg = block_sum(dg, sh);
    if (trace && tid == 0) {
      trace[2 * pass] = off;
      trace[2 * pass + 1] = dg;
    }
    const float rmax = __uint_as_float(sh.rmax);
    const double floor = 1e-14 * sqrt(dg) / n;
    if (!(rmax < 0.1f)) break;
    // ---- Loewdin step ------------------------------------------------------------
    apply_small(V, D, n, ld, 1.f, true, reinterpret_cast<float2*>(T));
    for (int e = tid; e < upper; e += blockDim.x) {
      int i, j;
      if (!upper_element(e, m, n, i, j)) continue;
      if (i == j) {
        cd& d = D[(size_t)i * ld + i];
        d = {sh.w[i] * (1.0 + 2.0 * d.y), 0.0};
      } else {
        const float2 h = *reinterpret_cast<const float2*>(&D[(size_t)i * ld + j]);
        const double dd = sh.w[i] + sh.w[j];
        cd& u = D[(size_t)j * ld + i];
        u = {u.x + dd * h.x, u.y + dd * h.y};
        D[(size_t)i * ld + j] = {u.x, -u.y};
      }
    }
    __syncthreads();
    // ---- near-degenerate pairs exactly ----------------------------------------------
    for (int it = 0; it < 12; ++it) {
      bool strong = false;
      for (int e = tid; e < upper; e += blockDim.x) {
        int i, j;
        if (!upper_element(e, m, n, i, j) || i == j) continue;
        const cd u = D[(size_t)j * ld + i];
        const double b2 = u.x * u.x + u.y * u.y;
        const double g = kRatio * (D[(size_t)j * ld + j].x - D[(size_t)i * ld + i].x);
        strong |= b2 > floor * floor && b2 > g * g;
      }
      if (!__syncthreads_or(strong)) break;
      sweep_f64(D, V, n, ld, floor, kRatio, sh);
    }
    // ---- the others to first order -----------------------------------------------------
    float em = 0.f;
    for (int e = tid; e < upper; e += blockDim.x) {
      int i, j;
      if (!upper_element(e, m, n, i, j) || i == j) continue;
      const cd u = D[(size_t)j * ld + i];
      const double g = D[(size_t)j * ld + j].x - D[(size_t)i * ld + i].x;
      const double b2 = u.x * u.x + u.y * u.y;
      float2 E = make_float2(0.f, 0.f);
      if (b2 <= kRatio * kRatio * g * g && g != 0.0) {
        const double ig = 1.0 / g;
        E = make_float2((float)(u.x * ig), (float)(u.y * ig));
      } else if (b2 > floor * floor) {
        em = 1.f;                 // still strong: another pass
      }
      em = fmaxf(em, fmaxf(fabsf(E.x), fabsf(E.y)));
      *reinterpret_cast<float2*>(&D[(size_t)i * ld + j]) = E;
    }
    atomicMax(&sh.emax, __float_as_uint(em));
    for (int i = tid; i < n; i += blockDim.x) sh.w[i] = D[(size_t)i * ld + i].x;
    __syncthreads();
    const float emax = __uint_as_float(sh.emax);
    apply_small(V, D, n, ld, -1.f, false, reinterpret_cast<float2*>(T));
    done = emax <= 1e-8f && rmax <= 1e-8f;
    __syncthreads();
  }
  if (done) return;
  // ---- plain cyclic Jacobi ---------------------------------------------------------
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int r = e % n, c = e / n;
    V[(size_t)c * ld + r] = {r == c ? 1.0 : 0.0, 0.0};
    D[(size_t)c * ld + r] = C[(size_t)c * ld + r];
  }
  __syncthreads();
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0, dg = 0.0;
    for (int e = tid; e < n * n; e += blockDim.x) {
      const int r = e % n, c = e / n;
      const cd x = D[(size_t)c * ld + r];
      const double a2 = x.x * x.x + x.y * x.y;
      if (r == c) dg += a2; else off += a2;
    }
    off = block_sum(off, sh);
    dg = block_sum(dg, sh);
    if (off <= 1e-28 * dg || off == 0.0) break;
    sweep_f64(D, V, n, ld, 0.0, 0.0, sh);
  }
  for (int i = tid; i < n; i += blockDim.x) sh.w[i] = D[(size_t)i * ld + i].x;
  __syncthreads();
}

// All threads of the CTA must call this.  In: U = B, C = A.  Out: the upper
// factor of B in u_out (global, n x n, column-major; its inverse diagonal in
// sh.dinv), eigenvalues in sh.w (unsorted), reduced eigenvectors in U; C and
// W hold scratch.  sh.fail != 0 on return when B is not positive definite.
// trace (nullable) receives (off, diag) per refinement pass.
static __device__ __noinline__ void hegv_reduced(cd* U, cd* C, cd* W, cd* T, int n, int ld, bool u_factored,
                                                 cd* __restrict__ u_out, Shared& sh, double* trace) {
  const int tid = threadIdx.x;
  if (tid == 0) sh.fail = 0;
  __syncthreads();
  // ---- 1. Cholesky B = U^H U (right-looking, upper) -------------------------
  for (int j = 0; j < n; ++j) {
    if (tid == 0) {
      const double d = U[(size_t)j * ld + j].x;
      double u = d;
      if (!u_factored) {
        if (!(d > 0.0)) sh.fail = n + j + 1;
        u = sqrt(fmax(d, 1e-300));
        U[(size_t)j * ld + j] = {u, 0.0};
      }
      sh.dinv[j] = 1.0 / u;
    }
    if (u_factored) continue;
    __syncthreads();
    if (sh.fail) return;
    const double inv = sh.dinv[j];
    for (int i = j + 1 + tid; i < n; i += blockDim.x) {   // row j, columns i > j
      cd& u = U[(size_t)i * ld + j];
      u.x *= inv;
      u.y *= inv;
    }
    __syncthreads();
    // trailing update B(r,c) -= conj(U(j,r)) U(j,c) for j < r <= c
    const int t = n - j - 1, mt = (t + 1) & ~1;
    for (int e = tid; e < mt * (mt + 1) / 2; e += blockDim.x) {
      int r, c;
      if (!upper_element(e, mt, t, r, c)) continue;
      r += j + 1;
      c += j + 1;
      cd& x = U[(size_t)c * ld + r];
      x = csub(x, cmulc(U[(size_t)r * ld + j], U[(size_t)c * ld + j]));
    }
    __syncthreads();
  }
  __syncthreads();
  // ---- 2. C = U^{-H} A U^{-1} ------------------------------------------------
  // Y = U^{-H} A, row i of the result finished, then taken out of the rows below
  for (int i = 0; i < n; ++i) {
    const double inv = sh.dinv[i];
    for (int c = tid; c < n; c += blockDim.x) {
      cd& x = C[(size_t)c * ld + i];
      x.x *= inv;
      x.y *= inv;
    }
    __syncthreads();
    const int t = n - i - 1;
    for (int e = tid; e < t * n; e += blockDim.x) {
      const int r = i + 1 + e % t, c = e / t;
      cd& x = C[(size_t)c * ld + r];
      x = csub(x, cmulc(U[(size_t)r * ld + i], C[(size_t)c * ld + i]));
    }
    __syncthreads();
  }
  // C = Y U^{-1}, lower triangle (r >= c), column by column
  for (int j = 0; j < n; ++j) {
    const double inv = sh.dinv[j];
    for (int r = j + tid; r < n; r += blockDim.x) {
      cd& x = C[(size_t)j * ld + r];
      x.x *= inv;
      x.y *= inv;
    }
    __syncthreads();
    const int t = n - j - 1, mt = (t + 1) & ~1;
    for (int e = tid; e < mt * (mt + 1) / 2; e += blockDim.x) {
      int c, r;                                            // c <= r
      if (!upper_element(e, mt, t, c, r)) continue;
      r += j + 1;
      c += j + 1;
      cd& x = C[(size_t)c * ld + r];
      x = csub(x, cmul(C[(size_t)j * ld + r], U[(size_t)c * ld + j]));
    }
    __syncthreads();
  }
  float cmax = 0.f;
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int r = e % n, c = e / n;
    u_out[e] = r <= c ? U[(size_t)c * ld + r] : cd{0.0, 0.0};
    if (r > c) {
      const cd x = C[(size_t)c * ld + r];
      C[(size_t)r * ld + c] = {x.x, -x.y};
      cmax = fmaxf(cmax, fmaxf(fabsf((float)x.x), fabsf((float)x.y)));
    } else if (r == c) {
      C[(size_t)c * ld + c].y = 0.0;
      cmax = fmaxf(cmax, fabsf((float)C[(size_t)c * ld + c].x));
    }
  }
  if (tid == 0) sh.emax = 0u;
  __syncthreads();
  atomicMax(&sh.emax, __float_as_uint(cmax));
  __syncthreads();
  // ---- 3. FP32 eigenvectors (scaled to entries of at most 1) -----------------
  const float big = __uint_as_float(sh.emax);
  const double scale = big > 0.f && big < 3e38f ? 1.0 / (double)big : 1.0;
  float2* C32 = reinterpret_cast<float2*>(W);
  float2* V32 = C32 + (size_t)n * ld;
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int r = e % n, c = e / n;
    const cd x = C[(size_t)c * ld + r];
    C32[c * ld + r] = make_float2((float)(x.x * scale), (float)(x.y * scale));
  }
  __syncthreads();
  jacobi_f32(C32, V32, n, ld, sh);
  for (int e = tid; e < n * n; e += blockDim.x) {
    const int r = e % n, c = e / n;
    const float2 x = V32[c * ld + r];
    U[(size_t)c * ld + r] = {(double)x.x, (double)x.y};
  }
  __syncthreads();
  // ---- 4. refinement -------------------------------------------------------------
  refine(C, U, W, T, n, ld, sh, trace);
}

// Ascending order of sh.w into sh.order, ties by index and NaN (of a matrix that
// holds one) after every number: order is a permutation whatever w holds.
static __device__ __forceinline__ void sorted_order(int n, Shared& sh) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double wi = sh.w[i];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double wj = sh.w[j];
      const bool tie = wj == wi || (isnan(wj) && isnan(wi));
      rank += wj < wi || (isnan(wi) && !isnan(wj)) || (tie && j < i);
    }
    sh.order[rank] = i;
  }
  __syncthreads();
}

}  // namespace jac
}  // namespace olc
