// jacobi.cuh -- one-CTA cyclic Jacobi eigensolver for a symmetric matrix, as
// device routines shared by the batched eigensolver kernel (linalg.cu) and the
// per-molecule SCF kernels of the batch engine (batch.cu).
//
// An FP32 Jacobi gives start vectors, products on the tensor cores refine them to
// FP64, and a cyclic FP64 Jacobi finishes where that leaves something.  Each sweep runs
// the n'-1 rounds of a round-robin tournament (n' = n rounded
// up to even); a round rotates n'/2 disjoint index pairs at once.
// Converges when the off-diagonal Frobenius norm falls below
// tol * ||A||_F.  Replaces the eigen step of DSYEV/DSYGV (src/scf/scf.f90:692,
// 478, 848).
#pragma once
#include "fixmm.cuh"

namespace mq {

__device__ __forceinline__ void rr_pair(int np, int r, int k, int &p, int &q) {
  // circle method: player 0 fixed, players 1..np-1 rotate
  const int m = np - 1;
  if (k == 0) {
    p = 0;
    q = 1 + (r % m);
  } else {
    p = 1 + (r + k) % m;
    q = 1 + (r - k + m) % m;
  }
  if (p > q) {
    int t = p;
    p = q;
    q = t;
  }
}

// Sum (largest) over the block of one value per thread, in every thread (red:
// 32 entries).  One warp adds the warps' sums: each FP64 addition occupies its
// SM for 16 clocks per warp, so sixteen warps each adding sixteen sums would
// take 4000.
template <class T, class Op>
__device__ __forceinline__ T jac_block_reduce(T v, T *red, T zero, Op op) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    T t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : zero;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = op(t, __shfl_xor_sync(0xffffffffu, t, o));
    __syncwarp();
    if (threadIdx.x == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}
__device__ __forceinline__ double jac_block_sum(double v, double *red) {
  return jac_block_reduce(v, red, 0.0, [](double a, double b) { return a + b; });
}
__device__ __forceinline__ float jac_block_sum(float v, double *red) {
  return jac_block_reduce(v, reinterpret_cast<float *>(red), 0.f, [](float a, float b) { return a + b; });
}
__device__ __forceinline__ double jac_block_max(double v, double *red) {
  return jac_block_reduce(v, red, 0.0, [](double a, double b) { return fmax(a, b); });
}

// acc(i, j, (X Y)_ij) of two n x n FP32 matrices
template <class Acc>
__device__ __forceinline__ void jac_mm_f32(int n, const float *X, const float *Y, Acc acc) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int j = w; j < n; j += nw)
    for (int i = lane; i < n; i += 32) {
      float s = 0.f;
#pragma unroll 4
      for (int l = 0; l < n; ++l) s = fmaf(X[i + n * l], Y[l + n * j], s);
      acc(i, j, s);
    }
}

// pair k of round r as rr_pair gives it (r < np - 1), without integer division
__device__ __forceinline__ void rr_pair_fast(int np, int r, int k, int &p, int &q) {
  const int m = np - 1;
  int a = r + k, b = r - k;
  if (a >= m) a -= m;
  if (b < 0) b += m;
  a += 1;
  b = k == 0 ? 0 : b + 1;
  p = min(a, b);
  q = max(a, b);
}

// Tangent of the Jacobi angle that annihilates apq, from aqq - app, in FP32
// with the approximate reciprocal and square root (any angle near it
// converges); apq != 0.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float tangent_f32(float diff, float apq) {
  // 2 apq / (|diff| + sqrt(diff^2 + 4 apq^2)), signed: one reciprocal
  const float b = 2.f * apq, t = fabsf(b) * rcp_approx(fabsf(diff) + sqrt_approx(fmaf(diff, diff, b * b)));
  return copysignf(1.f, diff) * copysignf(1.f, apq) * fminf(t, 1.f);
}

// FP32 cyclic Jacobi of A0 (n x n, n <= 128, destroyed with its twin A1), Vf <-
// the rotations: the start vectors of jacobi_block.  A round rotates n'/2
// disjoint pairs as independent 2 x 2 blocks (rows {p, q} of pair P, columns
// {u, v} of pair Q).  Every warp computes all the round's angles itself, a pair
// per lane (the lanes are idle otherwise), and writes the blocks of its pairs Q
// to the other copy of A, so that a round costs one barrier.  Ends at an
// off-diagonal norm of 1e-6 ||A||_F, near FP32's floor, or when a late sweep no
// longer halves it.
template <int CH>  // pairs per lane: n <= 64 CH
static __device__ __forceinline__ void jacobi_block_f32(int n, float *A0, float *A1, float *Vf, double *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int np = n + (n & 1), half = np / 2;
  float fro = 0.f;
  for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) fro += A0[idx] * A0[idx];
  const float stop = 1e-12f * jac_block_sum(fro, red);
  float last = INFINITY;
  for (int sweep = 0; sweep < 12; ++sweep) {
    float off = 0.f;
    for (int j = w; j < n; j += nw)
      for (int i = lane; i < n; i += 32)
        if (i != j) off += A0[i + n * j] * A0[i + n * j];
    off = jac_block_sum(off, red);
    if (!(off > stop) || (sweep > 6 && off > 0.25f * last)) return;
    last = off;
    for (int r = 0; r < np - 1; ++r) {
      const float *__restrict__ Ai = A0;
      float *__restrict__ Ao = A1;
      float cs[CH], sn[CH];
      int pp[CH], qq[CH];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        rr_pair_fast(np, r, min(lane + 32 * c, half - 1), pp[c], qq[c]);
        cs[c] = 1.f;
        sn[c] = 0.f;
        if (qq[c] < n) {
          const int p = pp[c], q = qq[c];
          const float apq = Ai[p + n * q], app = Ai[p + n * p], aqq = Ai[q + n * q];
          if (fabsf(apq) > 1e-9f * (fabsf(app) + fabsf(aqq))) {
            const float t = tangent_f32(aqq - app, apq);
            asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(cs[c]) : "f"(fmaf(t, t, 1.f)));
            sn[c] = t * cs[c];
          }
        } else {  // the dummy index: unit rotation, both copies of the row get the same value
          qq[c] = pp[c];
        }
      }
      for (int Q = w; Q < half; Q += nw) {
        const float cq = __shfl_sync(0xffffffffu, CH == 1 || Q < 32 ? cs[0] : cs[CH - 1], Q & 31);
        const float sq = __shfl_sync(0xffffffffu, CH == 1 || Q < 32 ? sn[0] : sn[CH - 1], Q & 31);
        int u, v;
        rr_pair_fast(np, r, Q, u, v);
        const bool vv = v < n;
        const int cu = n * u, cv = n * (vv ? v : u);
        float x[2 * CH], y[2 * CH];  // V's columns u and v
#pragma unroll
        for (int c = 0; c < 2 * CH; ++c) {
          const int i = lane + 32 * c;
          x[c] = i < n ? Vf[cu + i] : 0.f;
          y[c] = i < n ? Vf[cv + i] : 0.f;
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          const int p = pp[c], q = qq[c];
          const float apu = Ai[cu + p], aqu = Ai[cu + q], apv = Ai[cv + p], aqv = Ai[cv + q];
          const float bpu = cs[c] * apu - sn[c] * aqu, bqu = sn[c] * apu + cs[c] * aqu;
          const float bpv = cs[c] * apv - sn[c] * aqv, bqv = sn[c] * apv + cs[c] * aqv;
          if (lane + 32 * c < half) {
            Ao[cu + p] = cq * bpu - sq * bpv;
            Ao[cu + q] = cq * bqu - sq * bqv;
            if (vv) {
              Ao[cv + p] = sq * bpu + cq * bpv;
              Ao[cv + q] = sq * bqu + cq * bqv;
            }
          }
        }
#pragma unroll
        for (int c = 0; c < 2 * CH; ++c) {
          const int i = lane + 32 * c;
          if (i < n && vv) {
            Vf[cu + i] = cq * x[c] - sq * y[c];
            Vf[cv + i] = sq * x[c] + cq * y[c];
          }
        }
      }
      float *t = A0;
      A0 = A1;
      A1 = t;
      __syncthreads();
    }
  }
}

// Scratch of jacobi_block and of the products beside it: two fixed-point copies
// of an n x n matrix, two exponents per row and a sine and cosine per pair.
__host__ __device__ constexpr int jacobi_work(int n) {  // doubles, even
  return 2 * n * 2 * fx_ld(n) + (n + 2 * (n + 1) + 1) / 2 * 2;
}
struct JacobiWork {
  uint4 *U1, *U2;
  double *cs;
  int *e1, *e2;
  __device__ __forceinline__ JacobiWork(double *work, int n)
      : U1(reinterpret_cast<uint4 *>(work)), U2(U1 + n * fx_ld(n)), cs(reinterpret_cast<double *>(U2 + n * fx_ld(n))),
        e1(reinterpret_cast<int *>(cs + 2 * ((n + 1) / 2))), e2(e1 + n) {}
};

// Diagonalise A in place (n x n, n <= 128, column-major, shared or global
// memory of this CTA), V <- its eigenvectors.  red: 32 doubles, work:
// jacobi_work(n) doubles of this CTA on a 16-byte boundary (shared or global
// memory).  Returns false when max_sweeps did not reach the tolerance
// ||offdiag||_F <= tol ||A||_F, or A is not finite (V is then NaN).
//
// A cold FP64 Jacobi is bound by FP64 issue (two multiply-adds per clock and
// SM): nine sweeps of 6 n^3.  So the sweeps run in FP32 for start vectors, and
// FP64 work is products on the tensor cores (fixmm.cuh: within rounding of the rows'
// norms, as the whole solve is of ||A||):
//   V <- V (I - E/2 + 3/8 E^2 [- 5/16 E^3]), E = V^T V - I   orthonormal to rounding
//     (||E|| grows with n to 5e-5; without the cubic term max |V^T V - I| is 5e-16 at
//     n = 15, 5e-15 at 56 and 1e-14 at 64, with it 1e-15 to 2e-15: taken above 64)
//   A <- V^T A V                                off-diagonals 1e-6 ||A||_F
//   twice: P = I + E + E^2/2 [+ E^3/8] with the first-order rotations E_ij =
//     a_ij / (a_jj - a_ii) of the pairs with |E_ij| <= 3e-4; V <- V P, A <- P^T A P
//     (the second step's E is quadratically smaller)
// Nothing after the steps restores orthogonality, and what they leave of it is a power of
// the norm of E, not of its largest entry: E is antisymmetric, so P^T P - I = E^4/4
// without and -E^6/64 with the cubic term.  The norm is bounded by r = ||E||_F / sqrt(2)
// (singular values come in pairs; a dense E has r two to four times the norm), and the
// term taken above r = 4e-4 (6e-15, some 2e-16).  Fock matrices of an SCF of (H2O)8 have r
// around 3e-4.  Levels spaced 1e-5 to 5e-4 of the norm give ||E|| = 1e-3 to 2e-3 (r up to
// 1e-2): max |V^T V - I| 1.5e-12 at n = 110 without the term, 2e-14 with it, as a cold
// FP64 Jacobi.  Above r = 6e-3 (7e-16) only the pairs with |E_ij| <= 6e-3 / n are
// rotated, whose norm is below that.
// Pairs that this leaves (near-degenerate levels) go to FP64 Jacobi sweeps, which
// check the stopping rule of a cold solve and skip every rotation below
// tol ||A||_F / n: none where all levels are 1e-2 of the norm apart, two or three
// where they are closer.
static __device__ bool jacobi_block(int n, double *A, double *V, double *red, double *work, int max_sweeps,
                                    double tol) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int n2 = n * n;
  const JacobiWork jw(work, n);
  uint4 *U1 = jw.U1, *U2 = jw.U2;
  double *cs = jw.cs;
  int *e1 = jw.e1, *e2 = jw.e2;
  double big = 0.0, fro = 0.0;
  for (int idx = tid; idx < n2; idx += blockDim.x) big = fmax(big, fabs(A[idx]));
  big = jac_block_max(big, red);
  // a power of two that brings A into FP32's range and its squares into FP64's
  const double scale = big > 1e-290 && big < 1e290 ? exp2(-(double)ilogb(big)) : 1.0;
  for (int idx = tid; idx < n2; idx += blockDim.x) fro = fma(A[idx] * scale, A[idx] * scale, fro);
  fro = jac_block_sum(fro, red);
  if (!isfinite(fro)) {  // infinities or NaN in A
    for (int idx = tid; idx < n2; idx += blockDim.x) V[idx] = fro - fro;
    __syncthreads();
    return false;
  }
  const double stop2 = tol * tol * fro, skip = tol * sqrt(fro) / (n * scale);
  const int np = n + (n & 1), half = np / 2;
  auto off_norm2 = [&]() {
    double off = 0.0;
    for (int j = w; j < n; j += nw)
      for (int i = j + 1 + lane; i < n; i += 32) {
        const double x = A[i + (size_t)n * j] * scale;
        off = fma(x, x, off);
      }
    return 2.0 * jac_block_sum(off, red);
  };
  auto mirror = [&]() {  // (a congruence is symmetric but for the rounding of its halves)
    __syncthreads();
    for (int j = w; j < n; j += nw)
      for (int i = j + 1 + lane; i < n; i += 32) A[j + (size_t)n * i] = A[i + (size_t)n * j];
    __syncthreads();
  };
  auto col = [&](const double *x) { return [=](int r, int k) { return x[k + (size_t)n * r]; }; };
  auto row = [&](const double *x) { return [=](int r, int k) { return x[r + (size_t)n * k]; }; };
  {
    float *Vf = reinterpret_cast<float *>(V), *Af = Vf + n2;
    for (int idx = tid; idx < n2; idx += blockDim.x) {
      Af[idx] = (float)(A[idx] * scale);
      Vf[idx] = idx % (n + 1) == 0 ? 1.f : 0.f;
    }
    __syncthreads();
    if (n <= 64) jacobi_block_f32<1>(n, Af, reinterpret_cast<float *>(work), Vf, red);
    else jacobi_block_f32<2>(n, Af, reinterpret_cast<float *>(work), Vf, red);
    __syncthreads();
    double *W = reinterpret_cast<double *>(U2);
    for (int idx = tid; idx < n2; idx += blockDim.x) W[idx] = (double)Vf[idx];
    for (int i = tid; i < n; i += blockDim.x) e1[i] = 1;  // |entries| of a rotation < 2
    __syncthreads();
    cta_fix(n, n, true, e1, U1, col(W));
    __syncthreads();
    cta_fix_mm(n, n, n, U1, e1, U1, e1, [&](int i, int j, double v) { V[i + n * j] = v - (i == j ? 1.0 : 0.0); });
    __syncthreads();
    // ||E|| is below 1e-4: the FP32 rounding of its square and cube is below 1e-15
    float *Ef = reinterpret_cast<float *>(U1), *Qf = Ef + n2;
    for (int idx = tid; idx < n2; idx += blockDim.x) Ef[idx] = (float)V[idx];
    __syncthreads();
    const bool cubic = n > 64;
    if (cubic) {  // 3/8 E^2 - 5/16 E^3 = E (3/8 E - 5/16 E^2)
      jac_mm_f32(n, Ef, Ef, [&](int i, int j, float s) { Qf[i + n * j] = 0.375f * Ef[i + n * j] - 0.3125f * s; });
      __syncthreads();
    }
    const double c2 = cubic ? 1.0 : 0.375;
    jac_mm_f32(n, Ef, cubic ? Qf : Ef, [&](int i, int j, float s) {
      V[i + (size_t)n * j] = (i == j ? 1.0 : 0.0) - 0.5 * V[i + (size_t)n * j] + c2 * (double)s;
    });
    __syncthreads();
    cta_fix(n, n, false, e1, U1, row(W));
    __syncthreads();
    cta_fix(n, n, true, e1, U2, col(V));
    __syncthreads();
    cta_fix_mm(n, n, n, U1, e1, U2, e1, [&](int i, int j, double v) { V[i + n * j] = v; });
    __syncthreads();
    // A <- V^T (A V)
    for (int i = tid; i < n; i += blockDim.x) e2[i] = 1;
    cta_row_exp(n, n, A, n, 1, e1);
    __syncthreads();
    cta_fix(n, n, true, e1, U1, col(A));
    cta_fix(n, n, true, e2, U2, col(V));
    __syncthreads();
    cta_fix_mm(n, n, n, U1, e1, U2, e2, [&](int i, int j, double v) { A[i + n * j] = v; });
    __syncthreads();
    cta_row_exp(n, n, A, n, 1, e1);
    __syncthreads();
    cta_fix(n, n, true, e1, U1, col(A));
    __syncthreads();
    cta_fix_mm(n, n, n, U2, e2, U1, e1, [&](int i, int j, double v) { A[i + n * j] = v; });
    mirror();
  }
  for (int step = 0; step < 2; ++step) {
    const double off2 = off_norm2();
    if (off2 <= stop2) return true;
    constexpr float EMAX = 3e-4f, RCUBIC = 4e-4f, RMAX = 6e-3f;
    constexpr int EEXP = -11;  // EMAX < 2^EEXP
    float emax = EMAX;
    auto E = [&](int i, int j) {
      const double a = A[i + (size_t)n * j], gap = A[j + (size_t)n * j] - A[i + (size_t)n * i];
      const float x = (float)(a * scale), g = (float)(gap * scale);
      const float e = __fdividef(x, g);
      return i != j && fabsf(e) <= emax ? e : 0.f;  // (x / 0 is not taken)
    };
    for (int i = tid; i < n; i += blockDim.x) e1[i] = EEXP, e2[i] = 1;
    __syncthreads();
    float f2 = 0.f;
    auto columns = [&]() {  // of E
      cta_fix(n, n, true, e1, U2, [&](int c, int k) {
        const float e = E(k, c);
        f2 = fmaf(e, e, f2);
        return (double)e;
      });
    };
    columns();
    const float r = sqrtf(0.5f * jac_block_sum(f2, red));
    if (r > RMAX) {
      emax = RMAX / n;
      columns();
      __syncthreads();
    }
    double *P = reinterpret_cast<double *>(U1);
    cta_fix_mm(n, n, n, U2, e1, U2, e1, [&](int i, int j, double v) {  // v = (E^T E)_ij = -(E^2)_ij
      P[i + n * j] = (i == j ? 1.0 : 0.0) + (double)E(i, j) - 0.5 * v;
    });
    __syncthreads();
    if (r > RCUBIC) {  // E^3/8 is below 3e-8: FP32
      float *Ef = reinterpret_cast<float *>(U2), *Qf = Ef + n2;
      for (int j = w; j < n; j += nw)
        for (int i = lane; i < n; i += 32) {
          const float e = E(i, j);
          Ef[i + n * j] = e;
          Qf[i + n * j] = (float)(2.0 * (P[i + n * j] - (i == j ? 1.0 : 0.0) - (double)e));  // (E^2)_ij
        }
      __syncthreads();
      jac_mm_f32(n, Ef, Qf, [&](int i, int j, float s) { P[i + n * j] += 0.125 * (double)s; });
      __syncthreads();
    }
    cta_fix(n, n, true, e2, U2, col(P));  // the columns of P
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) e1[i] = 1;
    __syncthreads();
    cta_fix(n, n, false, e1, U1, row(V));
    __syncthreads();
    cta_fix_mm(n, n, n, U1, e1, U2, e2, [&](int i, int j, double v) { V[i + n * j] = v; });
    __syncthreads();
    cta_row_exp(n, n, A, n, 1, e1);
    __syncthreads();
    cta_fix(n, n, true, e1, U1, col(A));
    __syncthreads();
    cta_fix_mm(n, n, n, U1, e1, U2, e2, [&](int i, int j, double v) { A[i + n * j] = v; });
    __syncthreads();
    cta_row_exp(n, n, A, n, 1, e1);
    __syncthreads();
    cta_fix(n, n, true, e1, U1, col(A));
    __syncthreads();
    cta_fix_mm(n, n, n, U2, e2, U1, e1, [&](int i, int j, double v) { A[i + n * j] = v; });
    mirror();
  }
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (off_norm2() <= stop2) return true;
    for (int r = 0; r < np - 1; ++r) {
      int any = 0;
      for (int k = tid; k < half; k += blockDim.x) {
        int p, q;
        rr_pair_fast(np, r, k, p, q);
        double c = 1.0, s = 0.0;
        if (q < n) {
          const double apq = A[p + (size_t)n * q];
          // rotations below tol ||A||_F / n are skipped (all such pairs
          // together stay under the stopping threshold)
          if (fabs(apq) > skip) {
            // the tangent in FP32, the rotation orthogonal to FP64 rounding:
            // what it leaves of apq (1e-7 of it) is kept in A
            const double diff = (A[q + (size_t)n * q] - A[p + (size_t)n * p]) * scale;
            const double t = (double)tangent_f32((float)diff, (float)(apq * scale)), t2 = t * t;
            c = t2 < 1e-6 ? fma(t2, fma(t2, fma(t2, -0.3125, 0.375), -0.5), 1.0) : rsqrt(1.0 + t2);
            s = t * c;
            any = 1;
          }
        }
        cs[2 * k] = c;
        cs[2 * k + 1] = s;
      }
      if (!__syncthreads_or(any)) continue;
      // blocks (P, Q), P >= Q, of A and their mirror images, one per thread
      for (int idx = tid; idx < half * (half + 1) / 2; idx += blockDim.x) {
        int P = (int)((sqrtf(8.f * (float)idx + 1.f) - 1.f) * 0.5f);
        if (P * (P + 1) / 2 > idx) --P;
        if ((P + 1) * (P + 2) / 2 <= idx) ++P;
        const int Q = idx - P * (P + 1) / 2;
        const double cP = cs[2 * P], sP = cs[2 * P + 1], cQ = cs[2 * Q], sQ = cs[2 * Q + 1];
        if (sP == 0.0 && sQ == 0.0) continue;
        int p, q, u, v;
        rr_pair_fast(np, r, P, p, q);
        rr_pair_fast(np, r, Q, u, v);
        const bool qv = q < n, vv = v < n;
        double *au = A + (size_t)n * u, *av = A + (size_t)n * (vv ? v : u);
        if (P == Q) {  // the rotated 2 x 2 block
          const double app = au[u], aqq = av[v], apq = au[v];
          const double bpp = cP * app - sP * apq, bqp = sP * app + cP * apq;
          const double bpq = cP * apq - sP * aqq, bqq = sP * apq + cP * aqq;
          au[u] = cP * bpp - sP * bpq;
          av[v] = sP * bqp + cP * bqq;
          au[v] = av[u] = cP * bqp - sP * bqq;
          continue;
        }
        const double apu = au[p], aqu = qv ? au[q] : 0.0, apv = vv ? av[p] : 0.0, aqv = qv && vv ? av[q] : 0.0;
        const double bpu = cP * apu - sP * aqu, bqu = sP * apu + cP * aqu;
        const double bpv = cP * apv - sP * aqv, bqv = sP * apv + cP * aqv;
        const double npu = cQ * bpu - sQ * bpv, npv = sQ * bpu + cQ * bpv;
        const double nqu = cQ * bqu - sQ * bqv, nqv = sQ * bqu + cQ * bqv;
        au[p] = npu;
        A[u + (size_t)n * p] = npu;
        if (qv) {
          au[q] = nqu;
          A[u + (size_t)n * q] = nqu;
        }
        if (vv) {
          av[p] = npv;
          A[v + (size_t)n * p] = npv;
        }
        if (qv && vv) {
          av[q] = nqv;
          A[v + (size_t)n * q] = nqv;
        }
      }
      // V, one warp per pair
      for (int Q = w; Q < half; Q += nw) {
        const double cQ = cs[2 * Q], sQ = cs[2 * Q + 1];
        if (sQ == 0.0) continue;
        int u, v;
        rr_pair_fast(np, r, Q, u, v);
        double *vu = V + (size_t)n * u, *v2 = V + (size_t)n * v;
        for (int i = lane; i < n; i += 32) {
          const double x = vu[i], y = v2[i];
          vu[i] = cQ * x - sQ * y;
          v2[i] = sQ * x + cQ * y;
        }
      }
      __syncthreads();
    }
  }
  return false;
}

// Rank of eigenvalue i among the diagonal of A (ascending, ties by index): the
// ranks are a permutation of 0 .. n - 1 whatever the diagonal holds, since
// callers place i at its rank.  The bit patterns, ordered as the numbers are,
// give NaN a place too.
__device__ __forceinline__ int jacobi_rank(int n, const double *A, int i) {
  auto key = [&](int j) {
    const long long b = __double_as_longlong(A[j + (size_t)n * j]);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
  };
  const long long ki = key(i);
  int rank = 0;
  for (int j = 0; j < n; ++j) {
    const long long kj = key(j);
    rank += kj < ki || (kj == ki && j < i);
  }
  return rank;
}

// Eigenvalues ascending into w, eigenvectors into the matching columns of Vout,
// each with its largest component positive.
static __device__ void jacobi_sorted_out(int n, const double *A, const double *V, double *w, double *Vout) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int rank = jacobi_rank(n, A, i);
    w[rank] = A[i + (size_t)n * i];
    double big = 0.0;
    for (int k = 0; k < n; ++k)
      if (fabs(V[k + (size_t)n * i]) > fabs(big)) big = V[k + (size_t)n * i];
    const double sg = big < 0 ? -1.0 : 1.0;
    for (int k = 0; k < n; ++k) Vout[k + (size_t)n * rank] = sg * V[k + (size_t)n * i];
  }
}

}  // namespace mq
