// jacobi.cuh -- one-CTA cyclic Jacobi eigensolver for a symmetric matrix, as
// device routines shared by the batched eigensolver kernel (linalg.cu) and the
// per-molecule SCF kernels of the batch engine (batch.cu).
//
// Each sweep runs the n'-1 rounds of a round-robin tournament (n' = n rounded
// up to even); a round rotates n'/2 disjoint index pairs at once: rotation
// angles, then rows, then columns of A and V, with a block barrier between
// phases.  Converges when the off-diagonal Frobenius norm falls below
// tol * ||A||_F.  Replaces the eigen step of DSYEV/DSYGV (src/scf/scf.f90:692,
// 478, 848).
#pragma once

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

// Sum over the block of one value per thread (red: blockDim.x/32 doubles).
__device__ __forceinline__ double jac_block_sum(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
  return t;
}

// Largest value of one per thread over the block.
__device__ __forceinline__ double jac_block_max(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = fmax(t, red[w]);
  return t;
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

// ---- FP64 products of one CTA, column-major, leading dimension = row count.
// GB300 issues two FP64 multiply-adds per clock and SM, so the point is to
// spend FP64 issue slots on nothing else: each thread forms a 2 x 4 block of
// the product (8 independent chains, 6 loads per 8 multiply-adds), with one
// integer division per block.
constexpr int MM_C = 4;

// C (m x n) = f A (m x k) op(B), op(B) = B (k x n) or, TB, the transpose of
// B (n x k); with `cols` the columns of B are taken in that order
template <bool TB = false>
static __device__ __forceinline__ void cta_mm(int m, int n, int k, const double *A, const double *B, double *C,
                                              double f = 1.0, const int *cols = nullptr) {
  const size_t sb = TB ? n : 1;
  const int hi = (m + 1) / 2, nj = (n + MM_C - 1) / MM_C;
  for (int t = threadIdx.x; t < hi * nj; t += blockDim.x) {
    const int tj = t / hi, i0 = t - tj * hi, i1 = i0 + hi < m ? i0 + hi : i0, j0 = tj * MM_C;
    const double *b[MM_C];
    double s0[MM_C], s1[MM_C];
#pragma unroll
    for (int c = 0; c < MM_C; ++c) {
      const int j = min(j0 + c, n - 1);
      b[c] = TB ? B + j : B + (size_t)k * (cols ? cols[j] : j);
      s0[c] = s1[c] = 0.0;
    }
#pragma unroll 4
    for (int l = 0; l < k; ++l) {
      const double a0 = A[i0 + (size_t)m * l], a1 = A[i1 + (size_t)m * l];
#pragma unroll
      for (int c = 0; c < MM_C; ++c) {
        const double x = b[c][sb * l];
        s0[c] = fma(a0, x, s0[c]);
        s1[c] = fma(a1, x, s1[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < MM_C; ++c)
      if (j0 + c < n) {
        C[i0 + (size_t)m * (j0 + c)] = f * s0[c];
        C[i1 + (size_t)m * (j0 + c)] = f * s1[c];
      }
  }
}

// C (n x n) = A^T B, all n x n.  A thread's rows are the columns i0, i1 of A; its
// sum starts at row (thread) mod n, so that neighbouring threads read
// addresses n + 1 apart (no shared-memory bank conflicts).
static __device__ __forceinline__ void cta_mm_tn(int n, const double *A, const double *B, double *C) {
  const int hi = (n + 1) / 2, nj = (n + MM_C - 1) / MM_C;
  for (int t = threadIdx.x; t < hi * nj; t += blockDim.x) {
    const int tj = t / hi, i0 = t - tj * hi, i1 = i0 + hi < n ? i0 + hi : i0, j0 = tj * MM_C;
    const double *a0 = A + (size_t)n * i0, *a1 = A + (size_t)n * i1;
    const double *b[MM_C];
    double s0[MM_C], s1[MM_C];
#pragma unroll
    for (int c = 0; c < MM_C; ++c) {
      b[c] = B + (size_t)n * min(j0 + c, n - 1);
      s0[c] = s1[c] = 0.0;
    }
    int l = i0;
#pragma unroll 4
    for (int s = 0; s < n; ++s) {
      const double x0 = a0[l], x1 = a1[l];
#pragma unroll
      for (int c = 0; c < MM_C; ++c) {
        const double x = b[c][l];
        s0[c] = fma(x0, x, s0[c]);
        s1[c] = fma(x1, x, s1[c]);
      }
      l = l + 1 < n ? l + 1 : 0;
    }
#pragma unroll
    for (int c = 0; c < MM_C; ++c)
      if (j0 + c < n) {
        C[i0 + (size_t)n * (j0 + c)] = s0[c];
        C[i1 + (size_t)n * (j0 + c)] = s1[c];
      }
  }
}

// Tangent of the Jacobi angle that annihilates apq, from aqq - app, in FP32
// with the fast reciprocal and square root (any angle near it converges).
__device__ __forceinline__ float tangent_f32(float diff, float apq) {
  const float theta = __fdividef(diff, 2.f * apq), a = fabsf(theta);
  const float t = a > 1e15f ? __fdividef(0.5f, a) : __fdividef(1.f, a + __fsqrt_rn(fmaf(a, a, 1.f)));
  return copysignf(t, theta);
}
__device__ __forceinline__ float2 rotation_f32(float diff, float apq) {
  const float t = tangent_f32(diff, apq), c = rsqrtf(fmaf(t, t, 1.f));
  return make_float2(c, t * c);
}

// FP32 cyclic Jacobi of Af (n x n, destroyed), Vf <- the rotations: the start
// vectors of jacobi_block.  A round rotates n'/2 disjoint pairs as independent
// 2 x 2 blocks (rows {p, q} of pair P, columns {u, v} of pair Q), so it needs
// one barrier after the angles and one after the update; a warp's lanes run
// over P, whose p and q are runs of consecutive indices (no bank conflicts).
// Ends at an off-diagonal norm of 1e-6 ||A||_F, near FP32's floor, or when a
// late sweep no longer halves it.
static __device__ void jacobi_block_f32(int n, float *Af, float *Vf, float2 *cs, double *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int np = n + (n & 1), half = np / 2;
  float fro = 0.f;
  for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) fro += Af[idx] * Af[idx];
  const float stop = 1e-12f * (float)jac_block_sum(fro, red);
  float last = INFINITY;
  for (int sweep = 0; sweep < 12; ++sweep) {
    float off = 0.f;
    for (int j = w; j < n; j += nw)
      for (int i = lane; i < n; i += 32)
        if (i != j) off += Af[i + n * j] * Af[i + n * j];
    off = (float)jac_block_sum(off, red);
    if (!(off > stop) || (sweep > 6 && off > 0.25f * last)) return;
    last = off;
    for (int r = 0; r < np - 1; ++r) {
      for (int k = threadIdx.x; k < half; k += blockDim.x) {
        int p, q;
        rr_pair_fast(np, r, k, p, q);
        float2 v = make_float2(1.f, 0.f);
        if (q < n) {
          const float apq = Af[p + n * q], app = Af[p + n * p], aqq = Af[q + n * q];
          if (fabsf(apq) > 1e-9f * (fabsf(app) + fabsf(aqq))) {
            v = rotation_f32(aqq - app, apq);
          }
        }
        cs[k] = v;
      }
      __syncthreads();
      for (int Q = w; Q < half; Q += nw) {
        int u, v;
        rr_pair_fast(np, r, Q, u, v);
        const float2 cq = cs[Q];
        const bool vv = v < n;
        float *au = Af + n * u, *av = Af + n * (vv ? v : u);
        for (int P = lane; P < half; P += 32) {
          int p, q;
          rr_pair_fast(np, r, P, p, q);
          const float2 cp = cs[P];
          const bool qv = q < n;
          const float apu = au[p], aqu = qv ? au[q] : 0.f, apv = vv ? av[p] : 0.f, aqv = qv && vv ? av[q] : 0.f;
          const float bpu = cp.x * apu - cp.y * aqu, bqu = cp.y * apu + cp.x * aqu;
          const float bpv = cp.x * apv - cp.y * aqv, bqv = cp.y * apv + cp.x * aqv;
          au[p] = cq.x * bpu - cq.y * bpv;
          if (qv) au[q] = cq.x * bqu - cq.y * bqv;
          if (vv) av[p] = cq.y * bpu + cq.x * bpv;
          if (qv && vv) av[q] = cq.y * bqu + cq.x * bqv;
        }
        if (!vv || cq.y == 0.f) continue;
        float *vu = Vf + n * u, *v2 = Vf + n * v;
        for (int i = lane; i < n; i += 32) {
          const float x = vu[i], y = v2[i];
          vu[i] = cq.x * x - cq.y * y;
          v2[i] = cq.y * x + cq.x * y;
        }
      }
      __syncthreads();
    }
  }
}

// Diagonalise A in place (n x n, column-major, shared or global memory of this
// CTA), V <- its eigenvectors.  cs: n' doubles (a cosine and a sine per pair
// of a round, n' = n rounded up to even), red: blockDim.x/32 doubles, work:
// 2 n^2 doubles of this CTA (shared or global memory).  Returns false when
// max_sweeps did not reach the tolerance ||offdiag||_F <= tol ||A||_F.
//
// Bound by FP64 issue (two multiply-adds per clock and SM): a cold FP64 sweep
// of A and V costs 6 n^3 and nine were needed.  So the sweeps run in FP32 (64
// times the rate) for start vectors, which FP64 products make orthonormal to
// rounding and apply -- V <- V (I - E/2 + 3/8 E^2), E = V^T V - I, then
// A <- V^T A V (4 n^3 together) -- and the FP64 sweeps that follow start from
// off-diagonals of 1e-6 ||A||_F: two of 4 n^3 (A's lower blocks and their
// mirror images) and a check.  An FP64 division or square root takes a warp
// about a microsecond, so the tangents are FP32's.
static __device__ bool jacobi_block(int n, double *A, double *V, double *cs, double *red, double *work,
                                    int max_sweeps, double tol) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int n2 = n * n;
  double fro = 0.0, big = 0.0;
  for (int idx = tid; idx < n2; idx += blockDim.x) {
    fro += A[idx] * A[idx];
    big = fmax(big, fabs(A[idx]));
  }
  fro = jac_block_sum(fro, red);
  big = jac_block_max(big, red);
  const double stop2 = tol * tol * fro, skip = tol * sqrt(fro) / n;
  const int np = n + (n & 1), half = np / 2;
  // a power of two that brings A into FP32's range
  const double scale = big > 1e-290 && big < 1e290 ? exp2(-(double)ilogb(big)) : 1.0;
  {  // FP32 start vectors in V's space: the rotations, then the scaled matrix
    float *Vf = reinterpret_cast<float *>(V), *Af = Vf + n2;
    for (int idx = tid; idx < n2; idx += blockDim.x) {
      Af[idx] = (float)(A[idx] * scale);
      Vf[idx] = idx % (n + 1) == 0 ? 1.f : 0.f;
    }
    __syncthreads();
    jacobi_block_f32(n, Af, Vf, reinterpret_cast<float2 *>(cs), red);
    __syncthreads();
    double *W = work + n2;
    for (int idx = tid; idx < n2; idx += blockDim.x) W[idx] = (double)Vf[idx];
    __syncthreads();
    cta_mm_tn(n, W, W, work);
    __syncthreads();
    // E in FP32 (E is about 1e-6: its square's FP32 rounding is below 1e-19)
    for (int idx = tid; idx < n2; idx += blockDim.x) Vf[idx] = (float)(work[idx] - (idx % (n + 1) == 0 ? 1.0 : 0.0));
    __syncthreads();
    for (int j = w; j < n; j += nw)
      for (int i = lane; i < n; i += 32) {
        float s = 0.f;
        for (int l = 0; l < n; ++l) s = fmaf(Vf[i + n * l], Vf[l + n * j], s);
        const double d = i == j ? 1.0 : 0.0;
        work[i + n * j] = d - 0.5 * (work[i + n * j] - d) + 0.375 * (double)s;
      }
    __syncthreads();
    cta_mm(n, n, n, W, work, V);
    __syncthreads();
    cta_mm(n, n, n, A, V, work);
    __syncthreads();
    cta_mm_tn(n, V, work, A);
    __syncthreads();
    // (V^T A V is symmetric but for the rounding of its two halves)
    for (int j = w; j < n; j += nw)
      for (int i = j + 1 + lane; i < n; i += 32) A[j + (size_t)n * i] = A[i + (size_t)n * j];
    __syncthreads();
  }
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    double off = 0.0;
    for (int j = w; j < n; j += nw)
      for (int i = j + 1 + lane; i < n; i += 32) off = fma(A[i + (size_t)n * j], A[i + (size_t)n * j], off);
    off = 2.0 * jac_block_sum(off, red);
    if (off <= stop2) return true;
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

// Rank of eigenvalue i among the diagonal of A (ascending, ties by index).
__device__ __forceinline__ int jacobi_rank(int n, const double *A, int i) {
  const double wi = A[i + (size_t)n * i];
  int rank = 0;
  for (int j = 0; j < n; ++j) {
    const double wj = A[j + (size_t)n * j];
    rank += (wj < wi) || (wj == wi && j < i);
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
