// dgemm.cu -- every FP64 GEMM of the library: C = alpha op(A) op(B) + beta C,
// column-major, as BLAS DGEMM, optionally strided-batched (blockIdx.z).
//
// FP64 issue on this GPU is two multiply-adds per clock and SM, so the products
// are formed on the tensor cores from fixed-point digits (fixmm.cuh): 36 digit
// products per multiply-add at the 1024 per clock and SM that mma.sync gives, 28
// multiply-adds per clock and SM at best.  Their error is bounded by the largest
// elements of the row and the column, which is what the library's own steps need
// (energies, projectors, eigenvectors).  mq_dgemm promises BLAS's DGEMM, whose error is
// bounded by sum |a||b| of each element (GRADED): there the magnitudes are multiplied
// too (one more digit product), and an element whose sum falls below 2^-5 of 2^(ea + eb),
// the fixed point's unit, is summed in FP64 from the operands, in four interleaved sums
// (K/4 roundings).  At that line the digits' bound is K 2^-53.8 sum |a||b|.  Order 512:
// 53 us with random elements, 302 us with every element summed in FP64 (232 us of FP64
// issue); order 224: 18 and 76 us.
//
// A CTA of 8 warps forms 32 x 32 tiles of C: it reads 32 rows of op(A) and 32
// columns of op(B) over up to 128 of K into registers, finds their exponents,
// leaves them in shared memory as fixed-point pairs, and each warp accumulates a
// 16 x 8 block of digit products.  Sums over more than one chunk of K are
// rounded to FP64 per chunk and added in order.  Each CTA keeps the 32 columns
// of the operand with fewer tiles and goes through tiles of the other (X), so
// that the tall products of the four-index transform cut the small operand once
// per CTA.  The small tile leaves two CTAs per SM, whose load and digit phases
// run under each other's products, and spreads a product of order ~200 over
// many SMs; larger tiles (64 x 64, one CTA per SM) were slower on both.
//
// A chunk of K takes a CTA 8.5 us, most of it latency, so a single product of few
// tiles and more than three chunks splits K over the SMs; the parts go to a workspace
// and are added in order: 32 x 32 x 512 37 -> 15 us, 32 x 32 x 100000 6635 -> 91,
// 200 x 200 x 4096 255 -> 82.  (The library's own products have K up to their order, and at
// four chunks more tiles than SMs.)
//
// A row or column with an infinity or NaN has no fixed-point form either: its elements
// of C are summed in FP64 as well.
#include <algorithm>
#include <type_traits>

#include "fixmm.cuh"
#include "internal.h"

namespace mq {

constexpr int GX_K = 128;          // K chunk (exact up to FX_KMAX)
constexpr int GX_LD = GX_K / 2;    // pairs per row
constexpr int GX_T = 32;           // tile
constexpr int GX_THREADS = 256;

// The 32 rows of an operand's K chunk as fixed-point pairs.  ROWFAST: element
// (r, k) at x[r + ld k], else at x[k + ld r]; nr rows and kc elements exist.
// Leaves the rows' exponents in e (fields: scratch).
template <bool ROWFAST>
__device__ __forceinline__ void gx_load(const double *__restrict__ x, size_t ld, int nr, int kc, int *fields, int *e,
                                        uint4 *U) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int pairs = (kc + 15) / 16 * 8;
  auto put = [&](int r, int kp, double a, double b, int ex) {
    U[r * GX_LD + fx_pos(r, kp)] =
        ex == FX_BAD ? make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u) : fx_pair(fx_fix(a, ex), fx_fix(b, ex));
  };
  if (ROWFAST) {  // lanes over the rows, warps over the pairs
    constexpr int NW = GX_THREADS / 32, PER = GX_LD / NW;
    if (tid < GX_T) fields[tid] = 0;
    double v[PER][2];
    int f = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int k = 2 * (w + NW * i);
      v[i][0] = lane < nr && k < kc ? x[lane + ld * k] : 0.0;
      v[i][1] = lane < nr && k + 1 < kc ? x[lane + ld * (k + 1)] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) f = max(f, max(fx_field(v[i][0]), fx_field(v[i][1])));
    __syncthreads();
    if (f) atomicMax(fields + lane, f);
    __syncthreads();
    const int ex = fx_row_exp(fields[lane]);
    if (w == 0) e[lane] = ex;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (w + NW * i < pairs) put(lane, w + NW * i, v[i][0], v[i][1], ex);
  } else {  // a warp per row
    constexpr int PER = GX_T / (GX_THREADS / 32);
    double v[PER][4];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int r = w * PER + j;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = 2 * lane + (i & 1) + 64 * (i >> 1);
        v[j][i] = r < nr && k < kc ? x[k + ld * r] : 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int r = w * PER + j;
      const int f = max(max(fx_field(v[j][0]), fx_field(v[j][1])), max(fx_field(v[j][2]), fx_field(v[j][3])));
      const int ex = fx_row_exp(__reduce_max_sync(0xffffffffu, f));
      if (lane == 0) e[r] = ex;
      if (lane < pairs) put(r, lane, v[j][0], v[j][1], ex);
      if (lane + 32 < pairs) put(r, lane + 32, v[j][2], v[j][3], ex);
    }
  }
}

// C(r, c) at C[r sr + c sc]: rows r < mx of X, columns c < ny of Y
template <bool XROW, bool YROW, bool GRADED>
__global__ void __launch_bounds__(GX_THREADS, 2) dgemm_kernel(int mx, int ny, int k, double alpha,
                                                              const double *__restrict__ X, size_t ldx, long long sX,
                                                              const double *__restrict__ Y, size_t ldy, long long sY,
                                                              double beta, double *__restrict__ C, size_t sr,
                                                              size_t sc, long long sC, int kper,
                                                              double *__restrict__ W) {
  extern __shared__ __align__(16) unsigned char gx_smem[];
  uint4 *UX = reinterpret_cast<uint4 *>(gx_smem), *UY = UX + GX_T * GX_LD;
  __shared__ int fields[2 * GX_T], ex[GX_T], ey[GX_T];
  const int tiles = (mx + GX_T - 1) / GX_T, c0 = blockIdx.y * GX_T;
  // blockIdx.z: the part of K whose sums go to W, or the member of the batch
  const int kbeg = W ? blockIdx.z * kper : 0, kend = W ? min(k, kbeg + kper) : k;
  if (!W) {
    X += sX * blockIdx.z;
    Y += sY * blockIdx.z;
    C += sC * blockIdx.z;
  }
  const double *Yc = Y + (YROW ? (size_t)c0 : ldy * c0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int wr = (w & 1) * 16, wc = (w >> 1) * 8;
  const bool one = kend - kbeg <= GX_K;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int r0 = tile * GX_T;
    const double *Xr = X + (XROW ? (size_t)r0 : ldx * r0);
    double sum[4];
    for (int kb = kbeg; kb < kend || kb == kbeg; kb += GX_K) {
      const int kc = min(GX_K, kend - kb);
      __syncthreads();  // the previous operands have been read
      gx_load<XROW>(Xr + (XROW ? ldx * kb : (size_t)kb), ldx, min(GX_T, mx - r0), kc, fields, ex, UX);
      if (!one || tile == (int)blockIdx.x)
        gx_load<YROW>(Yc + (YROW ? ldy * kb : (size_t)kb), ldy, min(GX_T, ny - c0), kc, fields + GX_T, ey, UY);
      __syncthreads();
      float acc[FX_DIG][4], mag[4];
      fx_tile<GRADED>(UX, UY, GX_LD, GX_T, GX_T, wr, wc, (kc + 15) / 16, acc, &mag);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = wr + g + 8 * (i >> 1), c = wc + 2 * t + (i & 1);
        double x = 0.0;
        if (ex[r] != FX_BAD && ey[c] != FX_BAD && (!GRADED || mag[i] >= 0x1p23f)) {
          float v[FX_DIG];
#pragma unroll
          for (int L = 0; L < FX_DIG; ++L) v[L] = acc[L][i];
          x = fx_combine(v, ex[r], ey[c]);
        } else if (r0 + r < mx && c0 + c < ny) {
          double x4[4] = {0.0, 0.0, 0.0, 0.0};
          auto term = [&](int l, double s) {
            return fma(Xr[XROW ? r + ldx * l : l + ldx * r], Yc[YROW ? c + ldy * l : l + ldy * c], s);
          };
          int l = kb;
          for (; l + 3 < kb + kc; l += 4)
#pragma unroll
            for (int u = 0; u < 4; ++u) x4[u] = term(l + u, x4[u]);
          for (; l < kb + kc; ++l) x4[0] = term(l, x4[0]);
          x = (x4[0] + x4[1]) + (x4[2] + x4[3]);
        }
        sum[i] = kb > kbeg ? sum[i] + x : x;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + wr + g + 8 * (i >> 1), c = c0 + wc + 2 * t + (i & 1);
      if (r >= mx || c >= ny) continue;
      if (W) {
        W[(size_t)mx * ny * blockIdx.z + r + (size_t)mx * c] = sum[i];
        continue;
      }
      double *cp = C + sr * r + sc * c;
      const double x = alpha == 1.0 ? sum[i] : alpha * sum[i];
      *cp = beta == 0.0 ? x : fma(beta, *cp, x);
    }
  }
}

// C = alpha (sum of the parts, in order) + beta C; elements as dgemm_kernel's
__global__ void dgemm_parts_kernel(int mx, int ny, int parts, double alpha, const double *__restrict__ W, double beta,
                                   double *__restrict__ C, size_t sr, size_t sc) {
  const size_t mn = (size_t)mx * ny, idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= mn) return;
  double t = W[idx];
  for (int p = 1; p < parts; ++p) t += W[mn * p + idx];
  double *cp = C + sr * (idx % mx) + sc * (idx / mx);
  const double x = alpha == 1.0 ? t : alpha * t;
  *cp = beta == 0.0 ? x : fma(beta, *cp, x);
}

int dgemm_batched(mq_ctx *c, char ta, char tb, int m, int n, int k, double alpha, const double *A, int lda,
                  long long sA, const double *B, int ldb, long long sB, double beta, double *C, int ldc,
                  long long sC, int batch, bool graded) {
  if (m <= 0 || n <= 0 || batch <= 0) return MQ_OK;
  if (batch > 65535) return set_err(c, MQ_EINVAL, "dgemm: more than 65535 batched products");
  const bool TA = ta == 'T' || ta == 't', TB = tb == 'T' || tb == 't';
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  // X: the operand with more tiles
  const bool swap = n > m;
  const int mx = swap ? n : m, ny = swap ? m : n;
  const bool xrow = swap ? TB : !TA, yrow = swap ? !TA : TB;
  const int xt = (mx + GX_T - 1) / GX_T, yt = (ny + GX_T - 1) / GX_T;
  if (yt > 65535) return set_err(c, MQ_EINVAL, "dgemm: too many output tiles");
  // a few waves of two CTAs per SM, each with as many tiles of X as that leaves
  const long long want = std::max<long long>(1, (8LL * sms + (long long)yt * batch - 1) / ((long long)yt * batch));
  const long long tiles = (long long)xt * yt;
  const int chunks = (k + GX_K - 1) / GX_K;
  int parts = 1, kper = 0;
  double *W = nullptr;
  if (batch == 1 && chunks > 3 && tiles < sms) {
    const int most = std::min(chunks, (int)(2 * sms / tiles)), per = (chunks + most - 1) / most;
    parts = (chunks + per - 1) / per;
    kper = per * GX_K;
    // (products queued on the aux stream have sums of their own)
    W = (double *)buf(c, c->aux && c->stream == c->aux ? "dgemm_parts_aux" : "dgemm_parts",
                      sizeof(double) * parts * (size_t)mx * ny);
    if (!W) return MQ_ENOMEM;
  }
  const size_t sr = swap ? ldc : 1, sc = swap ? 1 : ldc;
  const dim3 grid((unsigned)std::min<long long>(xt, want), yt, W ? parts : batch);
  const size_t sm = sizeof(uint4) * 2 * GX_T * GX_LD;
  auto pick = [&](auto g) {
    constexpr bool G = decltype(g)::value;
    return xrow ? (yrow ? dgemm_kernel<true, true, G> : dgemm_kernel<true, false, G>)
                : (yrow ? dgemm_kernel<false, true, G> : dgemm_kernel<false, false, G>);
  };
  auto kern = graded ? pick(std::true_type{}) : pick(std::false_type{});
  MQ_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  kern<<<grid, GX_THREADS, sm, c->stream>>>(mx, ny, k, alpha, swap ? B : A, swap ? ldb : lda, swap ? sB : sA,
                                            swap ? A : B, swap ? lda : ldb, swap ? sA : sB, beta, C, sr, sc, sC, kper,
                                            W);
  c->stats.launches += 1;
  if (W) {
    dgemm_parts_kernel<<<(unsigned)(((size_t)mx * ny + 255) / 256), 256, 0, c->stream>>>(mx, ny, parts, alpha, W, beta,
                                                                                       C, sr, sc);
    c->stats.launches += 1;
  }
  MQ_CUDA(c, cudaGetLastError());
  return MQ_OK;
}

}  // namespace mq
