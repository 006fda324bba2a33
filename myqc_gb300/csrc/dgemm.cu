// dgemm.cu -- every FP64 GEMM of the library: C = alpha op(A) op(B) + beta C,
// column-major, as BLAS DGEMM, optionally strided-batched (blockIdx.z).
//
// FP64 issue on this GPU is two multiply-adds per clock and SM, so the products
// are formed on the tensor cores from fixed-point digits (fixmm.cuh), correct to
// FP64 rounding or better.  A CTA forms a TM x TN tile of C: per chunk of up to
// 128 of K it reads its rows of op(A) and columns of op(B) into registers,
// finds their exponents, leaves them in shared memory as fixed-point pairs, and
// each warp accumulates a 16 x 8 NT block of digit products; the chunk's sums
// are rounded to FP64 and added over the chunks in FP64, in order.  Bound by
// integer issue (cutting and recombining digits) and the tensor pipe.
//
// Tiles of 64 x 64 serve products with enough of them to fill the SMs; others
// take 32 x 32, which spread a product of order ~200 over more SMs.
//
// A row or column with an infinity or NaN has no fixed-point form: its elements
// of C are summed in FP64 from the operands as they are.
#include <algorithm>

#include "fixmm.cuh"
#include "internal.h"

namespace mq {

constexpr int GX_K = 128;          // K chunk (exact up to FX_KMAX)
constexpr int GX_LD = GX_K / 2;    // pairs per row
constexpr int GX_BAD = 4000;       // exponent that marks a row with a non-finite element

// TR rows of an operand's K chunk as fixed-point pairs.  ROWFAST: element (r, k)
// at x[r + ld k], else at x[k + ld r]; nr rows and kc elements exist.  Leaves
// the rows' exponents in e (fields: TR ints of scratch).
template <int TR, bool ROWFAST, int THREADS>
__device__ __forceinline__ void gx_load(const double *__restrict__ x, size_t ld, int nr, int kc, int *fields, int *e,
                                        uint4 *U) {
  const int tid = threadIdx.x;
  auto put = [&](int r, int kp, double a, double b, int ex) {
    U[r * GX_LD + fx_pos(r, kp)] =
        ex == GX_BAD ? make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u) : fx_pair(fx_fix(a, ex), fx_fix(b, ex));
  };
  auto exponent = [](int f) { return f == 0x7ff ? GX_BAD : fx_exp(f); };
  if (ROWFAST) {
    constexpr int GR = THREADS / TR, PER = GX_K / GR;  // threads per row, elements per thread
    const int r = tid % TR, k0 = (tid / TR) * PER;
    if (tid < TR) fields[tid] = 0;
    double v[PER];
    int f = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = r < nr && k0 + i < kc ? x[r + ld * (k0 + i)] : 0.0;
#pragma unroll
    for (int i = 0; i < PER; ++i) f = max(f, fx_field(v[i]));
    __syncthreads();
    if (f) atomicMax(fields + r, f);
    __syncthreads();
    const int ex = exponent(fields[r]);
    if (tid < TR) e[tid] = ex;
#pragma unroll
    for (int i = 0; i < PER; i += 2) put(r, (k0 + i) / 2, v[i], v[i + 1], ex);
  } else {
    const int lane = tid & 31, w = tid >> 5;
    constexpr int NW = THREADS / 32;
#pragma unroll 4
    for (int r = w; r < TR; r += NW) {
      double v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = 2 * lane + (i & 1) + 64 * (i >> 1);
        v[i] = r < nr && k < kc ? x[k + ld * r] : 0.0;
      }
      const int f = max(max(fx_field(v[0]), fx_field(v[1])), max(fx_field(v[2]), fx_field(v[3])));
      const int ex = exponent(__reduce_max_sync(0xffffffffu, f));
      if (lane == 0) e[r] = ex;
      put(r, lane, v[0], v[1], ex);
      put(r, lane + 32, v[2], v[3], ex);
    }
  }
}

template <int TM, int TN, bool TA, bool TB>
__global__ void __launch_bounds__(TM * 4) dgemm_kernel(int m, int n, int k, double alpha, const double *__restrict__ A,
                                                       int lda, long long sA, const double *__restrict__ B, int ldb,
                                                       long long sB, double beta, double *__restrict__ C, int ldc,
                                                       long long sC) {
  constexpr int THREADS = TM * 4, WM = TM / 16, WN = THREADS / 32 / WM, NT = TN / WN / 8;
  extern __shared__ __align__(16) unsigned char gx_smem[];
  uint4 *UA = reinterpret_cast<uint4 *>(gx_smem), *UB = UA + TM * GX_LD;
  __shared__ int fields[TM + TN], ea[TM], eb[TN];
  const int tiles_m = (m + TM - 1) / TM;
  const int r0 = (int)(blockIdx.x % tiles_m) * TM, c0 = (int)(blockIdx.x / tiles_m) * TN;
  A += sA * blockIdx.z;  // the batch's operands
  B += sB * blockIdx.z;
  C += sC * blockIdx.z;
  const double *Ar = TA ? A + (size_t)lda * r0 : A + r0, *Bc = TB ? B + c0 : B + (size_t)ldb * c0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int wr = (w % WM) * 16, wc = (w / WM) * (8 * NT);
  double sum[NT][4];
  for (int kb = 0; kb < k || kb == 0; kb += GX_K) {
    const int kc = min(GX_K, k - kb);
    if (kb) __syncthreads();  // the previous chunk's operands have been read
    gx_load<TM, !TA, THREADS>(TA ? Ar + kb : Ar + (size_t)lda * kb, lda, min(TM, m - r0), kc, fields, ea, UA);
    gx_load<TN, TB, THREADS>(TB ? Bc + (size_t)ldb * kb : Bc + kb, ldb, min(TN, n - c0), kc, fields + TM, eb, UB);
    __syncthreads();
    float acc[NT][FX_DIG][4];
    fx_tile<NT>(UA, UB, GX_LD, TM, TN, wr, wc, (kc + 15) / 16, acc);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = wr + g + 8 * (i >> 1), c = wc + 8 * j + 2 * t + (i & 1);
        double x;
        if (ea[r] != GX_BAD && eb[c] != GX_BAD) {
          float v[FX_DIG];
#pragma unroll
          for (int L = 0; L < FX_DIG; ++L) v[L] = acc[j][L][i];
          x = fx_combine(v, ea[r], eb[c]);
        } else {
          x = 0.0;
          if (r0 + r < m && c0 + c < n) for (int l = kb; l < kb + kc; ++l)
            x = fma(TA ? A[l + (size_t)lda * (r0 + r)] : A[r0 + r + (size_t)lda * l],
                    TB ? B[c0 + c + (size_t)ldb * l] : B[l + (size_t)ldb * (c0 + c)], x);
        }
        sum[j][i] = kb ? sum[j][i] + x : x;
      }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + wr + g + 8 * (i >> 1), c = c0 + wc + 8 * j + 2 * t + (i & 1);
      if (r >= m || c >= n) continue;
      double *cp = C + r + (size_t)ldc * c;
      const double x = alpha == 1.0 ? sum[j][i] : alpha * sum[j][i];
      *cp = beta == 0.0 ? x : fma(beta, *cp, x);
    }
}

template <int TM, int TN>
static int launch_gemm(mq_ctx *c, bool TA, bool TB, dim3 grid, int m, int n, int k, double alpha, const double *A,
                       int lda, long long sA, const double *B, int ldb, long long sB, double beta, double *C, int ldc,
                       long long sC) {
  const size_t sm = sizeof(uint4) * (TM + TN) * GX_LD;
  auto kern = TA ? (TB ? dgemm_kernel<TM, TN, true, true> : dgemm_kernel<TM, TN, true, false>)
                 : (TB ? dgemm_kernel<TM, TN, false, true> : dgemm_kernel<TM, TN, false, false>);
  MQ_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  kern<<<grid, TM * 4, sm, c->stream>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC);
  c->stats.launches += 1;
  MQ_CUDA(c, cudaGetLastError());
  return MQ_OK;
}

int dgemm_batched(mq_ctx *c, char ta, char tb, int m, int n, int k, double alpha, const double *A, int lda,
                  long long sA, const double *B, int ldb, long long sB, double beta, double *C, int ldc,
                  long long sC, int batch) {
  if (m <= 0 || n <= 0 || batch <= 0) return MQ_OK;
  if (batch > 65535) return set_err(c, MQ_EINVAL, "dgemm: more than 65535 batched products");
  const bool TA = ta == 'T' || ta == 't', TB = tb == 'T' || tb == 't';
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  auto tiles = [&](long long tm, long long tn) { return ((m + tm - 1) / tm) * ((n + tn - 1) / tn); };
  if (tiles(32, 32) > 2147483647LL) return set_err(c, MQ_EINVAL, "dgemm: too many output tiles");
  const long long t64 = tiles(64, 64);
  if (n > 32 && t64 * batch >= 2 * sms)
    return launch_gemm<64, 64>(c, TA, TB, dim3((unsigned)t64, 1, batch), m, n, k, alpha, A, lda, sA, B, ldb, sB, beta,
                               C, ldc, sC);
  return launch_gemm<32, 32>(c, TA, TB, dim3((unsigned)tiles(32, 32), 1, batch), m, n, k, alpha, A, lda, sA, B, ldb, sB,
                             beta, C, ldc, sC);
}

}  // namespace mq
