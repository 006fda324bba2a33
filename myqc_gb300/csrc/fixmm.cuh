// fixmm.cuh -- FP64 matrix products on the tensor cores, as exact integer
// products of fixed-point operands (the splitting of Ozaki, Ogita, Oishi and
// Rump, Numer. Algorithms 59, 95 (2012), on FP16 digits).
//
// Each row of op(A) and each column of op(B) is scaled by a power of two to
// |x| < 2^62 and cut to an integer (every element within 2^9 of the row's
// largest stays exact), cut into eight digits of eight bits,
// x = sum_k s_k 256^(7-k), -128 <= s_k <= 127, |s_0| <= 64.  FP16 holds a digit
// exactly, a digit product is an integer of at most 2^14, and the sum of one
// level (the products s_k s'_l with k + l = L) over K <= 144 stays below 2^24,
// so the FP32 accumulators of mma.sync hold every level exactly in any order.
// The levels L = 0..7 (36 digit products) are combined as integers and rounded
// to FP64 once.  What is dropped, in units of 2^(ea + eb), a row's and a column's
// power of two (up to four times the product of their largest elements):
//   the cutting of both operands                       at most K 2^-61
//   levels 8 to 14 (level 8: 7 products of 2^14 2^48 in 2^124)   K 2^-59.2
// together at most K 2^-58.8, sqrt(K) 2^-62 for digits without a pattern.  So the error is
// bounded by the rows' norms, not element by element: an element of C is correct to
// rounding down to about K 2^-6 of 2^(ea + eb), below that it keeps fewer bits, and an
// operand's element 2^-62 below its row's largest is lost, as are subnormals.
// An FP64 sum rounds after each of its K additions, by 2^-53 sum |a||b| each.  Where that
// bound has to hold for every element (dgemm.cu, mq_dgemm), sum |a||b| is formed
// beside the product from the leading digits (fx_tile<true>).
//
// Why: this GPU issues two FP64 multiply-adds per clock and SM.  36 digit
// products take the tensor cores a small part of that time; operands of up to a few hundred
// rows do not fill the larger tiles of tcgen05.mma and would have to be staged
// in shared memory seven times over, whereas the fragments of mma.sync are
// built in registers from one 8-byte integer per element: byte k of x + (128 in
// every byte) is s_k + 128; with 0x64 above it, it is the FP16 number
// 1024 + s_k + 128, and one subtraction per two elements gives the digits.  Two
// neighbouring elements' bytes are stored alternating, so that one byte
// permutation forms the pair of a fragment register.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace mq {

constexpr int FX_DIG = 8;
constexpr int FX_KMAX = 144;  // (6 * 128^2 + 2 * 64 * 128) * 144 < 2^24
constexpr unsigned long long FX_BIAS = 0x8080808080808080ull;
constexpr int FX_BITS = 62;

// Position of the pair of elements (2 kp, 2 kp + 1) in row r of fixed-point
// pairs: within each run of 8 pairs (128 bytes) the rows are permuted so that
// neither a fragment's 16-byte loads (4 neighbouring pairs of 2 neighbouring
// rows per quarter warp) nor a quarter warp's stores of one pair of 8
// neighbouring rows meet a bank conflict.
__device__ __forceinline__ int fx_pos(int r, int kp) { return kp ^ (((r & 1) << 2) | ((r >> 1) & 3)); }

// x * 2^(FX_BITS - e) cut to an integer, biased; |x| < 2^e, e = fx_exp(field of
// the row's largest element)
__device__ __forceinline__ unsigned long long fx_fix(double x, int e) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int E = (int)(hi >> 20) & 0x7ff;
  const unsigned h = (hi & 0xfffffu) | 0x100000u;
  // the significand with its leading bit at 2^61, moved down to the row's scale
  // (unsigned: an element above its row's scale, an infinity or NaN under a fixed
  // exponent, is cut to 0)
  unsigned long long m = ((unsigned long long)(h << 9 | lo >> 23) << 32 | lo << 9) >> min((unsigned)(e + 1022 - E), 63u);
  if (E == 0) m = 0;
  return ((int)hi < 0 ? 0ull - m : m) + FX_BIAS;
}
// e with |x| < 2^e for every x of exponent field <= E (0 for a zero row)
__device__ __forceinline__ int fx_exp(int E) { return E == 0 ? -1100 : E - 1022; }
__device__ __forceinline__ int fx_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// The exponent of a row with an infinity or NaN, which has no fixed-point form:
// the products with it are NaN, or summed in FP64 from the operands as they are
// where those are at hand (dgemm.cu, fock.cu).
constexpr int FX_BAD = 4000;
__device__ __forceinline__ int fx_row_exp(int E) { return E == 0x7ff ? FX_BAD : fx_exp(E); }

// Two biased integers with their bytes alternating, lowest first
__device__ __forceinline__ uint4 fx_pair(unsigned long long u0, unsigned long long u1) {
  const unsigned l0 = (unsigned)u0, h0 = (unsigned)(u0 >> 32), l1 = (unsigned)u1, h1 = (unsigned)(u1 >> 32);
  return make_uint4(__byte_perm(l0, l1, 0x5140), __byte_perm(l0, l1, 0x7362), __byte_perm(h0, h1, 0x5140),
                    __byte_perm(h0, h1, 0x7362));
}

// Digit k of a pair of elements as an FP16 pair
__device__ __forceinline__ unsigned fx_digit(const uint4 &u, int k) {
  const int by = FX_DIG - 1 - k;  // byte of digit k
  const unsigned word = (by >> 1) == 0 ? u.x : (by >> 1) == 1 ? u.y : (by >> 1) == 2 ? u.z : u.w;
  const unsigned w = __byte_perm(word, 0x64646464u, by & 1 ? 0x4342 : 0x4140);
  const __half2 off = __half2half2(__ushort_as_half(0x6480));  // 1024 + 128
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&w), off);
  return *reinterpret_cast<const unsigned *>(&h);
}

__device__ __forceinline__ void fx_mma(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// acc[L] += the digit products of level L of a 16 x 16 fragment A (pairs (row g,
// k), (g + 8, k), (g, k + 8), (g + 8, k + 8)) and a 16 x 8 fragment B.  A's
// digits are formed as they are used, B's are kept.
__device__ __forceinline__ void fx_block(float (&acc)[FX_DIG][4], const uint4 (&a)[4], const uint4 (&b)[2]) {
  unsigned bd[2][FX_DIG];
#pragma unroll
  for (int k = 0; k < FX_DIG; ++k) {
    bd[0][k] = fx_digit(b[0], k);
    bd[1][k] = fx_digit(b[1], k);
  }
#pragma unroll
  for (int x = 0; x < FX_DIG; ++x) {
    const unsigned av[4] = {fx_digit(a[0], x), fx_digit(a[1], x), fx_digit(a[2], x), fx_digit(a[3], x)};
#pragma unroll
    for (int y = 0; y + x < FX_DIG; ++y) {
      const unsigned bv[2] = {bd[0][y], bd[1][y]};
      fx_mma(acc[x + y], av, bv);
    }
  }
}

// sum_L v_L 256^(7-L) * 2^(ea + eb - 2 FX_BITS + 8 * 7), rounded to nearest.
// Integers throughout: an FP64 instruction would occupy its SM for 16 clocks
// per warp, and the result of a product needs five of them.
__device__ __forceinline__ double fx_combine(const float *v, int ea, int eb) {
  auto four = [](const float *q) {
    return ((long long)__float2int_rn(q[0]) << 24) + ((long long)__float2int_rn(q[1]) << 16) +
           ((long long)__float2int_rn(q[2]) << 8) + __float2int_rn(q[3]);
  };
  const long long lo = four(v + 4);
  long long h = four(v) + (lo >> 32);  // the sum is h 2^32 + l, |h| < 2^45, 0 <= l < 2^32
  unsigned l = (unsigned)lo;
  const bool neg = h < 0;
  if (neg) {
    h = ~h + (l == 0);
    l = 0u - l;
  }
  if (h == 0 && l == 0) return 0.0;
  // the leading 64 bits: m 2^x with the top bit of m set
  const int z = h ? __clzll(h) : 64 + __clz(l);
  const unsigned long long m = z >= 32 ? ((unsigned long long)h << 32 | l) << (z - 32)
                                       : ((unsigned long long)h << z | l >> (32 - z));
  // (h 2^32 + l < 2^77, so z >= 19; the sum is m 2^(32 - z))
  const int e = 32 - z + 63 + ea + eb - 2 * FX_BITS + 56;  // binary exponent of the leading bit
  const unsigned long long r = (m >> 11) + ((m >> 10) & 1);  // 53 bits, maybe 2^53 after rounding
  if (e > -1022 && e < 1023) {
    const long long bits = ((long long)(e + 1022) << 52) + (long long)r;
    return __longlong_as_double(neg ? bits | (long long)0x8000000000000000ull : bits);
  }
  // at the ends of the exponent range: scaled by FP64 products
  const double x = (double)r * (neg ? -1.0 : 1.0);
  const int s = e - 52, s1 = max(min(s / 2, 1000), -1000), s2 = max(min(s - s1, 1000), -1000);
  return x * __hiloint2double((s1 + 1023) << 20, 0) * __hiloint2double((s2 + 1023) << 20, 0);
}

// The magnitudes of a pair in units of 2^(e - 14), to 2^-11 of themselves or one half
__device__ __forceinline__ unsigned fx_mag(const uint4 &u) {
  const unsigned d0 = fx_digit(u, 0), d1 = fx_digit(u, 1);
  const __half2 h = __habs2(__hfma2(*reinterpret_cast<const __half2 *>(&d0), __half2half2(__ushort_as_half(0x5c00)),
                                    *reinterpret_cast<const __half2 *>(&d1)));  // 256 s_0 + s_1
  return *reinterpret_cast<const unsigned *>(&h);
}

// A 16 x 8 tile: rows of UA (fragment rows r0 + g, r0 + g + 8; clamped to
// na - 1), columns = rows of UB (c0 + g, clamped), K = 16 ksteps.
// MAG: mag = sum |a||b| in units of 2^(ea + eb - 28).
template <bool MAG = false>
__device__ __forceinline__ void fx_tile(const uint4 *UA, const uint4 *UB, int ld, int na, int nb, int r0, int c0,
                                        int ksteps, float (&acc)[FX_DIG][4], float (*mag)[4] = nullptr) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ra = min(r0 + g, na - 1), rb = min(r0 + g + 8, na - 1), cb = min(c0 + g, nb - 1);
#pragma unroll
  for (int L = 0; L < FX_DIG; ++L)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[L][i] = 0.f;
  if constexpr (MAG)
#pragma unroll
    for (int i = 0; i < 4; ++i) (*mag)[i] = 0.f;
#pragma unroll 1
  for (int ks = 0; ks < ksteps; ++ks) {
    const int k0 = 8 * ks + t;
    const uint4 a[4] = {UA[(size_t)ra * ld + fx_pos(ra, k0)], UA[(size_t)rb * ld + fx_pos(rb, k0)],
                        UA[(size_t)ra * ld + fx_pos(ra, k0 + 4)], UA[(size_t)rb * ld + fx_pos(rb, k0 + 4)]};
    const uint4 b[2] = {UB[(size_t)cb * ld + fx_pos(cb, k0)], UB[(size_t)cb * ld + fx_pos(cb, k0 + 4)]};
    fx_block(acc, a, b);
    if constexpr (MAG) {
      const unsigned am[4] = {fx_mag(a[0]), fx_mag(a[1]), fx_mag(a[2]), fx_mag(a[3])}, bm[2] = {fx_mag(b[0]), fx_mag(b[1])};
      fx_mma(*mag, am, bm);
    }
  }
}

// ---- One CTA's products.  Row r < nr of a matrix, X(r, k) at x[r rs + k ks],
// k < nk, becomes fx_ld(nk) fixed-point pairs (zeros behind nk) under the
// exponent e[r]; neighbouring threads take neighbouring elements of the faster
// index.  (No barrier inside: e must be visible to all, after one.)
__host__ __device__ constexpr int fx_ld(int nk) { return (nk + 15) / 16 * 8; }

static __device__ __forceinline__ void cta_row_exp(int nr, int nk, const double *x, int rs, int ks, int *e) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (ks == 1) {  // a warp per row
    for (int r = w; r < nr; r += nw) {
      int m = 0;
      for (int k = lane; k < nk; k += 32) m = max(m, fx_field(x[(size_t)r * rs + k]));
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) e[r] = fx_row_exp(m);
    }
  } else {  // 4 threads per row, 8 neighbouring rows per warp
    for (int r0 = 8 * w; r0 < nr; r0 += 8 * nw) {
      const int r = r0 + (lane & 7);
      int m = 0;
      if (r < nr)
        for (int k = lane >> 3; k < nk; k += 4) m = max(m, fx_field(x[(size_t)r * rs + (size_t)k * ks]));
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
      if (r < nr && lane < 8) e[r] = fx_row_exp(m);
    }
  }
}
// elem(r, k) is X(r, k); `fast_k`: k is the faster index
template <class Elem>
static __device__ __forceinline__ void cta_fix(int nr, int nk, bool fast_k, const int *e, uint4 *U, Elem elem) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, ld = fx_ld(nk);
  auto put = [&](int r, int kp) {
    const int k = 2 * kp, ex = e[r];
    const unsigned long long u0 = k < nk ? fx_fix(elem(r, k), ex) : FX_BIAS;
    const unsigned long long u1 = k + 1 < nk ? fx_fix(elem(r, k + 1), ex) : FX_BIAS;
    U[(size_t)r * ld + fx_pos(r, kp)] = fx_pair(u0, u1);
  };
  if (fast_k) {
    for (int r = w; r < nr; r += nw)
      for (int kp = lane; kp < ld; kp += 32) put(r, kp);
  } else {
    for (int kp = w; kp < ld; kp += nw)
      for (int r = lane; r < nr; r += 32) put(r, kp);
  }
}

// Both: the rows X(r, k) = x[r rs + k ks] with their exponents, ready for all
// threads (begins and ends with a barrier)
static __device__ __forceinline__ void cta_fix_rows(int nr, int nk, const double *x, int rs, int ks, int *e, uint4 *U) {
  __syncthreads();
  cta_row_exp(nr, nk, x, rs, ks, e);
  __syncthreads();
  cta_fix(nr, nk, ks == 1, e, U, [=](int r, int k) { return x[(size_t)r * rs + (size_t)k * ks]; });
  __syncthreads();
}

// store(i, j, value) of the na x nb product of the fixed-point rows UA and UB;
// NaN where a row's exponent is FX_BAD
template <class Store>
static __device__ __forceinline__ void cta_fix_mm(int na, int nb, int nk, const uint4 *UA, const int *ea,
                                                  const uint4 *UB, const int *eb, Store store) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, g = lane >> 2, t = lane & 3;
  const int tm = (na + 15) / 16, tn = (nb + 7) / 8;
  for (int tile = w; tile < tm * tn; tile += nw) {
    const int tj = tile / tm, ti = tile - tj * tm;
    float acc[FX_DIG][4];
    fx_tile(UA, UB, fx_ld(nk), na, nb, 16 * ti, 8 * tj, (nk + 15) / 16, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 16 * ti + g + 8 * (i >> 1), cc = 8 * tj + 2 * t + (i & 1);
      float v[FX_DIG];
#pragma unroll
      for (int L = 0; L < FX_DIG; ++L) v[L] = acc[L][i];
      if (r < na && cc < nb) {
        const int xa = ea[r], xb = eb[cc];
        store(r, cc, xa == FX_BAD || xb == FX_BAD ? __longlong_as_double(0x7ff8000000000000ll) : fx_combine(v, xa, xb));
      }
    }
  }
}

}  // namespace mq
