// Restart combination out_c = sum_i V_i Y[i][c] (BVMultInPlace in SLEPc's
// Krylov-Schur restart) for real storage: the default form.
//
// In FP64 FMAs the combination is bound by GB300's FP64 unit (16 x 8 FMAs per
// row), and half the outputs in 64-bit integer products beside it by the
// integer multiplier: 5.9 ms per 8 outputs at 40.1M rows, against 1.1 ms for
// its memory traffic.  Here the products run on the tensor cores in exact
// digits:
//  * a row's entries in 68-bit fixed point against the row's largest exponent,
//    a coefficient column against its own, both as six balanced 10-bit digits
//    and a last one of ten bits (FP16 holds them exactly);
//  * mma.m16n8k16 on 16 rows x 16 columns x 8 outputs: the 28 digit products
//    i + j <= 6, one FP32 accumulator per weight ("level") i + j.  A level
//    sum is an exact integer for levels 0..4 (at most 16 x 2^20 = 2^24); levels
//    5 and 6 are folded into one and may round in its last bit, 2^-66 of the
//    scales;
//  * the levels are combined in 64-bit integers and rounded to FP64 with
//    integer operations.
// The cut digits and products stay below m 2^-64.6 of (row scale) x (column
// scale).  A value below 2^-11 of the scales none of whose products reaches that
// either is computed again in FP64 (combine_small), so that every entry is as
// good as an FP64 chain's: within (m + 1) 2^-53 sum |V_i Y_ic|, and the column
// itself where one coefficient is a power of two and the others are 0.  With 58
// bits and no second look, an entry 2^-k below its row's largest kept 58 - k.
// Rows that are not finite or lie below 2^-951 are FP64 throughout.
//
// mma.sync and not tcgen05: the operands are made in registers, one row pair
// per thread, and the fragment layout lets the thread that loads and splits
// the entries also own the accumulators of the same rows, so nothing passes
// through shared memory.  The splitting and rounding bound the kernel.  At 40.1M
// rows and 16 columns: 8 outputs 5.90 -> 3.02 ms, 9 outputs 7.13 -> 3.99 ms, 15
// outputs 4.40 ms (58 bits: 2.39, 3.25 and 3.54 ms).  Conversion costs more
// than 16 FP64 FMAs per entry group, so the Gram-Schmidt dots and updates, one
// FMA per entry, stay FP64.
//
// Fragment layout: lane = 4 g + t; A rows g and g + 8 are rows 2 g and
// 2 g + 1 of the 16-row tile (one 16-byte load brings both), K index =
// column.
#include "ed_internal.h"
#include "ed_device.cuh"
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include <cstring>

namespace {

constexpr int CB_DIG = 7, CB_LEV = 7;
constexpr int CB_MAXM = 127;
constexpr int CB_CELL = 4;  // 16-byte words per lane and cell: 14 words of digits
constexpr int CB_THREADS = 128;
constexpr int CB_MINB = 4;  // 128 registers: nine outputs, 40.1M rows, 3 blocks 4.49 ms, 4 3.99

template <int NC>
struct CombineArgs {
  const double* v[16 * NC];
  double* out[16];
  double y[16 * NC][16];  // Y of this launch's outputs, zero padded
};

// An entry as digits of trunc(|v| 2^(68 - E)), |v| < 2^E, E = emax - 1022:
//  q  the upper six: trunc(v 2^(58 - E)) with 512 added to each 10-bit digit, so
//     digit d of the balanced representation is field 5 - d minus 512 (|q| <
//     2^58 keeps the top one below 258);
//  r  the next ten bits, with the sign of v (hw).  Only an entry more than five
//     binades below emax has any.
struct Digits {
  unsigned long long q;
  uint32_t r, hw;
};
constexpr unsigned long long CB_BIAS = 0x0802008020080200ull;  // sum 512 2^(10 i), i = 0..5
static_assert(CB_BIAS == (512ull | 512ull << 10 | 512ull << 20 | 512ull << 30 | 512ull << 40 | 512ull << 50), "");

// emax >= CB_EMIN: an entry with e = 0 (zero, subnormal) is shifted out of q and r.
constexpr int CB_EMIN = 72;
__device__ __forceinline__ Digits digits10(double v, int emax) {
  const uint32_t hw = (uint32_t)__double2hiint(v), lw = (uint32_t)__double2loint(v);
  // mantissa 2^5 (58 bits) >> (emax - e)
  const uint32_t mh = (__funnelshift_l(lw, hw, 5) & 0x01FFFFFFu) | 0x02000000u;
  const unsigned long long mant = ((unsigned long long)mh << 32) | (lw << 5);
  const int sh = emax - (int)((hw >> 20) & 0x7FFu);
  const unsigned long long q = mant >> min(sh, 63);
  const long long s = (int)hw >> 31;  // 0 or -1: CB_BIAS + q or CB_BIAS - q
  Digits d;
  d.q = (q ^ (unsigned long long)s) + (CB_BIAS - (unsigned long long)s);
  d.r = (uint32_t)((mant << 5) >> min((uint32_t)(sh - 5), 63u)) & 0x3FFu;  // sh < 5: all shifted out
  d.hw = hw;
  return d;
}

// digit D of two entries as FP16 pair (x low, y high)
template <int D>
__device__ __forceinline__ uint32_t digit_pair(const Digits& x, const Digits& y) {
  constexpr bool tail = D == CB_DIG - 1;
  constexpr int s = tail ? 0 : 10 * (CB_DIG - 2 - D);
  const uint32_t a = tail ? x.r : (uint32_t)(x.q >> s), b = tail ? y.r : (uint32_t)(y.q >> s);
  uint32_t h;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(h) : "r"(a), "r"(b), "r"(0x5410u));
  h = (tail ? h : h & 0x03FF03FFu) | 0x64006400u;  // 1024 + field
  const float off = tail ? -1024.0f : -1536.0f;
  const __half2 r = __hadd2(*reinterpret_cast<__half2*>(&h), __floats2half2_rn(off, off));
  uint32_t w = *reinterpret_cast<const uint32_t*>(&r);
  if (tail) {
    uint32_t sg;  // the sign bits
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(sg) : "r"(x.hw), "r"(y.hw), "r"(0x7632u));
    w ^= sg & 0x80008000u;
  }
  return w;
}

template <int D = 0>
__device__ __forceinline__ void digit_pairs(const Digits& x, const Digits& y, uint32_t (&o)[CB_DIG]) {
  o[D] = digit_pair<D>(x, y);
  if constexpr (D + 1 < CB_DIG) digit_pairs<D + 1>(x, y, o);
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
      "%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// T 2^X rounded to the nearest FP64 (integer operations)
__device__ __forceinline__ double fx64_to_double(long long T, int X) {
  const unsigned long long neg = (unsigned long long)T & 0x8000000000000000ull;
  unsigned long long u = (unsigned long long)(T < 0 ? -T : T);
  const int z = __clzll((long long)u);
  u <<= z & 63;
  int bexp = X + 63 - z + 1023;
  // 53 bits and the rounding bit; a carry moves into the exponent field
  unsigned long long r = ((unsigned long long)(unsigned)(bexp - 1) << 52) + (u >> 11) + ((u >> 10) & 1ull);
  if (bexp >= 0x7FF) r = 0x7FF0000000000000ull;
  if (bexp <= 0 || z == 64) r = 0ull;
  return __longlong_as_double((long long)(r | neg));
}

// Rows r0, r0 + 1 of a column (0 past the end).
template <bool VEC>
__device__ __forceinline__ double2 load2(const double* p, int64_t r, int64_t n) {
  if (VEC) {
    if (r + 1 < n) return __ldg((const double2*)(p + r));
    return make_double2(r < n ? __ldg(p + r) : 0.0, 0.0);
  }
  return make_double2(r < n ? __ldg(p + r) : 0.0, r + 1 < n ? __ldg(p + r + 1) : 0.0);
}

__device__ __forceinline__ int biased_exp(double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7FF); }

// Digit products of one 16-column group and 8 outputs, by level.
__device__ __forceinline__ void combine_mma(const uint32_t (&a)[4][CB_DIG], const uint32_t (&b)[2 * CB_DIG],
                                            float (&acc)[CB_LEV][4]) {
#pragma unroll
  for (int l = 0; l < CB_LEV; ++l)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[l][k] = 0.0f;
#pragma unroll
  for (int i = 0; i < CB_DIG; ++i)
#pragma unroll
    for (int l = CB_LEV - 1; l >= 0; --l)
      if (l >= i && l - i < CB_DIG)
        mma16816(acc[l], a[0][i], a[1][i], a[2][i], a[3][i], b[l - i], b[CB_DIG + l - i]);
}

// Levels 0..4, and 5 with 6 folded in, as integers.
__device__ __forceinline__ int combine_level(const float (&acc)[CB_LEV][4], int l, int q) {
  return __float2int_rn(l < 5 ? acc[l][q] : fmaf(acc[6][q], 0x1p-10f, acc[5][q]));
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// The value of the levels of one accumulator entry.  |T| < m 2^56 < 2^63 in
// the unit 2^(E + F - 116 + 60), E, F = biased - 1022; a value that leaves room
// takes level 5 in full.  small: the value is below 2^-11 of 2^(E + F) or of
// the normal range, and combine_small decides.
__device__ __forceinline__ double combine_value(const int (&L)[6], int X, bool fast, bool& small) {
  // l0 2^40 + l1 2^30 as (l0 2^10 + l1) 2^30; multiply-adds, since the ALU is
  // what the kernel waits for
  const long long t = mad_wide(L[3], 1 << 10, mad_wide(L[2], 1 << 20, (long long)L[4]));
  const long long u = mad_wide(L[0], 1 << 10, (long long)L[1]);
  long long T = t + (long long)((unsigned long long)u << 30);
  const int hi = (int)(T >> 32);
  small = (uint32_t)(hi + (1 << 13)) < (1u << 14);       // |T| < 2^45
  const bool room = (uint32_t)(hi + (1 << 20)) < (1u << 21);  // |T| < 2^52
  T = room ? (T << 10) + L[5] : T + ((L[5] + 512) >> 10);
  X -= room ? 10 : 0;
  // in range of every T: the conversion unit (idle otherwise) rounds, and the
  // scale is an addition to the exponent field
  if (fast) {
    const double d = __ll2double_rn(T);
    const int h = __double2hiint(d);
    return __hiloint2double(h == 0 ? 0 : h + (X << 20), __double2loint(d));
  }
  const double d = fx64_to_double(T, X);
  small |= (__double2hiint(d) & 0x7FF00000) == 0;
  return d;
}

// Scales of a row pair with the exponents e0, e1 and an output's F, and
// whether every value there is in the normal range.
__device__ __forceinline__ bool combine_fast(int X0, int X1) {
  return __all_sync(0xffffffffu, min(X0, X1) > -1010 && max(X0, X1) < 960);
}

template <bool VEC, typename Args>
__device__ __forceinline__ void combine_out(const Args& A, int o, double2 res, int nout, int64_t row, int64_t n) {
  if (o >= nout || row >= n) return;
  if (VEC && row + 1 < n) {
    *(double2*)(A.out[o] + row) = res;
  } else {
    A.out[o][row] = res.x;
    if (row + 1 < n) A.out[o][row + 1] = res.y;
  }
}

// This lane's coefficient digits of a 16-column group and 8 outputs.
__device__ __forceinline__ void combine_b(const uint4* __restrict__ sB, int cell, int lane, uint32_t (&b)[2 * CB_DIG]) {
  const uint4* p = sB + (cell * 32 + lane) * CB_CELL;
#pragma unroll
  for (int q = 0; q < CB_CELL; ++q) {
    const uint4 w = p[q];
    b[4 * q] = w.x;
    b[4 * q + 1] = w.y;
    if (4 * q + 2 < 2 * CB_DIG) {
      b[4 * q + 2] = w.z;
      b[4 * q + 3] = w.w;
    }
  }
}

// Coefficient digits of every (group, 8 outputs) cell to shared memory (cell c
// * NT + nt, CB_CELL words per lane), and the exponents of this lane's
// outputs.  All warps of the block; ends with a barrier.
template <int NT, typename Args>
__device__ __forceinline__ void combine_setup(const Args& A, int m, uint4* sB, int (&F)[NT][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warp = threadIdx.x >> 5;
  const int ng = (m + 15) / 16;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    int f = 0;
    for (int i = t; i < m; i += 4) f = max(f, biased_exp(A.y[i][8 * nt + g]));
    f = max(f, __shfl_xor_sync(0xffffffffu, f, 1));
    f = max(max(f, __shfl_xor_sync(0xffffffffu, f, 2)), CB_EMIN);  // smaller coefficients count as 0: their results are small
    for (int c = warp; c < ng; c += CB_THREADS / 32) {
      uint32_t d[2][CB_DIG];
      for (int h = 0; h < 2; ++h) {
        const int i = 16 * c + 2 * t + 8 * h;
        digit_pairs(digits10(A.y[i][8 * nt + g], f), digits10(A.y[i + 1][8 * nt + g], f), d[h]);
      }
      uint4* p = sB + ((c * NT + nt) * 32 + lane) * CB_CELL;
      p[0] = make_uint4(d[0][0], d[0][1], d[0][2], d[0][3]);
      p[1] = make_uint4(d[0][4], d[0][5], d[0][6], d[1][0]);
      p[2] = make_uint4(d[1][1], d[1][2], d[1][3], d[1][4]);
      p[3] = make_uint4(d[1][5], d[1][6], 0u, 0u);
    }
    F[nt][0] = __shfl_sync(0xffffffffu, f, 8 * t);
    F[nt][1] = __shfl_sync(0xffffffffu, f, 8 * t + 4);
  }
  __syncthreads();
}

__device__ __forceinline__ void combine_digits(const double2 (&v)[4], int e0, int e1, uint32_t (&a)[4][CB_DIG]) {
  // A registers: (row 2g, k lo), (row 2g + 1, k lo), (2g, k hi), (2g + 1, k hi)
  digit_pairs(digits10(v[0].x, e0), digits10(v[1].x, e0), a[0]);
  digit_pairs(digits10(v[0].y, e1), digits10(v[1].y, e1), a[1]);
  digit_pairs(digits10(v[2].x, e0), digits10(v[3].x, e0), a[2]);
  digit_pairs(digits10(v[2].y, e1), digits10(v[3].y, e1), a[3]);
}

// Rows in FP64 (the four lanes of a row pair).
template <typename Args>
__device__ __noinline__ void combine_row_fp64(const Args& A, int m, int nout, int t, bool slow0, bool slow1,
                                              int64_t row, int64_t n) {
  for (int h = 0; h < 2; ++h) {
    if (!(h ? slow1 : slow0) || row + h >= n) continue;
    for (int o = t; o < nout; o += 4) {
      double s = 0.0;
      for (int i = 0; i < m; ++i) s = fma(A.v[i][row + h], A.y[i][o], s);
      A.out[o][row + h] = s;
    }
  }
}

// Small values, looked at again 32 at a time (a warp's list of row 16 + output):
// FP64 where no product reaches 2^-11 of the scales 2^(E + F) that the digits
// were cut against, or the value may leave the normal range.  Where one does, the
// value is small because the products cancel, and its error is below m 2^-53 of
// that product.  Random orthonormal columns have 0.1% of such values; the restarts
// of a disordered N=24 solve up to 13%, two thirds of them then FP64: its 19
// restarts take 2.4 ms of 63.6 for this.  One at a time, as they were met, the
// random ones took 13% of the kernel; 5.0 ms of the solve with the coefficients
// read from the kernel's parameters and the entries read twice.
constexpr int CB_LIST = 64;
template <typename Args>
__device__ __noinline__ void combine_small(const Args& A, int m, const double (*Y)[16], const unsigned long long* list,
                                           int count) {
  __syncwarp();  // the list, and the values stored before
  for (int q = threadIdx.x & 31; q < count; q += 32) {
    const int64_t r = (int64_t)(list[q] >> 4);
    const int o = (int)(list[q] & 15u);
    int ev = CB_EMIN, ey = CB_EMIN, ep = 0;  // largest exponents: entry, coefficient, product
    double s = 0.0;
#pragma unroll 8
    for (int i = 0; i < m; ++i) {  // one pass: the loads are what a round waits for
      const double v = A.v[i][r], c = Y[i][o];
      const int x = biased_exp(v), y = biased_exp(c);
      ev = max(ev, x);
      ey = max(ey, y);
      ep = max(ep, x + y);
      s = fma(v, c, s);
    }
    if (ep < ev + ey - 9 || ev + ey < 2044 - 950) A.out[o][r] = s;
  }
  __syncwarp();  // the list is free
}

// Bit 4 nt + 2 k + h: this lane's output 8 nt + 2 t + k of row + h.  The outputs
// there are (a padded one is 0, and small):
__device__ __forceinline__ unsigned combine_mine(int nout) {
  unsigned mine = 0u;
#pragma unroll
  for (int b = 0; b < 8; b += 2)
    if (8 * (b >> 2) + 2 * (int)(threadIdx.x & 3) + ((b >> 1) & 1) < nout) mine |= 3u << b;
  return mine;
}

// Notes the values of need, one of every lane at a time.  All lanes of the warp.
template <typename Args>
__device__ __forceinline__ void combine_note(const Args& A, int m, const double (*Y)[16], unsigned need, int64_t row,
                                             int64_t n, unsigned long long* list, int& count) {
  const int lane = threadIdx.x & 31, t = lane & 3;
  if (row >= n) need = 0u;
  if (row + 1 >= n) need &= 0x55u;
  for (unsigned mk = __ballot_sync(0xffffffffu, need); mk; mk = __ballot_sync(0xffffffffu, need)) {
    if (count + __popc(mk) > CB_LIST) {
      combine_small(A, m, Y, list, count);
      count = 0;
    }
    if (need) {
      const int b = __ffs(need) - 1, o = 8 * (b >> 2) + 2 * t + ((b >> 1) & 1);
      list[count + __popc(mk & ((1u << lane) - 1u))] = (unsigned long long)(row + (b & 1)) << 4 | (unsigned)o;
      need &= need - 1u;
    }
    count += __popc(mk);
  }
}

// A row pair from the largest high words (sign cleared) of this lane's entries:
// e, the exponents for the digits; slow, a row that is not finite or has nothing
// above 2^-951; keep, the bits of need (combine_small) that rows with digits may
// set (a row of zeros is exact).  lo: entries whose low word is not zero.
struct RowPair {
  int e0, e1;
  bool slow0, slow1;
  unsigned keep;
};
__device__ __forceinline__ RowPair combine_rows(uint32_t w0, uint32_t w1, bool lo0, bool lo1) {
#pragma unroll
  for (int s = 1; s <= 2; s <<= 1) {
    w0 = max(w0, __shfl_xor_sync(0xffffffffu, w0, s));
    w1 = max(w1, __shfl_xor_sync(0xffffffffu, w1, s));
  }
  if (__any_sync(0xffffffffu, w0 == 0u || w1 == 0u)) {  // low words count where all high ones are zero
    const unsigned b0 = __ballot_sync(0xffffffffu, lo0), b1 = __ballot_sync(0xffffffffu, lo1);
    const int q = threadIdx.x & 28;
    w0 |= (b0 >> q) & 15u ? 1u : 0u;
    w1 |= (b1 >> q) & 15u ? 1u : 0u;
  }
  RowPair p;
  p.e0 = (int)(w0 >> 20);
  p.e1 = (int)(w1 >> 20);
  p.slow0 = w0 != 0u && (p.e0 == 0x7FF || p.e0 < CB_EMIN);
  p.slow1 = w1 != 0u && (p.e1 == 0x7FF || p.e1 < CB_EMIN);
  p.keep = (w0 != 0u && !p.slow0 ? 0x55u : 0u) | (w1 != 0u && !p.slow1 ? 0xAAu : 0u);
  p.e0 = max(p.e0, CB_EMIN);
  p.e1 = max(p.e1, CB_EMIN);
  return p;
}

// NC: groups of 16 columns; NT: groups of 8 outputs.  VEC: every column and
// output is 16-byte aligned.
template <int NC, int NT, bool VEC>
__global__ void __launch_bounds__(CB_THREADS, NC == 1 ? CB_MINB : 3) k_combine(const __grid_constant__ CombineArgs<NC> A,
                                                                         int m, int nout, int64_t n) {
  __shared__ uint4 sB[NC * NT * 32 * CB_CELL];
  __shared__ double sY[16 * NC][16];  // the coefficients, for combine_small
  __shared__ unsigned long long lists[CB_THREADS / 32][CB_LIST];
  unsigned long long* list = lists[threadIdx.x >> 5];
  int count = 0;
  const unsigned mine = combine_mine(nout);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  int F[NT][2];  // exponents of outputs 8 nt + 2 t, + 1
  for (int k = threadIdx.x; k < 16 * NC * 16; k += CB_THREADS) sY[k >> 4][k & 15] = A.y[k >> 4][k & 15];
  combine_setup<NT>(A, 16 * NC, sB, F);  // ends with a barrier
  const double* col[NC][4];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) col[c][k] = A.v[16 * c + 2 * t + (k & 1) + 8 * (k >> 1)];
  const int64_t stride = (int64_t)gridDim.x * (CB_THREADS / 32) * 16;
  int64_t r = ((int64_t)blockIdx.x * (CB_THREADS / 32) + (threadIdx.x >> 5)) * 16;
  double2 nx[NC][4];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      nx[c][k] = col[c][k] && r < n ? load2<VEC>(col[c][k], r + 2 * g, n) : make_double2(0.0, 0.0);
  for (; r < n; r += stride) {
    const int64_t row = r + 2 * g;
    uint32_t w0 = 0u, w1 = 0u;
    bool lo0 = false, lo1 = false;
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w0 = max(w0, (uint32_t)__double2hiint(nx[c][k].x) & 0x7FFFFFFFu);
        w1 = max(w1, (uint32_t)__double2hiint(nx[c][k].y) & 0x7FFFFFFFu);
      }
    if (__any_sync(0xffffffffu, w0 == 0u || w1 == 0u)) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          lo0 |= __double2loint(nx[c][k].x) != 0;
          lo1 |= __double2loint(nx[c][k].y) != 0;
        }
    }
    const RowPair rp = combine_rows(w0, w1, lo0, lo1);
    const int x0 = rp.e0, x1 = rp.e1;
    uint32_t a[NC][4][CB_DIG];
#pragma unroll
    for (int c = 0; c < NC; ++c) combine_digits(nx[c], x0, x1, a[c]);
    if (r + stride + 16 <= n) {  // the next tile, loaded while this one is multiplied
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (col[c][k]) nx[c][k] = load2<VEC>(col[c][k], row + stride, INT64_MAX);
    } else if (r + stride < n) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (col[c][k]) nx[c][k] = load2<VEC>(col[c][k], row + stride, n);
    }
    const bool full = r + 16 <= n;
    unsigned need = 0u;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float acc[NC][CB_LEV][4];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        uint32_t b[2 * CB_DIG];
        combine_b(sB, c * NT + nt, lane, b);
        combine_mma(a[c], b, acc[c]);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (8 * nt + k >= nout) break;  // no lane has an output here
        const int X0 = x0 + F[nt][k] - 2044 - 56, X1 = x1 + F[nt][k] - 2044 - 56;
        const bool fast = combine_fast(X0, X1);
        double2 res;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int L[6];
#pragma unroll
          for (int l = 0; l < 6; ++l) {
            L[l] = combine_level(acc[0], l, 2 * h + k);
            if (NC > 1) L[l] += combine_level(acc[NC - 1], l, 2 * h + k);
          }
          bool small;
          const double d = combine_value(L, h ? X1 : X0, fast, small);
          if (h) res.y = d; else res.x = d;
          need |= (small ? 1u : 0u) << (4 * nt + 2 * k + h);
        }
        combine_out<VEC>(A, 8 * nt + 2 * t + k, res, nout, row, full ? INT64_MAX : n);
      }
    }
    need &= rp.keep & mine;
    if (__any_sync(0xffffffffu, need)) combine_note(A, m, sY, need, row, n, list, count);
    __syncwarp();  // the stores above come first
    if (rp.slow0 || rp.slow1) combine_row_fp64(A, m, nout, t, rp.slow0, rp.slow1, row, n);
    __syncwarp();
  }
  if (count) combine_small(A, m, sY, list, count);
}

// More than 32 columns: the row exponents from a first read of the columns,
// then one group of 16 at a time (read again, from the caches).
template <bool VEC>
__global__ void __launch_bounds__(CB_THREADS, 3) k_combine_many(const __grid_constant__ CombineArgs<8> A, int m, int nout,
                                                                int64_t n) {
  extern __shared__ uint4 sBd[];
  __shared__ unsigned long long lists[CB_THREADS / 32][CB_LIST];
  unsigned long long* list = lists[threadIdx.x >> 5];
  int count = 0;
  const unsigned mine = combine_mine(nout);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ng = (m + 15) / 16, NT = (nout + 7) / 8;
  int F[2][2];
  double(*sY)[16] = (double(*)[16])(sBd + ng * 2 * 32 * CB_CELL);  // the coefficients, for combine_small
  for (int k = threadIdx.x; k < m * 16; k += CB_THREADS) sY[k >> 4][k & 15] = A.y[k >> 4][k & 15];
  combine_setup<2>(A, m, sBd, F);  // ends with a barrier
  const int64_t stride = (int64_t)gridDim.x * (CB_THREADS / 32) * 16;
  for (int64_t r = ((int64_t)blockIdx.x * (CB_THREADS / 32) + (threadIdx.x >> 5)) * 16; r < n; r += stride) {
    const int64_t row = r + 2 * g;
    uint32_t w0 = 0u, w1 = 0u;
    bool lo0 = false, lo1 = false;
#pragma unroll 4
    for (int i = t; i < m; i += 4) {
      const double2 v = load2<VEC>(A.v[i], row, n);
      w0 = max(w0, (uint32_t)__double2hiint(v.x) & 0x7FFFFFFFu);
      w1 = max(w1, (uint32_t)__double2hiint(v.y) & 0x7FFFFFFFu);
      lo0 |= __double2loint(v.x) != 0;
      lo1 |= __double2loint(v.y) != 0;
    }
    const RowPair rp = combine_rows(w0, w1, lo0, lo1);
    const int e0 = rp.e0, e1 = rp.e1;
    unsigned need = 0u;
    int L[2][6][4];
    for (int c = 0; c < ng; ++c) {
      double2 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = 16 * c + 2 * t + (k & 1) + 8 * (k >> 1);
        v[k] = i < m ? load2<VEC>(A.v[i], row, n) : make_double2(0.0, 0.0);
      }
      uint32_t a[4][CB_DIG];
      combine_digits(v, e0, e1, a);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        if (nt < NT) {
          uint32_t b[2 * CB_DIG];
          float acc[CB_LEV][4];
          combine_b(sBd, c * 2 + nt, lane, b);
          combine_mma(a, b, acc);
#pragma unroll
          for (int l = 0; l < 6; ++l)
#pragma unroll
            for (int q = 0; q < 4; ++q) L[nt][l][q] = (c ? L[nt][l][q] : 0) + combine_level(acc, l, q);
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (8 * nt + k >= nout) break;
        const int X0 = e0 + F[nt][k] - 2044 - 56, X1 = e1 + F[nt][k] - 2044 - 56;
        const bool fast = combine_fast(X0, X1);
        double2 res;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int Lq[6];
#pragma unroll
          for (int l = 0; l < 6; ++l) Lq[l] = L[nt][l][2 * h + k];
          bool small;
          const double d = combine_value(Lq, h ? X1 : X0, fast, small);
          if (h) res.y = d; else res.x = d;
          need |= (small ? 1u : 0u) << (4 * nt + 2 * k + h);
        }
        combine_out<VEC>(A, 8 * nt + 2 * t + k, res, nout, row, n);
      }
    need &= rp.keep & mine;
    if (__any_sync(0xffffffffu, need)) combine_note(A, m, sY, need, row, n, list, count);
    __syncwarp();  // the stores above come first
    if (rp.slow0 || rp.slow1) combine_row_fp64(A, m, nout, t, rp.slow0, rp.slow1, row, n);
    __syncwarp();
  }
  if (count) combine_small(A, m, sY, list, count);
}

template <int NC, int NT, bool VEC>
int combine_launch(ed_ctx* ctx, const CombineArgs<NC>& A, int m, int nout, int64_t n) {
  auto go = [&](auto kern, size_t smem) -> int {
    if (smem > 0) ED_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    ED_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, CB_THREADS, smem));
    const int64_t tiles = (n + 15) / 16, b = (tiles + CB_THREADS / 32 - 1) / (CB_THREADS / 32);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)ctx->num_sms * std::max(1, per_sm)));
    kern<<<grid, CB_THREADS, smem, ctx->stream>>>(A, m, nout, n);
    ED_CHECK_LAUNCH(ctx);
    return ED_OK;
  };
  if constexpr (NC > 2) return go(k_combine_many<VEC>, sizeof(uint4) * (size_t)((m + 15) / 16) * 2 * 32 * CB_CELL + sizeof(double) * 16 * (size_t)m);
  else return go(k_combine<NC, NT, VEC>, 0);
}

template <int NC>
int combine_nc(ed_ctx* ctx, const double* const* cols, int m, const double* Y, int ldY, int l, double* const* out,
               int64_t n) {
  bool vec = true;
  for (int i = 0; i < m; ++i) vec = vec && ((uintptr_t)cols[i] & 15) == 0;
  for (int c = 0; c < l; ++c) vec = vec && ((uintptr_t)out[c] & 15) == 0;
  // 16 outputs per pass over V (two groups of 8 share its loads and digits)
  for (int c0 = 0; c0 < l; c0 += 16) {
    const int nout = std::min(16, l - c0);
    CombineArgs<NC> A;
    memset(&A, 0, sizeof(A));
    for (int i = 0; i < m; ++i) {
      A.v[i] = cols[i];
      for (int c = 0; c < nout; ++c) A.y[i][c] = Y[(size_t)i * ldY + c0 + c];
    }
    for (int c = 0; c < nout; ++c) A.out[c] = out[c0 + c];
    int rc;
    if (nout <= 8) rc = vec ? combine_launch<NC, 1, true>(ctx, A, m, nout, n) : combine_launch<NC, 1, false>(ctx, A, m, nout, n);
    else rc = vec ? combine_launch<NC, 2, true>(ctx, A, m, nout, n) : combine_launch<NC, 2, false>(ctx, A, m, nout, n);
    ED_TRY(rc);
  }
  return ED_OK;
}

}  // namespace

int ed_combine(ed_ctx* ctx, const double* const* cols, int m, const double* Y, int ldY, int l, double* const* out,
               int64_t n) {
  if (m < 1 || m > CB_MAXM || n < 1) return ED_ENOTSUP;
  for (int i = 0; i < m; ++i)
    for (int c = 0; c < l; ++c)
      if (!std::isfinite(Y[(size_t)i * ldY + c])) return ED_ENOTSUP;  // the FP64 form propagates it
  if (m <= 16) return combine_nc<1>(ctx, cols, m, Y, ldY, l, out, n);
  if (m <= 32) return combine_nc<2>(ctx, cols, m, Y, ldY, l, out, n);
  return combine_nc<8>(ctx, cols, m, Y, ldY, l, out, n);
}
