// Correlations of a real state (the solver's eigenvectors are real): every
// S^z S^z moment and every flip sum from two passes over the state, for all
// pairs of sites at once.  They serve the four operators of ExpectVal
// (src/spinOperators/correlation.cpp:38-299), the sublattice magnetisations
// and the energy gradients.
//
// S^z moments.  w_r = psi_r^2 (FP64) as a 128-bit integer at the scale
// 2^(124 - e), sum_r w_r < 2^e, which holds every w_r above 2^(e - 72)
// exactly; all sums are exact integer sums.  A state splits into its high
// half c1 and its low half c0 (the two-table rank: the states of one c1 are
// one run of rows, in the order of the low halves of equal popcount), so
// every pair moment follows from three small tables:
//   W0[c0]    = sum over c1 of w          (k_corr_cols: a thread owns c0)
//   M[i][c1]  = sum over c0 with bit i of w, i a low site
//   M[w0][c1] = sum over c0 of w          (k_corr_rows: a warp owns c1)
// That is one 128-bit add per row and low site instead of one per row and
// pair: at N=28 (40.1M rows, 406 pairs) 0.44 ms instead of 13.4 ms for the
// 26 passes of 16 pairs before.
//
// Flip sums.  F_ij = sum over rows with bit i set and j clear of psi_r
// psi_r' equals sum_t phi_i(t) phi_j(t) over the states t with one spin less
// up, phi_i(t) = psi(t + spin i) (0 where i is up in t): a Gram matrix with
// N rows, and N gathers of half-empty columns per t serve all N^2 / 2 pairs.
// As FP64 FMAs it would be bound by the FP64 unit (7.4 ms at N=28), so it
// runs on the tensor cores in exact 8-bit digits (k_corr_gram): 2.5 ms at
// N=28 (seven digits; now eight and a second product, 10% of the call more)
// instead of 31.6 ms for 26 passes of 16 pairs before.  Small flip sums are formed
// again in FP64, so a list's length does not change their accuracy.  All S.S of
// the N=28 state: 47.5 -> 3.23 ms; the energy gradient over 96 bonds at N=24: 10.9
// -> 0.35 ms.
#include "ed_internal.h"
#include "ed_device.cuh"
#include "ed_halves.cuh"
#include "ed_umma.cuh"
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace {

constexpr int CR_SITES = 32;      // sites padded to 32

// 128-bit integer accumulators (two 64-bit words, add with carry)
__device__ __forceinline__ void add128(unsigned long long& lo, unsigned long long& hi, unsigned long long alo,
                                       unsigned long long ahi) {
  asm("add.cc.u64 %0, %0, %2;\n\taddc.u64 %1, %1, %3;" : "+l"(lo), "+l"(hi) : "l"(alo), "l"(ahi));
}

// w >= 0 (finite) as the 128-bit integer round(w 2^S); exact when w's last
// bit is at or above 2^-S.  w < 2^(124 - S) keeps it below 2^124.
__device__ __forceinline__ void fx128(double w, int S, unsigned long long& lo, unsigned long long& hi) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(w);
  const int E = (int)((bits >> 52) & 0x7FF);
  const unsigned long long mant = (bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int sh = E - 1075 + S;  // w 2^S = mant 2^sh
  lo = 0ull;
  hi = 0ull;
  if (E == 0) return;  // zero or below 2^-1022
  if (sh >= 64) {
    hi = mant << (sh - 64);
  } else if (sh > 0) {
    lo = mant << sh;
    hi = mant >> (64 - sh);
  } else if (sh == 0) {
    lo = mant;
  } else if (sh > -54) {
    lo = (mant + (1ull << (-sh - 1))) >> (-sh);
  }
}

struct CorrHeader {
  double W;        // sum psi_r^2
  double B;        // sum |w_r| (two vectors; with one it is W)
  int imag;        // some imaginary part is not zero
  int emax;        // largest biased exponent of a real part
  int nonfinite;   // some part is not finite
  unsigned done;   // blocks finished
  int err;         // a wait of k_corr_gram ran out
};

// One pass over psi (TWO: and lam): the real parts to pr (pl), the sum of
// squares of psi (TWO: and sum |lam psi|), psi's largest exponent and the
// flags.  Four rows in flight per thread; bound by memory (24 bytes per row and
// vector).  The last block sums the block partials in order.
template <bool TWO>
__global__ void __launch_bounds__(256) k_corr_prep(const double2* __restrict__ psi, const double2* __restrict__ lam,
                                                   int64_t n, double* __restrict__ pr, double* __restrict__ pl,
                                                   CorrHeader* __restrict__ hdr, double* __restrict__ part) {
  constexpr int NA = TWO ? 2 : 1;
  double acc[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) acc[k] = 0.0;
  int im = 0, nf = 0, em = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r0 < n; r0 += 4 * stride) {
    double xa[4];
#pragma unroll
    for (int k = 0; k < NA; ++k) {
      const double2* src = k ? lam : psi;
      double* dst = k ? pl : pr;
      double2 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = r0 + u * stride < n ? src[r0 + u * stride] : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r0 + u * stride < n) dst[r0 + u * stride] = v[u].x;
        const int e = (int)((__double_as_longlong(v[u].x) >> 52) & 0x7FF);
        if (k == 0) em = max(em, e);
        nf |= e == 0x7FF;
        im |= v[u].y != 0.0;  // a NaN counts as not zero
        if (k == 0) xa[u] = v[u].x;
        acc[k] = fma(fabs(v[u].x), fabs(xa[u]), acc[k]);
      }
    }
  }
  em = (int)__reduce_max_sync(0xffffffffu, (unsigned)em);
  nf = (int)__reduce_or_sync(0xffffffffu, (unsigned)nf);
  im = (int)__reduce_or_sync(0xffffffffu, (unsigned)im);
  if ((threadIdx.x & 31) == 0) {
    if (em > 0) atomicMax(&hdr->emax, em);
    if (nf) atomicOr(&hdr->nonfinite, 1);
    if (im) atomicOr(&hdr->imag, 1);
  }
  __shared__ double sh[32 * NA];
  __shared__ bool last;
  ed_block_reduce<NA>(acc, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NA; ++k) part[k * gridDim.x + blockIdx.x] = acc[k];
    __threadfence();
    last = atomicAdd(&hdr->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) {
    t[k] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) t[k] += __ldcg(part + k * gridDim.x + b);
  }
  __syncthreads();  // sh free
  ed_block_reduce<NA>(t, sh);
  if (threadIdx.x == 0) {
    hdr->W = t[0];
    hdr->B = t[NA - 1];
  }
}

// The row's weight w = x y as a signed 128-bit integer (y = x with one vector).
template <bool TWO>
__device__ __forceinline__ void weight128(double x, double y, int S, unsigned long long& lo, unsigned long long& hi) {
  if (!TWO) {
    fx128(x * x, S, lo, hi);
    return;
  }
  const double w = x * y;
  fx128(fabs(w), S, lo, hi);
  if (w < 0.0) {
    lo = ~lo;
    hi = ~hi;
    add128(lo, hi, 1ull, 0ull);
  }
}

// W0: thread = one low half, loop over a segment of the high halves of its
// class: 256 consecutive rows per block and high half, so the reads are
// coalesced; bound by memory.  The 128-bit sum of a segment is added to the
// table as four 32-bit limbs in 64-bit integers (order does not matter).
constexpr int COLS_SEG = 64;  // most high halves per block
template <bool TWO>
__global__ void __launch_bounds__(256) k_corr_cols(const double* __restrict__ pr, const double* __restrict__ pl,
                                                   const CorrGeom g,
                                                   const uint16_t* __restrict__ lows,
                                                   const uint32_t* __restrict__ highs,
                                                   const uint32_t* __restrict__ t1, int S, int nseg,
                                                   unsigned long long* __restrict__ W0) {
  int k = 0;
  while (k < g.w0 && (int)blockIdx.x >= g.prefix[k + 1]) ++k;
  const int item = (int)blockIdx.x - g.prefix[k];
  const int seg = item / g.chunks[k], o = (item - seg * g.chunks[k]) * 256 + (int)threadIdx.x;
  const int h0 = seg * nseg, h1 = min(g.nhigh[k], h0 + nseg);
  __shared__ uint32_t base[COLS_SEG];
  for (int h = h0 + threadIdx.x; h < h1; h += blockDim.x) base[h - h0] = t1[highs[g.high_off[k] + h]];
  __syncthreads();
  if (o >= g.nlow[k]) return;
  unsigned long long lo = 0ull, hi = 0ull;
  for (int h = 0; h < h1 - h0; h += 4) {
    double x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool on = h + u < h1 - h0;
      x[u] = on ? pr[(size_t)base[h + u] + o] : 0.0;
      y[u] = TWO && on ? pl[(size_t)base[h + u] + o] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      unsigned long long wl, wh;
      weight128<TWO>(x[u], y[u], S, wl, wh);
      add128(lo, hi, wl, wh);
    }
  }
  unsigned long long* d = W0 + (size_t)lows[g.low_off[k] + o] * 4;
  atomicAdd(d, lo & 0xFFFFFFFFull);
  atomicAdd(d + 1, lo >> 32);
  atomicAdd(d + 2, hi & 0xFFFFFFFFull);
  atomicAdd(d + 3, (unsigned long long)((long long)hi >> 32));  // signed
}

// round(v 2^(62 - E)) for |v| < 2^E, E = emax - 1022, plus 128 in each byte:
// byte i is then digit i + 128 of the balanced base-256 representation, digits
// in [-128, 127] (|q| <= 2^62).  Halves round to even: half of the entries ten
// binades below the largest are halves, and rounding them up added to the sums of
// a state of one sign.
constexpr unsigned long long GRAM_ZERO = 0x8080808080808080ull;
__device__ __forceinline__ unsigned long long gram_entry(double v, int emax) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((b >> 52) & 0x7FF);
  if (e == 0) return GRAM_ZERO;
  const unsigned long long mant = (unsigned long long)(b & 0xFFFFFFFFFFFFFll) | 0x10000000000000ull;
  const int sh = e - emax + 9;  // <= 9
  unsigned long long q;
  if (sh >= 0) q = mant << sh;
  else if (sh > -60) q = (mant + (1ull << (-sh - 1)) - 1ull + ((mant >> -sh) & 1ull)) >> (-sh);
  else q = 0ull;
  return b < 0 ? GRAM_ZERO - q : GRAM_ZERO + q;
}

// M: warp = one high half, its run of rows; lane 0 ends with the sums over
// the low halves with bit i set (i < w0) and over all.  The bit tests and
// adds of the 14 low sites (four 32-bit adds each) are most of the work.
// QUANT: each entry is then replaced by its digits for k_corr_gram.
template <bool QUANT, bool TWO>
__global__ void __launch_bounds__(128) k_corr_rows(double* __restrict__ pr, const double* __restrict__ pl, int w0,
                                                   int w1, int nup,
                                                   const CorrGeom g, const uint16_t* __restrict__ lows,
                                                   const uint32_t* __restrict__ t1, int S, int emax,
                                                   ulonglong2* __restrict__ M) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int c1 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c1 < (1 << w1); c1 += nwarps) {
    const int k = nup - __popc(c1);
    if (k < 0 || k > w0) {
      if (lane <= w0) M[((size_t)lane << w1) + c1] = make_ulonglong2(0ull, 0ull);
      continue;
    }
    unsigned long long lo[CR_MAXW0 + 1], hi[CR_MAXW0 + 1];
#pragma unroll
    for (int i = 0; i <= CR_MAXW0; ++i) lo[i] = hi[i] = 0ull;
    const int n = g.nlow[k];
    const uint16_t* lw = lows + g.low_off[k];
    double* p = pr + t1[c1];
    const double* py = pl + t1[c1];
    double xn = lane < n ? p[lane] : 0.0, yn = TWO && lane < n ? py[lane] : 0.0;
    uint32_t cn = lane < n ? lw[lane] : 0u;
    for (int o = lane; o < n; o += 32) {
      const double x = xn, y = yn;
      const uint32_t c0 = cn;
      if (o + 32 < n) {
        xn = p[o + 32];
        if (TWO) yn = py[o + 32];
        cn = lw[o + 32];
      }
      unsigned long long wl, wh;
      weight128<TWO>(x, y, S, wl, wh);
#pragma unroll
      for (int i = 0; i < CR_MAXW0; ++i)
        if ((c0 >> i) & 1u) add128(lo[i], hi[i], wl, wh);
      add128(lo[CR_MAXW0], hi[CR_MAXW0], wl, wh);
      if (QUANT) ((unsigned long long*)p)[o] = gram_entry(x, emax);
    }
#pragma unroll
    for (int i = 0; i <= CR_MAXW0; ++i) {
      if (i < w0 || i == CR_MAXW0) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
          const unsigned long long ol = __shfl_down_sync(0xffffffffu, lo[i], s);
          const unsigned long long oh = __shfl_down_sync(0xffffffffu, hi[i], s);
          add128(lo[i], hi[i], ol, oh);
        }
        if (lane == 0) M[((size_t)(i < w0 ? i : w0) << w1) + c1] = make_ulonglong2(lo[i], hi[i]);
      }
    }
  }
}

// P[a (a + 1) / 2 + b], b <= a: sum of w over the states with sites a and b
// up; the last entry: the sum over all states.  One block per entry.
__global__ void __launch_bounds__(256) k_corr_moments(const unsigned long long* __restrict__ W0,
                                                      const ulonglong2* __restrict__ M, int w0, int w1, int npairs,
                                                      ulonglong2* __restrict__ P) {
  const int q = blockIdx.x;
  int a = 0;
  while ((a + 1) * (a + 2) / 2 <= q) ++a;
  const int b = q - a * (a + 1) / 2;
  unsigned long long lo = 0ull, hi = 0ull;
  if (q < npairs && a < w0) {  // both low
    const uint32_t m = (1u << a) | (1u << b);
    for (int c = threadIdx.x; c < (1 << w0); c += blockDim.x) {
      if ((c & m) != m) continue;
      const unsigned long long* d = W0 + (size_t)c * 4;
      add128(lo, hi, d[0], 0ull);
      add128(lo, hi, d[1] << 32, d[1] >> 32);
      add128(lo, hi, 0ull, d[2]);
      add128(lo, hi, 0ull, d[3] << 32);
    }
  } else {
    // a high (or everything): rows of M over the high halves with the bits
    const bool all = q >= npairs;
    const uint32_t m = all ? 0u : (1u << (a - w0)) | (b >= w0 ? 1u << (b - w0) : 0u);
    const ulonglong2* row = M + ((size_t)((!all && b < w0) ? b : w0) << w1);
    for (int c = threadIdx.x; c < (1 << w1); c += blockDim.x) {
      if (((uint32_t)c & m) != m) continue;
      const ulonglong2 v = row[c];
      add128(lo, hi, v.x, v.y);
    }
  }
  __shared__ unsigned long long sl[8], sh[8];
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const unsigned long long ol = __shfl_down_sync(0xffffffffu, lo, s), oh = __shfl_down_sync(0xffffffffu, hi, s);
    add128(lo, hi, ol, oh);
  }
  if ((threadIdx.x & 31) == 0) {
    sl[threadIdx.x >> 5] = lo;
    sh[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) add128(lo, hi, sl[w], sh[w]);
    P[q] = make_ulonglong2(lo, hi);
  }
}

// ---------------------------------------------------------------------------
// Gram matrix F = Phi Phi^T on the tensor cores.  phi_i(t) in 63-bit fixed
// point against the largest entry of the state, as eight balanced 8-bit digits,
// which FP16 holds exactly.  One tcgen05.mma has M = 128 rows (digits 0..3 x 32
// sites), N = 256 columns (digits 0..7 x 32 sites) and K = 16 states; the digits
// are symmetric in the two factors, so every product with a digit of 0..3 is
// among them or the transpose of one.  Of the products of digits 4..7 alone a
// second MMA (M = digits 4..7, N = digit 4) brings those that matter: (4, 4) is
// 2^-62 of the squared scale per state with a random sign, and without it the
// flip sums of a state of a few decades at N=24 had 5 times the error of FP64
// chains (6.5e-18 where the last rounding is 5.2e-19, as it is now); what is left,
// (5, 5) and below, is 2^-78.  It takes 6% of the kernel, the one set of
// accumulators 12%; two sets, with the first MMA split in halves, were slower (3.69
// against 3.23 ms for all pairs at N=28).  A digit product sum stays an exact
// integer in the FP32 accumulator over GRAM_GROUP stages (1024 states x 128^2 =
// 2^24), then four epilogue warps add it to 64-bit integers in shared memory.  The
// accumulators fill more than half of the TMEM, so there is one set; the producers,
// which bound the kernel, go on for two stages while it is read.
//
// The rounded entries leave a root mean square error of at most 2^-62 / sqrt(12)
// of 2^E times the norm: that of the last rounding of F for |F| >= 2^-9 2^E norm.
// Smaller flip sums (sharply peaked states) are formed again in FP64
// (ed_corr_real).  With 55 bits a flip sum of 6e-8 of a Neel-like state was off
// by 1e-13 of itself.
//
// A stage is 128 states t = (c1, 128 consecutive low halves of one popcount).
// The 16 producer warps take two sites each: a lane reads the entries of its
// site for 8 states (16 apart, so that a load instruction reads 128
// consecutive bytes for a high site), splits them with PRMT and one FP16 add
// per pair, and writes 16 bytes per digit: the K-major core-matrix row of its
// site.  The targets of a low site depend on the low half alone: they stay
// in registers while the stages run over the high halves.  The loads of the
// next stage are issued before the current one is converted.
// ---------------------------------------------------------------------------
constexpr int GRAM_DIG = 8;
constexpr int GRAM_AGAIN = 9;                                  // a flip sum below 2^-9 2^E norm: again in FP64
constexpr int GRAM_STATES = 128;
constexpr int GRAM_ROWS = GRAM_DIG * CR_SITES;                 // 256
constexpr int GRAM_N = GRAM_ROWS;
constexpr int GRAM_LBO = GRAM_ROWS * 16 + 16;                  // + 16: the 16-byte rows of 8 lanes miss each other's banks
constexpr int GRAM_STAGE = (GRAM_STATES / 8) * GRAM_LBO;       // 65792 bytes
constexpr int GRAM_GROUP = 8;                                  // stages per accumulation: 2^24 bound
constexpr int GRAM_PROD = 16, GRAM_THREADS = (GRAM_PROD + 5) * 32;
constexpr int GRAM_PLANE = 3;                                  // columns 0..3, 4..7, and digit 4 x digits 4..7
constexpr int GRAM_ACC = 128 * CR_SITES * GRAM_PLANE;          // 64-bit sums per CTA
constexpr int GRAM_LOW = GRAM_N;                               // TMEM column of the second MMA's sums
constexpr size_t GRAM_SMEM = 2 * (size_t)GRAM_STAGE + (size_t)GRAM_ACC * 8;

struct GramShared {
  uint64_t full[2], empty[2], tfull, tempty, done;
  uint32_t tmem;
};

// A place in the stage order: classes, then pieces of 128 low halves, then
// high halves.  Advanced one stage at a time (no division per stage).
struct GramAt {
  int k, tile, hi, nhigh, high_off, chunks;
  __device__ __forceinline__ void enter(const CorrGeom& g) {
    nhigh = g.nhigh[k];
    high_off = g.high_off[k];
    chunks = g.chunks[k];
  }
  __device__ __forceinline__ void start(const CorrGeom& g, int s) {
    k = 0;
    while (s >= g.prefix[k + 1]) ++k;
    enter(g);
    tile = (s - g.prefix[k]) / nhigh;
    hi = s - g.prefix[k] - tile * nhigh;
  }
  __device__ __forceinline__ void next(const CorrGeom& g) {
    if (++hi < nhigh) return;
    hi = 0;
    if (++tile < chunks) return;
    tile = 0;
    do {  // past the last class: stay there (the caller stops)
      if (k + 1 >= CR_CLASSES) return;
      ++k;
      enter(g);
    } while (nhigh == 0);
  }
};

__device__ __forceinline__ void gram_ld8(uint32_t taddr, uint32_t (&d)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7])
               : "r"(taddr));
}

// orders the uses of loaded registers after the wait before it
__device__ __forceinline__ void gram_loaded(uint32_t (&d)[8]) {
#pragma unroll
  for (int c = 0; c < 8; ++c) asm volatile("" : "+r"(d[c]));
}

__device__ __forceinline__ void gram_mma(uint32_t dcol, uint64_t a, uint64_t b, uint32_t idesc, uint32_t keep) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(dcol),
      "l"(a), "l"(b), "r"(idesc), "r"(keep));
}

__global__ void __launch_bounds__(GRAM_THREADS, 1) k_corr_gram(const unsigned long long* __restrict__ q,
                                                               const __grid_constant__ CorrGeom g, int nstages,
                                                               const uint16_t* __restrict__ t0,
                                                               const uint32_t* __restrict__ t1,
                                                               const uint16_t* __restrict__ lows,
                                                               const uint32_t* __restrict__ highs,
                                                               long long* __restrict__ part, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ GramShared S;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  long long* acc = (long long*)(smem + 2 * GRAM_STAGE);  // [site b][plane][TMEM lane]
  for (int i = tid; i < GRAM_ACC; i += GRAM_THREADS) acc[i] = 0ll;
  if (warp == GRAM_PROD + 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&S.full[i])), "r"(GRAM_PROD));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.empty[i])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.tfull)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&S.tempty)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.done)));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = S.tmem;
  // this CTA's stages: a contiguous piece, high halves innermost
  const int s0 = (int)((int64_t)nstages * blockIdx.x / gridDim.x);
  const int s1 = (int)((int64_t)nstages * (blockIdx.x + 1) / gridDim.x);
  if (warp < GRAM_PROD && 2 * warp >= g.N) {
    // Both sites lie past the last one: their digits are zero in every stage,
    // so both buffers get them once.  The wait for empty stays: without it a
    // warp could arrive twice in one phase of full.
    // All pairs at N=28 (2 of 16 warps): 2.95 -> 2.88 ms; all bonds at N=24
    // (4 of 16): 308 -> 295 us (the whole call).
    const int site = 2 * warp + (lane >> 4), l = lane & 15;
    for (int b = 0; b < 2; ++b)
      for (int d = 0; d < GRAM_DIG; ++d)
        *reinterpret_cast<uint4*>(smem + b * GRAM_STAGE + l * GRAM_LBO + site * 16 + d * (CR_SITES * 16)) =
            make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int s = s0; s < s1; ++s) {
      const int it = s - s0, st = it & 1;
      if (!mbar_wait(smem_u32(&S.empty[st]), ((it >> 1) & 1) ^ 1, TC_WAIT_POLLS)) {
        atomicExch(err, 1);
        break;
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&S.full[st])) : "memory");
    }
  } else if (warp < GRAM_PROD) {
    const int site = 2 * warp + (lane >> 4), l = lane & 15;
    const bool low = site < g.w0, high = !low && site < g.N;
    const uint32_t jbit = high ? 1u << (site - g.w0) : 0u;
    int off[8], cur_k = -1, cur_tile = -1;
    // targets of the 8 states of a (class, tile) for this site
    auto targets = [&](int k, int tile) {
      cur_k = k;
      cur_tile = tile;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int o = tile * GRAM_STATES + l + 16 * u;
        off[u] = -1;
        if (o < g.nlow[k]) {
          if (high) {
            off[u] = o;
          } else if (low) {
            const uint32_t c0 = lows[g.low_off[k] + o];
            if (!((c0 >> site) & 1u)) off[u] = (int)t0[c0 | (1u << site)];
          }
        }
      }
    };
    unsigned long long v[8], nx[8];
    auto gather = [&](uint32_t base, bool on, unsigned long long (&d)[8]) {
      const unsigned long long* p = q + base;
#pragma unroll
      for (int u = 0; u < 8; ++u) d[u] = on && off[u] >= 0 ? __ldg(p + off[u]) : GRAM_ZERO;
    };
    // A gather needs T1 of the stage's high half: the high half is read three
    // stages ahead and its T1 two, so that no load waits for the one before.
    // With the place advanced instead of divided for: all pairs at N=28 3.23 ->
    // 2.95 ms, all bonds at N=24 344 -> 314 us (the whole call).  Past the last
    // stage the place stays a valid one: an empty class has high_off 0.
    GramAt at1, at3;  // the places of stages s + 1 and s + 3
    uint32_t c1a = 0u, base1 = 0u;
    bool on1 = false;
    if (s0 < s1) {
      at3.start(g, s0);
      targets(at3.k, at3.tile);
      const uint32_t c1 = highs[at3.high_off + at3.hi];
      gather(t1[c1 | jbit], (c1 & jbit) == 0u, v);
      at3.next(g);
      at1 = at3;
      c1a = highs[at3.high_off + at3.hi];  // stage s0 + 1 (or any valid place past the end)
      base1 = t1[c1a | jbit];
      on1 = (c1a & jbit) == 0u;
      at3.next(g);
      c1a = highs[at3.high_off + at3.hi];  // s0 + 2
      at3.next(g);
    }
    const __half2 shift = __floats2half2_rn(-1152.0f, -1152.0f);
    for (int s = s0; s < s1; ++s) {
      const int it = s - s0, st = it & 1;
      if (s + 1 < s1) {
        if (at1.k != cur_k || at1.tile != cur_tile) targets(at1.k, at1.tile);
        gather(base1, on1, nx);
        at1.next(g);
        base1 = t1[c1a | jbit];              // stage s + 2
        on1 = (c1a & jbit) == 0u;
        c1a = highs[at3.high_off + at3.hi];  // s + 3
        at3.next(g);
      }
      if (!mbar_wait(smem_u32(&S.empty[st]), ((it >> 1) & 1) ^ 1, TC_WAIT_POLLS)) {
        atomicExch(err, 1);
        break;
      }
      unsigned char* dst = smem + st * GRAM_STAGE + l * GRAM_LBO + site * 16;
#pragma unroll
      for (int d = 0; d < GRAM_DIG; ++d) {
        const int by = GRAM_DIG - 1 - d;
        const uint32_t sel = (uint32_t)(by & 3) | ((uint32_t)((by & 3) + 4) << 8);
        uint32_t w[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const uint32_t x = by < 4 ? (uint32_t)v[2 * p] : (uint32_t)(v[2 * p] >> 32);
          const uint32_t y = by < 4 ? (uint32_t)v[2 * p + 1] : (uint32_t)(v[2 * p + 1] >> 32);
          // bytes (x, ?, y, ?) under the exponent of 1024, then 1024 + 128 off
          uint32_t h;
          asm("prmt.b32 %0, %1, %2, %3;" : "=r"(h) : "r"(x), "r"(y), "r"(sel));
          h = (h & 0x00FF00FFu) | 0x64006400u;
          const __half2 r = __hadd2(*reinterpret_cast<__half2*>(&h), shift);
          w[p] = *reinterpret_cast<const uint32_t*>(&r);
        }
        *reinterpret_cast<uint4*>(dst + d * (CR_SITES * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&S.full[st])) : "memory");
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = nx[u];
    }
  } else if (warp < GRAM_PROD + 4) {
    // epilogue: TMEM lane = digit i of the first factor (this warp's) x site a
    const int sub = warp - GRAM_PROD;
    const int ngroups = (s1 - s0 + GRAM_GROUP - 1) / GRAM_GROUP;
    for (int gq = 0; gq < ngroups; ++gq) {
      if (!mbar_wait(smem_u32(&S.tfull), gq & 1, TC_WAIT_POLLS)) {
        atomicExch(err, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t taddr = tmem + ((uint32_t)(sub * 32) << 16);
#pragma unroll 1
      for (int b0 = 0; b0 < CR_SITES; b0 += 8) {
        long long* ab = acc + (size_t)(b0 * GRAM_PLANE) * 128 + sub * 32 + lane;
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {  // digits 0..3, 4..7 of the second factor
          uint32_t d[4][8];
#pragma unroll
          for (int j = 0; j < 4; ++j) gram_ld8(taddr + (uint32_t)((4 * pl + j) * CR_SITES + b0), d[j]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 4; ++j) gram_loaded(d[j]);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            long long t = 0ll;
#pragma unroll
            for (int j = 0; j < 4; ++j) t = t * 256 + (long long)__float2int_rz(__uint_as_float(d[j][c]));
            ab[(c * GRAM_PLANE + pl) * 128] += t;
          }
        }
        uint32_t d[8];  // digit 4 + sub of the first factor x digit 4
        gram_ld8(taddr + (uint32_t)(GRAM_LOW + b0), d);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        gram_loaded(d);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          ab[(c * GRAM_PLANE + 2) * 128] += (long long)__float2int_rz(__uint_as_float(d[c]));
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&S.tempty)) : "memory");
    }
  } else if (lane == 0) {
    const uint32_t idesc = umma_idesc_f16(128, GRAM_N), idesc_low = umma_idesc_f16(128, CR_SITES);
    const uint32_t base = smem_u32(smem);
    for (int s = s0; s < s1; ++s) {
      const int it = s - s0, st = it & 1, gq = it / GRAM_GROUP, in = it % GRAM_GROUP;
      if (!mbar_wait(smem_u32(&S.full[st]), (it >> 1) & 1, TC_WAIT_POLLS) ||
          (in == 0 && !mbar_wait(smem_u32(&S.tempty), (gq & 1) ^ 1, TC_WAIT_POLLS))) {
        atomicExch(err, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      // rows 0 .. 127 of a stage are digits 0..3, rows 128 .. 255 digits 4..7
      auto rows = [&](int ks, int r) { return umma_desc(base + st * GRAM_STAGE + ks * 2 * GRAM_LBO + r * 16, GRAM_LBO, 128); };
#pragma unroll
      for (int ks = 0; ks < GRAM_STATES / 16; ++ks) {
        const uint32_t keep = in > 0 || ks > 0 ? 1u : 0u;
        gram_mma(tmem, rows(ks, 0), rows(ks, 0), idesc, keep);
        gram_mma(tmem + (uint32_t)GRAM_LOW, rows(ks, 128), rows(ks, 128), idesc_low, keep);
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&S.empty[st]))
                   : "memory");
      if (in == GRAM_GROUP - 1 || s + 1 == s1)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&S.tfull))
                     : "memory");
    }
    // every MMA issued has completed before the TMEM is freed
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(&S.done))
                 : "memory");
    if (!mbar_wait(smem_u32(&S.done), 0, TC_WAIT_POLLS)) atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  for (int i = tid; i < GRAM_ACC; i += GRAM_THREADS) part[(size_t)blockIdx.x * GRAM_ACC + i] = acc[i];
  if (warp == GRAM_PROD + 4)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// Sums over the CTAs and the digits i, as 128-bit integers in units of 2^32
// q-units: out[b][a] = digit pairs (i, j <= 3), out[1024 + 32 b + a] = (i, j = 4..7),
// out[2048 + ..] = (4, 4), out[3072 + ..] = (5, 4) and (6, 4) ((7, 4) lies below the
// unit).  Block = site b, thread = plane and TMEM lane (i, a).
__global__ void __launch_bounds__(128 * GRAM_PLANE) k_corr_gram_sum(const long long* __restrict__ part, int ncta,
                                                                    ulonglong2* __restrict__ out) {
  const int b = blockIdx.x, plane = threadIdx.x >> 7, ln = threadIdx.x & 127, i = ln >> 5;
  const long long* p = part + (size_t)(b * GRAM_PLANE + plane) * 128 + ln;
  unsigned long long lo = 0ull, hi = 0ull;
  for (int c = 0; c < ncta; ++c) {
    const long long x = p[(size_t)c * GRAM_ACC];
    add128(lo, hi, (unsigned long long)x, (unsigned long long)(x >> 63));
  }
  const int sh = (plane == 0 ? 56 : plane == 1 ? 24 : 16) - 8 * i;  // 0 .. 56, below 0: (7, 4)
  if (sh > 0) {
    hi = (hi << sh) | (lo >> (64 - sh));
    lo <<= sh;
  }
  __shared__ unsigned long long sl[128 * GRAM_PLANE], sh_[128 * GRAM_PLANE];
  sl[threadIdx.x] = lo;
  sh_[threadIdx.x] = hi;
  __syncthreads();
  if (ln >= 32) return;
  ulonglong2* o = out + (size_t)plane * 1024 + b * 32 + ln;
  if (plane < 2) {
    for (int w = 1; w < 4; ++w) add128(lo, hi, sl[threadIdx.x + 32 * w], sh_[threadIdx.x + 32 * w]);
    *o = make_ulonglong2(lo, hi);
  } else {
    *o = make_ulonglong2(lo, hi);
    lo = sl[threadIdx.x + 32];
    hi = sh_[threadIdx.x + 32];
    add128(lo, hi, sl[threadIdx.x + 64], sh_[threadIdx.x + 64]);
    o[1024] = make_ulonglong2(lo, hi);
  }
}

// Flip sums directly, ED_CORR_FEW pairs per pass (grid.y, masks in fm): every
// antiparallel row is paired with its partner, so only rows with bit i set and bit j clear
// contribute.  Lane l of a warp serves pair l / 2: a ballot per pair marks
// the contributing rows among the warp's 32, and the pair's two lanes take
// alternate marked rows (state, psi and rank halves by shuffle), four
// gathers in flight each.  A row and pair that contribute nothing cost no FMA
// and no gather.  TWO: sum over the same rows of (lam_r psi_r' + lam_r' psi_r)
// / 2 with lam in pl.  A lane adds FL_FOLD chunks in a plain chain; the chains of
// a lane, the lanes and the blocks are joined as pairs, so that few long chains
// (16 pairs share the lanes) do not round more than the one row per thread and
// term of the general kernels: 1.6-1.7 times their error at N=24 as plain chains,
// 0.6-1.0 times so.  Two blocks per SM (three with two vectors, whose loads per
// gather are two), all resident: the registers then hold the loads in flight.  16
// bonds of a gradient at N=28 2.25 -> 2.22 ms, at N=16 93 -> 100 us; mixed
// expectations of 96 bonds at N=24 1.23 -> 1.26 ms.  partial[(pass ED_CORR_FEW + g) nblk + blk]: pairs.
struct FlipMasks {
  int n;
  uint32_t m[ED_CORR_FEW];   // (1 << i) | (1 << j)
  uint32_t bi[ED_CORR_FEW];  // 1 << i
  uint32_t ml[ED_CORR_FEW];  // m & (2^w0 - 1)
  uint32_t mh[ED_CORR_FEW];  // m >> w0
};

constexpr int FL_U = 4;
constexpr int FL_FOLD = 4;
template <bool TWO>
__global__ void __launch_bounds__(256, TWO ? 3 : 2) k_expect_flip_r(const uint32_t* __restrict__ states,
                                                       const double* __restrict__ pr, const double* __restrict__ pl,
                                                       int64_t dim, const uint16_t* __restrict__ t0,
                                                       const uint32_t* __restrict__ t1, int w0,
                                                       const FlipMasks* __restrict__ fm,
                                                       double2* __restrict__ partial, int nblk) {
  __shared__ FlipMasks pm;
  if (threadIdx.x < sizeof(FlipMasks) / 4) ((uint32_t*)&pm)[threadIdx.x] = ((const uint32_t*)(fm + blockIdx.y))[threadIdx.x];
  partial += (size_t)blockIdx.y * ED_CORR_FEW * nblk;
  extern __shared__ uint16_t t0s[];
  for (int i = threadIdx.x; i < (1 << w0); i += blockDim.x) t0s[i] = t0[i];
  __syncthreads();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int gl = lane >> 1, par = lane & 1;  // this lane's pair and its turn
  const bool gl_on = gl < pm.n;
  const uint32_t my_m = pm.m[gl], my_ml = pm.ml[gl], my_mh = pm.mh[gl];
  uint32_t mm[ED_CORR_FEW], mb[ED_CORR_FEW];
#pragma unroll
  for (int g = 0; g < ED_CORR_FEW; ++g) {
    mm[g] = pm.m[g];
    mb[g] = g < pm.n ? pm.bi[g] : 0xFFFFFFFFu;  // past the list: never met
  }
  // the chains before the current one, in shared memory: registers are what keeps
  // loads in flight
  __shared__ double2 shf[8 * 32];
  shf[threadIdx.x] = make_double2(0.0, 0.0);
  double fl = 0.0;  // the current chain
  int chunk = 0;
  bool folded = false;
  const uint32_t low = (1u << w0) - 1u;
  const int64_t step = (((int64_t)gridDim.x * blockDim.x) >> 5) * 32;
  int64_t base = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32;
  uint32_t s_n = 0u;
  double x_n = 0.0, y_n = 0.0;
  if (base + lane < dim) {
    s_n = states[base + lane];
    x_n = pr[base + lane];
    if (TWO) y_n = pl[base + lane];
  }
  for (; base < dim; base += step) {
    const int64_t r = base + lane;
    const bool valid = r < dim;
    const uint32_t s = s_n;
    const double x = x_n, y = y_n;
    s_n = 0u;  // rows past the end: never marked
    x_n = 0.0;
    if (base + step + lane < dim) {
      s_n = states[base + step + lane];
      x_n = pr[base + step + lane];
      if (TWO) y_n = pl[base + step + lane];
    }
    const uint32_t r0 = valid ? (uint32_t)t0s[s & low] : 0u;  // rank(s) = r0 + T1[s_hi]
    const uint32_t r1 = (uint32_t)r - r0;                    // = T1[s_hi]
    uint32_t L = 0u;
#pragma unroll
    for (int g = 0; g < ED_CORR_FEW; ++g) {
      const bool lead = valid && (s & mm[g]) == mb[g];
      const uint32_t bal = __ballot_sync(FULL, lead);
      L = gl == g ? bal : L;
    }
    if (!gl_on) L = 0u;
    if (par) L &= L - 1u;  // the pair's second lane starts at its second marked row
    const int mine = (__popc(L) + 1) >> 1;
    const int T = __reduce_max_sync(FULL, (unsigned)mine);
    for (int t = 0; t < T; t += FL_U) {
      int k[FL_U];
      bool has[FL_U];
#pragma unroll
      for (int u = 0; u < FL_U; ++u) {
        has[u] = L != 0u;
        k[u] = has[u] ? __ffs(L) - 1 : lane;
        L &= L - 1u;  // taken
        L &= L - 1u;  // the other lane's
      }
      double xk[FL_U], q[FL_U], yk[FL_U], ql[FL_U];
#pragma unroll
      for (int u = 0; u < FL_U; ++u) {
        const uint32_t sk = __shfl_sync(FULL, s, k[u]);
        const uint32_t r0k = __shfl_sync(FULL, r0, k[u]);
        const uint32_t r1k = __shfl_sync(FULL, r1, k[u]);
        xk[u] = __shfl_sync(FULL, x, k[u]);
        if (TWO) yk[u] = __shfl_sync(FULL, y, k[u]);
        q[u] = ql[u] = 0.0;
        if (has[u]) {
          const uint32_t f = sk ^ my_m;
          const uint32_t c = (my_ml ? (uint32_t)t0s[f & low] : r0k) + (my_mh ? __ldg(&t1[f >> w0]) : r1k);
          q[u] = __ldg(&pr[c]);
          if (TWO) ql[u] = __ldg(&pl[c]);
        }
      }
#pragma unroll
      for (int u = 0; u < FL_U; ++u)
        if (has[u]) fl = TWO ? fma(yk[u], q[u], fma(xk[u], ql[u], fl)) : fma(xk[u], q[u], fl);
    }
    if (++chunk == FL_FOLD) {
      double2 p = shf[threadIdx.x];
      ed_pair_add(p.x, p.y, fl, 0.0);
      shf[threadIdx.x] = p;
      fl = 0.0;
      chunk = 0;
      folded = true;
    }
  }
  {
    double2 p = shf[threadIdx.x];
    if (folded) ed_pair_add(p.x, p.y, fl, 0.0);
    else p.x = fl;
    shf[threadIdx.x] = p;
  }
  __syncthreads();
  // one warp: a lane adds its place of the eight warps, then the pair's two lanes
  // (64 FP64 instructions; 16 threads per pair in four steps are 256, which
  // bounded 80 pairs of short vectors)
  if (threadIdx.x >= 32) return;
  double2 p = shf[lane];
#pragma unroll
  for (int w = 1; w < 8; ++w) ed_pair_add(p.x, p.y, shf[w * 32 + lane].x, shf[w * 32 + lane].y);
  const double x = __shfl_xor_sync(FULL, p.x, 1), xl = __shfl_xor_sync(FULL, p.y, 1);
  ed_pair_add(p.x, p.y, x, xl);
  if (!par) partial[(size_t)gl * nblk + blockIdx.x] = TWO ? make_double2(0.5 * p.x, 0.5 * p.y) : p;
}

// out[pair]: the sum rounded to FP64, and what that left
__global__ void __launch_bounds__(128) k_flip_sum(const double2* __restrict__ partial, int nblk,
                                                  double2* __restrict__ out) {
  double h = 0.0, l = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    const double2 v = partial[(size_t)blockIdx.x * nblk + b];
    ed_pair_add(h, l, v.x, v.y);
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const double x = __shfl_down_sync(0xffffffffu, h, s), xl = __shfl_down_sync(0xffffffffu, l, s);
    ed_pair_add(h, l, x, xl);
  }
  __shared__ double2 sh[4];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_double2(h, l);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w) ed_pair_add(h, l, sh[w].x, sh[w].y);
    const double f = h + l;
    out[blockIdx.x] = make_double2(f, l - (f - h));
  }
}

typedef unsigned __int128 u128;

// Signed 128-bit to double: |error| below 2^-52 of the value.
double i128_to_double(u128 z) {
  const bool neg = (__int128)z < 0;
  if (neg) z = ~z + 1;
  const double d = std::fma((double)(uint64_t)(z >> 64), 0x1p64, (double)(uint64_t)z);
  return neg ? -d : d;
}

// The nearest double and what is left of z, as a double (|z| below 2^126).
double i128_split(u128 z, double& rest) {
  const double d = (double)(__int128)z;
  rest = (double)((__int128)z - (__int128)d);
  return d;
}

// T - 2 A, A = the weight of the antiparallel states of (i, j)
u128 zz_sum(const ed_corr& c, int i, int j) {
  const int a = std::max(i, j), b = std::min(i, j);
  const u128 A = c.P[a * (a + 1) / 2 + a] + c.P[b * (b + 1) / 2 + b] - 2 * c.P[a * (a + 1) / 2 + b];
  return c.T - 2 * A;
}

}  // namespace

double ed_corr::zz(int i, int j) const {
  if (i == j) return i128_to_double(T) * inv_scale;
  return i128_to_double(zz_sum(*this, i, j)) * inv_scale;
}

// Both parts are exact integers (Gram form).  Rounded apart and then added, the
// root mean square error at N=20 was 6% above that of an FP64 flip sum; rounded
// once it is 1.62e-17 of the largest value, as with the FP64 sum.
double ed_corr::sisj(int i, int j, int64_t q) const {
  double zl;
  const double f = 0.25 * inv_scale, z = i128_split(zz_sum(*this, i, j), zl) * f;
  const double s = z + F[q], t = s - z;
  const double e = (z - (s - t)) + (F[q] - t);  // z + F = s + e (Knuth's TwoSum)
  return s + (e + (zl * f + Fl[q]));
}

double ed_corr::up(int i) const { return i128_to_double(P[i * (i + 1) / 2 + i]) * inv_scale; }
double ed_corr::down(int i) const { return i128_to_double(T - P[i * (i + 1) / 2 + i]) * inv_scale; }
double ed_corr::sz(int i) const { return 0.5 * (i128_to_double(2 * P[i * (i + 1) / 2 + i] - T) * inv_scale); }

int ed_corr_real(const ed_basis* b, const double2* lam, const double2* psi, bool want_zz, const int32_t* pairs,
                 int64_t np, ed_corr& out) {
  const bool two = lam != psi;
  ed_ctx* ctx = b->ctx;
  const int64_t dim = b->dim;
  const int N = b->nspins, w0 = b->lin_w0, w1 = N - w0;
  // flip sums wanted: distinct sites only
  std::vector<int64_t> flips;
  for (int64_t p = 0; p < np; ++p)
    if (pairs[2 * p] != pairs[2 * p + 1]) flips.push_back(p);
  // up to 16 pairs are one pass of the direct kernel (1.2 ms at N=28, 0.08 ms
  // at N=24); the Gram kernel serves all pairs for 2.8 and 0.2 ms, so it takes
  // every longer list.  Two vectors take direct passes.
  const bool gram = !two && (int64_t)flips.size() > ED_CORR_FEW;
  const bool few = !gram && !flips.empty();
  // passes of the direct kernel per launch; behind the Gram kernel, for the
  // pairs it leaves (GRAM_AGAIN)
  int64_t npass = ((int64_t)flips.size() + ED_CORR_FEW - 1) / ED_CORR_FEW;
  if (gram) npass = std::min<int64_t>(npass, 32);
  if (npass > 65535) return ED_ENOTSUP;  // grid.y
  const int nprep = (int)std::max<int64_t>(1, std::min<int64_t>((dim + 1023) / 1024, (int64_t)ctx->num_sms * 8));
  // all blocks of a pass resident at once
  const int nflip = (int)std::max<int64_t>(1, std::min<int64_t>((dim + 255) / 256, (int64_t)ctx->num_sms * (two ? 3 : 2)));
  // long segments where there is work for every SM (fewer table adds), short
  // ones below, where the chain of loads is what takes time (21 us at N=16
  // with 64)
  const int seg = dim < (int64_t)1 << 20 ? 8 : COLS_SEG;
  const CorrGeom gc = corr_geom(b, b->nup, 256, [seg](int nh) { return (nh + seg - 1) / seg; });
  const CorrGeom gg = corr_geom(b, b->nup - 1, GRAM_STATES, [](int nh) { return nh; });
  const int nstages = gg.prefix[CR_CLASSES];
  const int ncta = std::max(1, std::min(ctx->num_sms, (nstages + GRAM_GROUP - 1) / GRAM_GROUP));
  const int npairs = N * (N + 1) / 2;
  // workspace: header, results, tables, the compact copy
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 255) & ~(size_t)255;
    return o;
  };
  const size_t o_hdr = take(sizeof(CorrHeader));
  const size_t o_W0 = take(want_zz ? sizeof(unsigned long long) * 4 << w0 : 0);
  const size_t o_zero = at;  // cleared up to here
  const size_t o_P = take(sizeof(ulonglong2) * (size_t)(npairs + 1));
  const size_t o_G = take(sizeof(ulonglong2) * 4096);
  const size_t o_f = take(sizeof(double2) * ED_CORR_FEW * (size_t)npass);
  const size_t o_res = at;  // read back: header .. here
  const size_t o_part = take(sizeof(double) * 2 * (size_t)nprep);
  const size_t o_M = take((sizeof(ulonglong2) * (size_t)(w0 + 1)) << w1);
  const size_t o_fm = take(sizeof(FlipMasks) * (size_t)npass);
  const size_t o_fp = take(sizeof(double2) * (size_t)ED_CORR_FEW * (size_t)npass * nflip);
  const size_t o_gp = take(gram ? sizeof(long long) * (size_t)GRAM_ACC * ncta : 0);
  const size_t o_pr = take(sizeof(double) * (size_t)dim);
  const size_t o_pl = take(two ? sizeof(double) * (size_t)dim : 0);
  ed_workspace ws(ctx, at);
  if (!ws.ptr) return ED_ENOMEM;
  char* base = (char*)ws.ptr;
  CorrHeader* hdr = (CorrHeader*)(base + o_hdr);
  double* pr = (double*)(base + o_pr);
  double* pl = (double*)(base + o_pl);
  ED_CUDA(cudaMemsetAsync(base, 0, o_zero, ctx->stream));
  if (two) k_corr_prep<true><<<nprep, 256, 0, ctx->stream>>>(psi, lam, dim, pr, pl, hdr, (double*)(base + o_part));
  else k_corr_prep<false><<<nprep, 256, 0, ctx->stream>>>(psi, psi, dim, pr, pr, hdr, (double*)(base + o_part));
  ED_CHECK_LAUNCH(ctx);
  CorrHeader hh;
  ED_CUDA(cudaMemcpyAsync(&hh, hdr, sizeof(hh), cudaMemcpyDeviceToHost, ctx->stream));
  ED_CUDA(cudaStreamSynchronize(ctx->stream));
  out.real = hh.imag == 0;
  // sum_r |w_r| = B < 2^e: every w_r and every integer sum stays below 2^124 at
  // the scale 2^(124 - e) (the rounding of B moves it by far less than the
  // spare bits).  Below 2^-900 products and scales run out of exponents: the
  // general kernels answer.
  const double B = hh.B;
  if (!out.real || hh.nonfinite || !std::isfinite(B)) return ED_ENOTSUP;
  if ((want_zz || gram) && B < 0x1p-900) return ED_ENOTSUP;
  out.N = N;
  out.W = hh.W;
  int e = 0;
  if (B > 0.0) std::frexp(B, &e);
  const int S = 124 - e;
  out.inv_scale = std::ldexp(1.0, -S);
  if (want_zz) {
    auto kern = two ? k_corr_cols<true> : k_corr_cols<false>;
    kern<<<gc.prefix[CR_CLASSES], 256, 0, ctx->stream>>>(pr, pl, gc, b->d_lin_lows, b->d_lin_highs, b->d_lin_t1, S,
                                                         seg, (unsigned long long*)(base + o_W0));
    ED_CHECK_LAUNCH(ctx);
  }
  // flip sums of flips[list[0 .. count - 1]] to o_f, count <= npass ED_CORR_FEW
  auto direct = [&](const size_t* list, size_t count) -> int {
    const size_t np_ = (count + ED_CORR_FEW - 1) / ED_CORR_FEW;
    std::vector<FlipMasks> fm(np_);
    memset(fm.data(), 0, sizeof(FlipMasks) * fm.size());
    const uint32_t low = (1u << w0) - 1u;
    for (size_t t = 0; t < count; ++t) {
      FlipMasks& pm = fm[t / ED_CORR_FEW];
      const int g = pm.n++;
      const int i = pairs[2 * flips[list[t]]], j = pairs[2 * flips[list[t]] + 1];
      pm.m[g] = (1u << i) | (1u << j);
      pm.bi[g] = 1u << i;
      pm.ml[g] = pm.m[g] & low;
      pm.mh[g] = pm.m[g] >> w0;
    }
    ED_CUDA(cudaMemcpyAsync(base + o_fm, fm.data(), sizeof(FlipMasks) * fm.size(), cudaMemcpyHostToDevice,
                            ctx->stream));
    const size_t smem = sizeof(uint16_t) * ((size_t)1 << w0);
    auto kern = two ? k_expect_flip_r<true> : k_expect_flip_r<false>;
    kern<<<dim3(nflip, (unsigned)np_), 256, smem, ctx->stream>>>(b->d_states, pr, pl, dim, b->d_lin_t0, b->d_lin_t1,
                                                                 w0, (const FlipMasks*)(base + o_fm),
                                                                 (double2*)(base + o_fp), nflip);
    ED_CHECK_LAUNCH(ctx);
    k_flip_sum<<<(unsigned)count, 128, 0, ctx->stream>>>((const double2*)(base + o_fp), nflip, (double2*)(base + o_f));
    ED_CHECK_LAUNCH(ctx);
    return ED_OK;
  };
  std::vector<size_t> list(flips.size());
  for (size_t t = 0; t < list.size(); ++t) list[t] = t;
  if (few) ED_TRY(direct(list.data(), list.size()));
  if (want_zz || gram) {
    const int gr = std::max(1, std::min((1 << w1) / 4, ctx->num_sms * 16));
    auto kern = gram ? k_corr_rows<true, false> : two ? k_corr_rows<false, true> : k_corr_rows<false, false>;
    kern<<<gr, 128, 0, ctx->stream>>>(pr, pl, w0, w1, b->nup, gc, b->d_lin_lows, b->d_lin_t1, S, hh.emax,
                                      (ulonglong2*)(base + o_M));
    ED_CHECK_LAUNCH(ctx);
  }
  if (want_zz) {
    k_corr_moments<<<npairs + 1, 256, 0, ctx->stream>>>((const unsigned long long*)(base + o_W0),
                                                       (const ulonglong2*)(base + o_M), w0, w1, npairs,
                                                       (ulonglong2*)(base + o_P));
    ED_CHECK_LAUNCH(ctx);
  }
  if (gram && nstages > 0) {
    ED_CUDA(cudaFuncSetAttribute(k_corr_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GRAM_SMEM));
    k_corr_gram<<<ncta, GRAM_THREADS, GRAM_SMEM, ctx->stream>>>((const unsigned long long*)pr, gg, nstages, b->d_lin_t0,
                                                               b->d_lin_t1, b->d_lin_lows, b->d_lin_highs,
                                                               (long long*)(base + o_gp), &hdr->err);
    ED_CHECK_LAUNCH(ctx);
    k_corr_gram_sum<<<CR_SITES, 128 * GRAM_PLANE, 0, ctx->stream>>>((const long long*)(base + o_gp), ncta,
                                                       (ulonglong2*)(base + o_G));
    ED_CHECK_LAUNCH(ctx);
  }
  std::vector<char> res(o_res);
  ED_CUDA(cudaMemcpyAsync(res.data(), base, o_res, cudaMemcpyDeviceToHost, ctx->stream));
  ED_CUDA(cudaStreamSynchronize(ctx->stream));
  memcpy(&hh, res.data() + o_hdr, sizeof(hh));
  if (hh.err) return ed_fail(ED_ECUDA, "correlation Gram matrix: completion wait timed out");
  auto get = [&](size_t o) {
    uint64_t w[2];
    memcpy(w, res.data() + o, sizeof(w));
    return ((u128)w[1] << 64) | w[0];
  };
  if (want_zz) {
    out.P.resize(npairs);
    for (int q = 0; q < npairs; ++q) out.P[q] = get(o_P + 16 * (size_t)q);
    out.T = get(o_P + 16 * (size_t)npairs);
    if (!two) out.W = i128_to_double(out.T) * out.inv_scale;  // exact, rounded once
  }
  out.F.assign(np, 0.0);
  out.Fl.assign(np, 0.0);
  list.clear();
  const double least = gram ? std::ldexp(std::sqrt(out.W), hh.emax - 1022 - GRAM_AGAIN) : 0.0;
  for (size_t t = 0; t < flips.size(); ++t) {
    const int i = pairs[2 * flips[t]], j = pairs[2 * flips[t] + 1];
    if (few) {
      double2 f;
      memcpy(&f, res.data() + o_f + sizeof(f) * t, sizeof(f));
      out.F[flips[t]] = f.x;
      out.Fl[flips[t]] = f.y;
      if (!std::isfinite(f.x)) return ED_ENOTSUP;  // a pair makes NaN of an infinity: the general kernels answer
    } else if (nstages > 0) {
      // F 2^(2 (62 - E) - 32), E = emax - 1022
      const size_t ij = i * 32 + j, ji = j * 32 + i;
      const u128 x = get(o_G + 16 * ij) + get(o_G + 16 * (1024 + ij)) + get(o_G + 16 * (1024 + ji)) +
                     get(o_G + 16 * (2048 + ij)) + get(o_G + 16 * (3072 + ij)) + get(o_G + 16 * (3072 + ji));
      const int sh = 2 * (hh.emax - 1022) - 124 + 32;
      double rest;
      out.F[flips[t]] = std::ldexp(i128_split(x, rest), sh);
      out.Fl[flips[t]] = std::ldexp(rest, sh);
      if (std::fabs(out.F[flips[t]]) < least) list.push_back(t);
    }
  }
  if (list.empty()) return ED_OK;
  // small flip sums again in FP64; the digits took the real parts' place
  k_corr_prep<false><<<nprep, 256, 0, ctx->stream>>>(psi, psi, dim, pr, pr, hdr, (double*)(base + o_part));
  ED_CHECK_LAUNCH(ctx);
  const size_t most = (size_t)npass * ED_CORR_FEW;
  for (size_t t0 = 0; t0 < list.size(); t0 += most) {
    const size_t cnt = std::min(most, list.size() - t0);
    ED_TRY(direct(list.data() + t0, cnt));
    std::vector<double2> f(cnt);
    ED_CUDA(cudaMemcpyAsync(f.data(), base + o_f, sizeof(double2) * cnt, cudaMemcpyDeviceToHost, ctx->stream));
    ED_CUDA(cudaStreamSynchronize(ctx->stream));
    for (size_t t = 0; t < cnt; ++t) {
      out.F[flips[list[t0 + t]]] = f[t].x;
      out.Fl[flips[list[t0 + t]]] = f[t].y;
    }
  }
  return ED_OK;
}
