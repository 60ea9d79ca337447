// Expansion steps of the real-storage Krylov-Schur solve.
//
// A step is four kernels and no host round trip: H.v with x^T y (ed_hv_lin.cu,
// ed_hv_jit.cu), the local Lanczos projection with the Gram-Schmidt dots, the
// update with the new norm, and the scaling with the fixed-point copy for the
// next H.v.  Every reduction ends in the kernel that needs it: the last block
// to finish sums the block partials in a fixed order.  The coefficients, the
// refinement test (DGKS), the test for an invariant subspace and the scale
// live in device memory (KrState); where a step needs the host (a refinement
// pass, an invariant subspace, an exponent the high word of max |w| does not
// determine) it sets `stop`, the kernels queued behind it return at once and
// the host takes that step over.  Before, each step waited for the host three
// times and took three reduction kernels: 130 us per step at 13k rows.
#include "ed_internal.h"
#include "ed_device.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>

#define KR_THREADS 256
#define KR_GROUP 16  // columns per dots launch

struct ColPtrsR {
  const double* p[128];
};

struct KrCols {
  const double* p[KR_GROUP];
};

// For short vectors (kr_dependent; DEP) the kernels of a step are launched as
// programmatic dependents: the blocks of one become resident while the one
// before drains.  A solve of the 16-site chain 2.91 -> 2.52 ms.  Each begins with kr_wait,
// before it reads or writes any memory: it returns when the grid before has
// completed and its writes are visible, so the order of the stream is kept.
// Every block runs it, so a grid completes only after the one before it.
__device__ __forceinline__ void kr_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Reads in these kernels go through kr_ld: the kernel before may still write
// when a block becomes resident, so a read-only (.nc) load, which the compiler
// may choose for a const restrict pointer and move above the wait, is not
// allowed.  volatile keeps the order against kr_wait, .cg reads from L2.
template <bool DEP>
__device__ __forceinline__ double kr_ld(const double* p) {
  if (!DEP) return *p;
  double v;
  asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
template <bool DEP>
__device__ __forceinline__ int kr_ld(const int* p) {
  if (!DEP) return *p;
  int v;
  asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
// lets the next grid's blocks become resident (they wait in kr_wait)
__device__ __forceinline__ void kr_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... K, typename... A>
static int kr_launch(ed_ctx* ctx, bool dep, void (*kern)(K...), int nblk, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nblk);
  cfg.blockDim = dim3(KR_THREADS);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dep ? 1 : 0;
  ED_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<K>(args)...));
  ctx->kernels++;
  return ED_OK;
}

static ColPtrsR kr_cols(const double* const* cols, int nv) {
  ColPtrsR c;
  for (int i = 0; i < 128; ++i) c.p[i] = nullptr;
  for (int i = 0; i < nv && i < 128; ++i) c.p[i] = cols[i];
  return c;
}

// Sums of NI <= 16 items per thread over the block: 16 threads per item add
// 16 values each from shared memory, then four shuffle steps.  Every FP64 add
// costs issue slots of GB300's slow FP64 unit, and a shuffle tree over 8 warps
// spends 5 adds of 32 lanes per warp and item (45 warp adds per item against
// 10 here).  Threads with (threadIdx.x & 15) == 0 return their item's sum.
__device__ __forceinline__ double block_sums16(const double (&acc)[KR_GROUP], int ni, double* sh) {
#pragma unroll
  for (int k = 0; k < KR_GROUP; ++k)
    if (k < ni) sh[k * (KR_THREADS + 1) + threadIdx.x] = acc[k];
  __syncthreads();
  const int item = threadIdx.x >> 4, l = threadIdx.x & 15;
  double a = 0.0;
  if (item < ni) {
    double t[16];  // pairwise: half the rounding of one after the other, as many adds
#pragma unroll
    for (int q = 0; q < 16; ++q) t[q] = sh[item * (KR_THREADS + 1) + l + 16 * q];
#pragma unroll
    for (int w = 8; w > 0; w >>= 1)
#pragma unroll
      for (int q = 0; q < w; ++q) t[q] += t[q + w];
    a = t[0];
  }
#pragma unroll
  for (int s = 8; s > 0; s >>= 1) a += __shfl_down_sync(0xffffffffu, a, s, 16);
  return a;
}

// Sum over the block's 256 threads (all threads call it; thread 0 has it): 32
// lanes add 8 values each, then one shuffle tree.
__device__ __forceinline__ double block_sum256(double v, double* sh) {
  __syncthreads();  // sh free
  sh[threadIdx.x] = v;
  __syncthreads();
  double a = 0.0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < KR_THREADS / 32; ++q) a += sh[threadIdx.x + 32 * q];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) a += __shfl_down_sync(0xffffffffu, a, k);
  }
  return a;
}

// Rounding of the dots.  Half as many threads with more registers each would mean
// chains twice as long, so a thread adds its rows in two: with one, and two blocks
// per SM, the root mean square error of 16 dots of 10M rows was 1.32 times that of
// four blocks per SM.  One more FP64 add per column and thread, so only from 32 rows
// on (2.7M rows, 16 columns: 116 -> 123 us), 16 for up to eight columns, which
// memory bounds; four chains cost a solve at N=24 1.3% more.  Below, the sums over
// threads and blocks round more, and those are pairwise and in four chains.  Errors
// of 16 dots in units of 1e-16 / sqrt(n), one chain and sequential sums -> now (four blocks
// per SM): 13k rows 2.14 -> 1.95 (1.97), 185k 2.71 -> 2.22 (2.21), 705k 2.85 -> 2.27
// (2.23), 2.7M 3.11 -> 2.46 (2.49), 10.4M 5.14 -> 3.61 (3.77).  Steps of the first
// chain, of all steps of rows each:
__device__ __forceinline__ int64_t kr_chain(int64_t steps, int rows, int cols) {
  return steps * rows < (cols > 8 ? 32 : 16) ? steps : (steps + 1) / 2;
}

// Blocks per SM of k_kr_dots: registers for the loads of a row in flight.
__host__ __device__ constexpr int kr_dots_per_sm(int ng) { return ng > 8 ? 2 : 3; }

// w <- w - a vj - b vjm1 (LOCAL, written back), then out[i] = V_i^T w for the
// NG columns of cp.  a and b from the device where a_dev / b_dev are given.
// One instance per column count: the loads of a row (of several rows for few
// columns) are then issued together, without a test per column; bound by the
// FP64 unit (NG + 2 FMAs per row) from about 6 columns on, by memory below.
template <int NG, bool LOCAL, bool DEP>
__global__ void __launch_bounds__(KR_THREADS, kr_dots_per_sm(NG)) k_kr_dots(const __grid_constant__ KrCols cp, double* __restrict__ w,
                                                           int64_t n, const double* __restrict__ vj, double a,
                                                           const double* __restrict__ a_dev,
                                                           const double* __restrict__ vjm1, double b,
                                                           const double* __restrict__ b_dev,
                                                           double* __restrict__ partial, double* __restrict__ out,
                                                           unsigned* __restrict__ counter,
                                                           const int* __restrict__ stop) {
  constexpr int U = NG <= 3 ? 4 : NG <= 8 ? 2 : 1;  // rows in flight per thread
  if (DEP) {
    kr_next();
    kr_wait();
  }
  if (stop && kr_ld<DEP>(stop)) return;
  if (LOCAL && a_dev) a = kr_ld<DEP>(a_dev);
  if (LOCAL && b_dev) b = kr_ld<DEP>(b_dev);
  double acc[KR_GROUP];
#pragma unroll
  for (int k = 0; k < KR_GROUP; ++k) acc[k] = 0.0;
  __shared__ double sh[NG * (KR_THREADS + 1)];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t half = r + kr_chain((n + U * stride - 1) / (U * stride), U, NG) * (U * stride);
  bool two = false;  // the first chain's sums are in this thread's places of sh
  for (; r + (U - 1) * stride < n; r += U * stride) {
    if (r == half) {
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        sh[g * (KR_THREADS + 1) + threadIdx.x] = acc[g];
        acc[g] = 0.0;
      }
      two = true;
    }
    double v[U][NG], wv[U], p[U], q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t ru = r + u * stride;
      wv[u] = kr_ld<DEP>(w + ru);
      p[u] = LOCAL ? kr_ld<DEP>(vj + ru) : 0.0;
      q[u] = LOCAL && vjm1 ? kr_ld<DEP>(vjm1 + ru) : 0.0;
#pragma unroll
      for (int g = 0; g < NG; ++g) v[u][g] = kr_ld<DEP>(cp.p[g] + ru);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (LOCAL) {
        wv[u] = fma(-a, p[u], wv[u]);
        if (vjm1) wv[u] = fma(-b, q[u], wv[u]);
        w[r + u * stride] = wv[u];
      }
#pragma unroll
      for (int g = 0; g < NG; ++g) acc[g] = fma(v[u][g], wv[u], acc[g]);
    }
  }
  if (U > 1) {
    for (; r < n; r += stride) {
      double wv = kr_ld<DEP>(w + r);
      if (LOCAL) {
        wv = fma(-a, kr_ld<DEP>(vj + r), wv);
        if (vjm1) wv = fma(-b, kr_ld<DEP>(vjm1 + r), wv);
        w[r] = wv;
      }
#pragma unroll
      for (int g = 0; g < NG; ++g) acc[g] = fma(kr_ld<DEP>(cp.p[g] + r), wv, acc[g]);
    }
  }
  if (two) {
#pragma unroll
    for (int g = 0; g < NG; ++g) acc[g] += sh[g * (KR_THREADS + 1) + threadIdx.x];
  }
  const int item = threadIdx.x >> 4, l = threadIdx.x & 15;
  const double s = block_sums16(acc, NG, sh);
  if (l == 0 && item < NG) partial[(size_t)item * gridDim.x + blockIdx.x] = s;
  if (!ed_last_block(counter)) return;
  double t = 0.0;
  if (item < NG) {
    double c[4] = {0.0, 0.0, 0.0, 0.0};  // four chains of blocks
    for (unsigned q = l; q < gridDim.x; q += 64) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (q + 16 * k < gridDim.x) c[k] += __ldcg(partial + (size_t)item * gridDim.x + q + 16 * k);
    }
    t = (c[0] + c[1]) + (c[2] + c[3]);
  }
#pragma unroll
  for (int k = 8; k > 0; k >>= 1) t += __shfl_down_sync(0xffffffffu, t, k, 16);
  if (l == 0 && item < NG) out[item] = t;
}

// ||w||^2, four rows in flight per thread.
__global__ void __launch_bounds__(KR_THREADS) k_kr_norm2(const double* __restrict__ w, int64_t n,
                                                         double* __restrict__ partial, double* __restrict__ out,
                                                         unsigned* __restrict__ counter) {
  double acc[1] = {0.0};
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += 4 * stride) {
    double x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = r + u * stride < n ? w[r + u * stride] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[0] = fma(x[u], x[u], acc[0]);
  }
  __shared__ double sh[KR_THREADS];
  const double bs = block_sum256(acc[0], sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = bs;
  if (!ed_last_block(counter)) return;
  double t = 0.0;
  for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) t += __ldcg(partial + q);
  t = block_sum256(t, sh);
  if (threadIdx.x == 0) *out = t;
}

// fl(max |w| s) has one biased exponent for every max |w| with this high word,
// or -1 (ed_fx64_emax_scaled).
__device__ __forceinline__ int kr_emax_scaled(double absmax_hi, double s) {
  const double u = __longlong_as_double((long long)((unsigned long long)__double_as_longlong(absmax_hi) | 0xFFFFFFFFull));
  const double ml = absmax_hi * s, mu = u * s;
  if (!isfinite(ml) || !isfinite(mu) || !(s > 0.0)) return -1;
  const int el = (int)(((unsigned long long)__double_as_longlong(ml) >> 52) & 0x7FF);
  const int eu = (int)(((unsigned long long)__double_as_longlong(mu) >> 52) & 0x7FF);
  return el == eu ? el : -1;
}

// w <- w - sum_i V_i c_i with ||w||^2 and the high word of max |w|; the last
// block then closes the step (see the top of the file).  One instance per
// column count up to KR_GROUP: the loads of a row are issued together.  NV = 0:
// any count, two rows per thread, columns unrolled by four.  Bound by the FP64
// unit for large n, by the chain of latencies for small n: against NV = 0 for
// every count, a solve of the 16-site chain (13k rows) 3.00 -> 2.93 ms, of the
// N=28 lattice 476.9 -> 470.9 ms.
template <int NV, bool DEP>
__global__ void __launch_bounds__(KR_THREADS, NV > 8 ? 3 : 4) k_kr_update(const ColPtrsR cp, int nv, double* __restrict__ w, int64_t n,
                                                          double* __restrict__ partial, KrState* __restrict__ st,
                                                          const double* __restrict__ hv, int j,
                                                          int* __restrict__ gmax) {
  if (DEP) {
    kr_next();
    kr_wait();
  }
  if (kr_ld<DEP>(&st->stop)) return;
  __shared__ double sh_h[128];
  for (int i = threadIdx.x; i < nv; i += blockDim.x) sh_h[i] = kr_ld<DEP>(&st->c[i]);
  __syncthreads();
  double acc[1] = {0.0};
  unsigned int amax = 0u;  // high word of max |w|
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if (NV > 0) {
    constexpr int U = NV <= 3 ? 4 : NV <= 8 ? 2 : 1;  // rows in flight per thread
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t half = r + kr_chain((n + U * stride - 1) / (U * stride), U, NV) * (U * stride);
    double before = 0.0;  // the first chain
    for (; r < n; r += U * stride) {
      if (r == half) {
        before = acc[0];
        acc[0] = 0.0;
      }
      double v[U][NV + 1], x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t ru = r + u * stride;
        const bool in = ru < n;
        x[u] = in ? kr_ld<DEP>(w + ru) : 0.0;
#pragma unroll
        for (int i = 0; i < NV; ++i) v[u][i] = in ? kr_ld<DEP>(cp.p[i] + ru) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int i = 0; i < NV; ++i) x[u] = fma(-v[u][i], sh_h[i], x[u]);
        if (r + u * stride < n) {
          w[r + u * stride] = x[u];
          acc[0] = fma(x[u], x[u], acc[0]);
          amax = ed_absmax_hi(amax, x[u]);
        }
      }
    }
    acc[0] += before;
  } else {
    for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r0 < n; r0 += 2 * stride) {
      const int64_t r1 = r0 + stride;
      const bool has1 = r1 < n;
      double w0 = kr_ld<DEP>(w + r0);
      double w1 = has1 ? kr_ld<DEP>(w + r1) : 0.0;
#pragma unroll 4
      for (int i = 0; i < nv; ++i) {
        const double* col = cp.p[i];
        const double c = sh_h[i];
        w0 = fma(-kr_ld<DEP>(col + r0), c, w0);
        if (has1) w1 = fma(-kr_ld<DEP>(col + r1), c, w1);
      }
      w[r0] = w0;
      acc[0] = fma(w0, w0, acc[0]);
      amax = ed_absmax_hi(amax, w0);
      if (has1) {
        w[r1] = w1;
        acc[0] = fma(w1, w1, acc[0]);
        amax = ed_absmax_hi(amax, w1);
      }
    }
  }
  __shared__ double sh[KR_THREADS];
  __shared__ unsigned int shm[8];
  double bs = block_sum256(acc[0], sh);
  amax = __reduce_max_sync(0xffffffffu, amax);
  if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < KR_THREADS / 32; ++q) amax = max(amax, shm[q]);
    partial[blockIdx.x] = bs;
    partial[gridDim.x + blockIdx.x] = ed_absmax_hi_value(amax);
  }
  if (!ed_last_block(&st->counter)) return;
  double t = 0.0;
  amax = 0u;
  for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) {
    t += __ldcg(partial + q);
    amax = ed_absmax_hi(amax, __ldcg(partial + gridDim.x + q));
  }
  const double n2 = block_sum256(t, sh);
  amax = __reduce_max_sync(0xffffffffu, amax);
  if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  // one warp closes the step; FP64 instructions are slow, so as few in a row
  // as possible: the tests compare squares
  amax = __reduce_max_sync(0xffffffffu, threadIdx.x < KR_THREADS / 32 ? shm[threadIdx.x] : 0u);
  double c2 = 0.0;
  for (int i = threadIdx.x; i < nv; i += 32) c2 = fma(sh_h[i], sh_h[i], c2);
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) c2 += __shfl_down_sync(0xffffffffu, c2, k);
  if (threadIdx.x == 0) {
    const double nw = sqrt(n2), mx = ed_absmax_hi_value(amax), y2 = kr_ld<DEP>(hv + 2);
    const double s = 1.0 / nw;
    const int emax = kr_emax_scaled(mx, s);
    st->step = j;
    st->y2 = y2;
    st->wmax = mx;
    st->alpha[j] = kr_ld<DEP>(hv) + sh_h[j];
    st->beta[j] = nw;
    st->s = s;
    st->emax = emax;
    int why = KR_RUN;
    // the squared norm before the update is n2 + sum c_i^2 (Pythagoras against
    // the orthonormal basis): refine below 1/sqrt(2) of it
    if (!(n2 >= 0.5 * (n2 + c2))) why = KR_REFINE;
    else if (n2 <= 1e-26 * y2) why = KR_INVARIANT;
    else if (emax < 0) why = KR_EXPONENT;
    if (why != KR_RUN) {
      st->stop = why;  // the kernels queued behind, H.v among them, return
    } else {
      gmax[0] = emax;
      gmax[1] = 0;
      gmax[2] = 0;
    }
  }
}

// dst = w s and its fixed-point copy for the next H.v (k_scale_quantize_r with
// the scale and exponent from the device).
template <bool DEP>
__global__ void __launch_bounds__(KR_THREADS) k_kr_scale(const double* __restrict__ w, double* __restrict__ dst,
                                                         int64_t n, const KrState* __restrict__ st, int sbits,
                                                         long long* __restrict__ xq) {
  if (DEP) {
    kr_next();
    kr_wait();
  }
  if (kr_ld<DEP>(&st->stop)) return;
  const double s = kr_ld<DEP>(&st->s);
  const int emax = kr_ld<DEP>(&st->emax);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r0 < n; r0 += 2 * stride) {
    const int64_t r1 = r0 + stride;
    const double v0 = kr_ld<DEP>(w + r0) * s, v1 = r1 < n ? kr_ld<DEP>(w + r1) * s : 0.0;
    dst[r0] = v0;
    xq[r0] = ed_fx64_entry(v0, emax, sbits);
    if (r1 < n) {
      dst[r1] = v1;
      xq[r1] = ed_fx64_entry(v1, emax, sbits);
    }
  }
}

// Blocks of a pass over n rows: at most per_sm per SM.
static int kr_blocks(ed_ctx* ctx, int64_t n, int per_sm) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + KR_THREADS - 1) / KR_THREADS, (int64_t)ctx->num_sms * per_sm));
}

// Dependent launches pay where a kernel is hardly longer than the gap before
// it; with long passes the L2 loads they need cost more than the gap.  Per step
// of a 16-column solve on 152 SMs, plain -> dependent: 3432 rows 41.3 -> 35.2
// us, 12870 45.7 -> 39.6, 48620 51.4 -> 47.1, 184756 69.2 -> 67.7, 705432 143.3
// -> 144.1, 2704156 313-316 either way.  The line, 311296 rows there, is eight
// rows per thread of one block per SM.
static bool kr_dependent(const ed_ctx* ctx, int64_t n) { return n <= (int64_t)ctx->num_sms * KR_THREADS * 8; }

// partials, results and the counter in the reduction buffer:
// [items][nblk] | out[items] ; the counter is the context's
static int kr_dots(ed_ctx* ctx, const double* const* cols, int nv, double* w, int64_t n, const double* vj, double a,
                   const double* a_dev, const double* vjm1, double b, const double* b_dev, double* out, const int* stop) {
  const int nblk = kr_blocks(ctx, n, 4);
  const bool dep = kr_dependent(ctx, n);
  ED_TRY(ed_ensure_reduce(ctx, (size_t)KR_GROUP * nblk + 256));
  ED_TRY(ed_ensure_counter(ctx));
  double* partial = ctx->d_red;
  for (int v0 = 0; v0 < nv; v0 += KR_GROUP) {
    KrCols cp;
    for (int i = 0; i < KR_GROUP; ++i) cp.p[i] = v0 + i < nv ? cols[v0 + i] : nullptr;
    const bool local = v0 == 0 && vj;
    if (!local) a_dev = b_dev = vjm1 = nullptr;
    const int nb = kr_blocks(ctx, n, kr_dots_per_sm(std::min(KR_GROUP, nv - v0)));
    int rc = ED_OK;
    auto go = [&](auto kern) {
      rc = kr_launch(ctx, dep, kern, nb, cp, w, n, local ? vj : nullptr, a, a_dev, vjm1, b, b_dev, partial, out + v0,
                     ctx->d_counter, stop);
    };
#define KR_DOTS(NG)                                                                 \
  case NG:                                                                          \
    if (dep) local ? go(k_kr_dots<NG, true, true>) : go(k_kr_dots<NG, false, true>); \
    else local ? go(k_kr_dots<NG, true, false>) : go(k_kr_dots<NG, false, false>);   \
    break;
    switch (std::min(KR_GROUP, nv - v0)) {
      KR_DOTS(1) KR_DOTS(2) KR_DOTS(3) KR_DOTS(4) KR_DOTS(5) KR_DOTS(6) KR_DOTS(7) KR_DOTS(8)
      KR_DOTS(9) KR_DOTS(10) KR_DOTS(11) KR_DOTS(12) KR_DOTS(13) KR_DOTS(14) KR_DOTS(15) KR_DOTS(16)
    }
#undef KR_DOTS
    ED_TRY(rc);
  }
  return ED_OK;
}

int ed_multidot_r(ed_ctx* ctx, const double* const* cols, int nv, double* w, int64_t n, const double* vj, double a,
                  const double* vjm1, double b, double* h_host, double* wnorm2_host) {
  if (nv > 127) return ed_fail(ED_ENOTSUP, "at most 127 basis vectors");
  const int nblk = kr_blocks(ctx, n, 4);
  const size_t part = (size_t)KR_GROUP * nblk;
  ED_TRY(ed_ensure_reduce(ctx, part + 256));
  ED_TRY(ed_ensure_counter(ctx));
  double* out = ctx->d_red + part;
  if (nv > 0) ED_TRY(kr_dots(ctx, cols, nv, w, n, vj, a, nullptr, vjm1, b, nullptr, out, nullptr));
  if (wnorm2_host) {
    k_kr_norm2<<<nblk, KR_THREADS, 0, ctx->stream>>>(w, n, ctx->d_red, out + nv, ctx->d_counter);
    ED_CHECK_LAUNCH(ctx);
  }
  const int items = nv + (wnorm2_host ? 1 : 0);
  if (items == 0) return ED_OK;
  ED_CUDA(cudaMemcpyAsync(ctx->h_red, out, sizeof(double) * items, cudaMemcpyDeviceToHost, ctx->stream));
  ED_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int i = 0; i < nv; ++i) h_host[i] = ctx->h_red[i];
  if (wnorm2_host) *wnorm2_host = ctx->h_red[nv];
  return ED_OK;
}

// Queues step j: H.v of cols[j] (its fixed-point copy is in place or is made
// here), projection, update and scaling into cols[j + 1].  Nothing waits.
int ed_kr_step(ed_ham* h, double* const* cols, int j, bool three_term, double* w, KrState* st) {
  ed_ctx* ctx = h->ctx;
  const int64_t n = h->basis->dim;
  const double* hv = nullptr;
  ED_TRY(ed_launch_hv_dot_dev(h, cols[j], w, &st->stop, &hv));
  ED_TRY(kr_dots(ctx, cols, j + 1, w, n, cols[j], 0.0, hv, three_term ? cols[j - 1] : nullptr, 0.0,
                 three_term ? &st->beta[j - 1] : nullptr, st->c, &st->stop));
  const int nv = j + 1;
  const bool dep = kr_dependent(ctx, n);
  const int nblk = kr_blocks(ctx, n, nv > 8 && nv <= KR_GROUP ? 3 : 4);  // all resident
  int rc = ED_OK;
  auto update = [&](auto kern) {
    rc = kr_launch(ctx, dep, kern, nblk, kr_cols(cols, nv), nv, w, n, ctx->d_red, st, hv, j, h->d_gmax);
  };
#define KR_UPDATE(NV)                                                    \
  case NV:                                                               \
    dep ? update(k_kr_update<NV, true>) : update(k_kr_update<NV, false>); \
    break;
  switch (nv) {
    KR_UPDATE(1) KR_UPDATE(2) KR_UPDATE(3) KR_UPDATE(4) KR_UPDATE(5) KR_UPDATE(6) KR_UPDATE(7) KR_UPDATE(8)
    KR_UPDATE(9) KR_UPDATE(10) KR_UPDATE(11) KR_UPDATE(12) KR_UPDATE(13) KR_UPDATE(14) KR_UPDATE(15) KR_UPDATE(16)
    default:
      dep ? update(k_kr_update<0, true>) : update(k_kr_update<0, false>);
  }
#undef KR_UPDATE
  ED_TRY(rc);
  ED_TRY(kr_launch(ctx, dep, dep ? k_kr_scale<true> : k_kr_scale<false>, kr_blocks(ctx, n, 8), w, cols[j + 1], n, st, ed_fx64_sbits(h), (long long*)h->d_xq));
  h->xq_src = cols[j + 1];
  return ED_OK;
}
