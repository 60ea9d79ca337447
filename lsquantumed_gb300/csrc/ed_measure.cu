// Measurements: correlation expectation values (SzSz / SpSm / SmSp / SiSj,
// src/spinOperators/correlation.cpp:38-299) and DSF coefficients
// c_{i,n} = <v_n | S_i | psi0> (include/phys.tmpl_func.hpp:161-186 with
// Sqz / Sqp from include/spinOperators/spinOPft.tmpl_func.hpp).
//
// The reference builds a sparse operator matrix per (i, j) and runs MatMult +
// VecDot; here each pass over the basis evaluates a group of pairs at once,
// gathering psi at the rank of the flipped state.  The PETSc VecDot
// convention is kept: ExpectVal = sum_s psi_s * conj((O psi)_s).
#include "ed_internal.h"
#include "ed_device.cuh"
#include "ed_halves.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>

#define MEAS_G 8
#define MEAS_GR 16  // pairs per pass when psi is real

struct PairGroup {
  int n;
  int32_t i[MEAS_GR], j[MEAS_GR];
};

// Groups of up to G pairs per pass over the basis.  Ranks of flipped states
// come from the basis's two-table rank (T0 in shared memory, T1 through the
// read-only cache).  REAL: psi has zero imaginary parts (then every result is
// real and only real parts are accumulated; G = 16 pairs share one pass); a
// real psi normally takes ed_corr_real (ed_corr.cu), and this form only when
// its compact copy does not fit or psi is not finite.
template <int G, bool REAL>
__global__ void __launch_bounds__(256) k_expect(const uint32_t* __restrict__ states, const double2* __restrict__ psi,
                                                int64_t dim, const uint16_t* __restrict__ t0,
                                                const uint32_t* __restrict__ t1, int w0, int op, const PairGroup pg,
                                                double* __restrict__ partial, int nblk) {
  extern __shared__ uint16_t t0s[];
  for (int i = threadIdx.x; i < (1 << w0); i += blockDim.x) t0s[i] = t0[i];
  __syncthreads();
  constexpr int NA = REAL ? G : 2 * G;
  double acc[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) acc[k] = 0.0;
  const uint32_t low = (1u << w0) - 1u;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < dim; r += stride) {
    const uint32_t s = states[r];
    const double2 p = psi[r];
    const double w = REAL ? p.x * p.x : fma(p.x, p.x, p.y * p.y);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (g < pg.n) {
        const int i = pg.i[g], j = pg.j[g];
        const uint32_t a = (s >> i) & 1u, b = (s >> j) & 1u;
        double cr = 0.0, ci = 0.0;
        // S^z_i S^z_j part: psi * conj(0.25 * (+-1) * psi)
        if (op == ED_OP_SZSZ || op == ED_OP_SISJ) cr += (a ^ b) ? -0.25 * w : 0.25 * w;
        if (op != ED_OP_SZSZ) {
          const double half = (op == ED_OP_SISJ) ? 0.5 : 1.0;
          if (i == j) {
            // S+S- = n_i (a = 1), S-S+ = 1 - n_i (a = 0)
            const bool on = (op == ED_OP_SPSM) ? (a == 1u) : (op == ED_OP_SMSP) ? (a == 0u) : true;
            if (on) cr += half * w;
          } else {
            const bool on = (op == ED_OP_SPSM) ? (a == 0u && b == 1u) : (op == ED_OP_SMSP) ? (a == 1u && b == 0u) : (a != b);
            if (on) {
              const uint32_t f = s ^ ((1u << i) | (1u << j));
              const uint32_t c = (uint32_t)t0s[f & low] + __ldg(&t1[f >> w0]);
              const double2 q = __ldg(&psi[c]);
              // psi_r * conj(psi_c)
              if (REAL) {
                cr += half * (p.x * q.x);
              } else {
                cr += half * fma(p.x, q.x, p.y * q.y);
                ci += half * fma(p.y, q.x, -p.x * q.y);
              }
            }
          }
        }
        if (REAL) {
          acc[g] += cr;
        } else {
          acc[2 * g] += cr;
          acc[2 * g + 1] += ci;
        }
      }
    }
  }
  __shared__ double sh[NA * 32];
  ed_block_reduce<NA>(acc, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NA; ++k) partial[(size_t)k * nblk + blockIdx.x] = acc[k];
  }
}

__global__ void k_sum_partials(const double* __restrict__ partial, int nblk, int items, double* __restrict__ out) {
  const int item = blockIdx.x;
  if (item >= items) return;
  __shared__ double sh[256];
  double a = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) a += partial[(size_t)item * nblk + b];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[item] = sh[0];
}

template <int G, bool REAL>
static int expect_g(const ed_basis* b, int op, const double2* psi, const int32_t* pairs, int64_t np, double2* out) {
  ed_ctx* ctx = b->ctx;
  const int64_t dim = b->dim;
  const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>((dim + 255) / 256, (int64_t)ctx->num_sms * 4));
  const int items = REAL ? G : 2 * G;
  const int64_t groups = (np + G - 1) / G;
  ED_TRY(ed_ensure_reduce(ctx, (size_t)items * nblk + (size_t)items * groups + 8));
  const size_t smem = sizeof(uint16_t) * ((size_t)1 << b->lin_w0);
  double* out_dev = ctx->d_red + (size_t)items * nblk;  // [group][item], one read-back for all
  for (int64_t p0 = 0; p0 < np; p0 += G) {
    PairGroup pg;
    memset(&pg, 0, sizeof(pg));
    pg.n = (int)std::min<int64_t>(G, np - p0);
    for (int g = 0; g < pg.n; ++g) {
      pg.i[g] = pairs[2 * (p0 + g)];
      pg.j[g] = pairs[2 * (p0 + g) + 1];
    }
    k_expect<G, REAL><<<nblk, 256, smem, ctx->stream>>>(b->d_states, psi, dim, b->d_lin_t0, b->d_lin_t1, b->lin_w0, op,
                                                        pg, ctx->d_red, nblk);
    ED_CHECK_LAUNCH(ctx);
    k_sum_partials<<<items, 256, 0, ctx->stream>>>(ctx->d_red, nblk, items, out_dev + p0 / G * items);
    ED_CHECK_LAUNCH(ctx);
  }
  ED_CUDA(cudaMemcpyAsync(ctx->h_red, out_dev, sizeof(double) * (size_t)(items * groups), cudaMemcpyDeviceToHost,
                          ctx->stream));
  ED_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int64_t p = 0; p < np; ++p) {
    const double* h = ctx->h_red + p / G * items;
    const int g = (int)(p % G);
    out[p] = REAL ? make_double2(h[g], 0.0) : make_double2(h[2 * g], h[2 * g + 1]);
  }
  return ED_OK;
}

int ed_launch_expect_pairs(const ed_basis* b, int op, const double2* psi, const int32_t* pairs, int64_t np,
                           double2* out) {
  // a real psi: S^z moments and flip sums of all pairs at once (ed_corr.cu);
  // for a real psi <S+_i S-_j> = <S-_i S+_j> = F_ij, i != j
  ed_corr c;
  bool diag = false;
  for (int64_t p = 0; p < np; ++p) diag |= pairs[2 * p] == pairs[2 * p + 1];
  const bool zz = op == ED_OP_SZSZ || op == ED_OP_SISJ || diag;
  const int rc = ed_corr_real(b, psi, psi, zz, pairs, op == ED_OP_SZSZ ? 0 : np, c);
  if (rc == ED_OK) {
    for (int64_t p = 0; p < np; ++p) {
      const int i = pairs[2 * p], j = pairs[2 * p + 1];
      double v = 0.0;
      if (op == ED_OP_SZSZ) v = 0.25 * c.zz(i, j);
      if (op == ED_OP_SISJ) v = i == j ? 0.75 * c.zz(i, i) : c.sisj(i, j, p);  // + (S+S- + S-S+) / 2
      if (op == ED_OP_SPSM) v = i == j ? c.up(i) : c.F[p];
      if (op == ED_OP_SMSP) v = i == j ? c.down(i) : c.F[p];
      out[p] = make_double2(v, 0.0);
    }
    return ED_OK;
  }
  if (rc != ED_ENOMEM && rc != ED_ENOTSUP) return rc;
  bool real = c.real;
  if (rc == ED_ENOMEM) ED_TRY(ed_is_real(b->ctx, psi, b->dim, &real));
  if (real) return expect_g<MEAS_GR, true>(b, op, psi, pairs, np, out);
  return expect_g<MEAS_G, false>(b, op, psi, pairs, np, out);
}

// ---------------------------------------------------------------------------
// DSF coefficients.  One launch handles up to MEAS_G sites for one target
// vector v_n.
//   Sqz: c_{i,n} = sum_r conj(v_n[r]) * 0.5 * (b_i(s_r) ? 1 : -1) * psi0[r]
//   Sqp: c_{i,n} = sum_{r: b_i(s_r) = 0} conj(v_n[rank1(s_r | 1<<i)]) * psi0[r]
// ---------------------------------------------------------------------------
template <int K1>
__global__ void __launch_bounds__(256) k_dsf(const uint32_t* __restrict__ states0, const double2* __restrict__ psi0,
                                             int64_t dim0, const RankTables rt1, int op, int i0, int ni,
                                             const double2* __restrict__ v, double* __restrict__ partial, int nblk) {
  extern __shared__ uint32_t stab[];
  if (op == 1) ed_load_tables(stab, rt1);
  double acc[2 * MEAS_G];
#pragma unroll
  for (int k = 0; k < 2 * MEAS_G; ++k) acc[k] = 0.0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < dim0; r += stride) {
    const uint32_t s = states0[r];
    const double2 p = psi0[r];
    if (op == 0) {
      const double2 q = v[r];
      // conj(q) * p
      const double pr = fma(q.x, p.x, q.y * p.y), pi = fma(q.x, p.y, -q.y * p.x);
#pragma unroll
      for (int g = 0; g < MEAS_G; ++g) {
        if (g < ni) {
          const double sg = ((s >> (i0 + g)) & 1u) ? 0.5 : -0.5;
          acc[2 * g] = fma(sg, pr, acc[2 * g]);
          acc[2 * g + 1] = fma(sg, pi, acc[2 * g + 1]);
        }
      }
    } else {
#pragma unroll
      for (int g = 0; g < MEAS_G; ++g) {
        if (g < ni && !((s >> (i0 + g)) & 1u)) {
          const uint32_t c = ed_rank<K1>(s | (1u << (i0 + g)), stab, rt1);
          const double2 q = __ldg(&v[c]);
          acc[2 * g] += fma(q.x, p.x, q.y * p.y);
          acc[2 * g + 1] += fma(q.x, p.y, -q.y * p.x);
        }
      }
    }
  }
  __shared__ double sh[2 * MEAS_G * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < 2 * MEAS_G; ++k) {
    double a = acc[k];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) sh[k * 32 + wid] = a;
  }
  __syncthreads();
  if (wid == 0) {
    for (int k = 0; k < 2 * MEAS_G; ++k) {
      double a = lane < nw ? sh[k * 32 + lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
      if (lane == 0) partial[(size_t)k * nblk + blockIdx.x] = a;
    }
  }
}

template <int K1>
static int dsf_k(const ed_basis* b0, const ed_basis* b1, int op, const double2* psi0, const double2* vecs, int nev,
                 double2* c_host) {
  ed_ctx* ctx = b0->ctx;
  const int64_t dim0 = b0->dim, dim1 = b1->dim;
  const int N = b0->nspins, groups = (N + MEAS_G - 1) / MEAS_G;
  const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>((dim0 + 255) / 256, (int64_t)ctx->num_sms * 2));
  const int items = 2 * MEAS_G;
  const size_t total = (size_t)items * groups * nev;
  ED_TRY(ed_ensure_reduce(ctx, (size_t)items * nblk + total + 8));
  size_t smem = op == 1 ? (size_t)b1->rt.total * sizeof(uint32_t) : 0;
  ED_CUDA(cudaFuncSetAttribute(k_dsf<K1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(56 * 1024)));
  double* out_dev = ctx->d_red + (size_t)items * nblk;  // [n][group][item], one read-back for all
  for (int n = 0; n < nev; ++n) {
    const double2* v = vecs + (size_t)n * dim1;
    for (int q = 0; q < groups; ++q) {
      const int i0 = q * MEAS_G, ni = std::min(MEAS_G, N - i0);
      k_dsf<K1><<<nblk, 256, smem, ctx->stream>>>(b0->d_states, psi0, dim0, b1->rt, op, i0, ni, v, ctx->d_red, nblk);
      ED_CHECK_LAUNCH(ctx);
      k_sum_partials<<<items, 256, 0, ctx->stream>>>(ctx->d_red, nblk, items,
                                                     out_dev + ((size_t)n * groups + q) * items);
      ED_CHECK_LAUNCH(ctx);
    }
  }
  ED_CUDA(cudaMemcpyAsync(ctx->h_red, out_dev, sizeof(double) * total, cudaMemcpyDeviceToHost, ctx->stream));
  ED_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int n = 0; n < nev; ++n)
    for (int i = 0; i < N; ++i) {
      const double* h = ctx->h_red + ((size_t)n * groups + i / MEAS_G) * items + 2 * (i % MEAS_G);
      c_host[(size_t)i * nev + n] = make_double2(h[0], h[1]);
    }
  return ED_OK;
}

// ---------------------------------------------------------------------------
// The same coefficients from the runs of the two-table rank.  k_dsf spends an
// FP64 FMA pair per row and site and reads psi and v once per 8 sites.
// Sqz: sum_r sigma_i(r) q_r, q = conj(v) psi, needs q summed over the low
// halves of each c1 (high sites) and over the high halves of each c0 (low
// sites) only: two FP64 FMAs per row of a real v instead of N pairs.
//  * k_dsfz_high: a warp takes the run of one c1; lane j keeps site w0 + j's
//    signed sum;
//  * k_dsfz_low: a thread owns one low half and loops over a segment of the
//    high halves; the block then forms the signed sums of the low sites.
// Both take DZ_V vectors at a time, so psi is read once per DZ_V.
// Real vectors (eigenvectors of the real H) need only the products of the
// real parts; any nonzero imaginary part raises *imag and the host runs the
// complex form.
// The signed sums cancel, so the large unsigned ones may not round: a thread's
// rows are added in chains of DZ_ROWS, and everything after is exact to 2^-70 of
// the largest term or kept as a pair, up to the last rounding of c.  The root
// mean square (largest) error against quad sums, relative to the largest c, N=20
// and 24, ten real states of a few decades: 0.62-0.65e-16 (1.9-2.5e-16) against
// 1.10-1.41e-16 (3.7-3.9e-16) with k_dsf; ten complex ones 0.82-0.88e-16
// (3.5-3.6e-16) against 1.03-1.18e-16 (4.1-5.2e-16).  With the warps' and blocks'
// sums rounded to FP64 it was 1.43-1.60e-16 (5.9-6.8e-16) and 1.30-1.48e-16
// (7.3-7.5e-16).  N=24, ten real vectors, the call: 3.78 ms with k_dsf, 0.395
// with those roundings, 0.480 so (the two reads of the vectors, 0.95 GB, take 0.14).
// ---------------------------------------------------------------------------
#define DZ_V 5
#define DZ_SEG 32
#define DZ_BITS 54
#define DZ_MORE 20
#define DZ_EMIN (DZ_BITS + DZ_MORE)
#define DZ_ROWS 16  // rows per plain FP64 chain

// 2^(em - 1022 - DZ_BITS), the last place of fixed point against em, for em >=
// DZ_EMIN; and the factor to units of 2^-DZ_MORE of it
__device__ __forceinline__ double dsf_unit(int em) { return __longlong_as_double((long long)(em + 1 - DZ_BITS) << 52); }
__device__ __forceinline__ double dsf_more(int em) {
  return __longlong_as_double((long long)(2046 - (em + 1 - DZ_BITS - DZ_MORE)) << 52);
}

// The warp's sum of pairs, in every lane: as integers (54 + 20 bits against the
// largest), 12 FP64 operations where five steps of ed_pair_add are 40.
__device__ __forceinline__ void dsf_warp(double& h, double& l) {
  const int em = (int)__reduce_max_sync(
      0xffffffffu, (unsigned)(((unsigned long long)__double_as_longlong(h) >> 52) & 0x7FF));
  if (em == 0x7FF || em < DZ_EMIN) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      const double x = __shfl_xor_sync(0xffffffffu, h, s), xl = __shfl_xor_sync(0xffffffffu, l, s);
      ed_pair_add(h, l, x, xl);
    }
    return;
  }
  const double u = dsf_unit(em);
  long long q = ed_fx64_entry(h, em, DZ_BITS);
  long long r = __double2ll_rn((fma(-(double)q, u, h) + l) * dsf_more(em));
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    q += __shfl_xor_sync(0xffffffffu, q, s);
    r += __shfl_xor_sync(0xffffffffu, r, s);
  }
  const double hq = (double)q;
  h = hq * u;
  l = fma((double)r, 1.0 / (1 << DZ_MORE), (double)(q - (long long)hq)) * u;
}

// partial[(((n * gridDim.x) + blk) * 32 + j) * 4]: re, im of site w0 + j, as pairs
template <bool REAL>
__global__ void __launch_bounds__(128, REAL ? 5 : 3) k_dsfz_high(const double2* __restrict__ psi, const double2* __restrict__ vecs,
                                                   int64_t dim, int nev, int w0, int w1, int nup, const CorrGeom g,
                                                   const uint32_t* __restrict__ t1, double* __restrict__ partial,
                                                   int* __restrict__ imag) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n0 = blockIdx.y * DZ_V, nv = min(DZ_V, nev - n0);
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  constexpr int C = REAL ? 1 : 2;  // parts: re, im
  double hh[C][DZ_V], hl[C][DZ_V];  // the warp's signed sums of its runs
#pragma unroll
  for (int v = 0; v < DZ_V; ++v)
#pragma unroll
    for (int c = 0; c < C; ++c) hh[c][v] = hl[c][v] = 0.0;
  bool im = false;
  for (int c1 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c1 < (1 << w1); c1 += nwarps) {
    if (REAL && __any_sync(0xffffffffu, *(volatile int*)imag != 0)) break;  // the host asks for the complex form
    const int k = nup - __popc(c1);
    if (k < 0 || k > w0) continue;
    const int n = g.nlow[k];
    const double2* p = psi + t1[c1];
    const double2* q = vecs + (size_t)n0 * dim + t1[c1];
    double sh_[C][DZ_V], sl_[C][DZ_V];
#pragma unroll
    for (int v = 0; v < DZ_V; ++v)
#pragma unroll
      for (int c = 0; c < C; ++c) sh_[c][v] = sl_[c][v] = 0.0;
    for (int o0 = lane; o0 < n; o0 += 32 * DZ_ROWS) {
      double a[C][DZ_V];
#pragma unroll
      for (int v = 0; v < DZ_V; ++v)
#pragma unroll
        for (int c = 0; c < C; ++c) a[c][v] = 0.0;
      const int o1 = min(n, o0 + 32 * DZ_ROWS);
#pragma unroll 2
      for (int o = o0; o < o1; o += 32) {
        const double2 x = p[o];
        double2 y[DZ_V];
#pragma unroll
        for (int v = 0; v < DZ_V; ++v) y[v] = v < nv ? q[(size_t)v * dim + o] : make_double2(0.0, 0.0);
        if (REAL) im |= x.y != 0.0;
#pragma unroll
        for (int v = 0; v < DZ_V; ++v) {
          if (REAL) {
            im |= y[v].y != 0.0;
            a[0][v] = fma(y[v].x, x.x, a[0][v]);
          } else {  // conj(v) psi
            a[0][v] = fma(y[v].x, x.x, fma(y[v].y, x.y, a[0][v]));
            a[C - 1][v] = fma(y[v].x, x.y, fma(-y[v].y, x.x, a[C - 1][v]));
          }
        }
      }
#pragma unroll
      for (int v = 0; v < DZ_V; ++v)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (o0 == lane) sh_[c][v] = a[c][v];  // the first chain
          else ed_pair_add(sh_[c][v], sl_[c][v], a[c][v], 0.0);
        }
    }
    if (REAL && __any_sync(0xffffffffu, im)) {
      if (lane == 0) atomicOr(imag, 1);
      break;
    }
    const bool up = (c1 >> lane) & 1;
#pragma unroll
    for (int v = 0; v < DZ_V; ++v)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        double h = sh_[c][v], l = sl_[c][v];
        dsf_warp(h, l);
        ed_pair_add(hh[c][v], hl[c][v], up ? h : -h, up ? l : -l);
      }
  }
  __shared__ double2 sh[C][DZ_V][4][32];
#pragma unroll
  for (int v = 0; v < DZ_V; ++v)
#pragma unroll
    for (int c = 0; c < C; ++c) sh[c][v][wid][lane] = make_double2(hh[c][v], hl[c][v]);
  __syncthreads();
  for (int v = wid; v < nv; v += 4) {
    double2* d = (double2*)partial + (((size_t)(n0 + v) * gridDim.x + blockIdx.x) * 32 + lane) * 2;
    for (int c = 0; c < 2; ++c) {
      double2 t = make_double2(0.0, 0.0);
      if (c < C)
        for (int w = 0; w < 4; ++w) ed_pair_add(t.x, t.y, sh[c][v][w][lane].x, sh[c][v][w][lane].y);
      d[c] = t;
    }
  }
}

// partial[(((n * gridDim.x) + item) * 16 + i) * 4]: re, im of low site i, as pairs
template <bool REAL>
__global__ void __launch_bounds__(256) k_dsfz_low(const double2* __restrict__ psi, const double2* __restrict__ vecs,
                                                  int64_t dim, int nev, const CorrGeom g,
                                                  const uint16_t* __restrict__ lows,
                                                  const uint32_t* __restrict__ highs,
                                                  const uint32_t* __restrict__ t1, double* __restrict__ partial,
                                                  const int* __restrict__ imag) {
  if (REAL && *imag) return;  // k_dsfz_high met an imaginary part
  int k = 0;
  while (k < g.w0 && (int)blockIdx.x >= g.prefix[k + 1]) ++k;
  const int item = (int)blockIdx.x - g.prefix[k];
  const int seg = item / g.chunks[k], o = (item - seg * g.chunks[k]) * 256 + (int)threadIdx.x;
  const int h0 = seg * DZ_SEG, nh = min(DZ_SEG, g.nhigh[k] - h0);
  const int n0 = blockIdx.y * DZ_V, nv = min(DZ_V, nev - n0);
  __shared__ uint32_t base[DZ_SEG];
  __shared__ uint16_t c0[256];
  constexpr int C = REAL ? 1 : 2;
  __shared__ double sh[C][DZ_V][256];  // a column's sum, as fixed point
  __shared__ int sr2[C][DZ_V][256];    // and what its rounding left, in 2^-DZ_MORE of its unit
  __shared__ int emax[REAL ? 1 : 2][DZ_V];
  if (threadIdx.x < (REAL ? 1 : 2) * DZ_V) (&emax[0][0])[threadIdx.x] = 0;
  if (threadIdx.x < nh) base[threadIdx.x] = t1[highs[g.high_off[k] + h0 + threadIdx.x]];
  const bool on = o < g.nlow[k];
  c0[threadIdx.x] = on ? lows[g.low_off[k] + o] : (uint16_t)0;
  __syncthreads();
  double ar[DZ_V], ai[DZ_V], rr[DZ_V], ri[DZ_V];  // a column's sum and what its rounding left
#pragma unroll
  for (int v = 0; v < DZ_V; ++v) ar[v] = ai[v] = rr[v] = ri[v] = 0.0;
  if (on) {
    const double2* q = vecs + (size_t)n0 * dim;
    double sr[DZ_V], si[DZ_V], lr[DZ_V], li[DZ_V];  // chains of DZ_ROWS joined as pairs
#pragma unroll
    for (int v = 0; v < DZ_V; ++v) sr[v] = si[v] = lr[v] = li[v] = 0.0;
    auto join = [&](bool first) {
#pragma unroll
      for (int v = 0; v < DZ_V; ++v) {
        if (first) {
          sr[v] = ar[v];
          si[v] = ai[v];
        } else {
          ed_pair_add(sr[v], lr[v], ar[v], 0.0);
          if (!REAL) ed_pair_add(si[v], li[v], ai[v], 0.0);
        }
        ar[v] = ai[v] = 0.0;
      }
    };
#pragma unroll 2
    for (int h = 0; h < nh; ++h) {
      if (h > 0 && h % DZ_ROWS == 0) join(h == DZ_ROWS);
      const size_t r = (size_t)base[h] + o;
      const double2 x = psi[r];
      double2 y[DZ_V];
#pragma unroll
      for (int v = 0; v < DZ_V; ++v) y[v] = v < nv ? q[(size_t)v * dim + r] : make_double2(0.0, 0.0);
#pragma unroll
      for (int v = 0; v < DZ_V; ++v) {
        if (REAL) {
          ar[v] = fma(y[v].x, x.x, ar[v]);
        } else {
          ar[v] = fma(y[v].x, x.x, fma(y[v].y, x.y, ar[v]));
          ai[v] = fma(y[v].x, x.y, fma(-y[v].y, x.x, ai[v]));
        }
      }
    }
    join(nh <= DZ_ROWS);
#pragma unroll
    for (int v = 0; v < DZ_V; ++v) {
      // |rest| <= half the last bit of the sum
      ar[v] = sr[v];
      ed_pair_add(ar[v], rr[v], lr[v], 0.0);
      ai[v] = si[v];
      ed_pair_add(ai[v], ri[v], li[v], 0.0);
    }
  }
  // The signed sums cancel: exact, as 54-bit integers against the block's
  // largest column (256 of them stay below 2^62) and 20 bits more behind them.
  // FP64 adds are the scarcer unit too.  A column that is not finite: in FP64, as
  // it was.
#pragma unroll
  for (int v = 0; v < DZ_V; ++v)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int e = (int)(((unsigned long long)__double_as_longlong(c ? ai[v] : ar[v]) >> 52) & 0x7FF);
      const int m = (int)__reduce_max_sync(0xffffffffu, (unsigned)e);
      if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(&emax[c][v], m);
    }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < DZ_V; ++v)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const double x = c ? ai[v] : ar[v];
      const int em = emax[c][v];
      if (em == 0x7FF) {
        sh[c][v][threadIdx.x] = x;
      } else {
        const long long q = ed_fx64_entry(x, em, DZ_BITS);
        sh[c][v][threadIdx.x] = __longlong_as_double(q);
        // |rest| is at most 2 units; its unit is a normal number for em >= DZ_EMIN
        int r = 0;
        if (em >= DZ_EMIN) {
          const double rest = fma(-(double)q, dsf_unit(em), x) + (c ? ri[v] : rr[v]);
          r = __double2int_rn(rest * dsf_more(em));
        }
        sr2[c][v][threadIdx.x] = r;
      }
    }
  __syncthreads();
  // 16 threads per site: signed sums of the 256 columns
  const int i = threadIdx.x >> 4, l = threadIdx.x & 15;
  for (int v = 0; v < nv; ++v) {
    double2 rm[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
#pragma unroll
    for (int p = 0; p < C; ++p) {
      if (emax[p][v] == 0x7FF) {
        for (int c = l; c < 256; c += 16) rm[p].x += ((c0[c] >> i) & 1) ? sh[p][v][c] : -sh[p][v][c];
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) rm[p].x += __shfl_down_sync(0xffffffffu, rm[p].x, s, 16);
      } else {
        long long q = 0;
        int r = 0;
        for (int c = l; c < 256; c += 16) {
          const long long x = __double_as_longlong(sh[p][v][c]);
          const bool up = (c0[c] >> i) & 1;
          q += up ? x : -x;
          r += up ? sr2[p][v][c] : -sr2[p][v][c];
        }
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) {
          q += __shfl_down_sync(0xffffffffu, q, s, 16);
          r += __shfl_down_sync(0xffffffffu, r, s, 16);
        }
        const double h = (double)q;
        const double rest = (double)(q - (long long)h) + (double)r * (1.0 / (1 << DZ_MORE));
        rm[p] = make_double2(ldexp(h, emax[p][v] - 1022 - DZ_BITS), ldexp(rest, emax[p][v] - 1022 - DZ_BITS));
      }
    }
    if (l == 0) {
      double2* d = (double2*)partial + (((size_t)(n0 + v) * gridDim.x + blockIdx.x) * 16 + i) * 2;
      d[0] = rm[0];
      d[1] = rm[1];
    }
  }
}

// c[n * N + i] = f sum over the blocks of site i's partials (low sites in
// pl, high in ph); grid (sites, vectors)
__global__ void __launch_bounds__(128) k_dsf_sum(const double* __restrict__ pl, int nl, int wl,
                                                 const double* __restrict__ ph, int nh, int w0, double f,
                                                 double2* __restrict__ c) {
  const int i = blockIdx.x, n = blockIdx.y;
  const bool low = i < w0;
  const double2* p = (const double2*)(low ? pl : ph) + ((size_t)n * (low ? nl * wl : nh * 32) + (low ? i : i - w0)) * 2;
  const int cnt = low ? nl : nh, ld = (low ? wl : 32) * 2;
  double h[2] = {0.0, 0.0}, l[2] = {0.0, 0.0};
#pragma unroll 4
  for (int b = threadIdx.x; b < cnt; b += 128) {
    const double2 re = p[(size_t)b * ld], im = p[(size_t)b * ld + 1];
    ed_pair_add(h[0], l[0], re.x, re.y);
    ed_pair_add(h[1], l[1], im.x, im.y);
  }
  __shared__ double sh[4][4];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      const double x = __shfl_down_sync(0xffffffffu, h[k], s), xl = __shfl_down_sync(0xffffffffu, l[k], s);
      ed_pair_add(h[k], l[k], x, xl);
    }
    if ((threadIdx.x & 31) == 0) {
      sh[threadIdx.x >> 5][2 * k] = h[k];
      sh[threadIdx.x >> 5][2 * k + 1] = l[k];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w) {
      ed_pair_add(h[0], l[0], sh[w][0], sh[w][1]);
      ed_pair_add(h[1], l[1], sh[w][2], sh[w][3]);
    }
    c[(size_t)n * gridDim.x + i] = make_double2(f * (h[0] + l[0]), f * (h[1] + l[1]));
  }
}

// *any = 1 if some entry has a nonzero imaginary part (two arrays); the first one
// found ends the search
__global__ void k_any_imag(const double2* __restrict__ a, int64_t na, const double2* __restrict__ b, int64_t nb,
                           int* __restrict__ any) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int k = 0; k < 2; ++k) {
    const double2* v = k ? b : a;
    const int64_t n = k ? nb : na;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 - threadIdx.x < n; i0 += 8 * stride) {
      if (__any_sync(0xffffffffu, *(volatile int*)any != 0)) return;
      bool f = false;
#pragma unroll
      for (int u = 0; u < 8; ++u) f |= i0 + u * stride < n && v[i0 + u * stride].y != 0.0;
      if (__any_sync(0xffffffffu, f)) {
        if ((threadIdx.x & 31) == 0) atomicOr(any, 1);
        return;
      }
    }
  }
}

// Sqp for real vectors: a warp takes the run of one c1 of sector 0; every site
// that is down adds psi v(s + spin i).  A low site's target lies in the run
// of c1 in sector 1 at T0[c0 + site]; a high site's is the same offset of
// the run of c1 + site, so consecutive lanes read consecutive entries.  One
// pass over psi and v for all sites, one FMA per site that is down; grid.y
// is the vector.  partial[(((n * gridDim.x) + blk) * 32 + site) * 4].
__global__ void __launch_bounds__(128) k_dsfp_r(const double2* __restrict__ psi, const double2* __restrict__ vecs,
                                                int64_t dim1, int w0, int w1, int nup, const CorrGeom g,
                                                const uint16_t* __restrict__ lows, const uint16_t* __restrict__ t0,
                                                const uint32_t* __restrict__ t1a, const uint32_t* __restrict__ t1b,
                                                double* __restrict__ partial, const int* __restrict__ imag) {
  if (*imag) return;  // complex vectors: the general kernel answers
  extern __shared__ uint16_t t0s[];
  for (int i = threadIdx.x; i < (1 << w0); i += blockDim.x) t0s[i] = t0[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  const double2* v = vecs + (size_t)blockIdx.y * dim1;
  double acc[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0.0;
  for (int c1 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c1 < (1 << w1); c1 += nwarps) {
    const int k = nup - __popc(c1);
    if (k < 0 || k > w0) continue;
    const int n = g.nlow[k];
    const uint16_t* lw = lows + g.low_off[k];
    const double2* p = psi + t1a[c1];
    const uint32_t run = t1b[c1];                                             // low sites
    const uint32_t hrun = lane < w1 ? t1b[c1 | (1 << lane)] : 0u;  // high site `lane`
    for (int o = lane; o < ((n + 31) & ~31); o += 32) {
      const bool on = o < n;
      const double x = on ? p[o].x : 0.0;
      const uint32_t c0 = on ? lw[o] : 0xFFFFFFFFu;
#pragma unroll
      for (int i = 0; i < CR_MAXW0; ++i)
        if (i < w0 && !((c0 >> i) & 1u)) acc[i] = fma(__ldg(&v[(size_t)run + t0s[c0 | (1u << i)]].x), x, acc[i]);
#pragma unroll
      for (int j = 0; j < 32 - CR_MAXW0; ++j) {
        if (j < w1 && !((c1 >> j) & 1)) {
          const uint32_t b = __shfl_sync(0xffffffffu, hrun, j);
          if (on) acc[CR_MAXW0 + j] = fma(__ldg(&v[(size_t)b + o].x), x, acc[CR_MAXW0 + j]);
        }
      }
    }
  }
  __shared__ double sh[4][32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    double a = acc[i];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) a += __shfl_down_sync(0xffffffffu, a, s);
    if (lane == 0) sh[wid][i] = a;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double2* d = (double2*)partial + (((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 32 + lane) * 2;
    d[0] = make_double2((sh[0][lane] + sh[1][lane]) + (sh[2][lane] + sh[3][lane]), 0.0);
    d[1] = make_double2(0.0, 0.0);
  }
}

// ED_ENOTSUP (nothing returned): some vector is complex and the form asked
// for is the real one, or a result is not finite; ED_ENOMEM: no scratch.
template <bool REAL>
static int dsf_runs(const ed_basis* b0, const ed_basis* b1, int op, const double2* psi, const double2* vecs, int nev,
                    double2* c_host) {
  ed_ctx* ctx = b0->ctx;
  const int N = b0->nspins, w0 = b0->lin_w0, w1 = N - w0;
  const int nb = std::max(1, std::min((1 << w1) / 4, ctx->num_sms * 8));
  const CorrGeom g = corr_geom(b0, b0->nup, 256, [](int nh) { return (nh + DZ_SEG - 1) / DZ_SEG; });
  const int ni = g.prefix[CR_CLASSES];
  const size_t o_c = 256, o_h = o_c + ((sizeof(double2) * (size_t)N * nev + 255) & ~(size_t)255);
  const size_t o_l = o_h + 2 * sizeof(double2) * 32 * (size_t)nb * nev;
  ed_workspace ws(ctx, o_l + 2 * sizeof(double2) * 16 * (size_t)ni * nev);
  if (!ws.ptr) return ED_ENOMEM;
  char* base = (char*)ws.ptr;
  int* imag = (int*)base;
  double2* c = (double2*)(base + o_c);
  double *ph = (double*)(base + o_h), *pl = (double*)(base + o_l);
  ED_CUDA(cudaMemsetAsync(imag, 0, sizeof(int), ctx->stream));
  if (op == 0) {
    const dim3 gh(nb, (nev + DZ_V - 1) / DZ_V), gl(ni, (nev + DZ_V - 1) / DZ_V);
    k_dsfz_high<REAL><<<gh, 128, 0, ctx->stream>>>(psi, vecs, b0->dim, nev, w0, w1, b0->nup, g, b0->d_lin_t1, ph, imag);
    ED_CHECK_LAUNCH(ctx);
    k_dsfz_low<REAL><<<gl, 256, 0, ctx->stream>>>(psi, vecs, b0->dim, nev, g, b0->d_lin_lows, b0->d_lin_highs,
                                                  b0->d_lin_t1, pl, imag);
    ED_CHECK_LAUNCH(ctx);
    k_dsf_sum<<<dim3(N, nev), 128, 0, ctx->stream>>>(pl, ni, 16, ph, nb, w0, 0.5, c);
  } else {
    const int64_t n1 = b1->dim * nev;
    const int gi = (int)std::max<int64_t>(1, std::min<int64_t>((n1 + 1023) / 1024, (int64_t)ctx->num_sms * 8));
    k_any_imag<<<gi, 256, 0, ctx->stream>>>(psi, b0->dim, vecs, n1, imag);
    ED_CHECK_LAUNCH(ctx);
    const size_t smem = sizeof(uint16_t) * ((size_t)1 << w0);
    k_dsfp_r<<<dim3(nb, nev), 128, smem, ctx->stream>>>(psi, vecs, b1->dim, w0, w1, b0->nup, g, b0->d_lin_lows,
                                                        b0->d_lin_t0, b0->d_lin_t1, b1->d_lin_t1, ph, imag);
    ED_CHECK_LAUNCH(ctx);
    // all sites in ph, low ones at 0 .., high ones at CR_MAXW0 ..
    k_dsf_sum<<<dim3(N, nev), 128, 0, ctx->stream>>>(ph, nb, 32, ph + 4 * CR_MAXW0, nb, w0, 1.0, c);
  }
  ED_CHECK_LAUNCH(ctx);
  std::vector<char> res(o_h);
  ED_CUDA(cudaMemcpyAsync(res.data(), base, o_h, cudaMemcpyDeviceToHost, ctx->stream));
  ED_CUDA(cudaStreamSynchronize(ctx->stream));
  int h_imag = 0;
  memcpy(&h_imag, res.data(), sizeof(int));
  if (REAL && h_imag) return ED_ENOTSUP;
  const double2* h = (const double2*)(res.data() + o_c);
  // compensated sums make NaN of an infinity: the general kernel answers
  for (int64_t q = 0; q < (int64_t)N * nev; ++q)
    if (!std::isfinite(h[q].x) || !std::isfinite(h[q].y)) return ED_ENOTSUP;
  for (int n = 0; n < nev; ++n)
    for (int i = 0; i < N; ++i) c_host[(size_t)i * nev + n] = h[(size_t)n * N + i];
  return ED_OK;
}

int ed_launch_dsf(const ed_basis* b0, const ed_basis* b1, int op, const double2* psi0, const double2* vecs, int nev,
                  double2* c_host) {
  // the real form serves the solver's eigenvectors; a complex vector or a
  // non-finite entry takes the complex arithmetic
  const bool fits = nev <= 65535;  // grid.y
  int rc = fits ? dsf_runs<true>(b0, b1, op, psi0, vecs, nev, c_host) : ED_ENOTSUP;
  if (rc == ED_ENOTSUP && op == 0 && fits) rc = dsf_runs<false>(b0, b1, op, psi0, vecs, nev, c_host);
  if (rc != ED_ENOTSUP && rc != ED_ENOMEM) return rc;
  switch (b1->rt.K) {
    case 1: return dsf_k<1>(b0, b1, op, psi0, vecs, nev, c_host);
    case 2: return dsf_k<2>(b0, b1, op, psi0, vecs, nev, c_host);
    case 3: return dsf_k<3>(b0, b1, op, psi0, vecs, nev, c_host);
    default: return dsf_k<4>(b0, b1, op, psi0, vecs, nev, c_host);
  }
}
