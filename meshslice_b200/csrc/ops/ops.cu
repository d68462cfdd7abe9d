// Memory-bound kernels of the GPT block: LayerNorm (+ residual) over column-sharded features,
// GeLU, AdamW, vocab-parallel cross-entropy, embedding, gradient norm.  All of them stream
// 16-byte vectors (8 bf16) and keep statistics in fp32.
#include "ops.h"

#include <cuda_bf16.h>
#include <string.h>

#include <type_traits>

#include "../common/f32x2.cuh"
#include "../common/gelu.cuh"
#include "../common/pdl.cuh"

namespace msb {

namespace {

constexpr int kLnThreads = 256;
constexpr int kLnBwdThreads = 512;
constexpr int kLnGroupedMaxCols = 2048;   // rows up to this width run several per CTA in ln_bwd_kernel

// ---- cross-GPU row exchange (see RowExchange in ops.h) ----
__device__ __forceinline__ void ex_red_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ex_ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t ex_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Thread 0 of the CTA publishes "this CTA's rows are written" on every peer.
__device__ __forceinline__ void ex_signal(const RowExchange& ex) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    for (int p = 0; p < ex.n; ++p)
      if (p != ex.me) ex_red_release_sys(ex.counter[p], 1u);
  }
}
// All threads return true once every CTA of every peer has published; false after the deadline
// (the status word then says which kernel gave up: code 20 + kind).
__device__ __forceinline__ bool ex_wait(const RowExchange& ex, uint32_t kind) {
  int ok = 1;
  if (threadIdx.x == 0) {
    const uint64_t t0 = ex_timer_ns();
    uint32_t it = 0;
    while ((int32_t)(ex_ld_acquire_sys(ex.my_counter) - ex.target) < 0) {
      if ((++it & 0xf) == 0) {
        if (ex_timer_ns() - t0 > ex.timeout_ns) {
          ok = 0;
          if (atomicCAS(ex.status, 0u, 20u + kind) == 0u) {
            ex.status[1] = blockIdx.x;
            ex.status[2] = ex_ld_acquire_sys(ex.my_counter);
            ex.status[3] = ex.target;
          }
          break;
        }
        __nanosleep(128);
      }
    }
  }
  return __syncthreads_and(ok) != 0;
}
// Writes this GPU's W-float contribution of one row into its slot on every GPU of the group.
template <int W>
__device__ __forceinline__ void ex_put(const RowExchange& ex, int row, const float (&v)[W]) {
  for (int p = 0; p < ex.n; ++p) {
    float* d = ex.dst[p] + (int64_t)row * W;
#pragma unroll
    for (int i = 0; i < W; ++i) d[i] = v[i];
  }
}
// Source q's contribution of one row (L1 bypassed: peers wrote it).
__device__ __forceinline__ float ex_get(const RowExchange& ex, int q, int row, int width, int i) {
  return __ldcg(ex.slots + q * ex.stride + (int64_t)row * width + i);
}

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  f[0] = bf_lo(u.x); f[1] = bf_hi(u.x); f[2] = bf_lo(u.y); f[3] = bf_hi(u.y);
  f[4] = bf_lo(u.z); f[5] = bf_hi(u.z); f[6] = bf_lo(u.w); f[7] = bf_hi(u.w);
}
// Word i of a vector; its two bf16 as packed fp32 lanes; four such pairs as floats.
__device__ __forceinline__ uint32_t word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }
__device__ __forceinline__ uint64_t unpack2(uint32_t u) { return f32x2(bf_lo(u), bf_hi(u)); }
__device__ __forceinline__ void split4(const uint64_t (&v)[4], float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) split(v[i], f[2 * i], f[2 * i + 1]);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack2(f[0], f[1]); u.y = pack2(f[2], f[3]); u.z = pack2(f[4], f[5]); u.w = pack2(f[6], f[7]);
  return u;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Sum of two values over the CTA; every thread gets the result.  `red` holds 2 * 32 floats.
__device__ __forceinline__ void block_sum2(float& a, float& b, float* red) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) { red[w] = a; red[32 + w] = b; }
  __syncthreads();
  a = l < nw ? red[l] : 0.f;
  b = l < nw ? red[32 + l] : 0.f;
  a = warp_sum(a);
  b = warp_sum(b);
}
// The same for a loop over rows: `red` holds two such buffers that alternate, so that one barrier per row is enough (a
// thread that writes buffer p again has passed the barrier of the other one, after every read of p).
__device__ __forceinline__ void block_sum2_alt(float& a, float& b, float* red, int& parity) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  float* buf = red + parity * 64;
  parity ^= 1;
  if (l == 0) { buf[w] = a; buf[32 + w] = b; }
  __syncthreads();
  a = l < nw ? buf[l] : 0.f;
  b = l < nw ? buf[32 + l] : 0.f;
  a = warp_sum(a);
  b = warp_sum(b);
}
__device__ __forceinline__ float block_max(float a, float* red) {
  a = warp_max(a);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = a;
  __syncthreads();
  a = l < nw ? red[l] : -INFINITY;
  return warp_max(a);
}

// ------------------------------------------------------------------------------------------
// Row ring of the LayerNorm kernels: a thread copies the 16-byte vectors that it will read itself, two rows (one for the
// widest backward rows) ahead, into shared memory (cp.async), so rows travel while earlier ones are reduced and written, at
// no registers and without a barrier.  Layout [stage][input][vector of the thread][thread].
// ------------------------------------------------------------------------------------------
constexpr int ln_stages(bool backward, int maxv) { return backward && maxv > 3 ? 2 : 3; }
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
               ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------
// LayerNorm forward in two passes (column-sharded rows: mode 1 statistics, mode 2 the rest; a row on one device is
// ln_fwd_row_kernel's, below).  One CTA per row (grid-stride), row cached in registers.  Bound by HBM: it reads x (and res) and
// writes h (with res), or reads h and writes y.  32768 x 2048, statistics with residual: 92 us with loads of one row at a time, 64
// with the row ring (6.3 TB/s).  RING = false loads the row when it is due: ln_fwd_direct says where that is faster.
// (No minimum of blocks there: with one stated, of any number, the compiler takes 80 registers or spills instead of 40.)
// ------------------------------------------------------------------------------------------
template <int MAXV, bool RING>
__global__ void __launch_bounds__(kLnThreads, !RING ? 0 : MAXV == 1 ? 5 : MAXV == 2 ? 4 : 1)
ln_fwd_kernel(int mode, const uint4* __restrict__ x, const uint4* __restrict__ res,
              uint4* __restrict__ h_out, uint4* __restrict__ y, const uint4* __restrict__ gamma,
              const uint4* __restrict__ beta, float* __restrict__ stats,
              float* __restrict__ mean_rstd, int rows, int cols, int total_cols, float eps,
              const __grid_constant__ RowExchange ex) {
  extern __shared__ uint4 ring[];
  constexpr int S = ln_stages(false, MAXV);
  __shared__ float red[128];
  int parity = 0;
  const int nvec = cols >> 3, T = blockDim.x;
  const bool add = mode != 2 && res != nullptr;
  const int inputs = add ? 2 : 1;
  auto slot = [&](int stage, int input, int k) {
    return ring + ((stage * inputs + input) * MAXV + k) * T + threadIdx.x;
  };
  auto prefetch = [&](uint32_t row, int stage) {
    if (row < (uint32_t)rows) {
      const int64_t base = (int64_t)row * nvec;
#pragma unroll
      for (int k = 0; k < MAXV; ++k) {
        const int v = threadIdx.x + k * T;
        if (v < nvec) {
          cp_async16(slot(stage, 0, k), x + base + v);
          if (add) cp_async16(slot(stage, 1, k), res + base + v);
        }
      }
    }
    cp_async_commit();
  };
  // With an exchange (ex.n > 0) mode 1 writes the partial statistics of its rows to every GPU of
  // the mesh row and counts one arrival per CTA on every peer; mode 2 first waits (bounded) for
  // the arrivals of all peers' CTAs and then sums the sources' statistics in fixed order.
  const bool exchange = ex.n > 0;
  if (exchange && mode == 2 && !ex_wait(ex, 0u)) return;   // nothing of this CTA is under way yet
  if (RING) {
#pragma unroll
    for (int i = 0; i < S - 1; ++i) prefetch(blockIdx.x + i * gridDim.x, i);
  }
  int stage = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    float vals[MAXV][8];
    float s = 0.f, ss = 0.f;
    const int64_t base = (int64_t)row * nvec;
    if (RING) {
      prefetch((uint32_t)row + (S - 1) * gridDim.x, stage == 0 ? S - 1 : stage - 1);   // where the previous row was
      cp_async_wait<S - 1>();
    }
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int v = threadIdx.x + k * T;
      if (v < nvec) {
        unpack8(RING ? *slot(stage, 0, k) : x[base + v], vals[k]);
        if (add) {
          float r[8];
          unpack8(RING ? *slot(stage, 1, k) : res[base + v], r);
#pragma unroll
          for (int i = 0; i < 8; ++i) vals[k][i] += r[i];
        }
        if (mode != 2 && h_out != nullptr) {
          const uint4 hp = pack8(vals[k]);
          h_out[base + v] = hp;
          unpack8(hp, vals[k]);  // statistics of the rounded values the backward pass sees
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) { s += vals[k][i]; ss += vals[k][i] * vals[k][i]; }
      }
    }
    stage = stage + 1 == S ? 0 : stage + 1;
    if (mode == 1) {
      block_sum2_alt(s, ss, red, parity);
      if (threadIdx.x == 0) {
        if (exchange) {
          const float v2[2] = {s, ss};
          ex_put<2>(ex, row, v2);
        } else {
          stats[2 * row] = s;
          stats[2 * row + 1] = ss;
        }
      }
      continue;
    }
    if (exchange) {
      s = 0.f;
      ss = 0.f;
      for (int q = 0; q < ex.n; ++q) { s += ex_get(ex, q, row, 2, 0); ss += ex_get(ex, q, row, 2, 1); }
    } else {
      s = stats[2 * row];
      ss = stats[2 * row + 1];
    }
    const float mean = s / (float)total_cols, rstd = rsqrtf(fmaxf(ss / (float)total_cols - mean * mean, 0.f) + eps);
    if (threadIdx.x == 0 && mean_rstd != nullptr) {
      mean_rstd[2 * row] = mean;
      mean_rstd[2 * row + 1] = rstd;
    }
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int v = threadIdx.x + k * T;
      if (v < nvec) {
        float g[8], b[8], o[8];
        if (gamma != nullptr) unpack8(gamma[v], g);
        if (beta != nullptr) unpack8(beta[v], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float t = (vals[k][i] - mean) * rstd;
          if (gamma != nullptr) t *= g[i];
          if (beta != nullptr) t += b[i];
          o[i] = t;
        }
        y[base + v] = pack8(o);
      }
    }
  }
  if (exchange && mode == 1) ex_signal(ex);
}

// ------------------------------------------------------------------------------------------
// LayerNorm backward
// ------------------------------------------------------------------------------------------
// Sum of two values over the `gw` consecutive warps that share a row; every thread of the group gets the result.
// Alternating buffers as in block_sum2_alt.
__device__ __forceinline__ void group_sum2(float& a, float& b, float* red, int& parity, int gw) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  float* buf = red + parity * 64;
  parity ^= 1;
  if (l == 0) { buf[w] = a; buf[32 + w] = b; }
  __syncthreads();
  const int w0 = w / gw * gw;
  a = 0.f;
  b = 0.f;
  for (int i = 0; i < gw; ++i) { a += buf[w0 + i]; b += buf[32 + w0 + i]; }
}
// dst[0..4) += v: one 16-byte atomic where the address allows it.  Every CTA of the backward kernel ends with its sums
// of dgamma and dbeta, to the same addresses: one by one they took 45 us for 4096 columns, of 102 for 8192 rows.
__device__ __forceinline__ void add4(float* dst, float4 v) {
  if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
    atomicAdd(reinterpret_cast<float4*>(dst), v);
  } else {
    atomicAdd(dst, v.x);
    atomicAdd(dst + 1, v.y);
    atomicAdd(dst + 2, v.z);
    atomicAdd(dst + 3, v.w);
  }
}
__device__ __forceinline__ void add8(float* dst, const float (&v)[8]) {
  add4(dst, make_float4(v[0], v[1], v[2], v[3]));
  add4(dst + 4, make_float4(v[4], v[5], v[6], v[7]));
}

// A CTA of up to kLnBwdThreads threads walks the rows grid-stride.  A 4096-wide row is two 16-byte vectors per
// thread: the per-thread dgamma / dbeta accumulators (16 registers per vector) are what limits occupancy, so the rows
// ahead wait in the shared-memory ring and both passes over a row read it there; gamma is loaded once per CTA.  Bound by
// HBM (dy, h, dres read, dx written); 32768 x 4096 with dres: 254 us with loads of one row at a time, 192 us with the ring,
// 181 us with packed arithmetic and the normalised row kept between the two passes (65 % of the issue slots were taken; copy
// bandwidth would give 161); 8192 x 12288: 290, 146 and 136.
// GROUPED (rows of at most 256 vectors, e.g. column shards): the CTA works on blockDim.x / tpr rows at a time,
// `tpr` threads (whole warps) per row, and adds the row groups' dgamma / dbeta in shared memory before its one
// atomic per column, so that narrow rows neither idle most of a CTA nor multiply the atomics.
template <int MAXV, bool GROUPED>
__global__ void __launch_bounds__(kLnBwdThreads, MAXV == 1 ? 2 : 1)
ln_bwd_kernel(int mode, const uint4* dy, const uint4* h,
              const uint4* gamma, const float* mean_rstd,
              const uint4* dres, uint4* dx, float* stats,
              float* dgamma, float* dbeta, int rows, int cols,
              int total_cols, int tpr_arg, const __grid_constant__ RowExchange ex) {
  if (ex.n == 0) grid_trigger();
  grid_wait();
  static_assert(!GROUPED || MAXV == 1, "grouped rows are one vector per thread");
  constexpr bool kKeep = MAXV == 2;      // what both passes over a row need stays in registers where there is room for it
  extern __shared__ uint4 ring[];
  constexpr int S = ln_stages(true, MAXV);
  __shared__ float red[128];
  int parity = 0;
  __shared__ __align__(16) float comb[GROUPED ? 2 * kLnGroupedMaxCols : 1];
  const int nvec = cols >> 3;
  const int tpr = GROUPED ? tpr_arg : (int)blockDim.x;            // threads per row
  const int sub = GROUPED ? (int)threadIdx.x / tpr : 0;           // which of the CTA's rows
  const int tx = GROUPED ? (int)threadIdx.x - sub * tpr : (int)threadIdx.x;
  const int rows_per_cta = GROUPED ? (int)blockDim.x / tpr : 1;
  uint64_t accg[MAXV][4], accb[MAXV][4];
  uint4 pg[MAXV];
#pragma unroll
  for (int k = 0; k < MAXV; ++k) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { accg[k][i] = 0; accb[k][i] = 0; }
    const int v = tx + k * tpr;
    pg[k] = (gamma != nullptr && v < nvec) ? gamma[v] : make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
  }
  // exchange of the partial sums with the GPUs of the mesh row: see ln_fwd_kernel
  const bool exchange = ex.n > 0;
  if (exchange && mode == 2 && !ex_wait(ex, 1u)) return;   // nothing of this CTA is under way yet
  const bool want_param_grads = mode != 2 && dgamma != nullptr;
  const bool want_dres = mode != 1 && dres != nullptr;

  const int T = blockDim.x, inputs = want_dres ? 3 : 2;
  auto slot = [&](int stage, int input, int k) {
    return ring + ((stage * inputs + input) * MAXV + k) * T + threadIdx.x;
  };
  auto prefetch = [&](uint32_t row, int stage) {
    if (row < (uint32_t)rows) {
      const int64_t base = (int64_t)row * nvec;
#pragma unroll
      for (int k = 0; k < MAXV; ++k) {
        const int v = tx + k * tpr;
        if (v < nvec) {
          cp_async16(slot(stage, 0, k), dy + base + v);
          cp_async16(slot(stage, 1, k), h + base + v);
          if (want_dres) cp_async16(slot(stage, 2, k), dres + base + v);
        }
      }
    }
    cp_async_commit();
  };
  const uint32_t n_rows = rows, step = gridDim.x * rows_per_cta, first = blockIdx.x * rows_per_cta + sub;
#pragma unroll
  for (int i = 0; i < S - 1; ++i) prefetch(first + i * step, i);
  int stage = 0;
  float2 stat_next = make_float2(0.f, 0.f);   // (mean, rstd) of the next row
  if (first < n_rows) stat_next = make_float2(mean_rstd[2 * (int64_t)first], mean_rstd[2 * (int64_t)first + 1]);

  for (uint32_t r0 = blockIdx.x * rows_per_cta; r0 < n_rows; r0 += step) {
    const uint32_t row = r0 + sub;
    const bool live = row < n_rows;        // the last rows of a grouped CTA may be missing; barriers stay uniform
    const int64_t base = (int64_t)row * nvec;
    prefetch(row + (S - 1) * step, stage == 0 ? S - 1 : stage - 1);
    const float mean = stat_next.x, rstd = stat_next.y;
    if (row + step < n_rows)
      stat_next = make_float2(mean_rstd[2 * (int64_t)(row + step)], mean_rstd[2 * (int64_t)(row + step) + 1]);
    cp_async_wait<S - 1>();
    const uint64_t neg_mean = f32x2(-mean, -mean), rstd2 = f32x2(rstd, rstd);
    uint64_t sum1 = 0, sum2 = 0;
    uint64_t xs[kKeep ? MAXV : 1][4], gs[kKeep ? MAXV : 1][4];   // normalised row and dy * gamma
    const auto both = [&](int k, int i, const uint4& du, const uint4& hu, uint64_t& d, uint64_t& xh, uint64_t& g) {
      d = unpack2(word(du, i));
      xh = mul2(add2(unpack2(word(hu, i)), neg_mean), rstd2);
      g = mul2(d, unpack2(word(pg[k], i)));
    };
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int v = tx + k * tpr;
      if (live && v < nvec) {
        const uint4 du = *slot(stage, 0, k), hu = *slot(stage, 1, k);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint64_t d, xh, g;
          both(k, i, du, hu, d, xh, g);
          sum1 = add2(sum1, g);
          sum2 = fma2(g, xh, sum2);
          if (want_param_grads) { accg[k][i] = fma2(d, xh, accg[k][i]); accb[k][i] = add2(accb[k][i], d); }
          if (kKeep) { xs[k][i] = xh; gs[k][i] = g; }
        }
      }
    }
    float s1, s2, hi;
    split(sum1, s1, hi);
    s1 += hi;
    split(sum2, s2, hi);
    s2 += hi;
    if (mode == 2) {
      if (live) {
        if (exchange) {
          s1 = 0.f;
          s2 = 0.f;
          for (int q = 0; q < ex.n; ++q) { s1 += ex_get(ex, q, row, 2, 0); s2 += ex_get(ex, q, row, 2, 1); }
        } else {
          s1 = stats[2 * (int64_t)row];
          s2 = stats[2 * (int64_t)row + 1];
        }
      }
    } else {
      if (GROUPED) group_sum2(s1, s2, red, parity, tpr >> 5);
      else block_sum2_alt(s1, s2, red, parity);
      if (mode == 1) {
        if (tx == 0 && live) {
          if (exchange) {
            const float v2[2] = {s1, s2};
            ex_put<2>(ex, row, v2);
          } else {
            stats[2 * (int64_t)row] = s1;
            stats[2 * (int64_t)row + 1] = s2;
          }
        }
        stage = stage + 1 == S ? 0 : stage + 1;
        continue;
      }
    }
    const float m1 = s1 / (float)total_cols, m2 = s2 / (float)total_cols;
    const uint64_t neg_m1 = f32x2(-m1, -m1), neg_m2 = f32x2(-m2, -m2);
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int v = tx + k * tpr;
      if (live && v < nvec) {
        uint4 du = make_uint4(0u, 0u, 0u, 0u), hu = du, ru = du, o;
        if (!kKeep) {
          du = *slot(stage, 0, k);
          hu = *slot(stage, 1, k);
        }
        if (want_dres) ru = *slot(stage, 2, k);
        uint32_t* ow = &o.x;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint64_t d, xh, g;
          if (kKeep) { xh = xs[k][i]; g = gs[k][i]; }
          else both(k, i, du, hu, d, xh, g);
          const uint64_t t = fma2(xh, neg_m2, add2(g, neg_m1));
          float lo, hi;
          split(want_dres ? fma2(t, rstd2, unpack2(word(ru, i))) : mul2(t, rstd2), lo, hi);
          ow[i] = pack2(lo, hi);
        }
        __stcs(dx + base + v, o);
      }
    }
    stage = stage + 1 == S ? 0 : stage + 1;
  }
  if (exchange && mode == 1) ex_signal(ex);
  if (want_param_grads) {
    if (GROUPED) {
      for (int i = threadIdx.x; i < 2 * cols; i += blockDim.x) comb[i] = 0.f;
      __syncthreads();
      if (tx < nvec) {
        float fg[8], fb[8];
        split4(accg[0], fg);
        split4(accb[0], fb);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          atomicAdd(comb + tx * 8 + i, fg[i]);
          atomicAdd(comb + cols + tx * 8 + i, fb[i]);
        }
      }
      __syncthreads();
      const float4* c4 = reinterpret_cast<const float4*>(comb);
      for (int q = threadIdx.x; q < 2 * nvec; q += blockDim.x) {
        add4(dgamma + q * 4, c4[q]);
        if (dbeta != nullptr) add4(dbeta + q * 4, c4[2 * nvec + q]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < MAXV; ++k) {
        const int v = tx + k * tpr;
        if (v < nvec) {
          float f[8];
          split4(accg[k], f);
          add8(dgamma + v * 8, f);
          split4(accb[k], f);
          if (dbeta != nullptr) add8(dbeta + v * 8, f);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// LayerNorm of whole rows: W warps per row
// ------------------------------------------------------------------------------------------
// Bound by HBM or, while a call's tensors stay in L2, by latency.  A row is read once, into registers, by one warp (no barrier
// at all, four rows per CTA), four or eight warps (one barrier); every CTA has one set of rows, so what hides the latency is the
// number of CTAs, and no row waits for another one.  ln_fwd_row_shape / ln_bwd_row_shape choose W.  The kernels above walk
// their rows in persistent CTAs with a barrier per row; the same sizes there / here, us: forward 4099 x 1544 9.0 / 5.7, with
// residual 11.2 / 9.4, 32768 x 4096 119 / 81 (6.6 TB/s), with residual 172 / 158 (6.8 TB/s), 8192 x 12288 with residual
// 196 / 122, 512 x 512 2.5 / 2.1; backward without parameter gradients 4099 x 1544 15.0 / 6.8, with dres 16.4 / 8.2, 32768 x
// 2048 111 / 61 (6.6 TB/s), with dres 120 / 88.
constexpr int ln_row_warps(int w) { return w < 4 ? 4 : w; }     // warps of a CTA; rows of a CTA: ln_row_warps(w) / w

// Sum of two values over the W warps that share a row; every thread gets the result.  `red` is used once.
template <int W>
__device__ __forceinline__ void row_sum2(float& a, float& b, float2* red) {
  static_assert(W == 1 || W == ln_row_warps(W), "the barrier is the CTA's");
  a = warp_sum(a);
  b = warp_sum(b);
  if (W == 1) return;
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) red[w] = make_float2(a, b);
  __syncthreads();
  a = 0.f;
  b = 0.f;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const float2 v = red[i];
    a += v.x;
    b += v.y;
  }
}

template <int V, int W, bool RES>
__global__ void __launch_bounds__(32 * ln_row_warps(W))
ln_fwd_row_kernel(const uint4* x, const uint4* res, uint4* h_out, uint4* y,
                  const uint4* gamma, const uint4* beta, float* mean_rstd, int rows,
                  int cols, float eps) {
  grid_trigger();
  grid_wait();
  __shared__ float2 red[ln_row_warps(W)];
  const int warp = threadIdx.x >> 5, row = blockIdx.x * (ln_row_warps(W) / W) + warp / W;
  const int t = (warp % W) * 32 + (threadIdx.x & 31);            // this row's thread
  if (W < 4 && row >= rows) return;                              // (W >= 4: a CTA is one row, and there is one for each)
  const int nvec = cols >> 3;
  const int64_t base = (int64_t)row * nvec;
  uint4 u[V], r[RES ? V : 1];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = t + k * 32 * W;
    if (v < nvec) {
      u[k] = x[base + v];
      if (RES) r[k] = res[base + v];
    }
  }
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = t + k * 32 * W;
    if (v < nvec) {
      float f[8];
      unpack8(u[k], f);
      if (RES) {
        float g[8];
        unpack8(r[k], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] += g[i];
      }
      if (h_out != nullptr) {
        if (RES) u[k] = pack8(f);
        h_out[base + v] = u[k];
        unpack8(u[k], f);   // statistics of the rounded values the backward pass sees
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) { s += f[i]; ss += f[i] * f[i]; }
    }
  }
  // scale and shift are asked for one vector ahead of the stores, which no later load may pass
  uint4 gn = make_uint4(0u, 0u, 0u, 0u), bn = gn;
  const auto affine = [&](int v) {
    if (v < nvec && gamma != nullptr) gn = gamma[v];
    if (v < nvec && beta != nullptr) bn = beta[v];
  };
  affine(t);
  row_sum2<W>(s, ss, red);
  const float mean = s / (float)cols, rstd = rsqrtf(fmaxf(ss / (float)cols - mean * mean, 0.f) + eps);
  if (t == 0 && mean_rstd != nullptr) {
    mean_rstd[2 * (int64_t)row] = mean;
    mean_rstd[2 * (int64_t)row + 1] = rstd;
  }
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = t + k * 32 * W;
    if (v < nvec) {
      float f[8], g[8], b[8];
      unpack8(u[k], f);
      if (RES && h_out == nullptr) {          // the sum was not kept
        unpack8(r[k], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] += g[i];
      }
      unpack8(gn, g);
      unpack8(bn, b);
      if (k + 1 < V) affine(v + 32 * W);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float o = (f[i] - mean) * rstd;
        if (gamma != nullptr) o *= g[i];
        if (beta != nullptr) o += b[i];
        f[i] = o;
      }
      y[base + v] = pack8(f);
    }
  }
}

// dgamma += sum over the rows of dy * xhat, dbeta += sum of dy, for 32 columns and one of `slices` interleaved parts of the rows:
// four threads with a vector each per row, T / 4 rows at a time.
template <int T>
__device__ __forceinline__ void ln_column_sums(const uint4* dy, const uint4* h,
                                               const float* mean_rstd, int rows, int cols, float* dgamma,
                                               float* dbeta, int block, int slice, int slices) {
  __shared__ float part[T / 32][2][32];
  const int nvec = cols >> 3, sub = threadIdx.x & 3, v = block * 4 + sub;
  uint64_t g[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
  constexpr int kStep = T / 4, kAhead = 4;
  if (v < nvec) {
    for (int r0 = slice * kStep + (threadIdx.x >> 2); r0 < rows; r0 += slices * kStep * kAhead) {
      uint4 du[kAhead], hu[kAhead];
      float mean[kAhead], rstd[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const int64_t row = r0 + (int64_t)j * slices * kStep;
        const bool live = row < rows;
        du[j] = live ? dy[row * nvec + v] : make_uint4(0u, 0u, 0u, 0u);
        hu[j] = live ? h[row * nvec + v] : make_uint4(0u, 0u, 0u, 0u);
        mean[j] = live ? mean_rstd[2 * row] : 0.f;
        rstd[j] = live ? mean_rstd[2 * row + 1] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const uint64_t neg_mean = f32x2(-mean[j], -mean[j]), rstd2 = f32x2(rstd[j], rstd[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t d = unpack2(word(du[j], i));
          g[i] = fma2(d, mul2(add2(unpack2(word(hu[j], i)), neg_mean), rstd2), g[i]);
          b[i] = add2(b[i], d);
        }
      }
    }
  }
  float fg[8], fb[8];
  split4(g, fg);
  split4(b, fb);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      fg[i] += __shfl_xor_sync(0xffffffffu, fg[i], o);
      fb[i] += __shfl_xor_sync(0xffffffffu, fb[i], o);
    }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane < 4) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      part[warp][0][lane * 8 + i] = fg[i];
      part[warp][1][lane * 8 + i] = fb[i];
    }
  }
  __syncthreads();
  const int c = block * 32 + lane;
  if (warp < 2 && c < cols) {
    float* dst = warp == 0 ? dgamma : dbeta;
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < T / 32; ++i) sum += part[i][warp][lane];
    if (dst != nullptr) atomicAdd(dst + c, sum);
  }
}

// SUMS: the first `sum_ctas` CTAs add up dgamma and dbeta, from a second look at dy and h: `slices` of the rows for every 32 columns.
template <int V, int W, bool DRES, bool SUMS>
__global__ void __launch_bounds__(32 * ln_row_warps(W))
ln_bwd_row_kernel(const uint4* dy, const uint4* h, const uint4* gamma,
                  const float* mean_rstd, const uint4* dres, uint4* dx, int rows, int cols,
                  float* dgamma, float* dbeta, int sum_ctas, int slices) {
  grid_trigger();
  grid_wait();
  if (SUMS && (int)blockIdx.x < sum_ctas) {
    ln_column_sums<32 * ln_row_warps(W)>(dy, h, mean_rstd, rows, cols, dgamma, dbeta, blockIdx.x / slices, blockIdx.x % slices, slices);
    return;
  }
  const int cta = SUMS ? (int)blockIdx.x - sum_ctas : (int)blockIdx.x;
  __shared__ float2 red[ln_row_warps(W)];
  const int warp = threadIdx.x >> 5, row = cta * (ln_row_warps(W) / W) + warp / W;
  const int t = (warp % W) * 32 + (threadIdx.x & 31);
  if (W < 4 && row >= rows) return;
  const int nvec = cols >> 3;
  const int64_t base = (int64_t)row * nvec;
  uint4 d[V], hv[V], r[DRES ? V : 1];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = t + k * 32 * W;
    if (v < nvec) {
      d[k] = dy[base + v];
      hv[k] = h[base + v];
    }
  }
  const float mean = mean_rstd[2 * (int64_t)row], rstd = mean_rstd[2 * (int64_t)row + 1];
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = t + k * 32 * W;
    if (v < nvec) {
      float df[8], hf[8], gm[8];
      unpack8(d[k], df);
      unpack8(hv[k], hf);
      if (gamma != nullptr) unpack8(gamma[v], gm);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float g = gamma != nullptr ? df[i] * gm[i] : df[i];
        s1 += g;
        s2 += g * ((hf[i] - mean) * rstd);
      }
      if (DRES) r[k] = dres[base + v];
    }
  }
  uint4 gn = make_uint4(0u, 0u, 0u, 0u);      // scale, asked for one vector ahead of the stores
  const auto scale = [&](int v) {
    if (v < nvec && gamma != nullptr) gn = gamma[v];
  };
  scale(t);
  row_sum2<W>(s1, s2, red);
  const float m1 = s1 / (float)cols, m2 = s2 / (float)cols;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = t + k * 32 * W;
    if (v < nvec) {
      float df[8], hf[8], gm[8], o[8];
      unpack8(d[k], df);
      unpack8(hv[k], hf);
      unpack8(gn, gm);
      if (k + 1 < V) scale(v + 32 * W);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float g = gamma != nullptr ? df[i] * gm[i] : df[i];
        o[i] = rstd * (g - m1 - (hf[i] - mean) * rstd * m2);
      }
      if (DRES) {
        float rf[8];
        unpack8(r[k], rf);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += rf[i];
      }
      dx[base + v] = pack8(o);
    }
  }
}

// ------------------------------------------------------------------------------------------
// elementwise
// ------------------------------------------------------------------------------------------
__global__ void gelu_fwd_kernel(const uint4* x, uint4* y, int64_t nvec) {
  grid_trigger();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvec;
       i += (int64_t)gridDim.x * blockDim.x) {
    float f[8];
    unpack8(x[i], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = gelu_f(f[k]);
    y[i] = pack8(f);
  }
}
__global__ void gelu_bwd_kernel(const uint4* dy, const uint4* x,
                                uint4* dx, int64_t nvec) {
  grid_trigger();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvec;
       i += (int64_t)gridDim.x * blockDim.x) {
    float f[8], d[8];
    unpack8(x[i], f);
    unpack8(dy[i], d);
#pragma unroll
    for (int k = 0; k < 8; ++k) d[k] *= gelu_grad_f(f[k]);
    dx[i] = pack8(d);
  }
}
__global__ void add_kernel(const uint4* a, const uint4* b,
                           uint4* o, int64_t nvec) {
  grid_trigger();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvec;
       i += (int64_t)gridDim.x * blockDim.x) {
    float f[8], g[8];
    unpack8(a[i], f);
    unpack8(b[i], g);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] += g[k];
    o[i] = pack8(f);
  }
}
__global__ void cast_kernel(const float4* in, uint2* out, int64_t nvec,
                            int accumulate) {
  grid_trigger();
  grid_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvec;
       i += (int64_t)gridDim.x * blockDim.x) {
    float4 f = in[i];
    if (accumulate) {
      const uint2 c = out[i];
      f.x += bf_lo(c.x); f.y += bf_hi(c.x); f.z += bf_lo(c.y); f.w += bf_hi(c.y);
    }
    uint2 o;
    o.x = pack2(f.x, f.y);
    o.y = pack2(f.z, f.w);
    out[i] = o;
  }
}

// ------------------------------------------------------------------------------------------
// AdamW: 4 elements per thread
// ------------------------------------------------------------------------------------------
// Bound by HBM: 30 bytes an element.  One step per thread in as many CTAs as that takes: 188 M elements with their norm 1040 us
// with 2368 CTAs that walk the arrays, 995 with 9472, 957 so (6.7 TB/s); streaming hints or the order from the last element, whose
// gradient the norm has left in L2, to the first give nothing.
__global__ void adamw_kernel(uint2* param, float4* master,
                             float4* m, float4* v,
                             const void* grad, int grad_fp32, int64_t nvec, float lr,
                             float beta1, float beta2, float eps, float wd, float bc1, float bc2,
                             const float* grad_scale) {
  grid_trigger();
  grid_wait();
  const float gs = grad_scale != nullptr ? *grad_scale : 1.0f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvec;
       i += (int64_t)gridDim.x * blockDim.x) {
    float g[4];
    if (grad_fp32) {
      const float4 gg = reinterpret_cast<const float4*>(grad)[i];
      g[0] = gg.x; g[1] = gg.y; g[2] = gg.z; g[3] = gg.w;
    } else {
      const uint2 gg = reinterpret_cast<const uint2*>(grad)[i];
      g[0] = bf_lo(gg.x); g[1] = bf_hi(gg.x); g[2] = bf_lo(gg.y); g[3] = bf_hi(gg.y);
    }
    float4 p4 = master[i], m4 = m[i], v4 = v[i];
    float p[4] = {p4.x, p4.y, p4.z, p4.w};
    float mm[4] = {m4.x, m4.y, m4.z, m4.w};
    float vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float gk = g[k] * gs;
      mm[k] = beta1 * mm[k] + (1.f - beta1) * gk;
      vv[k] = beta2 * vv[k] + (1.f - beta2) * gk * gk;
      const float mh = mm[k] / bc1, vh = vv[k] / bc2;
      p[k] = p[k] - lr * (mh / (sqrtf(vh) + eps) + wd * p[k]);
    }
    master[i] = make_float4(p[0], p[1], p[2], p[3]);
    m[i] = make_float4(mm[0], mm[1], mm[2], mm[3]);
    v[i] = make_float4(vv[0], vv[1], vv[2], vv[3]);
    uint2 o;
    o.x = pack2(p[0], p[1]);
    o.y = pack2(p[2], p[3]);
    param[i] = o;
  }
}

// The clipping factor in one launch of one thread instead of seven of a scalar each (20 us of an optimizer step).
__global__ void clip_scale_kernel(const float* sq, int n, float max_norm, float* norm,
                                  float* scale) {
  grid_trigger();
  grid_wait();
  float s = 0.f;
  for (int i = 0; i < n; ++i) s += sq[i];
  const float len = sqrtf(s), f = max_norm / (len + 1e-6f);
  *norm = len;
  *scale = f > 1.0f ? 1.0f : f;    // NaN stays NaN
}

// Bound by HBM (with the write-back of what the step before left in L2).  Four vectors per thread in flight and 32 CTAs an SM, each
// with one atomic: the optimizer step of 188 M elements 957 -> 948 us (eight CTAs an SM 953, 128 951).
constexpr int kSumVec = 4;
__global__ void __launch_bounds__(256)
sumsq_kernel(const void* x, int is_fp32, int64_t nvec, float* out) {
  grid_trigger();
  grid_wait();
  __shared__ float red[64];
  float s = 0.f, dummy = 0.f;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < nvec; i0 += step * kSumVec) {
    float part[kSumVec];
    if (is_fp32) {
      float4 g[kSumVec];
#pragma unroll
      for (int j = 0; j < kSumVec; ++j)
        g[j] = i0 + j * step < nvec ? reinterpret_cast<const float4*>(x)[i0 + j * step] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < kSumVec; ++j) part[j] = g[j].x * g[j].x + g[j].y * g[j].y + g[j].z * g[j].z + g[j].w * g[j].w;
    } else {
      uint2 g[kSumVec];
#pragma unroll
      for (int j = 0; j < kSumVec; ++j)
        g[j] = i0 + j * step < nvec ? reinterpret_cast<const uint2*>(x)[i0 + j * step] : make_uint2(0u, 0u);
#pragma unroll
      for (int j = 0; j < kSumVec; ++j) {
        const float a = bf_lo(g[j].x), b = bf_hi(g[j].x), c = bf_lo(g[j].y), d = bf_hi(g[j].y);
        part[j] = a * a + b * b + c * c + d * d;
      }
    }
    s += (part[0] + part[1]) + (part[2] + part[3]);
  }
  block_sum2(s, dummy, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// ------------------------------------------------------------------------------------------
// vocab-parallel cross-entropy: one CTA per row
// ------------------------------------------------------------------------------------------
// Both kernels are bound by HBM and keep kCeVec vectors per thread in flight.  The partial pass reads a row once: every
// thread keeps the maximum of its elements and the sum of exponentials relative to it, and rescales the sum when a group
// of vectors raises the maximum (Milakov and Gimelshein, online softmax).  4096 rows x 50257: partial 124 us with two
// passes over the row, 82 us with one (four fifths of the issue slots taken), 67 us with maxima of packed bf16, packed
// differences and products and one-instruction exponentials; gradient 153 us with one vector in flight
// and a test per element, 132 us so (copy bandwidth: 62 and 124).
constexpr int kCeVec = 4;
static_assert(kCeVec == 4, "the sums below are written out");
// Larger of two bf16, twice (a NaN only where both are NaN: the sum shows the others).
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// 2^x in one instruction, results below 2^-126 zero: in a sum whose largest term is 1 they are nothing.
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// A thread's running maximum and sum of exp(x - m).
struct CeSum {
  float m = -INFINITY, s = 0.f;
  __device__ __forceinline__ void raise(float to) {
    if (to > m) {
      s *= __expf(m - to);                 // (0 while m is -inf: s is 0)
      m = to;
    }
  }
  __device__ __forceinline__ void add(const uint4 (&u)[kCeVec]) {
    uint32_t top = 0xff80ff80u;
#pragma unroll
    for (int j = 0; j < kCeVec; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) top = max_bf16x2(top, word(u[j], i));
    raise(fmaxf(bf_lo(top), bf_hi(top)));
    if (m > -INFINITY) {
      const uint64_t neg_m = f32x2(-m, -m), log2e = f32x2(1.4426950408889634f, 1.4426950408889634f);
      uint64_t part[kCeVec] = {};
#pragma unroll
      for (int j = 0; j < kCeVec; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float lo, hi;
          split(mul2(add2(unpack2(word(u[j], i)), neg_m), log2e), lo, hi);
          part[j] = add2(part[j], f32x2(exp2_ftz(lo), exp2_ftz(hi)));
        }
      float lo, hi;
      split(add2(add2(part[0], part[1]), add2(part[2], part[3])), lo, hi);
      s += lo + hi;
    } else {
      // while everything seen is -inf nothing counts, except that a NaN has to show
#pragma unroll
      for (int j = 0; j < kCeVec; ++j) {
        float f[8];
        unpack8(u[j], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += f[i] == f[i] ? 0.f : f[i];
      }
    }
  }
};
constexpr uint32_t kNegInf2 = 0xff80ff80u;   // two bf16 -inf
// (softmax - onehot) * scale of the eight logits of vector v; padding columns get 0.
__device__ __forceinline__ uint4 ce_grad_vector(const uint4& u, int v, int64_t t, int64_t valid, float mx, float inv, float scale) {
  float f[8];
  unpack8(u, f);
  if (v * 8 + 8 <= valid && (t >> 3) != v) {   // neither padding nor the target: most vectors
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __expf(f[i] - mx) * inv;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = v * 8 + i;
      float gsm = c < valid ? __expf(f[i] - mx) * inv : 0.f;
      if (c == t) gsm -= scale;
      f[i] = gsm;
    }
  }
  return pack8(f);
}
__global__ void __launch_bounds__(256)
ce_partial_kernel(const __nv_bfloat16* logits, int64_t ld,
                  const int64_t* targets, int rows, int cols, int col_offset,
                  int vocab, float* row_max, float* row_sumexp,
                  float* tgt_logit, const __grid_constant__ RowExchange ex) {
  if (ex.n == 0) grid_trigger();
  grid_wait();
  __shared__ float red[64];
  const int valid = max(0, min(cols, vocab - col_offset));
  const int nvec = valid >> 3;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* p = logits + (int64_t)row * ld;
    const uint4* pv = reinterpret_cast<const uint4*>(p);
    CeSum sum;
    for (int v0 = threadIdx.x; v0 < nvec; v0 += blockDim.x * kCeVec) {
      uint4 u[kCeVec];
#pragma unroll
      for (int j = 0; j < kCeVec; ++j) {
        const int v = v0 + j * blockDim.x;
        u[j] = v < nvec ? pv[v] : make_uint4(kNegInf2, kNegInf2, kNegInf2, kNegInf2);
      }
      sum.add(u);
    }
    for (int c = nvec * 8 + threadIdx.x; c < valid; c += blockDim.x) {
      const float f = __bfloat162float(p[c]);
      sum.raise(f);
      if (f != -INFINITY) sum.s += __expf(f - sum.m);
    }
    const float m = sum.m;
    float s = sum.s;
    const float mx = block_max(m, red);
    float dummy = 0.f;
    // a thread without elements adds nothing; a row of nothing but -inf has no sum (NaN), an empty one has 0
    s = valid == 0 ? 0.f : m == -INFINITY && mx > -INFINITY ? s : s * __expf(m - mx);
    block_sum2(s, dummy, red);
    if (threadIdx.x == 0) {
      const int64_t t = targets[row] - col_offset;
      const float tl = (t >= 0 && t < valid) ? __bfloat162float(p[t]) : 0.f;
      if (ex.n > 0) {        // publish (max, sum-exp relative to it, target logit) to the mesh row
        const float v3[3] = {mx, s, tl};
        ex_put<3>(ex, row, v3);
      } else {
        row_max[row] = mx;
        row_sumexp[row] = s;
        tgt_logit[row] = tl;
      }
    }
  }
  if (ex.n > 0) ex_signal(ex);
}

__global__ void __launch_bounds__(256)
ce_grad_kernel(__nv_bfloat16* logits, int64_t ld, const int64_t* targets,
               int rows, int cols, int col_offset, int vocab, const float* gmax,
               const float* gsumexp, float scale, float* row_loss,
               const float* tgt_logit, const __grid_constant__ RowExchange ex) {
  if (ex.n == 0) grid_trigger();
  grid_wait();
  const int nvec = cols >> 3;
  const int64_t valid = (int64_t)vocab - col_offset;       // columns before the padding
  if (ex.n > 0 && !ex_wait(ex, 2u)) return;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    __nv_bfloat16* p = logits + (int64_t)row * ld;
    uint4* pv = reinterpret_cast<uint4*>(p);
    float mx, se;
    if (ex.n > 0) {
      // combine the vocabulary slices of the mesh row in fixed order: global max, sum of the
      // rescaled partial sums, the one non-zero target logit; every GPU of the row gets the same
      mx = -INFINITY;
      for (int q = 0; q < ex.n; ++q) mx = fmaxf(mx, ex_get(ex, q, row, 3, 0));
      se = 0.f;
      float tl = 0.f;
      for (int q = 0; q < ex.n; ++q) {
        const float sq = ex_get(ex, q, row, 3, 1);
        if (sq > 0.f) se += sq * __expf(ex_get(ex, q, row, 3, 0) - mx);
        tl += ex_get(ex, q, row, 3, 2);
      }
      if (threadIdx.x == 0 && row_loss != nullptr) row_loss[row] = __logf(se) + mx - tl;
    } else {
      mx = gmax[row];
      se = gsumexp[row];
      if (threadIdx.x == 0 && row_loss != nullptr) row_loss[row] = logf(se) + mx - tgt_logit[row];
    }
    const float inv = scale / se;
    const int64_t t = targets[row] - col_offset;
    for (int v0 = threadIdx.x; v0 < nvec; v0 += blockDim.x * kCeVec) {
      uint4 u[kCeVec];
#pragma unroll
      for (int j = 0; j < kCeVec; ++j) {
        const int v = v0 + j * blockDim.x;
        if (v < nvec) u[j] = pv[v];
      }
#pragma unroll
      for (int j = 0; j < kCeVec; ++j) {
        const int v = v0 + j * blockDim.x;
        if (v < nvec) pv[v] = ce_grad_vector(u[j], v, t, valid, mx, inv, scale);
      }
    }
  }
}

// Both passes in one, for whole rows on one device: a row waits in shared memory between them (every thread copies the vectors
// that it reads itself, cp.async, kCeAhead groups of kCeVec ahead), so the logits are read once.  Two
// kernels / one, us: 4096 rows of 50257 211 / 167 (5.0 TB/s: two CTAs an SM, whose barriers between the passes leave gaps), 2048 of
// 30000 67 / 58, 1000 of 100000 104 / 98, 512 of 1000 6.8 / 4.4; with the sum of the row losses in one launch instead of two of the
// tensor library, a two-layer model of width 512, forward and backward, 454 / 431.
constexpr int kCeAhead = 4;
constexpr int kCeRowBytes = 200 * 1024;     // most of a row that is kept
__global__ void __launch_bounds__(512)
ce_row_kernel(__nv_bfloat16* logits, int64_t ld, const int64_t* targets, int cols, int vocab, float scale,
              float* row_loss) {
  extern __shared__ uint4 ring[];
  __shared__ float red[64];
  grid_trigger();
  grid_wait();
  const int T = blockDim.x, row = blockIdx.x, nvec = cols >> 3, valid = min(cols, vocab), nv = (valid + 7) >> 3;
  uint4* pv = reinterpret_cast<uint4*>(logits + (int64_t)row * ld);
  const int64_t t = targets[row];
  auto prefetch = [&](int v0) {
#pragma unroll
    for (int j = 0; j < kCeVec; ++j) {
      const int v = v0 + j * T;
      if (v < nv) cp_async16(ring + v, pv + v);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < kCeAhead; ++i) prefetch(threadIdx.x + i * T * kCeVec);
  CeSum sum;
  for (int v0 = threadIdx.x; v0 < nv; v0 += T * kCeVec) {
    prefetch(v0 + kCeAhead * T * kCeVec);
    cp_async_wait<kCeAhead>();
    uint4 u[kCeVec];
#pragma unroll
    for (int j = 0; j < kCeVec; ++j) {
      const int v = v0 + j * T;
      u[j] = v < nv ? ring[v] : make_uint4(kNegInf2, kNegInf2, kNegInf2, kNegInf2);
      if (v == nv - 1 && (valid & 7)) {      // columns beyond the vocabulary count as -inf
        uint32_t* w = &u[j].x;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (v * 8 + 2 * i >= valid) w[i] = kNegInf2;
          else if (v * 8 + 2 * i + 1 >= valid) w[i] = (w[i] & 0xffffu) | (kNegInf2 & 0xffff0000u);
        }
      }
    }
    sum.add(u);
  }
  cp_async_wait<0>();
  const float mx = block_max(sum.m, red);    // (its barriers make the whole row visible to every thread)
  float se = sum.m == -INFINITY && mx > -INFINITY ? sum.s : sum.s * __expf(sum.m - mx), dummy = 0.f;
  block_sum2(se, dummy, red);
  if (threadIdx.x == 0) {
    const float tl = t >= 0 && t < valid ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ring)[t]) : 0.f;
    row_loss[row] = logf(se) + mx - tl;
  }
  const float inv = scale / se;
  for (int v = threadIdx.x; v < nvec; v += T)
    pv[v] = ce_grad_vector(v < nv ? ring[v] : make_uint4(0u, 0u, 0u, 0u), v, t, valid, mx, inv, scale);
}

// out = sum of n values over divisor, in a fixed order, by one CTA.
__global__ void __launch_bounds__(1024)
sum_kernel(const float* x, int n, float divisor, float* out) {
  grid_trigger();
  grid_wait();
  __shared__ float red[64];
  float s = 0.f, dummy = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += x[i];
  block_sum2(s, dummy, red);
  if (threadIdx.x == 0) *out = s / divisor;
}

// ------------------------------------------------------------------------------------------
// embedding
// ------------------------------------------------------------------------------------------
// Four vectors of a row in flight before the first store: 8192 tokens of width 4096 26 us with one, 24 so.
constexpr int kEmbVec = 4;
__global__ void embedding_fwd_kernel(const int64_t* tokens,
                                     const uint4* tok_table,
                                     const uint4* pos_table, uint4* out,
                                     int n_tokens, int seq, int nvec) {
  grid_trigger();
  grid_wait();
  for (int t = blockIdx.x; t < n_tokens; t += gridDim.x) {
    const int64_t tok = tokens[t];
    const int pos = t % seq;
    const uint4* row = tok_table + tok * nvec;
    const uint4* at = pos_table + (int64_t)pos * nvec;
    for (int v0 = threadIdx.x; v0 < nvec; v0 += kEmbVec * blockDim.x) {
      uint4 u[kEmbVec], w[kEmbVec];
#pragma unroll
      for (int j = 0; j < kEmbVec; ++j) {
        const int v = v0 + j * blockDim.x;
        if (v < nvec) {
          u[j] = row[v];
          w[j] = at[v];
        }
      }
#pragma unroll
      for (int j = 0; j < kEmbVec; ++j) {
        const int v = v0 + j * blockDim.x;
        if (v >= nvec) continue;
        float a[8], b[8];
        unpack8(u[j], a);
        unpack8(w[j], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] += b[i];
        out[(int64_t)t * nvec + v] = pack8(a);
      }
    }
  }
}
// token table: scatter-add with fp32 vector atomics; position table: plain sum over the batch
__global__ void embedding_bwd_tok_kernel(const int64_t* tokens,
                                         const uint4* dout, float* dtok,
                                         int n_tokens, int nvec) {
  grid_trigger();
  grid_wait();
  for (int t = blockIdx.x; t < n_tokens; t += gridDim.x) {
    const int64_t tok = tokens[t];
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
      float a[8];
      unpack8(dout[(int64_t)t * nvec + v], a);
      float4* dst = reinterpret_cast<float4*>(dtok + (tok * nvec + v) * 8);
      atomicAdd(dst, make_float4(a[0], a[1], a[2], a[3]));
      atomicAdd(dst + 1, make_float4(a[4], a[5], a[6], a[7]));
    }
  }
}
__global__ void embedding_bwd_pos_kernel(const uint4* dout, float* dpos,
                                         int n_tokens, int seq, int nvec) {
  grid_trigger();
  grid_wait();
  const int64_t total = (int64_t)seq * nvec;
  const int nb = n_tokens / seq;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pos = i / nvec, v = i - pos * nvec;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = 0; b < nb; ++b) {
      float a[8];
      unpack8(dout[((int64_t)b * seq + pos) * nvec + v], a);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += a[k];
    }
    float* dst = dpos + i * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[k] += acc[k];
  }
}

// One CTA per row: as many threads as the row has 16-byte vectors (32..256), so that short
// column-sharded rows do not leave half of the CTA idle.
inline int ln_threads(int cols) {
  const int nvec = cols / 8;
  int t = (nvec + 31) / 32 * 32;
  if (t < 32) t = 32;
  if (t > kLnThreads) t = kLnThreads;
  return t;
}

// Launch shape of ln_bwd_kernel for a local width: threads per CTA, threads per row, rows per CTA, vectors per thread.
struct LnBwdShape { int threads, tpr, rows_per_cta, maxv; };
inline LnBwdShape ln_bwd_shape(int cols) {
  const int nvec = cols / 8;
  int tpr = (nvec + 31) / 32 * 32;
  if (tpr < 32) tpr = 32;
  if (cols <= kLnGroupedMaxCols) {
    const int g = kLnBwdThreads / tpr;
    return {g * tpr, tpr, g, 1};
  }
  // Two vectors per thread: the reductions and barriers of a row are shared by more of it than with one vector of twice
  // the threads (32768 x 4096 with dres: 244 us with 512 threads of one vector, 192 us so).
  tpr = ((nvec + 1) / 2 + 31) / 32 * 32;
  if (tpr > kLnBwdThreads) tpr = kLnBwdThreads;
  return {tpr, tpr, 1, (nvec + tpr - 1) / tpr};
}

// Shared memory of a row ring; CTAs of the forward kernel that an SM holds (by registers 1280 threads of one vector,
// 1024 of two, 512 of four, 256 of eight; at most 24 CTAs), with a residual: that is the grid of one resident wave, whose
// rows follow one another.
inline int ln_ring_bytes(bool backward, int inputs, int maxv, int threads) {
  return ln_stages(backward, maxv) * inputs * maxv * threads * 16;
}
inline int ln_fwd_maxv(int cols) {
  const int threads = ln_threads(cols), n = (cols / 8 + threads - 1) / threads;
  return n <= 1 ? 1 : n <= 2 ? 2 : n <= 4 ? 4 : 8;
}
inline int ln_fwd_resident(int cols) {
  const int threads = ln_threads(cols), maxv = ln_fwd_maxv(cols);
  const int by_regs = (maxv == 1 ? 1280 : maxv == 2 ? 1024 : maxv == 4 ? 512 : 256) / threads;
  const int by_smem = 224 * 1024 / (ln_ring_bytes(false, 2, maxv, threads) + 1280);
  int n = by_regs < by_smem ? by_regs : by_smem;
  return n < 1 ? 1 : n > 24 ? 24 : n;
}

// Rows of one vector per thread without the ring: while what a call moves stays in L2 there is no HBM latency to hide, and
// the way through shared memory costs more than it gives.  Repeated calls, ring / direct, us: statistics of 16384 x 1024 (32 MB)
// 14.5 / 12.4, with residual 12000 x 1024 (70 MB) 14.5 / 13.2, rows of 8192 x 2048 (64 MB) 18.6 / 16.5; beyond L2 the ring wins:
// statistics with residual of 8192 x 2048 (96 MB) 20.5 / 24.0, rows of 16384 x 2048 (128 MB) 35.8 / 36.9; below 8 MB there is
// nothing between them.  With inputs from HBM the ring is ahead by 0 to 2 us on most sizes, 4 with a residual (12000 x 1024 20.4 / 24.5).
// Wider rows keep the ring.
constexpr int64_t kLnDirectMin = 8 << 20, kLnDirectMax = 80 << 20;
inline bool ln_fwd_direct(int rows, int cols, int tensors) {
  const int64_t bytes = 2 * (int64_t)rows * cols * tensors;
  return ln_fwd_maxv(cols) == 1 && bytes >= kLnDirectMin && bytes <= kLnDirectMax;
}

// Warps per row and 16-byte vectors per thread of the row kernels (w = 0: the persistent kernel).  One warp as long as its
// vectors fit the registers that still leave enough warps per SM, four or eight beyond; with few rows more warps, down to a
// vector each, because a row's latency is all there is.  us for W = 1 / 4 / 8:
//   forward            32768 x 2048 42 / 51 / 71, x 4096 - / 81 / 106; 33 x 2048 2.9 / 2.2 / 2.0
//   with residual      65536 x 1024 82 / 89 / 133, 32768 x 1544 64 / 68 / 85, x 2048 85 / 81 / 94; 8192 x 6000 - / 63 / 62, x 8192 - /
//                      85 / 83
//   backward           32768 x 2048 61 / 63 / 77, x 4096 - / 117 / 129
//   with dres          65536 x 512 46 / 53 / 92, 32768 x 1024 52 / 41 / 56, x 3072 - / 132 / 145, x 4096 - / 192 / 172 (persistent 183),
//                      8192 x 8192 - / 125 / 110 (persistent 96): three tensors in registers beyond three vectors each are too many
struct LnRowShape { int v, w; };
struct LnRowMost { int w1, w4, w8; };     // most vectors per thread of a row of one, four, eight warps
constexpr LnRowMost kLnFwdMost{8, 8, 8}, kLnFwdResMost{7, 5, 8}, kLnBwdMost{8, 8, 8}, kLnBwdDresMost{2, 3, 3};
constexpr LnRowShape ln_row_shape(int rows, int cols, LnRowMost most) {
  const int nvec = cols / 8;
  const auto vectors = [&](int w) { return (nvec + 32 * w - 1) / (32 * w); };
  int w = vectors(1) <= most.w1 ? 1 : vectors(4) <= most.w4 ? 4 : vectors(8) <= most.w8 ? 8 : 0;
  if (w == 0) return {0, 0};
  while (w < 8 && vectors(w) > 1 && (int64_t)rows * w < 1024) w = w == 1 ? 4 : 8;
  return {vectors(w), w};
}
// dgamma and dbeta from a second look at dy and h, in CTAs of the same launch, instead of the persistent kernel's registers: that
// kernel ends with atomics of every CTA to the same addresses (5 us and more), and rows of up to 2048 columns wait there at a
// barrier each.  The second look is from L2 as long as the tensors stay there.  Persistent / here, us, with dres: 512 x 512
// 8.2 / 3.0, 4099 x 1544 22.1 / 11.2, 8192 x 2048 (34 MB a tensor) 40.8 / 30.0, 16384 x 2048 (67 MB) 70.4 / 66.0, 32768 x 1024 (67 MB)
// 67.0 / 76.6, 4099 x 3072 (25 MB) 27.1 / 24.4, 4099 x 4096 (34 MB) 33.3 / 33.0, 8192 x 4096 57.2 / 72.2; without dres 32768 x 2048
// (134 MB) 124 / 106, 4099 x 4096 26.4 / 24.9, 8192 x 4096 50.7 / 58.0.
inline bool ln_sums_from_second_look(int rows, int cols, bool dres) {
  const int64_t mb = 2 * (int64_t)rows * cols / 1000000;
  if (cols <= kLnGroupedMaxCols) return !dres || mb <= 64;
  return mb <= (dres ? 25 : 34);
}
// f(vectors, warps) as integral constants, for the shapes that ln_row_shape gives with `w1`, `w4`, `w8` and no others.
template <int w1, int w4, int w8, class F>
cudaError_t with_row_shape(LnRowShape s, F&& f) {
#define MSB_ROW(V, W, MOST) \
  if constexpr (V <= MOST)  \
    if (s.v == V && s.w == W) return f(std::integral_constant<int, V>{}, std::integral_constant<int, W>{});
#define MSB_ROWS(W, M) MSB_ROW(1, W, M) MSB_ROW(2, W, M) MSB_ROW(3, W, M) MSB_ROW(4, W, M) MSB_ROW(5, W, M) MSB_ROW(6, W, M) MSB_ROW(7, W, M) MSB_ROW(8, W, M)
  MSB_ROWS(1, w1) MSB_ROWS(4, w4) MSB_ROWS(8, w8)
#undef MSB_ROWS
#undef MSB_ROW
  return cudaErrorInvalidValue;
}

inline int grid_for(int64_t n, int threads, int cap = 148 * 16) {
  int64_t g = (n + threads - 1) / threads;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

// ------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------
// Shared memory beyond 48 KiB, of which the kernels here use at most 17 statically, has to be allowed per kernel and
// device.
static cudaError_t allow_smem(const void* kernel, int bytes) {
  return bytes <= 31 * 1024 ? cudaSuccess
                            : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Launch shapes.  In a row exchange every CTA ends in a system-wide fence and an add to the same counter of every peer,
// which takes longer than a row, and every CTA of the second pass polls its own: one resident wave with several rows a CTA
// (ce_partial_kernel: five CTAs an SM by registers).  4096 rows of 6400 logits in a group of eight: 254 us with a row per
// CTA, 83 with 740 CTAs (19 without an exchange).  On one device a row per CTA up to 32 per SM: blocks handed out as SMs get
// free leave no uneven last wave (4096 rows on 1184 CTAs: four rows each, three for some).
int ce_grid(int rows) { return rows < 148 * 5 ? rows : 148 * 5; }
static int ce_local_grid(int rows) { return rows < 148 * 32 ? rows : 148 * 32; }

static int ln_local_grid(int backward, int rows, int cols) {
  const int width = cols > 0 ? cols : 8 * kLnThreads;
  // narrow rows: three waves, because few rows per CTA leave the last one uneven (32768 x 1024 with residual: 53 us with
  // one wave, 48 with three, 65 without the ring)
  int cap = 148 * ln_fwd_resident(width) * (ln_fwd_maxv(width) == 1 ? 3 : 1);
  if (backward) {
    // one resident wave (1024 threads per SM at 64 registers, 512 at 128): every CTA ends with its atomics for
    // dgamma / dbeta, so CTAs beyond what is resident only add atomics
    const LnBwdShape sh = ln_bwd_shape(cols > 0 ? cols : 8 * kLnBwdThreads);
    cap = 148 * ((sh.maxv == 1 ? 1024 : 512) / sh.threads);
    const int groups = (rows + sh.rows_per_cta - 1) / sh.rows_per_cta;
    return groups < cap ? groups : cap;
  }
  return rows < cap ? rows : cap;
}
int ln_grid(int backward, int rows, int cols) {
  if (backward) return ln_local_grid(backward, rows, cols);   // already one wave
  const int resident = ln_fwd_resident(cols > 0 ? cols : 8 * kLnThreads), cap = 148 * (resident < 16 ? resident : 16);
  return rows < cap ? rows : cap;
}

cudaError_t ln_fwd(int mode, const void* x, const void* res, void* h_out, void* y,
                   const void* gamma, const void* beta, float* stats, float* mean_rstd, int rows,
                   int cols, int total_cols, float eps, cudaStream_t stream, const RowExchange* exch) {
  if (cols % 8 != 0 || cols > 8 * kLnThreads * 8) return cudaErrorInvalidValue;
  if (exch != nullptr && mode != 1 && mode != 2) return cudaErrorInvalidValue;
  if (rows <= 0 || (mode == 0 && total_cols != cols)) return cudaErrorInvalidValue;
  const int grid = exch != nullptr ? ln_grid(0, rows, cols) : ln_local_grid(0, rows, cols);
  RowExchange ex;
  if (exch != nullptr) ex = *exch; else memset(&ex, 0, sizeof(ex));
  auto X = reinterpret_cast<const uint4*>(x);
  auto R = reinterpret_cast<const uint4*>(res);
  auto H = reinterpret_cast<uint4*>(h_out);
  auto Y = reinterpret_cast<uint4*>(y);
  auto G = reinterpret_cast<const uint4*>(gamma);
  auto B = reinterpret_cast<const uint4*>(beta);
  const int threads = ln_threads(cols), maxv = ln_fwd_maxv(cols);
  const int inputs = mode != 2 && res != nullptr ? 2 : 1;
  const int tensors = inputs + (mode != 2 && h_out != nullptr ? 1 : 0) + (mode != 1 ? 1 : 0);
  if (mode == 0) {
    auto run = [&](auto kernel, int w) {
      const int per = ln_row_warps(w) / w;
      return launch_dependent(kernel, (rows + per - 1) / per, 32 * ln_row_warps(w), 0, stream, X, R, H, Y, G, B, mean_rstd, rows, cols, eps);
    };
    constexpr LnRowMost a = kLnFwdMost, b = kLnFwdResMost;
    return R == nullptr ? with_row_shape<a.w1, a.w4, a.w8>(ln_row_shape(rows, cols, a), [&](auto v, auto w) {
      return run(ln_fwd_row_kernel<v.value, w.value, false>, w.value);
    }) : with_row_shape<b.w1, b.w4, b.w8>(ln_row_shape(rows, cols, b), [&](auto v, auto w) {
      return run(ln_fwd_row_kernel<v.value, w.value, true>, w.value);
    });
  }
  if (exch == nullptr && ln_fwd_direct(rows, cols, tensors)) {
    ln_fwd_kernel<1, false><<<grid, threads, 0, stream>>>(mode, X, R, H, Y, G, B, stats, mean_rstd, rows, cols, total_cols, eps, ex);
    return cudaGetLastError();
  }
  const int smem = ln_ring_bytes(false, inputs, maxv, threads);
  auto run = [&](auto kernel) {
    const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, stream>>>(mode, X, R, H, Y, G, B, stats, mean_rstd, rows, cols, total_cols, eps, ex);
    return cudaGetLastError();
  };
  if (maxv == 1) return run(ln_fwd_kernel<1, true>);
  if (maxv == 2) return run(ln_fwd_kernel<2, true>);
  if (maxv == 4) return run(ln_fwd_kernel<4, true>);
  return run(ln_fwd_kernel<8, true>);
}

cudaError_t ln_bwd(int mode, const void* dy, const void* h, const void* gamma,
                   const float* mean_rstd, const void* dres, void* dx, float* stats, float* dgamma,
                   float* dbeta, int rows, int cols, int total_cols, cudaStream_t stream,
                   const RowExchange* exch) {
  if (cols % 8 != 0 || cols > 8 * kLnBwdThreads * 4) return cudaErrorInvalidValue;
  if (exch != nullptr && mode != 1 && mode != 2) return cudaErrorInvalidValue;
  const int grid = exch != nullptr ? ln_grid(1, rows, cols) : ln_local_grid(1, rows, cols);
  RowExchange ex;
  if (exch != nullptr) ex = *exch; else memset(&ex, 0, sizeof(ex));
  auto DY = reinterpret_cast<const uint4*>(dy);
  auto H = reinterpret_cast<const uint4*>(h);
  auto G = reinterpret_cast<const uint4*>(gamma);
  auto DR = reinterpret_cast<const uint4*>(dres);
  auto DX = reinterpret_cast<uint4*>(dx);
  const LnRowShape rs = ln_row_shape(rows, cols, DR != nullptr ? kLnBwdDresMost : kLnBwdMost);
  const bool sums = dgamma != nullptr;
  // dx may be written over dy or h: the second look would find it there
  const auto over = [&](const void* p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(dx), n = 2 * (uintptr_t)rows * cols;
    return a < b + n && b < a + n;
  };
  if (exch == nullptr && mode == 0 && total_cols == cols && (sums || dbeta == nullptr) && rs.w > 0 && rows > 0 &&
      (!sums || (ln_sums_from_second_look(rows, cols, DR != nullptr) && !over(dy) && !over(h)))) {
    auto run = [&](auto kernel, int w) {
      // column sums: at least 128 CTAs, and no more than eight steps of T rows for one
      const int T = 32 * ln_row_warps(w), per = ln_row_warps(w) / w;
      const int blocks = (cols + 31) / 32, most = (rows + T - 1) / T, few = (128 + blocks - 1) / blocks, deep = rows / (8 * T);
      const int want = few > deep ? few : deep, slices = !sums ? 1 : want < most ? want : most, sum_ctas = sums ? blocks * slices : 0;
      return launch_dependent(kernel, sum_ctas + (rows + per - 1) / per, T, 0, stream, DY, H, G, mean_rstd, DR, DX, rows, cols, dgamma,
                              dbeta, sum_ctas, slices);
    };
    constexpr LnRowMost a = kLnBwdMost, b = kLnBwdDresMost;
    return DR == nullptr ? with_row_shape<a.w1, a.w4, a.w8>(rs, [&](auto v, auto w) {
      return sums ? run(ln_bwd_row_kernel<v.value, w.value, false, true>, w.value) : run(ln_bwd_row_kernel<v.value, w.value, false, false>, w.value);
    }) : with_row_shape<b.w1, b.w4, b.w8>(rs, [&](auto v, auto w) {
      return sums ? run(ln_bwd_row_kernel<v.value, w.value, true, true>, w.value) : run(ln_bwd_row_kernel<v.value, w.value, true, false>, w.value);
    });
  }
  const LnBwdShape sh = ln_bwd_shape(cols);
  const int maxv = cols <= kLnGroupedMaxCols ? 1 : sh.maxv <= 2 ? 2 : sh.maxv;
  const int smem = ln_ring_bytes(true, mode != 1 && dres != nullptr ? 3 : 2, maxv, sh.threads);
  auto run = [&](auto kernel) {
    const cudaError_t e = allow_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    if (exch == nullptr)
      return launch_dependent(kernel, grid, sh.threads, smem, stream, mode, DY, H, G, mean_rstd, DR, DX, stats, dgamma, dbeta, rows,
                              cols, total_cols, sh.tpr, ex);
    kernel<<<grid, sh.threads, smem, stream>>>(mode, DY, H, G, mean_rstd, DR, DX, stats, dgamma, dbeta, rows, cols,
                                              total_cols, sh.tpr, ex);
    return cudaGetLastError();
  };
  if (cols <= kLnGroupedMaxCols) return run(ln_bwd_kernel<1, true>);
  if (maxv == 2) return run(ln_bwd_kernel<2, false>);
  if (maxv == 3) return run(ln_bwd_kernel<3, false>);
  return run(ln_bwd_kernel<4, false>);
}

cudaError_t gelu_fwd(const void* x, void* y, int64_t n, cudaStream_t stream) {
  if (n % 8) return cudaErrorInvalidValue;
  return launch_dependent(gelu_fwd_kernel, grid_for(n / 8, 256), 256, 0, stream, reinterpret_cast<const uint4*>(x), reinterpret_cast<uint4*>(y), n / 8);
}
cudaError_t gelu_bwd(const void* dy, const void* x, void* dx, int64_t n, cudaStream_t stream) {
  if (n % 8) return cudaErrorInvalidValue;
  return launch_dependent(gelu_bwd_kernel, grid_for(n / 8, 256), 256, 0, stream, reinterpret_cast<const uint4*>(dy), reinterpret_cast<const uint4*>(x), reinterpret_cast<uint4*>(dx), n / 8);
}
cudaError_t add_bf16(const void* a, const void* b, void* out, int64_t n, cudaStream_t stream) {
  if (n % 8) return cudaErrorInvalidValue;
  // a step per thread: 134 M elements 124 us with CTAs that walk the arrays, 113 so (the GeLU kernels, bound by issue slots, the
  // other way round: 113 and 131)
  return launch_dependent(add_kernel, grid_for(n / 8, 256, 1 << 22), 256, 0, stream, reinterpret_cast<const uint4*>(a), reinterpret_cast<const uint4*>(b), reinterpret_cast<uint4*>(out), n / 8);
}
cudaError_t cast_f32_to_bf16(const float* in, void* out, int64_t n, int accumulate, cudaStream_t stream) {
  if (n % 4) return cudaErrorInvalidValue;
  return launch_dependent(cast_kernel, grid_for(n / 4, 256), 256, 0, stream, reinterpret_cast<const float4*>(in), reinterpret_cast<uint2*>(out), n / 4, accumulate);
}

cudaError_t adamw_step(void* param, float* master, float* m, float* v, const void* grad,
                       int grad_fp32, int64_t n, float lr, float beta1, float beta2, float eps,
                       float weight_decay, float bias_corr1, float bias_corr2,
                       const float* grad_scale, cudaStream_t stream) {
  if (n % 4) return cudaErrorInvalidValue;
  return launch_dependent(adamw_kernel, grid_for(n / 4, 256, 1 << 22), 256, 0, stream, reinterpret_cast<uint2*>(param), reinterpret_cast<float4*>(master), reinterpret_cast<float4*>(m), reinterpret_cast<float4*>(v), grad, grad_fp32, n / 4, lr, beta1, beta2, eps, weight_decay, bias_corr1, bias_corr2, grad_scale);
}

cudaError_t clip_scale(const float* sq, int n, float max_norm, float* norm, float* scale, cudaStream_t stream) {
  if (n < 1) return cudaErrorInvalidValue;
  return launch_dependent(clip_scale_kernel, 1, 1, 0, stream, sq, n, max_norm, norm, scale);
}

cudaError_t sumsq(const void* x, int is_fp32, int64_t n, float* out, cudaStream_t stream) {
  if (n % 4) return cudaErrorInvalidValue;
  return launch_dependent(sumsq_kernel, grid_for(n / 4, 256, 148 * 32), 256, 0, stream, x, is_fp32, n / 4, out);
}

cudaError_t ce_partial(const void* logits, int64_t ld, const int64_t* targets, int rows, int cols,
                       int col_offset, int vocab, float* row_max, float* row_sumexp,
                       float* tgt_logit, cudaStream_t stream, const RowExchange* exch) {
  RowExchange ex;
  if (exch != nullptr) ex = *exch; else memset(&ex, 0, sizeof(ex));
  if (ld % 8) return cudaErrorInvalidValue;
  const int grid = exch != nullptr ? ce_grid(rows) : ce_local_grid(rows);
  if (exch == nullptr)
    return launch_dependent(ce_partial_kernel, grid, 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(logits), ld, targets, rows, cols, col_offset, vocab, row_max, row_sumexp, tgt_logit, ex);
  ce_partial_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(logits), ld, targets, rows, cols, col_offset, vocab, row_max, row_sumexp, tgt_logit, ex);
  return cudaGetLastError();
}
cudaError_t ce_grad(void* logits, int64_t ld, const int64_t* targets, int rows, int cols,
                    int col_offset, int vocab, const float* gmax, const float* gsumexp, float scale,
                    cudaStream_t stream, float* row_loss, const RowExchange* exch, const float* tgt_logit) {
  if (row_loss != nullptr && exch == nullptr && tgt_logit == nullptr) return cudaErrorInvalidValue;
  RowExchange ex;
  if (exch != nullptr) ex = *exch; else memset(&ex, 0, sizeof(ex));
  if (ld % 8 || cols % 8) return cudaErrorInvalidValue;
  const int grid = exch != nullptr ? ce_grid(rows) : ce_local_grid(rows);
  if (exch == nullptr)
    return launch_dependent(ce_grad_kernel, grid, 256, 0, stream, reinterpret_cast<__nv_bfloat16*>(logits), ld, targets, rows, cols, col_offset, vocab, gmax, gsumexp, scale, row_loss, tgt_logit, ex);
  ce_grad_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<__nv_bfloat16*>(logits), ld, targets, rows, cols, col_offset, vocab, gmax, gsumexp, scale, row_loss, tgt_logit, ex);
  return cudaGetLastError();
}

int ce_row_cols() { return kCeRowBytes / 2; }
cudaError_t ce_row(void* logits, int64_t ld, const int64_t* targets, int rows, int cols, int vocab, float scale, float* row_loss,
                   cudaStream_t stream) {
  if (ld % 8 || cols % 8 || rows <= 0 || vocab <= 0 || (cols < vocab ? cols : vocab) > ce_row_cols()) return cudaErrorInvalidValue;
  const int nv = ((cols < vocab ? cols : vocab) + 7) / 8, smem = nv * 16;
  const int threads = nv > 2048 ? 512 : 256;
  const cudaError_t e = smem <= 31 * 1024 ? cudaSuccess : allow_smem(reinterpret_cast<const void*>(ce_row_kernel), kCeRowBytes);
  if (e != cudaSuccess) return e;
  return launch_dependent(ce_row_kernel, rows, threads, smem, stream, reinterpret_cast<__nv_bfloat16*>(logits), ld, targets, cols, vocab,
                          scale, row_loss);
}
cudaError_t sum_over(const float* x, int n, float divisor, float* out, cudaStream_t stream) {
  if (n < 0) return cudaErrorInvalidValue;
  return launch_dependent(sum_kernel, 1, 1024, 0, stream, x, n, divisor, out);
}

cudaError_t embedding_fwd(const int64_t* tokens, const void* tok_table, const void* pos_table,
                          void* out, int n_tokens, int seq, int cols, cudaStream_t stream) {
  if (cols % 8) return cudaErrorInvalidValue;
  const int grid = n_tokens < 148 * 16 ? n_tokens : 148 * 16;
  return launch_dependent(embedding_fwd_kernel, grid, 128, 0, stream, tokens, reinterpret_cast<const uint4*>(tok_table), reinterpret_cast<const uint4*>(pos_table), reinterpret_cast<uint4*>(out), n_tokens, seq, cols / 8);
}
cudaError_t embedding_bwd(const int64_t* tokens, const void* dout, float* dtok, float* dpos,
                          int n_tokens, int seq, int cols, cudaStream_t stream) {
  if (cols % 8 || n_tokens % seq) return cudaErrorInvalidValue;
  const int grid = n_tokens < 148 * 16 ? n_tokens : 148 * 16;
  const cudaError_t e = launch_dependent(embedding_bwd_tok_kernel, grid, 128, 0, stream, tokens, reinterpret_cast<const uint4*>(dout), dtok, n_tokens, cols / 8);
  if (e != cudaSuccess) return e;
  return launch_dependent(embedding_bwd_pos_kernel, grid_for((int64_t)seq * (cols / 8), 256), 256, 0, stream, reinterpret_cast<const uint4*>(dout), dpos, n_tokens, seq, cols / 8);
}

}  // namespace msb
