// Flash-style attention forward / backward for head_dim 128 on tcgen05 (sm_100a): the score matrix
// lives in tensor memory only.
//
// Forward (attn_fwd2_kernel): persistent CTAs, two tiles of 128 query rows of a (sequence, head) at a time; S = Q K^T
//   into TMEM, online softmax in the log2 domain with lazy rescaling of O (only when the running
//   maximum grows by more than 2^8), P written back over S as packed bf16 and read by O += P V as
//   the TMEM operand.
// Backward (attn_bwd2_kernel): dK / dV are accumulated by the CTA that works
//   on 128 keys, dQ by the CTA that works on 128 queries; both recompute S and dP, keep P and dS in TMEM,
//   and never add to global memory: the gradients are bit-identical from run to run.
// All waits are bounded; a timeout records a code in `status` and the CTA leaves.
#include "attention.h"

#include <cuda_bf16.h>

#include <type_traits>

#include "../common/f32x2.cuh"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "../gemm/sm100_gemm.h"  // make_tensor_map_2d

namespace msb {

namespace {

constexpr int kD = 128;         // head dim
constexpr int kBlk = 128;       // query / key rows per tile
constexpr int kTile = kBlk * kD * 2;  // 32 KiB: one [128 x 128] bf16 tile = two swizzle halves
constexpr int kHalf = kTile / 2;
// A warp may touch the TMEM lanes 32 * (warp % 4) ... + 31: any four consecutive warps cover the 128 rows of a tile, whichever
// warp the element-wise work starts at.
constexpr uint32_t kErrAttn = 20;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

struct AttnArgs {
  float* lse;
  int batch, seq, heads, causal;
  int tiles_per_item; // fwd: query tiles that a CTA works on at a time (1 or 2)
  float scale;
  uint32_t* status;
  uint64_t timeout_ns;
};

__device__ __forceinline__ void report(uint32_t* status, uint32_t code, uint32_t d0, uint32_t d1) {
  if (atomicCAS(status, 0u, code) == 0u) {
    status[1] = blockIdx.x + (blockIdx.y << 12) + (blockIdx.z << 22);
    status[2] = d0;
    status[3] = d1;
  }
}

// Bounded wait of a whole warp: the lanes poll together (one transaction), the verdict is common.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, uint64_t tmo) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, tmo));
}

// 2^x on the special-function unit in one instruction (relative error 2^-22, denormal results
// flushed to zero: probabilities below 2^-126 are zero anyway).  exp2f() wraps the same
// instruction in range scaling that costs several more issue slots per element.
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The same on the FMA pipe, for the share of the exponentials that would queue for the special-function unit (16 results per
// cycle and SM): x = n + f with n the nearest whole number, 2^f by the polynomial of degree 5 with the smallest largest
// relative error on [-1/2, 1/2] (Remez exchange; 2^-23.7, with fp32 rounding 2^-22.2), times 2^n.  Below -125 the result is
// 2^-125 and not zero; NaN stays NaN.  x stays below 127 wherever the result is used.
__device__ __forceinline__ float exp2_fma(float x) {
  float t;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(t) : "f"(x), "f"(-125.0f));
  const float r = __fadd_rn(t, 12582912.0f);                 // 1.5 * 2^23: n in the low bits
  const float f = __fsub_rn(t, __fsub_rn(r, 12582912.0f));
  float p = 1.327647245e-03f;
  p = fmaf(p, f, 9.675540961e-03f);
  p = fmaf(p, f, 5.550713092e-02f);
  p = fmaf(p, f, 2.402212024e-01f);
  p = fmaf(p, f, 6.931469440e-01f);
  p = fmaf(p, f, 1.000000119e+00f);
  return p * __int_as_float((__float_as_int(r) << 23) + 0x3f800000);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// K-major view of a tile: rows = M or N index, contraction along the 128 columns.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile, int kstep) {
  return make_smem_desc(tile + (kstep >> 2) * kHalf + (kstep & 3) * 32, 16, 1024);
}
// MN-major view: rows = contraction index (16 per step), the 128 columns are the M or N index.
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile, int kstep) {
  return make_smem_desc(tile + kstep * 2048, kHalf, 1024);
}

__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col,
                                          int row) {
  tma_load_2d(dst, map, bar, col, row);
  tma_load_2d(dst + kHalf, map, bar, col + 64, row);
}

// ==========================================================================================
// forward: P stays in tensor memory, two query tiles per CTA
// ==========================================================================================
// One persistent CTA per SM works on items of two neighbouring 128-query tiles of one (sequence, head):
//   warp 0      TMA producer: Q of both tiles, then K_j / V_j through two-stage rings that both tiles read; asks the
//               hardware for the next item (cluster launch control: the grid has one block per item, a running CTA
//               takes over blocks that have not been launched)
//   warp 1      MMA issuer: S_t = Q_t K_j^T into TMEM columns [0,128) / [128,256); O_t += P_t V_j into [256,384) /
//               [384,512), with P read from TMEM (the A operand of tcgen05.mma may live in tensor memory)
//   warps 4-7   softmax and output of tile 0, warps 8-11 of tile 1: one thread per query row; P_j is written back over
//               S as packed bf16 (64 columns), so it never touches shared memory and needs no proxy fence
// The tensor pipe runs the MMAs in issue order, so S_t(j+1) may be issued right behind P_t(j) V(j) although it
// overwrites P_t(j), and a completed S_t(j+1) implies a completed P_t(j) V(j) (O_t is safe to rescale).
//
// What bounds it: a step (128 queries x 128 keys) needs 1024 cycles of the tensor pipe (64 per instruction) and 1024
// of the SFU (16 exponentials per cycle and SM), and a tile alternates between the two: about 2100 cycles of
// softmax, of which the read of S takes 400 because the other tile's products use tensor memory too, and 1500 until
// the next scores are there (768 of MMAs, the rest is latency of the hand-over).  Issue order keeps the two tiles
// apart, so that one's softmax runs under the other's products; two steps take about 3800 cycles.  Two CTAs per SM
// with a tile each and the same softmax fall into step instead, because the tensor pipe and the SFU then serve
// both at once: 298 us against 253 for 16 heads x 8192, causal (321 with two passes over S in tensor memory).
// A row of S is read once, into 128 registers; maxima take three inputs and multiply-adds and sums two lanes per
// instruction; P is handed over in two parts, so that six of the eight k-steps of P V run under the last quarter's
// exponentials, and half of the row's sum waits until P is on its way.  An item's output and the next item's first
// scores overlap: the roles only meet at the barriers.  Tried without gain: two threads per row (264 us, more
// barriers for the same tensor-memory traffic), a quarter to three eighths of the exponentials as a polynomial on
// the FMA pipe (263-289 us: the registers spill and the warp's issue slots are the limit).
// With outputs as TMA stores and one poll per wait: 230 us (1196 TFLOP/s) for 16 heads x 8192, causal; batch 4 x 2048,
// 32 heads: causal 202 -> 148 us (930), full 330 -> 233 us (1180).
constexpr int kFwdWarpStage = 32 * 128;   // output staging per softmax warp: 32 rows x 64 columns
constexpr size_t kFwd2Smem = 6 * kTile + 8 * kFwdWarpStage + 256 + 1024;
constexpr int kFwd2Threads = 384;
// registers per thread: 384 threads launch with 168; warps 0-3 give up what the softmax warps take
constexpr int kFwd2RegsLow = 96, kFwd2RegsHigh = 200;
static_assert(kFwd2RegsLow + 2 * kFwd2RegsHigh <= 3 * 168, "register shares exceed what the CTA is launched with");

// Cluster launch control: ask for a block of this grid that has not been launched (16-byte response into shared
// memory, announced on an mbarrier); after a refusal nothing more may be asked.
__device__ __forceinline__ void clc_try_cancel(void* resp, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(resp)), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool clc_read(const void* resp, uint32_t& x, uint32_t& y, uint32_t& z) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %3, 1, 0, p;\n\t"
      "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n\t}"
      : "=&r"(x), "=&r"(y), "=&r"(z), "=&r"(ok) : "r"(smem_u32(resp)) : "memory");
  return ok != 0;
}

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns: thread t of the warp writes row (lane base + t).
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// 16 lanes x 32 fp32 columns in the layout of a matrix fragment: thread t gets, of every group n of 8 columns, columns
// 2 (t % 4) and + 1 of rows t / 4 (r[4n], r[4n + 1]) and t / 4 + 8 (r[4n + 2], r[4n + 3]).
__device__ __forceinline__ void tmem_ld_16x32_frag(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// The same elements as packed bf16: r[2n] / r[2n + 1] are the two columns of rows t / 4 / t / 4 + 8; groups of 8 columns: 4 or 2.
__device__ __forceinline__ void tmem_st_16x32_frag(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_16x16_frag(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// shared -> global, one box of a tensor map; tracked by bulk groups
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(smem_u32(smem_src)), "r"(x), "r"(y) : "memory");
}
// A warp's staged box on its way: every lane's writes are visible to the copy engine before lane 0 starts it.
__device__ __forceinline__ void warp_store_box(const CUtensorMap* map, const void* stage, int32_t x, int32_t y) {
  fence_proxy_async_smem();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    tma_store_2d(map, stage, x, y);
    bulk_commit();
  }
}
// The staging area may be written again: the copy engine has read it.
__device__ __forceinline__ void warp_stage_free() {
  if ((threadIdx.x & 31) == 0) bulk_wait_read<0>();
  __syncwarp();
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// What an item is: tiles_per_item neighbouring tiles, longest causal items first.
struct FwdItem {
  int b, h, hi, n0, n1;   // sequence, head, block of tile 0 (tile 1: hi - 1), key blocks of the tiles (n1 = 0: no tile 1)
};
__device__ __forceinline__ FwdItem fwd_item(const AttnArgs& a, uint32_t x, uint32_t y, uint32_t z, int group) {
  FwdItem w;
  const int bh = (int)z * group + (int)x, nblk = a.seq / kBlk;
  w.b = bh / a.heads;
  w.h = bh - w.b * a.heads;
  w.hi = nblk - 1 - (int)y * a.tiles_per_item;
  w.n0 = a.causal ? w.hi + 1 : nblk;
  w.n1 = a.tiles_per_item == 2 && w.hi > 0 ? (a.causal ? w.hi : nblk) : 0;
  return w;
}

__global__ void __launch_bounds__(kFwd2Threads, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_out,
                 const __grid_constant__ AttnArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                 // [2] tiles
  uint8_t* sK = smem + 2 * kTile;     // [2] stages
  uint8_t* sV = smem + 4 * kTile;     // [2] stages
  uint8_t* sO = smem + 6 * kTile;     // [8] warps
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 8 * kFwdWarpStage);
  uint8_t* clc_resp = reinterpret_cast<uint8_t*>(bars);   // 16 bytes
  uint64_t* clc_full = bars + 2;
  uint64_t* clc_empty = bars + 3;
  uint64_t* q_full = bars + 4;        // all [2] from here
  uint64_t* q_empty = bars + 6;
  uint64_t* k_full = bars + 8;
  uint64_t* k_empty = bars + 10;
  uint64_t* v_full = bars + 12;
  uint64_t* v_empty = bars + 14;
  uint64_t* s_full = bars + 16;
  uint64_t* o_done = bars + 18;
  uint64_t* p_ready = bars + 20;      // [2 * tile + part]: columns [0,96) / [96,128) of P
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint64_t tmo = a.timeout_ns;
  const int group = gridDim.x;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_qkv);
    mbar_init(clc_full, 1);
    mbar_init(clc_empty, 10);         // producer and MMA thread, 8 softmax warps
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full + i, 1);
      mbar_init(q_empty + i, 1);
      mbar_init(k_full + i, 1);
      mbar_init(k_empty + i, 1);
      mbar_init(v_full + i, 1);
      mbar_init(v_empty + i, 1);
      mbar_init(s_full + i, 1);
      mbar_init(o_done + i, 1);
      mbar_init(p_ready + 2 * i, 128);
      mbar_init(p_ready + 2 * i + 1, 128);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  grid_trigger();
  grid_wait();

  // The next item as the producer got it: false when there is none (or on a timeout).
  uint32_t clc_phase = 0;
  auto next_item = [&](FwdItem& w) -> bool {
    uint32_t x, y, z;
    if (!mbar_wait(clc_full, clc_phase, 8 * tmo)) {
      report(a.status, kErrAttn + 6, 0, 0);
      return false;
    }
    clc_phase ^= 1;
    const bool more = clc_read(clc_resp, x, y, z);
    fence_proxy_async_smem();         // this read before the next response overwrites it
    if (more) w = fwd_item(a, x, y, z, group);
    return more;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFwd2RegsLow));
    FwdItem w = fwd_item(a, blockIdx.x, blockIdx.y, blockIdx.z, group);
    if (warp == 0 && elect_one()) {
      uint32_t c = 0;                 // K / V tiles loaded so far
      uint32_t qc[2] = {0, 0};        // Q tiles loaded so far
      bool ok = true, more = true;
      while (ok && more) {
        const int colq = w.h * 3 * kD, seq0 = w.b * a.seq;
        for (int t = 0; t < 2 && ok; ++t) {
          if (t == 1 && w.n1 == 0) break;
          if (!(ok = mbar_wait(q_empty + t, (qc[t] & 1) ^ 1, 8 * tmo))) break;
          ++qc[t];
          mbar_expect_tx(q_full + t, kTile);
          load_tile(sQ + t * kTile, &tm_qkv, q_full + t, colq, seq0 + (w.hi - t) * kBlk);
        }
        for (int j = 0; j < w.n0 && ok; ++j, ++c) {
          const uint32_t st = c & 1, ph = ((c >> 1) & 1) ^ 1;
          const int krow = seq0 + j * kBlk;
          if (!(ok = mbar_wait(k_empty + st, ph, 8 * tmo))) break;
          mbar_expect_tx(k_full + st, kTile);
          load_tile(sK + st * kTile, &tm_qkv, k_full + st, colq + kD, krow);
          if (!(ok = mbar_wait(v_empty + st, ph, 8 * tmo))) break;
          mbar_expect_tx(v_full + st, kTile);
          load_tile(sV + st * kTile, &tm_qkv, v_full + st, colq + 2 * kD, krow);
        }
        // Only now, with the item's last loads on their way, ask for the next item: a CTA that took one item ahead
        // would hold it back from a CTA that is free sooner.
        if (ok && (ok = mbar_wait(clc_empty, clc_phase ^ 1, 8 * tmo))) {
          mbar_expect_tx(clc_full, 16);
          clc_try_cancel(clc_resp, clc_full);
          more = next_item(w);
          mbar_arrive(clc_empty);
        }
        if (!ok) report(a.status, kErrAttn + 1, w.hi, c);
      }
    } else if (warp == 1 && elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_pv = make_idesc_bf16(128, 128, 0, 1);
      const uint64_t dq = desc_kmajor(smem_u32(sQ), 0), dk = desc_kmajor(smem_u32(sK), 0);
      const uint64_t dv = desc_mnmajor(smem_u32(sV), 0);
      constexpr uint64_t kTileOff = (uint64_t)(kTile >> 4);
      uint32_t kc = 0, vc = 0;        // K / V tiles consumed so far
      uint32_t qc[2] = {0, 0}, pc[2] = {0, 0};
      bool ok = true, more = true;
      auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t code, uint32_t d) -> bool {
        if (mbar_wait(bar, parity, 8 * tmo)) {
          tc_fence_after_sync();
          return true;
        }
        report(a.status, kErrAttn + code, d, kc);
        return false;
      };
      auto issue_s = [&](int t) {
        const uint64_t dqt = dq + t * kTileOff, dkt = dk + (kc & 1) * kTileOff;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint64_t off = (uint64_t)(((k >> 2) * kHalf + (k & 3) * 32) >> 4);
          umma_f16(tmem + t * 128, dqt + off, dkt + off, idesc_s, k != 0);
        }
        umma_commit(s_full + t);
      };
      while (ok && more) {
        const int n[2] = {w.n0, w.n1};
        for (int t = 0; t < 2 && ok; ++t) {
          if (n[t] == 0) continue;
          if (!(ok = wait(q_full + t, qc[t] & 1, 2, t))) break;
          ++qc[t];
          if (t == 0 && !(ok = wait(k_full + (kc & 1), (kc >> 1) & 1, 2, 2))) break;
          issue_s(t);
          if (n[t] == 1) umma_commit(q_empty + t);
        }
        if (!ok) break;
        umma_commit(k_empty + (kc & 1));
        ++kc;
        for (int j = 0; j < n[0] && ok; ++j) {
          if (!(ok = wait(v_full + (vc & 1), (vc >> 1) & 1, 4, 2))) break;
          const uint64_t dvs = dv + (vc & 1) * kTileOff;
          const bool both = j < n[1], both_next = j + 1 < n[1];
          for (int t = 0; t < 2; ++t) {
            if (j >= n[t]) continue;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              if (ok) ok = wait(p_ready + 2 * t + half, pc[t] & 1, 4, t);
              if (ok) {
#pragma unroll
                for (int k = half * 6; k < 6 + half * 2; ++k)   // 16 bf16 of a row of P = 8 TMEM columns per step
                  umma_f16_ts(tmem + 256 + t * 128, tmem + t * 128 + k * 8, dvs + (uint64_t)((k * 2048) >> 4), idesc_pv,
                              (j | k) != 0);
              }
            }
            if (!ok) break;
            ++pc[t];
            if (t == 1 || !both) umma_commit(v_empty + (vc & 1));
            if (j + 1 == n[t]) {
              umma_commit(o_done + t);
              continue;
            }
            if (t == 0 && !(ok = wait(k_full + (kc & 1), (kc >> 1) & 1, 3, t))) break;
            issue_s(t);
            if (j + 2 == n[t]) umma_commit(q_empty + t);
            if (t == 1 || !both_next) umma_commit(k_empty + (kc & 1));
          }
          ++vc;
          if (j + 1 < n[0]) ++kc;
        }
        if (ok) {
          more = next_item(w);
          mbar_arrive(clc_empty);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFwd2RegsHigh));
    // ---------------- softmax / output: one thread per query row ----------------
    const int t = (warp >> 2) - 1;            // this warpgroup's tile
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;           // row inside the tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t ts = tmem + t * 128 + lane_off, to = tmem + 256 + t * 128 + lane_off;
    const float sl2 = a.scale * kLog2e;
    const uint64_t sl2x2 = f32x2(sl2, sl2);
    uint8_t* stage = sO + (warp - 4) * kFwdWarpStage;
    uint32_t sc = 0, oc = 0;                  // S tiles / outputs of this tile so far
    bool ok = true, more = true;
    FwdItem w = fwd_item(a, blockIdx.x, blockIdx.y, blockIdx.z, group);
    while (more) {
      const int n_kv = t == 0 ? w.n0 : w.n1, i_blk = w.hi - t;
      float m_used = -INFINITY, l = 0.f;
      for (int j = 0; j < n_kv; ++j, ++sc) {
        if (!warp_wait(s_full + t, sc & 1, 8 * tmo)) {
          if (lane == 0) report(a.status, kErrAttn + 5, j, t);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        // the masked forms run for the diagonal block only: the other blocks carry no mask arithmetic
        const bool diag = a.causal && j == i_blk;
        uint32_t r[4][32];
        float mc[4];
        // the whole row with one wait: four loads in flight
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(ts + c * 32, r[c]);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float m0 = __uint_as_float(r[c][0]), m1 = __uint_as_float(r[c][1]);
#pragma unroll
          for (int i = 2; i + 3 < 32; i += 4) {
            m0 = max3(m0, __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
            m1 = max3(m1, __uint_as_float(r[c][i + 2]), __uint_as_float(r[c][i + 3]));
          }
          mc[c] = max3(fmaxf(m0, m1), __uint_as_float(r[c][30]), __uint_as_float(r[c][31]));
        }
        if (diag) {
          mc[0] = __uint_as_float(r[0][0]);
          mc[1] = mc[2] = mc[3] = -INFINITY;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i <= row) mc[c] = fmaxf(mc[c], __uint_as_float(r[c][i]));
        }
        const float m_blk = fmaxf(fmaxf(mc[0], mc[1]), fmaxf(mc[2], mc[3])) * sl2;
        if (j == 0) {
          m_used = m_blk;
        } else {
          // S_j is complete, hence P_{j-1} V_{j-1} is too: O may be rescaled in place
          const float m_new = fmaxf(m_used, m_blk);
          const bool need = (m_new - m_used) > 8.0f;
          if (__any_sync(0xffffffffu, need)) {
            const float alpha = need ? exp2f(m_used - m_new) : 1.0f;
            if (need) {
              l *= alpha;
              m_used = m_new;
            }
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t o[32];
              tmem_ld_32x32(to + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32(to + c * 32, o);
            }
          }
        }
        const uint64_t neg_m = f32x2(-m_used, -m_used);
        uint64_t sum[4];
        auto add_quarter = [&](int c) {
          sum[c] = f32x2(__uint_as_float(r[c][0]), __uint_as_float(r[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2)
            sum[c] = add2(sum[c], f32x2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])));
        };
        auto probabilities = [&](auto masked) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              float x0, x1;
              split(fma2(f32x2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), sl2x2, neg_m), x0, x1);
              x0 = fast_exp2(x0);
              x1 = fast_exp2(x1);
              if (masked.value) {
                if (c * 32 + i > row) x0 = 0.f;
                if (c * 32 + i + 1 > row) x1 = 0.f;
              }
              r[c][i] = __float_as_uint(x0);
              r[c][i + 1] = __float_as_uint(x1);
              pk[i >> 1] = pack_bf16(x0, x1);
            }
            // P columns [32c, 32c+32) as bf16 = TMEM columns [16c, 16c+16): over S columns already read
            tmem_st_32x16(ts + c * 16, pk);
            if (c < 2) add_quarter(c);
            if (c >= 2) {
              tmem_st_wait();
              tc_fence_before_sync();
              mbar_arrive(p_ready + 2 * t + c - 2);
            }
          }
        };
        if (diag) probabilities(std::true_type{});
        else probabilities(std::false_type{});
        // the row's sum; its second half is off the chain that the products wait for
        add_quarter(2);
        add_quarter(3);
        float s0, s1;
        split(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])), s0, s1);
        l += s0 + s1;
      }
      if (ok && n_kv > 0) {
        if (!warp_wait(o_done + t, oc & 1, 8 * tmo)) {
          if (lane == 0) report(a.status, kErrAttn + 7, t, 0);
          ok = false;
        }
        ++oc;
      }
      if (!ok) break;
      if (n_kv > 0) {
        tc_fence_after_sync();
        const float inv = 1.0f / l;
        // The warp's 32 rows leave through shared memory, 64 columns at a time, as TMA stores: nothing here waits for
        // the memory system (with plain stores a warp stalls when all SMs write their items at the same time).
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t o[2][32];
          tmem_ld_32x32(to + half * 64, o[0]);
          tmem_ld_32x32(to + half * 64 + 32, o[1]);
          warp_stage_free();
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 u;
              u.x = pack_bf16(__uint_as_float(o[c][q * 8 + 0]) * inv, __uint_as_float(o[c][q * 8 + 1]) * inv);
              u.y = pack_bf16(__uint_as_float(o[c][q * 8 + 2]) * inv, __uint_as_float(o[c][q * 8 + 3]) * inv);
              u.z = pack_bf16(__uint_as_float(o[c][q * 8 + 4]) * inv, __uint_as_float(o[c][q * 8 + 5]) * inv);
              u.w = pack_bf16(__uint_as_float(o[c][q * 8 + 6]) * inv, __uint_as_float(o[c][q * 8 + 7]) * inv);
              *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + q) ^ (lane & 7)) << 4)) = u;   // 128-byte swizzle
            }
          warp_store_box(&tm_out, stage, w.h * kD + half * 64, w.b * a.seq + i_blk * kBlk + q4 * 32);
        }
        a.lse[((int64_t)w.b * a.heads + w.h) * a.seq + i_blk * kBlk + row] = m_used * kLn2 + logf(l);
      }
      more = next_item(w);
      __syncwarp();                              // every lane has read the response
      if (lane == 0) mbar_arrive(clc_empty);
    }
    if (lane == 0) bulk_wait_all<0>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// ==========================================================================================
// backward
// ==========================================================================================
// delta[b, h, s] = -rowsum(dO * O) * scale and lse2[b, h, s] = -lse * log2(e): scaled and negated so that the
// element-wise passes of the backward kernels need one multiply-add each for the exponent and for dP * scale - delta.
// Bound by HBM (it reads O and dO once): 16 lanes with a 16-byte vector each take one head of kDeltaRows consecutive
// tokens, all loads requested before the first sum, and write neighbouring statistics.  33.5 M elements, cold: 52 us
// with a warp per (token, head) and 8 bytes per lane, 26 us so.
// kWide: `out` is 16-byte aligned (dout always is: the host refuses other addresses).
constexpr int kDeltaRows = 4;
static_assert(kBlk % kDeltaRows == 0, "sequences are whole groups of rows");
template <bool kWide>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const uint4* out, const uint4* dout, float* delta,
                  uint32_t groups, uint32_t seq, uint32_t heads, const float* lse, float* lse2,
                  float scale) {
  grid_wait();
  grid_trigger();
  const uint32_t sub = threadIdx.x & 15;
  const uint32_t w = blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4);   // (group of tokens, head)
  const bool live = w < groups;
  const uint32_t tg = w / heads, h = w - tg * heads;
  const int64_t t0 = (int64_t)tg * kDeltaRows;
  uint4 o[kDeltaRows], d[kDeltaRows];
#pragma unroll
  for (int i = 0; i < kDeltaRows; ++i) {
    o[i] = d[i] = make_uint4(0u, 0u, 0u, 0u);
    if (live) {
      const int64_t at = ((t0 + i) * heads + h) * 16 + sub;
      if (kWide) {
        o[i] = ld_stream(out + at);
      } else {
        const uint2* p = reinterpret_cast<const uint2*>(out) + at * 2;
        const uint2 lo = ld_stream(p), hi = ld_stream(p + 1);
        o[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
      }
      d[i] = ld_stream(dout + at);
    }
  }
  float mine = 0.f;                      // the sum of row `sub`
#pragma unroll
  for (int i = 0; i < kDeltaRows; ++i) {
    const uint32_t ov[4] = {o[i].x, o[i].y, o[i].z, o[i].w}, dv[4] = {d[i].x, d[i].y, d[i].z, d[i].w};
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      s += __uint_as_float(ov[k] << 16) * __uint_as_float(dv[k] << 16) +
           __uint_as_float(ov[k] & 0xffff0000u) * __uint_as_float(dv[k] & 0xffff0000u);
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (sub == i) mine = s;
  }
  if (live && sub < kDeltaRows) {
    const uint32_t b = tg / (seq / kDeltaRows);
    const int64_t idx = ((int64_t)b * heads + h) * seq + (t0 - (int64_t)b * seq) + sub;
    delta[idx] = -mine * scale;
    lse2[idx] = -lse[idx] * kLog2e;
  }
}

// ==========================================================================================
// backward: deterministic, P / dS stay in tensor memory
// ==========================================================================================
// The gradient is split by who accumulates it:
//   key-major    an item is 128 KEYS, whose CTA walks the query blocks and accumulates dV, dK in TMEM
//   query-major  an item is 128 QUERIES, whose CTA walks the key blocks and accumulates dQ in TMEM
// Both recompute S and dP (7 products per block pair instead of 5), but nothing is ever added to
// global memory: no fp32 dQ buffer, no memset, no atomics, and the result is bit-identical from run
// to run.  P and dS are written back over S and dP as packed bf16 and feed the gradient products
// as the TMEM (A) operand: they never touch shared memory.
//
// The products use full 128-wide blocks (eight instructions of 64 cycles each) and the kernels are organised
// around keeping the tensor pipe fed: the element-wise work is split in two phases (P from S; dS from
// dP and P) and the MMA warp issues the next block's S (and dP) where they do not depend on this block's phases:
//   key-major    P(i)? dV(i) S(i+1) | dS(i)? dK(i) dP(i+1) | ...       P^T is written over S^T, so S(i+1) follows dV(i)
//   query-major  S(j) read? S(j+1) dP(j+1) | dS(j)? dQ(j) | ...        P stays in registers: S is free once it is read
// Blocks follow one another across items: the next item's first S is issued like the next block's.
//
//   warp 0      TMA: the resident tile that S reads (K or Q), the three-stage ring of Q (with lse2) or K; asks for the next
//               item (cluster launch control, as in forward)
//   warp 18     TMA: the resident tile that dP reads (V or dO), the two-stage ring of dO (with delta) or V
//   warp 1      MMA issuer
//   warps 2-17  element-wise: four threads per TMEM lane, 32 of the 128 columns each
//
// What bounds it: the power cap first (1.4 to 1.65 GHz under these kernels: a block pair saved from waiting gives back half
// of it in clock), then, key-major, the chain S -> P -> dV -> S' (2750 cycles a pair, 2048 of them products) and, query-major,
// the 2000 cycles that a 32 KiB tile takes from L2 while every SM loads (1780 a pair, 1536 of products): K is held from the
// load to dQ, two blocks later, so its ring is the deeper one, and either ring has a producer of its own, because a stage of
// one is often free long before one of the other.  The place for that comes from the output: it is staged in the stage of
// the item's last dO or V.  Sixteen warps share a phase, each thread reads its 32 columns with one load and keeps P in fp32
// registers for dS; P^T is handed over in two parts.  Key-major, statistics vary along the columns: in the layout of a matrix
// fragment a thread has 8 different columns and not 32, so 8 shared loads of 8 bytes replace 16 of 16 (1590 wavefronts a pair
// became 490), and two exponentials of eight run on the FMA pipe (none of eight 363 -> 381 us, two 350, three 390 thousand
// cycles for the first case below).
// With one producer, rings of two stages each and a staging area: batch 4 x 2048, 32 heads, causal, 217 (key-major) and
// 173 us (query-major), now 219 and 165 (429 -> 421 us with the row sums); full 737 -> 716, 16 heads x 8192 causal 709 -> 671.
// The response is given back before the output leaves, not behind its copy: batch 64 x 128, 32 heads, full, forward and backward
// 206 -> 192 us (194 with the staging area).
// P^T through shared memory, so that S(i+1) need not wait for dV(i): no faster (3500 cycles; Q's ring has two stages then).
constexpr int kBwdPoly = 2;                 // key-major: exponentials of every eight that run on the FMA pipe
constexpr int kBwdWarps = 16;               // element-wise warps
constexpr int kBwdCols = kBlk * 4 / kBwdWarps;   // columns of a row per element-wise thread
constexpr int kBwdStage = 32 * kBwdCols * 2;     // output staging per element-wise warp
constexpr int kStatBytes = kBlk * 4;        // lse2 or delta of 128 queries
constexpr int kBwdAlignSlack = 256;
constexpr size_t kBwdBars = 7 * kTile + 5 * kStatBytes;   // where the barriers are
constexpr size_t kBwd2Smem = kBwdBars + 256 + kBwdAlignSlack;
static_assert(kBwdWarps * kBwdStage == kTile, "an item's staged output takes the place of a tile");
static_assert(kBwd2Smem <= 232448, "shared memory of a CTA");
constexpr int kBwd2Threads = 96 + 32 * kBwdWarps;

struct Bwd2Args {
  const float* lse2;    // -lse * log2(e)          (written by attn_delta_kernel)
  const float* delta;   // -rowsum(dO * O) * scale (written by attn_delta_kernel)
  uint32_t items;       // item i < items is key-major, items + i query-major
  int group;            // batch-heads of a block-order group
  int batch, seq, heads, causal;
  float scale;
  uint32_t* status;
  uint64_t timeout_ns;
};

struct BwdItem {
  int b, h, blk, i0, n_it;   // sequence, head, owned block, first streamed block, streamed blocks
};
template <bool kKeyMajor>
__device__ __forceinline__ BwdItem bwd_item(const Bwd2Args& a, uint32_t item) {
  BwdItem w;
  const uint32_t nblk = (uint32_t)a.seq / kBlk, i = kKeyMajor ? item : item - a.items, row = i / (uint32_t)a.group;
  const int bh = (int)(row / nblk) * a.group + (int)(i - row * (uint32_t)a.group), y = (int)(row % nblk);
  w.b = bh / a.heads;
  w.h = bh - w.b * a.heads;
  // same block order as the forward kernel: per group of batch-heads the longest tiles first (key block 0 / the
  // last query block stream the most); queries i0 .. nblk-1 for a key block, keys 0 .. blk for a query block
  w.blk = kKeyMajor || !a.causal ? y : (int)nblk - 1 - y;
  w.i0 = kKeyMajor && a.causal ? w.blk : 0;
  w.n_it = kKeyMajor ? (int)nblk - w.i0 : (a.causal ? w.blk + 1 : (int)nblk);
  return w;
}

// A CTA's run of items of one kind, from `item` on, until cluster launch control has none left or one of the other kind (the
// response stays in shared memory).  False after a timeout.  At its end every copy and every tcgen05 operation has arrived
// where it was announced, so the barriers can be set up anew for the next run.
// kKeyMajor = true:  resident tiles K, V (this item's 128 keys), streamed Q, dO; accumulators dV, dK.
//                    TMEM lanes = keys, columns = queries: lse / delta vary along the columns.
// kKeyMajor = false: resident tiles Q, dO (this item's 128 queries), streamed K, V; accumulator dQ.
//                    TMEM lanes = queries, columns = keys: lse / delta are per thread.
template <bool kKeyMajor>
__device__ __forceinline__ bool attn_bwd2_run(const CUtensorMap& tm_qkv, const CUtensorMap& tm_do, const CUtensorMap& tm_dqkv,
                                              const Bwd2Args& a, uint8_t* smem, uint32_t tmem, uint32_t item) {
  uint8_t* sR0 = smem;                      // resident: K (key-major) or Q
  uint8_t* sR1 = smem + kTile;              // resident: V (key-major) or dO
  // Streamed tiles, a ring each.  Q / K is read by the first and the last product of a block, dO (key-major) by the
  // second and third, V (query-major) by the second alone.
  constexpr uint32_t kRing0 = 3, kRing1 = 2;
  uint8_t* sS0 = smem + 2 * kTile;          // Q or K
  uint8_t* sS1 = smem + 5 * kTile;          // dO or V; between items the stage of an item's last block takes its output
  // key-major: lse2 travels with Q, delta with dO.  delta(i+2) takes the slot of delta(i): its producer waits for dS(i).
  float* sLse = reinterpret_cast<float*>(smem + 7 * kTile);   // [3][128]
  float* sDelta = sLse + 3 * kBlk;                            // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kBwdBars);   // up to 30: the tensor-memory address is behind them
  uint8_t* clc_resp = reinterpret_cast<uint8_t*>(bars);   // 16 bytes
  uint64_t* clc_full = bars + 2;
  uint64_t* clc_empty = bars + 3;
  uint64_t* res_full = bars + 4;            // [2] resident tiles: the one that S reads, the one that dP reads
  uint64_t* res_empty = bars + 6;           // [2]
  uint64_t* full0 = bars + 8;               // [3] rings
  uint64_t* empty0 = bars + 11;             // [3]
  uint64_t* full1 = bars + 14;              // [2]
  uint64_t* empty1 = bars + 16;             // [2]
  uint64_t* s_full = bars + 18;
  uint64_t* s_free = bars + 19;             // query-major: S is in registers
  uint64_t* dp_full = bars + 20;            // [2] (key-major uses [0] only)
  uint64_t* ds_ready = bars + 22;           // [2] dS is in TMEM, even and odd blocks
  uint64_t* p_ready = bars + 24;            // [2] key-major: the first / second 16 columns of every warp's P^T
  uint64_t* acc_done = bars + 26;           // [2] key-major: dV / dK; query-major: [1] dQ
  uint64_t* out_read = bars + 28;           // [2] the copy engine has read the output staged in a stage of ring 1

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint64_t tmo = a.timeout_ns;

  if (threadIdx.x == 0) {
    mbar_init(clc_full, 1);
    mbar_init(clc_empty, 3 + kBwdWarps);    // producers and MMA thread, element-wise warps
    for (int i = 0; i < 3; ++i) {
      mbar_init(full0 + i, 1);
      mbar_init(empty0 + i, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, kBwdWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(res_full + i, 1);
      mbar_init(res_empty + i, 1);
      mbar_init(full1 + i, 1);
      mbar_init(empty1 + i, 1);
      mbar_init(dp_full + i, 1);
      mbar_init(ds_ready + i, kBwdWarps);
      mbar_init(p_ready + i, kBwdWarps);
      mbar_init(acc_done + i, 1);
      mbar_init(out_read + i, kBwdWarps);
    }
    mbar_fence_init();
  }
  __syncthreads();
  // key-major:   S^T [0,128)  dP^T [128,256)  dV [256,384)  dK [384,512)
  // query-major: S [0,128)  dP buffers [128,256) [256,384)  dQ [384,512)
  const uint32_t t_dp = tmem + 128;
  const auto dp_buf = [](uint32_t q) -> uint32_t { return kKeyMajor ? 0 : q & 1; };         // of streamed block q
  const auto dp_phase = [](uint32_t q) -> uint32_t { return (kKeyMajor ? q : q >> 1) & 1; };
  const uint32_t t_acc0 = tmem + (kKeyMajor ? 256 : 384), t_acc1 = tmem + 384;

  BwdItem w = bwd_item<kKeyMajor>(a, item);
  bool ok = true;
  // The next item as the producer got it: false when there is none of this kind (or on a timeout).
  uint32_t items = 0;                       // items finished by this thread
  auto next_item = [&]() -> bool {
    uint32_t x, y, z;
    if (!mbar_wait(clc_full, items & 1, 8 * tmo)) {
      report(a.status, kErrAttn + 18, items, 0);
      ok = false;
      return false;
    }
    ++items;
    const bool more = clc_read(clc_resp, x, y, z) && (x < a.items) == kKeyMajor;
    fence_proxy_async_smem();               // this read before the next response overwrites it
    if (more) w = bwd_item<kKeyMajor>(a, x);
    return more;
  };
  uint32_t g = 0;                           // streamed blocks so far: stages and phases of the rings and the hand-overs

  if (warp == 0) {
    // resident tile of S, ring of Q or K, next items
    if (elect_one()) {
      bool more = true;
      while (ok && more) {
        const int colq = w.h * 3 * kD, seq0 = w.b * a.seq, rrow = seq0 + w.blk * kBlk;
        const int64_t stat0 = ((int64_t)w.b * a.heads + w.h) * a.seq;
        // the resident tile of S first, then the item's first streamed tile: S needs no more
        for (int it = -1; it < w.n_it && ok; ++it) {
          if (it < 0) {
            if (!(ok = mbar_wait(res_empty, (items & 1) ^ 1, 8 * tmo))) break;
            mbar_expect_tx(res_full, kTile);
            load_tile(sR0, &tm_qkv, res_full, kKeyMajor ? colq + kD : colq, rrow);           // K or Q
            continue;
          }
          const uint32_t st = g % kRing0;
          const int srow = (w.i0 + it) * kBlk;
          if (!(ok = mbar_wait(empty0 + st, ((g / kRing0) & 1) ^ 1, 8 * tmo))) break;
          mbar_expect_tx(full0 + st, kTile + (kKeyMajor ? kStatBytes : 0));
          load_tile(sS0 + st * kTile, &tm_qkv, full0 + st, kKeyMajor ? colq : colq + kD, seq0 + srow);
          if (kKeyMajor) bulk_g2s(sLse + st * kBlk, a.lse2 + stat0 + srow, kStatBytes, full0 + st);
          ++g;
        }
        if (ok && (ok = mbar_wait(clc_empty, (items & 1) ^ 1, 8 * tmo))) {
          mbar_expect_tx(clc_full, 16);
          clc_try_cancel(clc_resp, clc_full);
          more = next_item();
          mbar_arrive(clc_empty);
        }
      }
      // what is still under way (a timeout above is reported here too)
      for (uint32_t q = g; q < g + kRing0 && ok; ++q) ok = mbar_wait(empty0 + q % kRing0, ((q / kRing0) & 1) ^ 1, 8 * tmo);
      ok = ok && mbar_wait(res_empty, (items & 1) ^ 1, 8 * tmo);
      if (!ok) report(a.status, kErrAttn + 11, w.blk, g);
    }
  } else if (warp == 2 + kBwdWarps) {
    // resident tile of dP, ring of dO or V: by a thread of its own, because a stage of one ring is often free long before one of the other
    if (elect_one()) {
      bool more = true;
      uint32_t outs[2] = {0, 0};              // outputs staged in either stage so far
      bool staged[2] = {false, false};        // the last user of the stage was an item's output
      while (ok && more) {
        const int seq0 = w.b * a.seq, rrow = seq0 + w.blk * kBlk;
        const int64_t stat0 = ((int64_t)w.b * a.heads + w.h) * a.seq;
        if ((ok = mbar_wait(res_empty + 1, (items & 1) ^ 1, 8 * tmo))) {
          mbar_expect_tx(res_full + 1, kTile);
          if (kKeyMajor) load_tile(sR1, &tm_qkv, res_full + 1, w.h * 3 * kD + 2 * kD, rrow);     // V
          else load_tile(sR1, &tm_do, res_full + 1, w.h * kD, rrow);                            // dO
        }
        for (int it = 0; it < w.n_it && ok; ++it, ++g) {
          const uint32_t st = g % kRing1;
          const int srow = (w.i0 + it) * kBlk;
          if (!(ok = mbar_wait(empty1 + st, ((g / kRing1) & 1) ^ 1, 8 * tmo))) break;
          if (staged[st] && !(ok = mbar_wait(out_read + st, (outs[st] - 1) & 1, 8 * tmo))) break;
          staged[st] = false;
          mbar_expect_tx(full1 + st, kTile + (kKeyMajor ? kStatBytes : 0));
          if (kKeyMajor) {
            load_tile(sS1 + st * kTile, &tm_do, full1 + st, w.h * kD, seq0 + srow);                                // dO
            if (g > 1 && !(ok = mbar_wait(ds_ready + st, ((g - 2) >> 1) & 1, 8 * tmo))) break;
            bulk_g2s(sDelta + st * kBlk, a.delta + stat0 + srow, kStatBytes, full1 + st);
          } else {
            load_tile(sS1 + st * kTile, &tm_qkv, full1 + st, w.h * 3 * kD + 2 * kD, seq0 + srow);                  // V
          }
        }
        if (ok) {
          const uint32_t st = (g - 1) % kRing1;
          staged[st] = true;
          ++outs[st];
        }
        if (ok) {
          more = next_item();
          mbar_arrive(clc_empty);
        }
      }
      for (uint32_t q = g; q < g + kRing1 && ok; ++q) ok = mbar_wait(empty1 + q % kRing1, ((q / kRing1) & 1) ^ 1, 8 * tmo);
      ok = ok && mbar_wait(res_empty + 1, (items & 1) ^ 1, 8 * tmo);
      if (!ok) report(a.status, kErrAttn + 11, w.blk, g);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t id_s = make_idesc_bf16(128, 128, 0, 0);      // A K-major (smem) * B K-major
      const uint32_t id_g = make_idesc_bf16(128, 128, 0, 1);      // A (TMEM) * B MN-major
      // descriptors of the first k-step of each operand; the others are these plus constants
      const uint64_t dr0 = desc_kmajor(smem_u32(sR0), 0), dr1 = desc_kmajor(smem_u32(sR1), 0);
      const uint64_t ds0k = desc_kmajor(smem_u32(sS0), 0), ds1k = desc_kmajor(smem_u32(sS1), 0);
      const uint64_t ds0m = desc_mnmajor(smem_u32(sS0), 0), ds1m = desc_mnmajor(smem_u32(sS1), 0);
      constexpr uint64_t kStageOff = (uint64_t)(kTile >> 4);
      bool more = true;
      auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t code) -> bool {
        if (mbar_wait(bar, parity, 8 * tmo)) {
          tc_fence_after_sync();
          return true;
        }
        report(a.status, kErrAttn + code, g, items);
        return false;
      };
      // S (or S^T) / dP (or dP^T) of streamed block number q, once its tile is there and the block before is out of S (key-major:
      // the products that read its P^T were issued before)
      auto issue_s = [&](uint32_t q) -> bool {
        const uint32_t st = q % kRing0;
        if (!kKeyMajor && q > 0 && !wait(s_free, (q - 1) & 1, 19)) return false;
        if (!wait(full0 + st, (q / kRing0) & 1, 13)) return false;
        const uint64_t tile = ds0k + st * kStageOff;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint64_t off = (uint64_t)(((k >> 2) * kHalf + (k & 3) * 32) >> 4);
          umma_f16(tmem, dr0 + off, tile + off, id_s, k != 0);
        }
        umma_commit(s_full);
        return true;
      };
      auto issue_dp = [&](uint32_t q) -> bool {
        const uint32_t st = q % kRing1;
        if (!wait(full1 + st, (q / kRing1) & 1, 13)) return false;
        const uint64_t tile = ds1k + st * kStageOff;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint64_t off = (uint64_t)(((k >> 2) * kHalf + (k & 3) * 32) >> 4);
          umma_f16(t_dp + dp_buf(q) * 128, dr1 + off, tile + off, id_s, k != 0);
        }
        umma_commit(dp_full + dp_buf(q));
        if (!kKeyMajor) umma_commit(empty1 + st);         // V has no other reader
        return true;
      };
      // The first blocks of an item also wait for its resident tiles.  An item's last products of either kind free them.
      auto first_s = [&](uint32_t q) -> bool {
        if (!(wait(res_full, items & 1, 12) && issue_s(q))) return false;
        if (w.n_it == 1) umma_commit(res_empty);
        return true;
      };
      auto first_dp = [&](uint32_t q) -> bool {
        if (!(wait(res_full + 1, items & 1, 12) && issue_dp(q))) return false;
        if (w.n_it == 1) umma_commit(res_empty + 1);
        return true;
      };
      // acc += (P or dS in TMEM at `src`: a warp's columns packed from its first column) * streamed tile; the k-steps
      // of the first / second 16 columns of every warp
      auto issue_grad = [&](uint32_t acc, uint32_t src, uint64_t tile, int part, bool first) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          umma_f16_ts(acc, src + i * kBwdCols + part * 8, tile + (uint64_t)(((2 * i + part) * 2048) >> 4), id_g,
                      !(first && i == 0));
      };
      // Blocks follow one another across items: the next item's first S is issued where the next block's would be, and its
      // first dP behind this item's last product.
      ok = first_s(g) && first_dp(g);
      while (ok && more) {
        const int n = w.n_it;
        for (int it = 0; it < n && ok; ++it, ++g) {
          const bool last = it + 1 == n;
          const uint32_t st0 = g % kRing0, st1 = g % kRing1;
          if (kKeyMajor) {
            // dV += P^T dO (contraction over the queries)
            if (!(ok = wait(p_ready, g & 1, 14))) break;
            issue_grad(t_acc0, tmem, ds1m + st1 * kStageOff, 0, it == 0);
            if (!(ok = wait(p_ready + 1, g & 1, 14))) break;
            issue_grad(t_acc0, tmem, ds1m + st1 * kStageOff, 1, false);
            umma_commit(empty1 + st1);
            if (last) umma_commit(acc_done);
          }
          if (!last) {
            if (!(ok = issue_s(g + 1))) break;
            if (it + 2 == n) umma_commit(res_empty);
            if (!kKeyMajor) {
              if (!(ok = issue_dp(g + 1))) break;
              if (it + 2 == n) umma_commit(res_empty + 1);
            }
          } else {
            more = next_item();                           // w is the next item's from here on
            mbar_arrive(clc_empty);
            if (more && !(ok = first_s(g + 1))) break;
          }
          if (!(ok = wait(ds_ready + (g & 1), (g >> 1) & 1, 14))) break;
          const uint32_t acc = kKeyMajor ? t_acc1 : t_acc0, ds = t_dp + dp_buf(g) * 128;
          issue_grad(acc, ds, ds0m + st0 * kStageOff, 0, it == 0);     // dK += dS^T Q / dQ += dS K
          issue_grad(acc, ds, ds0m + st0 * kStageOff, 1, false);
          umma_commit(empty0 + st0);
          if (last) umma_commit(acc_done + 1);
          if (last) {
            if (more && !(ok = first_dp(g + 1))) break;
          } else if (kKeyMajor) {
            if (!(ok = issue_dp(g + 1))) break;
            if (it + 2 == n) umma_commit(res_empty + 1);
          }
        }
      }
    }
  } else {
    const int q4 = warp & 3;
    const int part = (warp - 2) >> 2;                     // which kBwdCols of the 128 columns
    const int row = q4 * 32 + lane;                       // TMEM lane: key (key-major) or query
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const uint64_t sl2 = f32x2(a.scale * kLog2e, a.scale * kLog2e), sc2 = f32x2(a.scale, a.scale);
    bool more = true;
    while (more) {
      const int me = w.blk * kBlk + row;                  // query-major: this lane's query
      const int me0 = w.blk * kBlk + q4 * 32 + (lane >> 2);   // key-major: the first of this thread's keys
      uint64_t my_lse2 = 0, my_delta = 0;
      if (!kKeyMajor) {
        const int64_t at = ((int64_t)w.b * a.heads + w.h) * a.seq + me;
        my_lse2 = f32x2(a.lse2[at], a.lse2[at]);
        my_delta = f32x2(a.delta[at], a.delta[at]);
      }
      for (int it = 0; it < w.n_it; ++it, ++g) {
        const uint32_t ts = tmem + lane_off + part * kBwdCols, tdp = ts + 128 + dp_buf(g) * 128;
        const int c0 = (w.i0 + it) * kBlk + part * kBwdCols;   // first streamed index of this thread's columns
        const uint32_t st0 = g % kRing0;
        // key-major: lse2 / delta of this thread's columns
        const float* my_lse = sLse + st0 * kBlk + part * kBwdCols + (lane & 3) * 2;
        const float* my_dlt = sDelta + (g & 1) * kBlk + part * kBwdCols + (lane & 3) * 2;
        // causal: a score survives when key <= query; only blocks that touch the diagonal pay for it
        const bool masked = a.causal && (kKeyMajor ? (c0 < me0 + 24) : (c0 + kBwdCols - 1 > me));
        float e[kBwdCols];                                // P of this thread's columns
        // ---- phase 1: P = exp2(S * scale * log2(e) - lse2) ----
        // (key-major: lse2 comes with Q and delta with dO, whose barriers order them for this thread)
        if (!warp_wait(s_full, g & 1, 8 * tmo) || (kKeyMajor && !warp_wait(full0 + st0, (g / kRing0) & 1, 8 * tmo))) {
          if (lane == 0) report(a.status, kErrAttn + 15, it, 0);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        {
          uint32_t rs[kBwdCols];
          if (kKeyMajor) {
            tmem_ld_16x32_frag(ts, rs);
            tmem_ld_16x32_frag(ts + (16u << 16), rs + 16);
          } else {
            tmem_ld_32x32(ts, rs);
          }
          tmem_ld_wait();
          if (!kKeyMajor) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_free);           // the next block's S may be computed
          }
          uint64_t st[4] = {my_lse2, my_lse2, my_lse2, my_lse2};
          if (kKeyMajor) {
#pragma unroll
            for (int n = 0; n < 4; ++n) st[n] = *reinterpret_cast<const uint64_t*>(my_lse + n * 8);
          }
          // key-major: columns of a fragment are in groups n of 8, elements 4 n + {0, 1} of this thread's first row of a
          // lane half, + {2, 3} of its second; by halves of 16 columns, so that P^T can be handed over in two parts
#pragma unroll
          for (int hp = 0; hp < 2; ++hp) {
#pragma unroll
            for (int i = 0; i < kBwdCols / 2; i += 2) {
              const int k = kKeyMajor ? (i >> 3) * 16 + hp * 8 + (i & 7) : hp * 16 + i;
              split(fma2(f32x2(__uint_as_float(rs[k]), __uint_as_float(rs[k + 1])), sl2, st[(k >> 2) & 3]), e[k], e[k + 1]);
              e[k] = kKeyMajor && i % 8 < kBwdPoly ? exp2_fma(e[k]) : fast_exp2(e[k]);
              e[k + 1] = kKeyMajor && i % 8 + 1 < kBwdPoly ? exp2_fma(e[k + 1]) : fast_exp2(e[k + 1]);
            }
            if (masked) {
#pragma unroll
              for (int i = 0; i < kBwdCols / 2; ++i) {
                const int k = kKeyMajor ? (i >> 3) * 16 + hp * 8 + (i & 7) : hp * 16 + i;
                if (kKeyMajor) {
                  const int key = me0 + (k >> 4) * 16 + (k >> 1 & 1) * 8, query = c0 + (k >> 2 & 3) * 8 + (lane & 3) * 2 + (k & 1);
                  if (key > query) e[k] = 0.f;
                } else if (c0 + k > me) {
                  e[k] = 0.f;
                }
              }
            }
            if (kKeyMajor) {
              // P^T over this warp's own S^T columns, packed from the first: the products that read the first 16
              // run under the exponentials of the second
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                uint32_t pk[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pk[i] = pack_bf16(e[h * 16 + hp * 8 + 2 * i], e[h * 16 + hp * 8 + 2 * i + 1]);
                tmem_st_16x16_frag(ts + hp * 8 + ((h * 16u) << 16), pk);
              }
              tmem_st_wait();
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(p_ready + hp);
            }
          }
        }
        // ---- phase 2: dS = P * (dP * scale - delta * scale) ----
        if (!warp_wait(dp_full + dp_buf(g), dp_phase(g), 8 * tmo) ||
            (kKeyMajor && !warp_wait(full1 + (g & 1), (g >> 1) & 1, 8 * tmo))) {
          if (lane == 0) report(a.status, kErrAttn + 16, it, 0);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        {
          uint32_t rp[kBwdCols], dk[16];
          uint64_t st[4] = {my_delta, my_delta, my_delta, my_delta};
          if (kKeyMajor) {
            tmem_ld_16x32_frag(tdp, rp);
            tmem_ld_16x32_frag(tdp + (16u << 16), rp + 16);
#pragma unroll
            for (int n = 0; n < 4; ++n) st[n] = *reinterpret_cast<const uint64_t*>(my_dlt + n * 8);
          } else {
            tmem_ld_32x32(tdp, rp);
          }
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < kBwdCols; k += 2) {
            float g0, g1;
            split(mul2(f32x2(e[k], e[k + 1]),
                       fma2(f32x2(__uint_as_float(rp[k]), __uint_as_float(rp[k + 1])), sc2, st[(k >> 2) & 3])), g0, g1);
            dk[k >> 1] = pack_bf16(g0, g1);
          }
          // dS over this thread's own dP columns
          if (kKeyMajor) {
            tmem_st_16x32_frag(tdp, dk);
            tmem_st_16x32_frag(tdp + (16u << 16), dk + 8);
          } else {
            tmem_st_32x16(tdp, dk);
          }
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(ds_ready + (g & 1));
        }
      }
      if (!ok) break;
      // Accumulators -> bf16 rows of dqkv: a warp's 32 rows x kBwdCols columns leave through shared memory as a TMA store
      // (with plain stores the warps stall for 4000 cycles when all SMs write their items at the same time).
      const int col = w.h * 3 * kD + part * kBwdCols, orow = w.b * a.seq + w.blk * kBlk + q4 * 32;
      const uint32_t phase = items & 1;
      const uint32_t out_st = (g - 1) & 1;
      uint8_t* stage = sS1 + out_st * kTile + (warp - 2) * kBwdStage;   // where the item's last dO or V was
      more = next_item();                        // w is the next item's from here on
      __syncwarp();                              // every lane has read the response: the one after may be asked for now
      if (lane == 0) mbar_arrive(clc_empty);
#pragma unroll 1
      for (int which = kKeyMajor ? 0 : 1; which < 2; ++which) {
        if (!warp_wait(acc_done + which, phase, 8 * tmo)) {
          if (lane == 0) report(a.status, kErrAttn + 17, which, 0);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        // key-major: acc0 = dV, acc1 = dK;  query-major: acc0 = dQ
        uint32_t r[kBwdCols];
        tmem_ld_32x32((kKeyMajor && which ? t_acc1 : t_acc0) + lane_off + part * kBwdCols, r);
        warp_stage_free();
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(r[q * 8 + 0]), __uint_as_float(r[q * 8 + 1]));
          v.y = pack_bf16(__uint_as_float(r[q * 8 + 2]), __uint_as_float(r[q * 8 + 3]));
          v.z = pack_bf16(__uint_as_float(r[q * 8 + 4]), __uint_as_float(r[q * 8 + 5]));
          v.w = pack_bf16(__uint_as_float(r[q * 8 + 6]), __uint_as_float(r[q * 8 + 7]));
          *reinterpret_cast<uint4*>(stage + lane * 64 + ((q ^ (lane >> 1 & 3)) << 4)) = v;   // 64-byte swizzle
        }
        warp_store_box(&tm_dqkv, stage, col + (kKeyMajor ? (which == 0 ? 2 * kD : kD) : 0), orow);
      }
      if (!ok) break;
      if (lane == 0) {
        bulk_wait_read<0>();
        mbar_arrive(out_read + out_st);          // the stage may take a tile again
      }
      tc_fence_before_sync();                    // the accumulators are read before the next P / dS is announced
      __syncwarp();
    }
  }
  tc_fence_before_sync();
  __syncwarp();
  const bool all = __syncthreads_and(ok) != 0;
  tc_fence_after_sync();
  if (threadIdx.x == 0 && all)
    for (int i = 2; i < 30; ++i) mbar_inval(bars + i);
  return all;
}

// A grid of key-major items, of query-major ones, or of both, all key-major items first: there query-major items, which need
// nothing of those, take SMs as they get free, and every CTA has waited for the row sums (and so for all that came before them
// in the stream) before it reads anything.  (Of two launches that overlap by programmatic dependence the second cannot wait for
// the row sums alone.)  A CTA of both kinds changes when cluster launch control gives it an item of the other one, in that
// order at most once; nothing depends on that.
template <bool kKey, bool kQuery>
__global__ void __launch_bounds__(kBwd2Threads, 1)
attn_bwd2_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do,
                 const __grid_constant__ CUtensorMap tm_dqkv, const __grid_constant__ Bwd2Args a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // the base is 1024-byte aligned in practice; there is no room for the full slack of an arbitrary one
  if (smem - smem_raw > kBwdAlignSlack) {
    grid_wait();
    if (threadIdx.x == 0) report(a.status, kErrAttn + 10, 0, 0);
    return;
  }
  uint8_t* clc_resp = smem + kBwdBars;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kBwdBars + 30 * 8);
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_qkv);
    tma_prefetch_desc(&tm_do);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  grid_wait();

  if (kKey && kQuery) {
    uint32_t item = blockIdx.x, y, z;
    bool more = true;
    while (more) {
      const bool ok = item < a.items ? attn_bwd2_run<true>(tm_qkv, tm_do, tm_dqkv, a, smem, tmem, item)
                                     : attn_bwd2_run<false>(tm_qkv, tm_do, tm_dqkv, a, smem, tmem, item);
      more = ok && clc_read(clc_resp, item, y, z);
      fence_proxy_async_smem();             // this read before the next response overwrites it
    }
  } else {
    attn_bwd2_run<kKey>(tm_qkv, tm_do, tm_dqkv, a, smem, tmem, blockIdx.x);
  }
  if (warp >= 2 && warp < 2 + kBwdWarps && lane == 0) bulk_wait_all<0>();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// The shared-memory attribute is per device: set it once on every device that launches.
cudaError_t configure_device() {
  static bool configured[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < 64 && configured[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(attn_fwd2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwd2Smem);
  if (e != cudaSuccess) return e;
  for (auto kernel : {attn_bwd2_kernel<true, true>, attn_bwd2_kernel<true, false>, attn_bwd2_kernel<false, true>}) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwd2Smem);
    if (e != cudaSuccess) return e;
  }
  if (dev >= 0 && dev < 64) configured[dev] = true;
  return cudaSuccess;
}

int sm_count() {
  static int count[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (count[dev] == 0 && cudaDeviceGetAttribute(&count[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return count[dev];
}

// Batch-heads per block-order group: the largest divisor of batch * heads that is at most 32.
int bh_group(int batch, int heads) {
  const int n = batch * heads;
  int g = 1;
  for (int d = 1; d <= 32; ++d)
    if (n % d == 0) g = d;
  return g;
}

}  // namespace

cudaError_t attention_fwd(const void* qkv, void* out, float* lse, int batch, int seq, int heads,
                          int causal, float scale, uint32_t* status, cudaStream_t stream) {
  if (seq % kBlk != 0 || batch <= 0 || heads <= 0 || (int64_t)batch * heads > 65535 || seq / kBlk > 65535)
    return cudaErrorInvalidValue;
  {
    cudaError_t e = configure_device();
    if (e != cudaSuccess) return e;
  }
  CUtensorMap tm;
  const uint64_t width = (uint64_t)heads * 3 * kD;
  if (make_tensor_map_2d(&tm, qkv, width, (uint64_t)batch * seq, width * 2, 64, kBlk) != 0)
    return cudaErrorInvalidValue;
  CUtensorMap to;
  const uint64_t wout = (uint64_t)heads * kD;
  if (make_tensor_map_2d(&to, out, wout, (uint64_t)batch * seq, wout * 2, 64, 32) != 0) return cudaErrorInvalidValue;
  AttnArgs a{};
  a.lse = lse;
  a.batch = batch; a.seq = seq; a.heads = heads; a.causal = causal;
  a.scale = scale;
  a.status = status;
  a.timeout_ns = 2000000000ull;
  const int grp = bh_group(batch, heads);
  const int nblk = seq / kBlk;
  // With no more tiles than SMs a tile per CTA leaves none idle and runs without a neighbour; beyond that pairs share
  // K and V and overlap.  One tile / two, us: 1 head x 8192 (64 tiles) 104 / 114, 8 x 2048 (128) 29.8 / 32.7, batch 3 x 640
  // with 5 heads (75) 12.4 / 14.2, batch 4 x 256 with 16 heads (128) 8.0 / 9.3; causal 104 / 114,
  // 30.0 / 32.8, 13.1 / 14.2 and 8.7 / 8.7.
  a.tiles_per_item = (int64_t)batch * heads * nblk <= sm_count() ? 1 : 2;
  dim3 grid(grp, (nblk + a.tiles_per_item - 1) / a.tiles_per_item, batch * heads / grp);
  return launch_dependent(attn_fwd2_kernel, grid, kFwd2Threads, kFwd2Smem, stream, tm, to, a);
}

cudaError_t attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse,
                          void* dqkv, float* dq_acc, float* delta, int batch, int seq, int heads,
                          int causal, float scale, uint32_t* status, cudaStream_t stream) {
  if (seq % kBlk != 0 || batch <= 0 || heads <= 0 || (int64_t)batch * heads > 65535 || seq / kBlk > 65535)
    return cudaErrorInvalidValue;
  // All that is refused is refused before the first launch: the row-sum kernel reads `dout` 16 and `out` at least 8 bytes
  // at a time, bulk copies read the statistics.
  const auto off = [](const void* p, uintptr_t align) { return (reinterpret_cast<uintptr_t>(p) & (align - 1)) != 0; };
  if (off(qkv, 16) || off(dout, 16) || off(dqkv, 16) || off(out, 8) || off(dq_acc, 16) || off(delta, 16))
    return cudaErrorInvalidValue;
  const int64_t items = (int64_t)batch * heads * (seq / kBlk);   // 256 KiB of tensors each
  if (items > 1 << 29) return cudaErrorInvalidValue;
  {
    cudaError_t e0 = configure_device();
    if (e0 != cudaSuccess) return e0;
  }
  const int64_t tokens = (int64_t)batch * seq;
  CUtensorMap tq, td;
  const uint64_t width = (uint64_t)heads * 3 * kD, wdo = (uint64_t)heads * kD;
  if (make_tensor_map_2d(&tq, qkv, width, (uint64_t)tokens, width * 2, 64, kBlk) != 0) return cudaErrorInvalidValue;
  if (make_tensor_map_2d(&td, dout, wdo, (uint64_t)tokens, wdo * 2, 64, kBlk) != 0) return cudaErrorInvalidValue;
  CUtensorMap tg;
  if (make_tensor_map_2d(&tg, dqkv, width, (uint64_t)tokens, width * 2, kBwdCols, 32, 64) != 0) return cudaErrorInvalidValue;
  {
    // -delta * scale into `delta`, -lse * log2(e) into the head of the `dq_acc` scratch
    const int64_t groups = tokens / kDeltaRows * heads;   // below 2^32: a group is 2 KiB of activations
    const int threads = 256, per_block = threads / 16;
    const int64_t blocks = (groups + per_block - 1) / per_block;
    auto kernel = off(out, 16) ? attn_delta_kernel<false> : attn_delta_kernel<true>;
    const cudaError_t e = launch_dependent(kernel, (unsigned)blocks, threads, 0, stream, reinterpret_cast<const uint4*>(out),
                                           reinterpret_cast<const uint4*>(dout), delta, (uint32_t)groups, (uint32_t)seq,
                                           (uint32_t)heads, lse, dq_acc, scale);
    if (e != cudaSuccess) return e;
  }
  // dK / dV per key block, dQ per query block
  Bwd2Args g{};
  g.lse2 = dq_acc;     // -lse * log2(e)
  g.delta = delta;     // -delta * scale
  g.items = (uint32_t)items;
  g.group = bh_group(batch, heads);
  g.batch = batch; g.seq = seq; g.heads = heads; g.causal = causal;
  g.scale = scale;
  g.status = status;
  g.timeout_ns = 2000000000ull;
  // One launch of both kinds where one kind leaves SMs free, two beyond: the kernel of both is slower by 4 % (96 registers).
  // Backward, two / one, us: batch 3 x 640, 5 heads (75 items) 35.5 / 27.5, 1 x 4096, 4 heads, causal (128) 92 / 63, 2 x 1024,
  // 8 heads (128) 34 / 25.6; 1 x 8192, 4 heads (256) 180 / 183, 1 x 4096, 16 heads (512) 191 / 198, 4 x 2048, 32 heads (2048)
  // 437 / 453, full 809 / 854.
  if (items <= sm_count()) return launch_dependent(attn_bwd2_kernel<true, true>, 2 * (unsigned)items, kBwd2Threads, kBwd2Smem, stream, tq, td, tg, g);
  const cudaError_t e = launch_dependent(attn_bwd2_kernel<true, false>, (unsigned)items, kBwd2Threads, kBwd2Smem, stream, tq, td, tg, g);
  if (e != cudaSuccess) return e;
  g.items = 0;
  return launch_dependent(attn_bwd2_kernel<false, true>, (unsigned)items, kBwd2Threads, kBwd2Smem, stream, tq, td, tg, g);
}

}  // namespace msb
