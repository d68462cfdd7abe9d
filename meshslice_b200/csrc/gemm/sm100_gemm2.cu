// Two-CTA variant of the local tcgen05 GEMM (no fused collectives): a cluster of two CTAs on
// neighbouring SMs computes one 256 x 256 tile with tcgen05.mma.cta_group::2.
//
// Each CTA loads 128 rows of A and 128 of the 256 B columns per k-block (32 KiB instead of 48 KiB
// per stage, so six stages and the output staging fit) and owns the 128 accumulator rows that land in its own TMEM.  Only
// the leader CTA (even rank) issues MMAs; it reads both CTAs' shared memory.  Synchronisation:
//   full[stage]    lives in the leader; both CTAs' TMA loads complete on it (the .cta_group::2
//                  load form with the leader barrier's cluster address); two arrivals: the leader's
//                  A producer and B producer each announce their operand's bytes
//   empty[stage]   one per CTA; one commit of the leader arrives on both
//   tfull[acc]     one per CTA, committed by the leader to both
//   tempty[acc]    lives in the leader, 8 arrivals: one per epilogue warp of both CTAs
// No load uses cluster multicast.  Every wait is bounded as in the one-CTA kernel.
#include <cuda_bf16.h>
#include <string.h>

#include "../common/gelu.cuh"
#include "../common/pdl.cuh"
#include "../common/ptx.cuh"
#include "out_turn.h"
#include "sm100_gemm.h"

namespace msb {

namespace {

constexpr uint32_t kAStage2 = kBM * kBK * 2;        // 16 KiB: this CTA's 128 rows of A
constexpr uint32_t b_stage2(int bn) { return (bn / 2) * kBK * 2; }   // this CTA's half of the tile's columns of B
constexpr uint32_t kOutBox = 32 * 128;              // a staged box: 32 rows of 128 bytes
constexpr uint32_t kOutStage = 4 * 2 * kOutBox;     // two per epilogue warp
constexpr int stages2(int bn) { return bn == 256 ? 6 : 8; }
constexpr uint32_t smem_alloc2(int bn) { return stages2(bn) * (kAStage2 + b_stage2(bn)) + kOutStage + 256 + 1024; }
constexpr int kThreads2 = 224;   // warps: A producer, MMA, 4x epilogue, B producer

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t leader_bar,
                                                 int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint32_t leader_bar,
                                                 int32_t x, int32_t y, int32_t z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(leader_bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the mbarrier at this offset of both CTAs' shared memory once all MMAs issued so far have finished.
__device__ __forceinline__ void umma_commit_both(uint32_t bar_addr) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar_addr), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ uint64_t desc_at(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

__device__ __forceinline__ void report2(const Gemm2Args& a, uint32_t code, uint32_t d0, uint32_t d1) {
  if (atomicCAS(a.status, 0u, code) == 0u) {
    a.status[1] = blockIdx.x;
    a.status[2] = d0;
    a.status[3] = d1;
  }
}

__device__ __forceinline__ float gelu_tanh2(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return 0.5f * x * (1.0f + t);
}
__device__ __forceinline__ uint32_t pk2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float blo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bhi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// Rows are a multiple of 16 bytes apart (ldc % 8 == 0 for both types), but the matrix may start anywhere.
__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

__device__ __forceinline__ void store32(void* base, int64_t ld, bool fp32, bool accumulate, int64_t row,
                                        int col0, int nvalid, float (&v)[32]) {
  if (fp32) {
    float* p = reinterpret_cast<float*>(base) + row * ld + col0;
    if (nvalid == 32 && aligned16(p)) {
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        float4 o = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        if (accumulate) {
          const float4 c = *reinterpret_cast<const float4*>(p + i);
          o.x += c.x; o.y += c.y; o.z += c.z; o.w += c.w;
        }
        *reinterpret_cast<float4*>(p + i) = o;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < nvalid) p[i] = accumulate ? p[i] + v[i] : v[i];
    }
  } else {
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(base) + row * ld + col0;
    if (nvalid == 32 && aligned16(p)) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint4 o;
        if (accumulate) {
          const uint4 c = *reinterpret_cast<const uint4*>(p + i);
          o.x = pk2(v[i] + blo(c.x), v[i + 1] + bhi(c.x));
          o.y = pk2(v[i + 2] + blo(c.y), v[i + 3] + bhi(c.y));
          o.z = pk2(v[i + 4] + blo(c.z), v[i + 5] + bhi(c.z));
          o.w = pk2(v[i + 6] + blo(c.w), v[i + 7] + bhi(c.w));
        } else {
          o.x = pk2(v[i], v[i + 1]);
          o.y = pk2(v[i + 2], v[i + 3]);
          o.z = pk2(v[i + 4], v[i + 5]);
          o.w = pk2(v[i + 6], v[i + 7]);
        }
        *reinterpret_cast<uint4*>(p + i) = o;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (i >= nvalid) continue;
        float x = v[i];
        if (accumulate) x += __bfloat162float(p[i]);
        p[i] = __float2bfloat16_rn(x);
      }
    }
  }
}

// 32 bf16 of a row as packed pairs; columns beyond `nvalid` are not read.
__device__ __forceinline__ void load32(const void* base, int64_t ld, int64_t row, int col0, int nvalid, uint32_t (&v)[16]) {
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(base) + row * ld + col0;
  if (nvalid == 32 && aligned16(p)) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 u = ld_stream(reinterpret_cast<const uint4*>(p) + i);
      v[4 * i] = u.x; v[4 * i + 1] = u.y; v[4 * i + 2] = u.z; v[4 * i + 3] = u.w;
    }
  } else {
    const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      v[i] = (2 * i < nvalid ? q[2 * i] : 0u) | (2 * i + 1 < nvalid ? (uint32_t)q[2 * i + 1] << 16 : 0u);
  }
}

// One box of a tensor map, shared -> global; the second form adds fp32 values to what is there (the sum that a register add
// would give, subnormal values included: test_gemm_fp32_accumulation_keeps_subnormals).
__device__ __forceinline__ void tma_store_box(const CUtensorMap* map, const void* src, int32_t x, int32_t y, bool add) {
  if (add)
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(smem_u32(src)), "r"(x), "r"(y) : "memory");
  else
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(smem_u32(src)), "r"(x), "r"(y) : "memory");
}
// Staging of one epilogue warp: two boxes, each free again once the copy engine has read it.  take() waits for all but
// the last `1 - taken` stores; OutTurn never names the box sent last.  With taken = 1 (the other box may be held unsent) no
// store may be outstanding.
struct OutStage {
  uint8_t* base;
  OutTurn turn;
  template <int taken = 0>
  __device__ __forceinline__ uint8_t* take(int lane) {
    if (lane == 0) bulk_wait_read<1 - taken>();
    __syncwarp();
    return base + turn.take() * kOutBox;
  }
  __device__ __forceinline__ void send(const CUtensorMap* map, const uint8_t* box, int lane, int32_t x, int32_t y, bool add) {
    turn.sent(box == base ? 0 : 1);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_box(map, box, x, y, add);
      bulk_commit();
    }
  }
};
__device__ __forceinline__ void stage_bf16(uint8_t* box, int lane, int half, const float (&v)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 o;
    o.x = pk2(v[q * 8 + 0], v[q * 8 + 1]);
    o.y = pk2(v[q * 8 + 2], v[q * 8 + 3]);
    o.z = pk2(v[q * 8 + 4], v[q * 8 + 5]);
    o.w = pk2(v[q * 8 + 6], v[q * 8 + 7]);
    *reinterpret_cast<uint4*>(box + lane * 128 + (((half * 4 + q) ^ (lane & 7)) << 4)) = o;   // 128-byte swizzle
  }
}
__device__ __forceinline__ void stage_f32(uint8_t* box, int lane, const float (&v)[32]) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<float4*>(box + lane * 128 + ((q ^ (lane & 7)) << 4)) =
        make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
}

// cluster tile t -> (256-row block, column block): panels of `group` blocks along M (or N, `along_n`), which the tiles of a
// panel sweep along the other dimension
__device__ __forceinline__ void tile2(int t, int tiles_m2, int tiles_n, int group, bool along_n, int& m2, int& nb) {
  const int across = along_n ? tiles_m2 : tiles_n, along = along_n ? tiles_n : tiles_m2;
  const int span = group * across;
  const int g = t / span;
  const int r = t - g * span;
  const int g0 = g * group;
  const int geff = min(group, along - g0);
  const int sweep = r / geff, in = g0 + (r - sweep * geff);
  m2 = along_n ? sweep : in;
  nb = along_n ? in : sweep;
}

}  // namespace

// BN: columns of a cluster tile (gemm2_tile_n chooses).  A launch works on one problem or on two independent ones: the tiles
// of the second follow those of the first, so that CTA pairs without a tile in the first one's last wave begin with the
// second.  The two gradients of a linear layer that way, in one launch and in two: 1992 x 4104 x 1032 (85 tiles of 32
// k-blocks and 136 of 17 on 74 pairs) 92.9 -> 81.9 us for the whole layer, 512 x 512 x 1536 38 -> 34, 4096 x 1024 x 51200 with
// its loss 1309 -> 1296; 8192 x 4096 x 16384 is under the power cap either way (2541 and 2537).
// kDGelu: a problem may have act 2.  An instance of its own: with it the kernel takes 230 registers instead of 94, and the
// layer of 1992 x 4104 x 1032, which has no GeLU, 81.9 us instead of 81.2.  The derivative here instead of a pass over the
// gradient (268 MB read twice and written in 160 us): decoder block of width 4096, 8192 tokens, 8817 -> 8643 us.
template <int BN, bool kDGelu>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads2, 1)
sm100_gemm2_kernel(const __grid_constant__ Gemm2Args a) {
  constexpr int kStages2 = stages2(BN);
  constexpr uint32_t kBStage2 = b_stage2(BN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  constexpr uint32_t kSmemB2 = kStages2 * kAStage2;
  constexpr uint32_t kSmemOut2 = kSmemB2 + kStages2 * kBStage2;
  constexpr uint32_t kSmemBar2 = kSmemOut2 + kOutStage;
  uint8_t* sA = smem;
  uint8_t* sB = smem + kSmemB2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSmemBar2);
  uint64_t* full_bar = bars;                    // [kStages2], used in the leader
  uint64_t* empty_bar = bars + kStages2;        // [kStages2], one set per CTA
  uint64_t* tfull_bar = bars + 2 * kStages2;    // [2], one set per CTA
  uint64_t* tempty_bar = tfull_bar + 2;         // [2], used in the leader
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();      // 0: leader
  const uint64_t tmo = a.timeout_ns;
  const int num_tiles = a.tiles[1];
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  // Tile t: its problem and its place in it.
  const auto place = [&](int t, bool& second, int& m2, int& nb) {
    second = t >= a.tiles[0];
    const Gemm2Problem& p0 = a.p[0];
    const Gemm2Problem& p1 = a.p[1];
    const int M = second ? p1.M : p0.M, N = second ? p1.N : p0.N;
    tile2(second ? t - a.tiles[0] : t, (M + 2 * kBM - 1) / (2 * kBM), (N + BN - 1) / BN, second ? p1.group : p0.group,
          (second ? p1.along_n : p0.along_n) != 0, m2, nb);
  };

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&a.p[0].a);
    tma_prefetch_desc(&a.p[0].b);
    for (int i = 0; i < kStages2; ++i) {
      mbar_init(full_bar + i, 2);    // the leader's two producers announce their operand's bytes
      mbar_init(empty_bar + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tfull_bar + i, 1);
      mbar_init(tempty_bar + i, 8);    // a lane of each epilogue warp of both CTAs
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2u * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  cluster_sync_all();      // barriers of both CTAs are initialised before any remote arrival
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_trigger();
  grid_wait();

  if (warp == 0 || warp == 6) {
    // ===================== TMA producers (both CTAs): warp 0 loads A, warp 6 loads B ==========
    // One thread issuing every load of a stage is what bounded the tensor pipe with MN-major
    // operands (two boxes per operand): the operands have a producer each, and an MN-major
    // operand is one 3-D box when its extent allows it.
    if (elect_one()) {
      const bool is_a = warp == 0;
      const uint32_t full0 = mapa_u32(smem_u32(full_bar), 0);     // the leader's barriers
      uint32_t stage = 0, phase = 0;
      bool ok = true, free = true;                                // `free`: the next stage was seen empty
      for (int t = cluster_id; t < num_tiles && ok; t += n_clusters) {
        bool second;
        int m2, nb;
        place(t, second, m2, nb);
        const Gemm2Problem* p = second ? &a.p[1] : &a.p[0];
        const CUtensorMap* map = is_a ? &p->a : &p->b;
        const bool mn_major = (is_a ? p->a_mn_major : p->b_mn_major) != 0, map3d = (is_a ? p->a_map3d : p->b_map3d) != 0;
        const int kblocks = (p->K + kBK - 1) / kBK;
        // this CTA's 128 rows of A / its half of the columns of B
        const int row = is_a ? (2 * m2 + (int)rank) * kBM : nb * BN + (int)rank * (BN / 2);
        const uint32_t bytes = is_a ? kAStage2 : kBStage2;
        uint8_t* ring = is_a ? sA : sB;
        const int boxes = is_a ? kBM / 64 : BN / 128;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!free && !mbar_wait(empty_bar + stage, phase ^ 1, 5 * tmo)) {
            report2(a, kTimeoutEmpty, t, kb);
            ok = false;
            break;
          }
          const uint32_t fb = full0 + stage * 8;
          const int k0 = kb * kBK;
          if (rank == 0) mbar_expect_tx(full_bar + stage, 2 * bytes);
          uint8_t* dst = ring + stage * bytes;
          if (!mn_major) {
            tma_load_2d_pair(dst, map, fb, k0, row);
          } else if (map3d) {
            tma_load_3d_pair(dst, map, fb, 0, k0, row >> 6);
          } else {
            for (int j = 0; j < boxes; ++j) tma_load_2d_pair(dst + j * (kBK * 128), map, fb, row + j * 64, k0);
          }
          if (++stage == kStages2) { stage = 0; phase ^= 1; }
          free = mbar_test(empty_bar + stage, phase ^ 1);
        }
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader only) =====================
    // What this thread does per k-block has to fit into the 512 (BN = 256) or 256 cycles that the four instructions
    // take on the tensor pipe: with the descriptors rebuilt for every instruction, two commits and the wait on the
    // critical path a k-block took 590 cycles whatever BN.  So only the low descriptor word changes, by additions; one
    // commit reaches both CTAs; and the next stage is looked at before this one is issued.
    if (rank == 0 && elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true, full = false;                               // `full`: the next stage was seen complete
      int it = 0;
      for (int t = cluster_id; t < num_tiles && ok; t += n_clusters, ++it) {
        const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
        if (!mbar_wait(tempty_bar + acc, acc_phase ^ 1, 6 * tmo)) {
          report2(a, kTimeoutTmemEmpty, t, acc);
          ok = false;
          break;
        }
        const uint32_t tmem_d = tmem_base + acc * BN;
        const Gemm2Problem* p = t >= a.tiles[0] ? &a.p[1] : &a.p[0];
        const int kblocks = (p->K + kBK - 1) / kBK;
        const bool a_mn = p->a_mn_major != 0, b_mn = p->b_mn_major != 0;
        const uint32_t idesc = make_idesc_bf16(2 * kBM, BN, a_mn, b_mn);
        const uint64_t da0 = make_smem_desc(smem_u32(sA), a_mn ? kBK * 128 : 16, 1024);
        const uint64_t db0 = make_smem_desc(smem_u32(sB), b_mn ? kBK * 128 : 16, 1024);
        const uint32_t da_hi = (uint32_t)(da0 >> 32), db_hi = (uint32_t)(db0 >> 32);
        const uint32_t a_kstep = (a_mn ? 16 * 128 : 32) >> 4;
        const uint32_t b_kstep = (b_mn ? 16 * 128 : 32) >> 4;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!full && !mbar_wait(full_bar + stage, phase, 4 * tmo)) {
            report2(a, kTimeoutFull, t, kb);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t da_lo = (uint32_t)da0 + stage * (kAStage2 >> 4);
          const uint32_t db_lo = (uint32_t)db0 + stage * (kBStage2 >> 4);
          const uint32_t eb = smem_u32(empty_bar + stage);
          if (++stage == kStages2) { stage = 0; phase ^= 1; }
          full = mbar_test(full_bar + stage, phase);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            umma_f16_pair(tmem_d, desc_at(da_lo + k * a_kstep, da_hi), desc_at(db_lo + k * b_kstep, db_hi), idesc,
                          (kb | k) != 0 ? 1u : 0u);
          umma_commit_both(eb);                 // the stage is free in both CTAs
        }
        if (ok) umma_commit_both(smem_u32(tfull_bar + acc));
      }
    }
  } else {
    // ===================== epilogue (both CTAs, own 128 rows) =====================
    const int q = warp & 3;
    OutStage out{smem + kSmemOut2 + q * 2 * kOutBox, {0}};
    bool ok = true;
    int it = 0;
    for (int t = cluster_id; t < num_tiles && ok; t += n_clusters, ++it) {
      bool second;
      int m2, nb;
      place(t, second, m2, nb);
      const Gemm2Problem& p = second ? a.p[1] : a.p[0];
      const __nv_bfloat16* bias = reinterpret_cast<const __nv_bfloat16*>(p.bias);
      void* const C = p.C;
      void* const C_pre = p.C_pre;
      const int64_t ldc = p.ldc;
      const int M = p.M, N = p.N, act = p.act;
      const bool fp32 = p.c_fp32 != 0, add = p.accumulate != 0, tma_c = p.tma_c != 0;
      const bool dual = act == 1 && C_pre != nullptr;       // two outputs: no store of one runs under the other's staging
      const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
      int okw = 1;
      if (lane == 0) okw = mbar_wait(tfull_bar + acc, acc_phase, 7 * tmo) ? 1 : 0;
      okw = __shfl_sync(0xffffffffu, okw, 0);
      if (!okw) {
        if (lane == 0) report2(a, kTimeoutTmemFull, t, acc);
        ok = false;
        break;
      }
      mbar_wait(tfull_bar + acc, acc_phase, tmo);
      tc_fence_after_sync();
      const int row0 = (2 * m2 + (int)rank) * kBM + q * 32;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
      const uint32_t te_leader = mapa_u32(smem_u32(tempty_bar + acc), 0);
      uint8_t* box = nullptr;
      uint8_t* box_pre = nullptr;
      // act 2: the result times the derivative of GeLU at C_pre, whose elements are asked for one step ahead
      const bool live = kDGelu && act == 2 && row0 + lane < M;
      uint32_t x_next[16];
      if (live) load32(C_pre, ldc, row0 + lane, nb * BN, min(32, N - nb * BN), x_next);
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        __syncwarp();
        tmem_ld_32x32(taddr + c * 32, r);
        tmem_ld_wait();
        if (c == BN / 32 - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(te_leader);     // accumulator drained: tell the leader's MMA warp
        }
        const int col0 = nb * BN + c * 32;
        const int nvalid = min(32, N - col0);
        if (row0 >= M || nb * BN + (c & ~1) * 32 >= N) continue;   // the two halves of a bf16 box go together
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
        if (bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < nvalid) v[i] += __bfloat162float(bias[col0 + i]);
        }
        if (live) {
          uint32_t x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = x_next[i];
          if (c + 1 < BN / 32 && col0 + 32 < N) load32(C_pre, ldc, row0 + lane, col0 + 32, min(32, N - col0 - 32), x_next);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            v[2 * i] *= gelu_grad_f(blo(x[i]));
            v[2 * i + 1] *= gelu_grad_f(bhi(x[i]));
          }
        }
        if (!tma_c) {
          if (row0 + lane >= M || nvalid <= 0) continue;
          if (act == 1) {
            if (C_pre != nullptr) store32(C_pre, ldc, false, false, row0 + lane, col0, nvalid, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = gelu_tanh2(v[i]);
          }
          store32(C, ldc, fp32, add, row0 + lane, col0, nvalid, v);
          continue;
        }
        // rows and columns beyond the matrix are clipped by the tensor map
        if (act == 1) {
          if (dual) {
            if ((c & 1) == 0) box_pre = out.take(lane);
            stage_bf16(box_pre, lane, c & 1, v);
            if (c & 1) out.send(&p.pre, box_pre, lane, col0 - 32, row0, false);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = gelu_tanh2(v[i]);
        }
        if (fp32) {
          if (nvalid <= 0) continue;
          box = dual ? out.take<1>(lane) : out.take(lane);
          stage_f32(box, lane, v);
          out.send(&p.c, box, lane, col0, row0, add);
        } else {
          if ((c & 1) == 0) box = dual ? out.take<1>(lane) : out.take(lane);
          stage_bf16(box, lane, c & 1, v);
          if (c & 1) out.send(&p.c, box, lane, col0 - 32, row0, false);
        }
      }
    }
    if (lane == 0) bulk_wait_all<0>();
  }

  // both CTAs are done with shared memory, barriers and TMEM of the pair
  tc_fence_before_sync();
  cluster_sync_all();
  tc_fence_after_sync();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * BN) : "memory");
}

template <int BN, bool kDGelu>
static cudaError_t launch2(const Gemm2Args& args, int grid, cudaStream_t stream) {
  static bool configured[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  constexpr int smem = (int)smem_alloc2(BN);
  if (dev < 64 && !configured[dev]) {
    e = cudaFuncSetAttribute(sm100_gemm2_kernel<BN, kDGelu>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  // the cluster shape (2,1,1) is part of the kernel's definition
  return launch_dependent(sm100_gemm2_kernel<BN, kDGelu>, grid, kThreads2, smem, stream, args);
}

// The tile width that ends sooner.  A 64-deep k-block takes about 390 cycles on 128 columns (the loads: 24 KiB
// a CTA) and 530 on 256 (the tensor pipe: 512), so a narrow tile counts three quarters of a wide one.  A CTA pair takes every
// n-th tile: the last pair to end is the one with one tile more of either problem (pair 0) or the first without.
// 2048 x 1024 x 4096 (32 wide tiles): 26.5 us wide, 19.6 narrow; 1024 x 2048 x 1024 11.9 and 8.7; 2048 x 2048 x 2048 (64
// wide tiles, one wave against two): wide, 16.3 us.
static int64_t last_end(const Gemm2Operands* o, int problems, int tile_n, int64_t pairs) {
  int64_t tiles[2] = {0, 0}, kb[2] = {0, 0};
  for (int i = 0; i < problems; ++i) {
    tiles[i] = ((o[i].M + 2 * kBM - 1) / (2 * kBM)) * ((o[i].N + tile_n - 1) / tile_n);
    kb[i] = (o[i].K + kBK - 1) / kBK;
  }
  const int64_t all = tiles[0] + tiles[1], at[3] = {0, tiles[0] % pairs, all % pairs};
  int64_t last = 0;
  for (int64_t i : at) {
    const int64_t n0 = (tiles[0] - i + pairs - 1) / pairs, n = (all - i + pairs - 1) / pairs;
    const int64_t end = n0 * kb[0] + (n - n0) * kb[1];
    last = end > last ? end : last;
  }
  return last;
}
int gemm2_tile_n(const Gemm2Operands* o, int problems, int sms) {
  const int64_t pairs = sms > 1 ? sms / 2 : 1;
  return 3 * last_end(o, problems, 128, pairs) < 4 * last_end(o, problems, 256, pairs) ? 128 : 256;
}

// The order of the tiles, by what they read from HBM: under the power cap that traffic costs clock.  A panel of sixteen
// blocks along one dimension is kept in L2 (33 MB at K = 4096) while the tiles sweep the other, so the panels' operand is
// read once and the other one once per panel: the dimension with the smaller sum.  Panels of eight / sixteen / thirty-two,
// sustained: 8192 x 16384 x 4096 815 / 788 / 871 us (along N: 824 / 803 / 886), 4096 x 51200 x 1024 345 / 336 / 336.
// Longer contractions keep panels of eight along M: 8192 x 4096 x 16384 833 / 840, 4096 x 16384 x 8192 added to fp32
// 864 / 876, 4096 x 4096 x 8192 235 / 236.  Every tile sums its contraction from the first k-block to the last, so that a
// result does not depend on which tiles a CTA pair had before; walking it backwards on every other tile, which finds the
// end of the contraction in L2, would give 822, 844 and 228.
Gemm2Order gemm2_order(int64_t M, int64_t N, int64_t K, int tile_n) {
  if (K > 4096) return {8, 0};
  const int64_t panels_m = (M + 16 * 256 - 1) / (16 * 256), panels_n = (N + 16 * tile_n - 1) / (16 * tile_n);
  return {16, N + panels_n * M < M + panels_m * N};
}

int gemm2_problem(Gemm2Problem* p, const Gemm2Operands& o, int tile_n) {
  memset(static_cast<void*>(p), 0, sizeof(*p));
  p->M = (int)o.M;
  p->N = (int)o.N;
  p->K = (int)o.K;
  p->a_mn_major = o.a_mn_major;
  p->b_mn_major = o.b_mn_major;
  p->C = o.C;
  p->ldc = o.ldc;
  p->c_fp32 = o.c_fp32;
  p->accumulate = o.accumulate;
  p->bias = o.bias;
  p->act = o.act;
  p->C_pre = o.C_pre;
  int r;
  if (!o.a_mn_major) r = make_tensor_map_2d(&p->a, o.A, o.K, o.M, o.lda * 2, kBK, kBM);
  else if (o.map3d && make_tensor_map_mn3d(&p->a, o.A, o.M, o.K, o.lda * 2, kBM / 64) == 0) { r = 0; p->a_map3d = 1; }
  else r = make_tensor_map_2d(&p->a, o.A, o.M, o.K, o.lda * 2, 64, kBK);
  if (r != 0) return r;
  if (!o.b_mn_major) r = make_tensor_map_2d(&p->b, o.B, o.K, o.N, o.ldb * 2, kBK, tile_n / 2);
  else if (o.map3d && make_tensor_map_mn3d(&p->b, o.B, o.N, o.K, o.ldb * 2, tile_n / 128) == 0) { r = 0; p->b_map3d = 1; }
  else r = make_tensor_map_2d(&p->b, o.B, o.N, o.K, o.ldb * 2, 64, kBK);
  if (r != 0) return r;
  // Output through shared memory and TMA where the tensor map allows it; bf16 accumulation adds before it rounds,
  // which the copy engine cannot do.
  p->tma_c = !(o.accumulate && !o.c_fp32) && make_tensor_map_out(&p->c, o.C, o.N, o.M, o.ldc, o.c_fp32 != 0) == 0 &&
             (o.act != 1 || o.C_pre == nullptr || make_tensor_map_out(&p->pre, o.C_pre, o.N, o.M, o.ldc, false) == 0);
  const Gemm2Order order = o.group > 0 ? Gemm2Order{o.group, 0} : gemm2_order(o.M, o.N, o.K, tile_n);
  p->group = order.group;
  p->along_n = order.along_n;
  return 0;
}

cudaError_t launch_sm100_gemm2(Gemm2Args& args, int problems, int tile_n, int sms, cudaStream_t stream) {
  int64_t tiles = 0;
  bool dgelu = false;
  for (int i = 0; i < 2; ++i) {
    if (i < problems) {
      const Gemm2Problem& p = args.p[i];
      dgelu = dgelu || p.act == 2;
      tiles += (int64_t)((p.M + 2 * kBM - 1) / (2 * kBM)) * ((p.N + tile_n - 1) / tile_n);
    }
    args.tiles[i] = (int)tiles;
  }
  int grid = (int)(2 * tiles < (sms & ~1) ? 2 * tiles : (sms & ~1));
  if (grid < 2) grid = 2;
  if (dgelu) return tile_n == 128 ? launch2<128, true>(args, grid, stream) : launch2<256, true>(args, grid, stream);
  return tile_n == 128 ? launch2<128, false>(args, grid, stream) : launch2<256, false>(args, grid, stream);
}

}  // namespace msb
