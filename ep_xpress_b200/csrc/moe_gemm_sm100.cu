// Grouped SwiGLU expert GEMM for sm_100a: tcgen05.mma on CTA pairs with TMEM accumulators,
// operands staged in shared memory by TMA, one elected thread issuing the MMAs.
//
// The reference ships no expert GEMM: its adapter calls a framework's Triton kernel
// around count-aware helper kernels (ep_xpress/adapters/sglang_valid.py:13-255). This
// file is the hand-written replacement for that whole runner:
//
//   align      received (row, slot) pairs whose expert lives on this rank are packed by
//              expert, bounded by the DEVICE valid_count (the job of
//              sglang_valid.py:13-161), and every expert's rows are cut into token tiles;
//   scatter    activation rows are copied into that expert-sorted order;
//   GEMM 1     act = silu(x W1_e) * (x W3_e): gate and up rows of the weights sit in one
//              tile, the epilogue pairs them up (the framework needs a separate activation
//              kernel, adapters/sglang/sglang-v0.5.21.patch:281-330);
//   GEMM 2     y = (act W2_e) * routing weight, rounded to BF16 per (row, slot);
//   slot sum   partial[row] = bf16(sum over the row's local slots, in slot order, FP32) -
//              the definition of a rank's partial (sglang_valid.py:206-222).
//
// Which operand is M: the WEIGHTS. tcgen05 fixes M (256 rows on a CTA pair) but takes any
// N = 16, 32, ... 256, and the number of tokens an expert got is the ragged dimension. With
// tokens as N a tile costs what its tokens cost: no row is padded beyond the next multiple of
// 16, so 32 experts with 32 tokens each stream their weights once instead of multiplying
// 256-row tiles that are 7/8 padding, and expert segments are packed without gaps.
// Measured (hidden 7168, inter 2048, 32 experts; tokens as 256-row M tiles -> tokens as N; us of
// GEMM 1 + GEMM 2): 16 tokens per expert 366 + 186 -> 280 + 146 (6.4-6.7 TB/s of weights: HBM
// bound), 1024 tokens 1285 + 676 -> 1290 + 650 (tensor bound,
// nothing to pad). Hidden 2048, inter 768, 128 experts x 64 tokens: 294 + 110 -> 148 + 74.
//
// All launches of the runner are chained by programmatic dependent launch: a kernel's prologue
// (barriers, TMEM, descriptors) and the dispatch of its CTAs overlap the tail of the one before.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "epx_device.cuh"
#include "moe_gemm.h"

namespace epx {
namespace {

constexpr int kTileK = 64;                 // 64 BF16 = one 128-byte swizzle row
constexpr int kTileM = 256;                // weight rows of a CTA pair's tile (128 per CTA)
constexpr int kMaxTileN = 256;             // tokens of a tile
constexpr int kABytes = 128 * kTileK * 2;  // one CTA's weight rows of a k-step
constexpr int kMaxStages = 12;
constexpr int kRingBytes = 7 * (kABytes + kMaxTileN / 2 * kTileK * 2);   // 224 KB: seven stages of the widest tile
constexpr size_t kGemmSmemBytes = kRingBytes + 1024;                      // + alignment of the swizzled tiles
constexpr int kMaxEpilogueShare = 4;       // epilogue warps per TMEM lane quadrant
constexpr int kGemmThreads = 64 + 128 * kMaxEpilogueShare;   // of the widest launch
constexpr int kAccumColumns = 256;
constexpr int kNMaps = 5;                  // boxes of 8, 16, 32, 64 and 128 token rows
constexpr unsigned long long kGemmWaitNs = 2000000000ull;   // bound of every pipeline wait: 2 s

// ---- PTX wrappers ----------------------------------------------------------------------
__device__ __forceinline__ bool elect_one() {
  unsigned pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  return mbarrier_wait_bounded(bar, parity, kGemmWaitNs);
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_load_32(unsigned taddr, unsigned (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (64 BF16) and
// 128-byte swizzled: 8-row groups are 1024 bytes apart (stride byte offset), the leading
// byte offset is unused for swizzled K-major layouts, descriptor version 1, layout type 2.
__device__ __forceinline__ unsigned long long smem_descriptor(const void* tile) {
  const unsigned long long address = smem_address(tile);
  return ((address & 0x3ffffull) >> 4) | (1ull << 16) | ((1024ull >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: D FP32, A/B BF16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ constexpr unsigned instruction_descriptor(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<unsigned>(n >> 3) << 17) |
         (static_cast<unsigned>(m >> 4) << 24);
}



__device__ __forceinline__ unsigned cluster_ctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory object in CTA `rank` of this cluster.
__device__ __forceinline__ unsigned peer_smem_address(const void* local, unsigned rank) {
  unsigned out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_address(local)), "r"(rank));
  return out;
}
__device__ __forceinline__ void mbar_arrive_cluster(unsigned cluster_address) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, unsigned bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_address(dst)), "l"(map), "r"(x), "r"(y), "r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(unsigned* smem_result, unsigned columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
               ::"r"(smem_address(smem_result)), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(unsigned address, unsigned columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc,
                                               unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// The weights of GEMM 1 as a five-dimensional box {64 k, 16 rows, gate/up, 4 blocks, expert}: 128
// rows of shared memory that alternate 16 gate rows with the 16 up rows of the same columns.
__device__ __forceinline__ void tma_load_5d_pair(void* dst, const CUtensorMap* map, int x, int block, int expert,
                                                 unsigned bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %3, %4, %5}], [%6];"
      ::"r"(smem_address(dst)), "l"(map), "r"(x), "r"(0), "r"(block), "r"(expert), "r"(bar_cluster) : "memory");
}
// Four rows of a row-major matrix (any four row indices) x one 64-column box, written to `dst`
// as four consecutive 128-byte rows; the tensor map has a box of {64, 1}. A row index at or
// beyond the matrix height reads zeros. No fan-out: the copy lands in this CTA only.
__device__ __forceinline__ void tma_gather4_pair(void* dst, const CUtensorMap* map, int x, int r0, int r1, int r2, int r3,
                                                 unsigned bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(smem_address(dst)), "l"(map), "r"(x), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(bar_cluster) : "memory");
}
// Arrives on the barrier at this offset in BOTH CTAs of the pair once every MMA issued so far by
// this thread has finished.
__device__ __forceinline__ void umma_commit_pair(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_address(bar)), "h"(static_cast<unsigned short>(3)) : "memory");
}

// ---- the grouped GEMM kernel -------------------------------------------------------------------
struct GemmParams {
  const int* counters;           // device: {token tiles in use, sorted rows in use}
  const int4* tiles;             // device: {expert, first sorted row, rows, -} of every token tile
  const float* row_scale;        // kMode 1: routing weight of every sorted row
  void* out;                     // bf16 [sorted rows, out_columns]
  int* error_flag;               // set to 1 when a bounded wait gave up
  int k_steps;                   // K / 64
  int m_tiles;                   // 256-row weight tiles of one expert
  int out_columns;               // row pitch of `out` in elements
  int b_rows;                    // token rows a stage has room for in one CTA (half of the widest tile)
  int stages;
  const int* gather_rows;        // null, or [sorted rows]: source row of every sorted position; the token operand
                                 // is then gathered from the unsorted matrix behind maps.b[0]
  int gather_height;             // rows of that matrix; an index at or above it reads zeros
};
struct GemmMaps {
  CUtensorMap a;
  CUtensorMap b[kNMaps];         // the token matrix with boxes of 8 << i rows
};

// Token tile `index` of the list that the align step wrote. Acquiring loads: they go to L2, so that a kernel
// that has not waited for the one before it yet never takes a stale line of the SM's L1 for the list.
__device__ __forceinline__ int4 acquire_tile(const int4* tiles, int index) {
  const unsigned long long* p = reinterpret_cast<const unsigned long long*>(tiles + index);
  const unsigned long long low = ld_acquire_gpu_u64(p), high = ld_acquire_gpu_u64(p + 1);
  return make_int4(static_cast<int>(low), static_cast<int>(low >> 32), static_cast<int>(high), static_cast<int>(high >> 32));
}

// Index of the smallest box that holds `half` token rows (a multiple of 8).
__device__ __forceinline__ int box_index(int half) {
  return half <= 8 ? 0 : (half <= 16 ? 1 : (half <= 32 ? 2 : (half <= 64 ? 3 : 4)));
}

// One 256 x N tile per CTA pair (a cluster of two), N = the tile's tokens rounded up to 16. Each
// CTA stages its own 128 weight rows and HALF of the tokens; the leader CTA's elected thread
// issues tcgen05.mma.cta_group::2, which reads both CTAs' shared memory and writes each CTA's 128
// accumulator rows into that CTA's own TMEM, and both CTAs run their own epilogue. Both producers
// complete their TMA loads on the LEADER's full barrier; the leader's commits release stages and
// hand over accumulators in both CTAs. No load fans out to more than one CTA.
//
// Persistent: pair c takes tiles c, c + pairs, ... in (token tile, weight tile) order, so the
// pairs that run together share one expert's tokens and, for experts with several token tiles,
// its weights in L2. Warp 0 feeds the ring, warp 1 issues MMAs, the others drain the accumulators
// (two buffers of 256 TMEM columns, so the epilogue of one tile overlaps the next main loop): up to four
// warps per TMEM lane quadrant, which take 32 tokens each in turn. The epilogue is about 500
// instructions per 32 tokens; with one warp per quadrant it took 16,000 cycles for a wide tile, longer
// than the main loop of K = 768 and as long as that of K = 2048, and stood alone at the end. (See
// epilogue_shares for narrower tiles.)
// Every wait is bounded and ends in an error flag, after which TMEM is still released.
//
// kMode 0: 256 weight rows = 128 gate and 128 up rows of the same columns, interleaved by 16, so
//          a gate row and its up row are 16 lanes apart in one warp: epilogue silu(gate) * up.
// kMode 1: 256 rows of W2, epilogue acc * row_scale.
template <int kMode>
__global__ void __launch_bounds__(kGemmThreads, 1)
grouped_gemm_kernel(const __grid_constant__ GemmMaps maps, const GemmParams p) {
  extern __shared__ __align__(1024) unsigned char gemm_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) &
                                                         ~static_cast<uintptr_t>(1023));
  __shared__ unsigned long long full_bar[kMaxStages], empty_bar[kMaxStages];
  __shared__ unsigned long long acc_full[2], acc_empty[2];
  __shared__ unsigned tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned rank = cluster_ctarank();           // 0 = leader
  const int shares = (static_cast<int>(blockDim.x) - 64) / 128;
  const int stages = p.stages;
  const int stage_bytes = kABytes + p.b_rows * kTileK * 2;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbarrier_init(full_bar + s, 1);                // leader's: one arrive.expect_tx + both CTAs' bytes
      mbarrier_init(empty_bar + s, 1);               // one commit from the leader per use
    }
    for (int b = 0; b < 2; ++b) {
      mbarrier_init(acc_full + b, 1);                // one commit from the leader per tile
      mbarrier_init(acc_empty + b, 8 * shares);        // leader's: the epilogue warps of both CTAs
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == 1) tmem_alloc_pair(&tmem_base_slot, 2 * kAccumColumns);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync();                                    // both CTAs' barriers exist before anyone signals
  tcgen05_fence_after();
  const unsigned tmem_base = tmem_base_slot;

  // The tile list comes from the align step, which is complete before the launch right behind it lets
  // this kernel start; only the tokens (and, when gathered, the list itself) are the previous kernel's.
  // So the producer fills its ring with the first tile's WEIGHTS while the previous kernel ends, and
  // waits before the first token load; it reads the list with acquiring loads until then. (One thread of
  // warp 0 waits in that mode, all threads of the other warps do, and the CTA leaves behind them all.)
  if (p.gather_rows != nullptr || warp != 0) {
    wait_for_previous();
    launch_dependents();
  }
  const int total = static_cast<int>(ld_acquire_gpu_u32(reinterpret_cast<const unsigned*>(p.counters))) * p.m_tiles;
  const int pair_id = blockIdx.x / 2, pairs = gridDim.x / 2;

  auto load_weights = [&](unsigned char* dst, int k, int expert, int mt, unsigned leader_full) {
    if (kMode == 0) tma_load_5d_pair(dst, &maps.a, k * kTileK, mt * 8 + static_cast<int>(rank) * 4, expert, leader_full);
    else tma_load_2d_pair(dst, &maps.a, k * kTileK, (expert * p.m_tiles + mt) * kTileM + static_cast<int>(rank) * 128, leader_full);
  };

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    // One ELECTED thread issues: the same loop under `if (lane == 0)` cost the tensor pipe a fifth of
    // its cycles (hidden 7168, inter 2048, 32 experts x 1024 tokens: 1431 + 746 us against 1290 + 646),
    // because without elect.sync the compiler cannot keep the copies' operands in uniform registers.
    int s = 0;
    unsigned parity = 1u;                            // of the stage's empty barrier: the first round passes at once
    if (p.gather_rows != nullptr) {
      // Gathered tokens: the whole warp takes part, every lane fetches four rows per k-step.
      bool go = true;
      for (int item = pair_id; item < total && go; item += pairs) {
        const int tt = item / p.m_tiles, mt = item - tt * p.m_tiles;
        const int4 tile = p.tiles[tt];
        const int half = ((tile.z + 15) & ~15) / 2;
        const bool fetch = 4 * lane < half;
        const int first = static_cast<int>(rank) * half + 4 * lane;
        int rows[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          rows[i] = fetch && first + i < tile.z ? p.gather_rows[tile.y + first + i] : p.gather_height;
        for (int k = 0; k < p.k_steps; ++k) {
          unsigned char* a_dst = smem + static_cast<size_t>(s) * stage_bytes;
          const unsigned leader_full = peer_smem_address(full_bar + s, 0);
          const bool ok = !failed && mbar_wait(empty_bar + s, parity);
          go = __all_sync(0xffffffffu, ok);
          if (!go) { failed = 1; break; }
          if (elect_one()) {
            if (rank == 0) mbarrier_arrive_expect_tx(full_bar + s, 2u * (kABytes + half * kTileK * 2));
            load_weights(a_dst, k, tile.x, mt, leader_full);
          }
          __syncwarp();
          if (fetch) tma_gather4_pair(a_dst + kABytes + lane * 512, maps.b, k * kTileK, rows[0], rows[1], rows[2], rows[3], leader_full);
          if (++s == stages) { s = 0; parity ^= 1u; }
        }
      }
    } else if (elect_one()) {
      int ahead = 0;                                 // k-steps of the first tile whose weights are under way
      if (pair_id < total) {
        const int tt = pair_id / p.m_tiles, mt = pair_id - tt * p.m_tiles;
        const int4 tile = acquire_tile(p.tiles, tt);
        const unsigned tx = 2u * (kABytes + (8u << box_index(((tile.z + 15) & ~15) / 2)) * kTileK * 2);
        for (; ahead < stages && ahead < p.k_steps; ++ahead) {
          if (rank == 0) mbarrier_arrive_expect_tx(full_bar + ahead, tx);
          load_weights(smem + static_cast<size_t>(ahead) * stage_bytes, ahead, tile.x, mt, peer_smem_address(full_bar + ahead, 0));
        }
      }
      wait_for_previous();
      for (int item = pair_id; item < total && !failed; item += pairs) {
        const int tt = item / p.m_tiles, mt = item - tt * p.m_tiles;
        const int4 tile = p.tiles[tt];
        const int half = ((tile.z + 15) & ~15) / 2;
        const int which = box_index(half);
        const CUtensorMap* map_b = maps.b + which;
        const unsigned tx = 2u * (kABytes + (8u << which) * kTileK * 2);
        const int b_row = tile.y + static_cast<int>(rank) * half;
        for (int k = 0; k < p.k_steps; ++k) {
          unsigned char* a_dst = smem + static_cast<size_t>(s) * stage_bytes;
          const unsigned leader_full = peer_smem_address(full_bar + s, 0);
          if (ahead > 0) {
            --ahead;
          } else {
            if (!mbar_wait(empty_bar + s, parity)) { failed = 1; break; }
            if (rank == 0) mbarrier_arrive_expect_tx(full_bar + s, tx);
            load_weights(a_dst, k, tile.x, mt, leader_full);
          }
          tma_load_2d_pair(a_dst + kABytes, map_b, k * kTileK, b_row, leader_full);
          if (++s == stages) { s = 0; parity ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader only) ----------------
    if (rank == 0 && elect_one()) {
      int s = 0;
      unsigned parity = 0u, local_tile = 0;
      for (int item = pair_id; item < total && !failed; item += pairs, ++local_tile) {
        const int n = (p.tiles[item / p.m_tiles].z + 15) & ~15;
        const unsigned idesc = instruction_descriptor(kTileM, n);
        const unsigned buffer = local_tile & 1u;
        if (!mbar_wait(acc_empty + buffer, ((local_tile >> 1) & 1u) ^ 1u)) { failed = 1; break; }
        tcgen05_fence_after();
        const unsigned tmem_d = tmem_base + buffer * kAccumColumns;
        for (int k = 0; k < p.k_steps; ++k) {
          if (!mbar_wait(full_bar + s, parity)) { failed = 1; break; }
          tcgen05_fence_after();
          const unsigned char* a_tile = smem + static_cast<size_t>(s) * stage_bytes;
          const unsigned long long a_desc = smem_descriptor(a_tile);
          const unsigned long long b_desc = smem_descriptor(a_tile + kABytes);
#pragma unroll
          for (int kk = 0; kk < kTileK / 16; ++kk)   // 16 BF16 = 32 bytes = 2 descriptor units per step
            umma_bf16_pair(tmem_d, a_desc + 2 * kk, b_desc + 2 * kk, idesc, (k | kk) != 0 ? 1u : 0u);
          umma_commit_pair(empty_bar + s);           // both CTAs may refill the stage
          if (++s == stages) { s = 0; parity ^= 1u; }
        }
        if (failed) break;
        umma_commit_pair(acc_full + buffer);         // both epilogues may read
      }
    }
  } else {
    // ---------------- epilogue (both CTAs, own 128 weight rows) ----------------
    // TMEM lane = weight row (output column), TMEM column = token.
    const int quadrant = warp & 3, share = (warp - 2) >> 2;
    unsigned local_tile = 0;
    for (int item = pair_id; item < total; item += pairs, ++local_tile) {
      const int tt = item / p.m_tiles, mt = item - tt * p.m_tiles;
      const int4 tile = p.tiles[tt];
      const unsigned buffer = local_tile & 1u;
      const bool ok = mbar_wait(acc_full + buffer, (local_tile >> 1) & 1u);
      if (!__all_sync(0xffffffffu, ok)) { failed = 1; break; }
      tcgen05_fence_after();
      const unsigned taddr = tmem_base + buffer * kAccumColumns + (static_cast<unsigned>(quadrant * 32) << 16);
      const int upper = lane >> 4;                   // kMode 0: lanes 0-15 hold gate rows, 16-31 their up rows
      const int column = kMode == 0 ? mt * 128 + static_cast<int>(rank) * 64 + quadrant * 16 + (lane & 15)
                                    : mt * kTileM + static_cast<int>(rank) * 128 + quadrant * 32 + lane;
      __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<long long>(tile.y) * p.out_columns + column;
#pragma unroll 1
      for (int c0 = 32 * share; c0 < tile.z; c0 += 32 * shares) {
        unsigned v[32];
        tmem_load_32(taddr + c0, v);
        tmem_load_wait();
        if (kMode == 0) {
          // A lane pair (l, l + 16) holds gate and up of 32 tokens: the lower lane finishes the first
          // sixteen of them, the upper lane the others.
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float mine = __uint_as_float(upper ? v[16 + i] : v[i]);
            const float theirs = __uint_as_float(__shfl_xor_sync(0xffffffffu, upper ? v[i] : v[16 + i], 16));
            const float gate = upper ? theirs : mine, up = upper ? mine : theirs;
            const int token = c0 + upper * 16 + i;
            if (token < tile.z)
              out[static_cast<long long>(token) * p.out_columns] = __float2bfloat16_rn((gate / (1.f + __expf(-gate))) * up);
          }
        } else {
          const float scale = c0 + lane < tile.z ? p.row_scale[tile.y + c0 + lane] : 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float w = __shfl_sync(0xffffffffu, scale, i);
            if (c0 + i < tile.z)
              out[static_cast<long long>(c0 + i) * p.out_columns] = __float2bfloat16_rn(__uint_as_float(v[i]) * w);
          }
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(peer_smem_address(acc_empty + buffer, 0));   // the leader's barrier
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync();                                    // the peer is done with this CTA's barriers and TMEM
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * kAccumColumns);
  }
  if (threadIdx.x == 0 && failed) atomicExch(p.error_flag, 1);
}

// ---- align / scatter / slot-sum helper kernels ---------------------------------------------------
constexpr int kAlignThreads = 1024;
constexpr int kMaxLocalExperts = 1024;
constexpr int kAlignClusterMax = 8;

// Rows to work on: the device's count bounded to [0, rows]. A negative count is an empty batch: as an
// unsigned number of a mover's items it would be four billion of them.
__device__ __forceinline__ int usable_rows(int valid_count, int rows) { return max(0, min(valid_count, rows)); }

// Exclusive prefix sum over the CTA's 1024 threads (`warp_sums` is 32 words of shared memory).
__device__ __forceinline__ int warp_inclusive_scan(int v, int lane) {
#pragma unroll
  for (int step = 1; step < 32; step <<= 1) {
    const int below = __shfl_up_sync(0xffffffffu, v, step);
    if (lane >= step) v += below;
  }
  return v;
}
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int upto = warp_inclusive_scan(v, lane);
  __syncthreads();
  if (lane == 31) warp_sums[warp] = upto;
  __syncthreads();
  const int sums = warp_inclusive_scan(warp_sums[lane], lane);      // every warp scans the 32 sums itself
  const int below = __shfl_sync(0xffffffffu, sums, (warp + 31) & 31);
  return (warp == 0 ? 0 : below) + upto - v;
}

// A chain of memory and barrier latencies, not bandwidth. One cluster of 1-8 CTAs packs the local
// (row, slot) pairs by expert: every CTA counts its share of the pairs per expert in shared memory (the counting atomic also ranks the pair inside the
// CTA), the CTAs read each other's counts through distributed shared memory, every CTA derives
// the same prefix sums, and the second pass writes each pair to expert base + CTA base + rank.
// Bounded by the device valid_count, never by a host-side count; order inside an expert is free
// (a row's results do not depend on it). 2048 pairs per CTA is where a second CTA starts to pay for
// the cluster barriers. 32576 pairs, most of them of other ranks' experts: 9 us; 32768 local ones
// inside a layer pass: 13 us, against 64 us for one CTA that counted, then counted again while
// scattering, plus 2.6 us for a launch that preset its outputs; 1024 pairs: 5.5 us against 8.1 + 1.3.
__global__ void __launch_bounds__(kAlignThreads) moe_align_kernel(const long long* __restrict__ local_ids,
                                                                  const float* __restrict__ weights,
                                                                  const int* __restrict__ valid_count, int rows,
                                                                  int topk, int experts, int max_sorted_rows,
                                                                  int tile_cap, int* sorted_row, float* sorted_scale,
                                                                  int* entry_pos, int4* tiles, int* counters,
                                                                  int* error_flag) {
  __shared__ int s_count[kMaxLocalExperts];
  __shared__ int s_base[kMaxLocalExperts];
  __shared__ int s_scan[32];
  unsigned cta, ctas;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cta));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
  const int tid = threadIdx.x;
  s_count[tid] = 0;
  __syncthreads();
  wait_for_previous();
  launch_dependents();
  const int pairs = usable_rows(*valid_count, rows) * topk;
  const int step = static_cast<int>(ctas) * kAlignThreads;
  constexpr int kBatch = 4;                          // independent loads in flight per thread
  // The first batch of a thread stays in registers between the two passes, weights included; up to
  // 32768 pairs there is no other and the second pass loads nothing.
  int held_id[kBatch], held_at[kBatch];
  float held_weight[kBatch];
  for (int first = static_cast<int>(cta) * kAlignThreads + tid, round = 0; first < pairs; first += kBatch * step, ++round) {
    long long id[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) id[b] = first + b * step < pairs ? local_ids[first + b * step] : -1;
    if (round == 0) {
#pragma unroll
      for (int b = 0; b < kBatch; ++b) held_weight[b] = first + b * step < pairs ? weights[first + b * step] : 0.f;
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const bool mine = id[b] >= 0 && id[b] < experts;
      const int at = mine ? atomicAdd(&s_count[id[b]], 1) : -1;
      if (round == 0) {
        held_id[b] = mine ? static_cast<int>(id[b]) : 0;
        held_at[b] = at;
      } else if (first + b * step < pairs) {
        entry_pos[first + b * step] = at;
      }
    }
  }
  cluster_sync();
  // Thread e: rows of expert e in the whole cluster and in the CTAs before this one.
  int mine = 0, before = 0;
  if (tid < experts) {
    unsigned v[kAlignClusterMax];
#pragma unroll
    for (unsigned c = 0; c < kAlignClusterMax; ++c) {  // all CTAs' counts in one round trip
      v[c] = 0;
      if (c < ctas)
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v[c]) : "r"(peer_smem_address(s_count + tid, c)) : "memory");
    }
#pragma unroll
    for (unsigned c = 0; c < kAlignClusterMax; ++c) {
      mine += static_cast<int>(v[c]);
      if (c < cta) before += static_cast<int>(v[c]);
    }
  }
  const int offset = block_exclusive_scan(mine, s_scan);
  s_base[tid] = offset + before;
  if (cta == 0) {
    // Token tiles: an expert's rows in equal parts of at most `tile_cap`, a multiple of 16 each.
    const int usable = max(0, min(mine, max_sorted_rows - offset));
    const int parts = (usable + tile_cap - 1) / tile_cap;
    const int part = parts > 0 ? ((usable + parts - 1) / parts + 15) / 16 * 16 : 0;
    const int at = block_exclusive_scan(parts, s_scan);
    for (int i = 0; i < parts; ++i)
      tiles[at + i] = make_int4(tid, offset + i * part, min(part, usable - i * part), 0);
    if (tid == kAlignThreads - 1) {
      counters[0] = at + parts;
      counters[1] = min(offset + mine, max_sorted_rows);
      if (offset + mine > max_sorted_rows) atomicExch(error_flag, 2);   // the caller's bound on local pairs was too small
    }
  }
  __syncthreads();
  for (int first = static_cast<int>(cta) * kAlignThreads + tid, round = 0; first < pairs; first += kBatch * step, ++round) {
    int at[kBatch], id[kBatch];
    float w[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int i = first + b * step;
      const bool held = round == 0;
      at[b] = held ? held_at[b] : (i < pairs ? entry_pos[i] : -1);
      id[b] = held ? held_id[b] : (i < pairs ? static_cast<int>(local_ids[i]) : -1);
      w[b] = held ? held_weight[b] : (i < pairs ? weights[i] : 0.f);
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int i = first + b * step;
      if (i >= pairs) continue;
      if (at[b] < 0) {
        if (round == 0) entry_pos[i] = -1;
        continue;
      }
      const int pos = s_base[id[b]] + at[b];
      if (pos < max_sorted_rows) {
        sorted_row[pos] = i / topk;
        sorted_scale[pos] = w[b];
      }
      entry_pos[i] = pos < max_sorted_rows ? pos : -1;
    }
  }
  cluster_sync();                                    // nobody leaves while a peer may still read its counts
}

// Both row movers work on units of 128 16-byte vectors (2 KB of a row, four vectors per lane), one
// unit per warp and pass: a single decode row is spread over several warps, and four independent
// 16-byte accesses per lane and slot cover the memory latency of a large batch.
constexpr int kUnitVecs = 128;
__device__ __forceinline__ int units_per_row(int vecs_per_row) { return (vecs_per_row + kUnitVecs - 1) / kUnitVecs; }

// sorted_x[entry_pos[row, slot]] = hidden[row] for every local slot: a row is read ONCE and stored to
// every expert it goes to. HBM bound: 4096 rows x 8 slots x 14 KB (529 MB) in 91 us = 5.8 TB/s;
// gathering per sorted position read each row eight times and wrote padding: 149 us.
__global__ void __launch_bounds__(256) moe_scatter_kernel(const uint4* __restrict__ hidden, const int* __restrict__ entry_pos,
                                                          const int* __restrict__ valid_count, uint4* __restrict__ sorted_x,
                                                          int rows, int topk, int vecs_per_row) {
  wait_for_previous();
  launch_dependents();
  const int lane = threadIdx.x & 31;
  const unsigned units = units_per_row(vecs_per_row);
  const unsigned items = usable_rows(*valid_count, rows) * units;
  const unsigned warps = gridDim.x * (blockDim.x / 32);
  for (unsigned item = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); item < items; item += warps) {
    const unsigned row = item / units;
    const int base = static_cast<int>(item - row * units) * kUnitVecs + lane;
    const int* positions = entry_pos + static_cast<long long>(row) * topk;
    const uint4* src = hidden + static_cast<long long>(row) * vecs_per_row;
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (base + u * 32 < vecs_per_row) v[u] = src[base + u * 32];
    for (int k0 = 0; k0 < topk; k0 += 32) {
      const int mine = k0 + lane < topk ? positions[k0 + lane] : -1;
      for (unsigned local = __ballot_sync(0xffffffffu, mine >= 0); local != 0; local &= local - 1) {
        const int pos = __shfl_sync(0xffffffffu, mine, __ffs(local) - 1);
        uint4* dst = sorted_x + static_cast<long long>(pos) * vecs_per_row;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (base + u * 32 < vecs_per_row) dst[base + u * 32] = v[u];
      }
    }
  }
}

// partial[row] = the row's local slots of y added in slot order. A warp takes kVecs vectors per lane of
// a row and keeps kSlots slots' loads in flight. Large batches are HBM bound with <4, 2> (2 KB units;
// 4096 rows x 8 slots, 529 MB: about 110 us); a decode batch is a chain of latencies, and <1, 8> makes
// the eight slots of a row one round trip instead of four and spreads it over four times the warps.
template <int kVecs, int kSlots>
__global__ void __launch_bounds__(256) moe_slot_sum_kernel(const uint4* __restrict__ y, const int* __restrict__ entry_pos,
                                                           const int* __restrict__ valid_count, uint4* __restrict__ partial,
                                                           int rows, int topk, int vecs_per_row) {
  wait_for_previous();
  launch_dependents();
  const int lane = threadIdx.x & 31;
  const unsigned units = (vecs_per_row + 32 * kVecs - 1) / (32 * kVecs);
  const unsigned items = usable_rows(*valid_count, rows) * units;
  const unsigned warps = gridDim.x * (blockDim.x / 32);
  for (unsigned item = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); item < items; item += warps) {
    const unsigned row = item / units;
    const int base = static_cast<int>(item - row * units) * 32 * kVecs + lane;
    const int* positions = entry_pos + static_cast<long long>(row) * topk;
    unsigned long long acc[kVecs][4];
#pragma unroll
    for (int u = 0; u < kVecs; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[u][i] = 0ull;
    for (int k0 = 0; k0 < topk; k0 += 32) {
      const int mine = k0 + lane < topk ? positions[k0 + lane] : -1;
      unsigned local = __ballot_sync(0xffffffffu, mine >= 0);
      while (local != 0) {
        uint4 v[kSlots][kVecs] = {};
        unsigned taken = 0;
#pragma unroll
        for (int j = 0; j < kSlots; ++j) {
          if (local == 0) break;                       // warp-uniform
          const uint4* src = y + static_cast<long long>(__shfl_sync(0xffffffffu, mine, __ffs(local) - 1)) * vecs_per_row;
          local &= local - 1;
          taken |= 1u << j;
#pragma unroll
          for (int u = 0; u < kVecs; ++u)
            if (base + u * 32 < vecs_per_row) v[j][u] = src[base + u * 32];
        }
#pragma unroll
        for (int j = 0; j < kSlots; ++j) {
          if (!((taken >> j) & 1u)) break;
#pragma unroll
          for (int u = 0; u < kVecs; ++u) {
            acc[u][0] = add_f32x2(acc[u][0], bf16x2_to_f32x2(v[j][u].x));
            acc[u][1] = add_f32x2(acc[u][1], bf16x2_to_f32x2(v[j][u].y));
            acc[u][2] = add_f32x2(acc[u][2], bf16x2_to_f32x2(v[j][u].z));
            acc[u][3] = add_f32x2(acc[u][3], bf16x2_to_f32x2(v[j][u].w));
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      if (base + u * 32 >= vecs_per_row) continue;
      unsigned out[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float lo, hi;
        unpack_f32x2(acc[u][i], lo, hi);
        out[i] = pack_bf16x2(lo, hi);
      }
      partial[static_cast<long long>(row) * vecs_per_row + base + u * 32] = make_uint4(out[0], out[1], out[2], out[3]);
    }
  }
}

// ---- tensor maps ----------------------------------------------------------------------------------
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void* entry = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &result) != cudaSuccess ||
        result != cudaDriverEntryPointSuccess)
      entry = nullptr;
    return reinterpret_cast<EncodeTiled>(entry);
  }();
  return fn;
}

// Row-major BF16 matrix [rows, columns]; box = box_rows x 64 columns, 128-byte swizzle.
bool make_map(CUtensorMap* map, const void* base, long long rows, long long columns, int box_rows) {
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(columns), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(columns) * 2};
  const cuuint32_t box[2] = {kTileK, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t element_strides[2] = {1, 1};
  return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                        element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// w13 [experts, gate/up, inter, hidden] as {hidden, 16 rows, gate/up, inter / 16, experts}; a box of
// {64, 16, 2, 4, 1} is 128 shared-memory rows: 16 gate rows, their 16 up rows, the next 16 gate rows ...
bool make_gate_up_map(CUtensorMap* map, const void* base, int experts, int inter, int hidden) {
  const cuuint64_t row = static_cast<cuuint64_t>(hidden) * 2;
  const cuuint64_t dims[5] = {static_cast<cuuint64_t>(hidden), 16, 2, static_cast<cuuint64_t>(inter / 16),
                              static_cast<cuuint64_t>(experts)};
  const cuuint64_t strides[4] = {row, row * inter, row * 16, row * inter * 2};
  const cuuint32_t box[5] = {kTileK, 16, 2, 4, 1};
  const cuuint32_t element_strides[5] = {1, 1, 1, 1, 1};
  return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box,
                        element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Ring geometry: small batches use narrow token boxes and more stages.
void set_ring(GemmParams* params, int tile_cap) {
  params->b_rows = tile_cap / 2;
  const int stages = kRingBytes / (kABytes + params->b_rows * kTileK * 2);
  params->stages = stages < kMaxStages ? stages : kMaxStages;
}

// Epilogue warps per quadrant: as many as tiles may need, each with 32 tokens. Narrow tiles are bound by
// the weights' stream, and idle warps at the accumulator's barrier slow it down (hidden 7168, inter 2048,
// 32 experts of 32 tokens: four warps 454 us a layer, two 446; 16 experts of 254 tokens, hidden 2048,
// inter 768: one 88, two 83, four 78 us).
int epilogue_shares(const GemmParams& params) {
  const int cap = 2 * params.b_rows;
  return cap >= kMaxTileN ? kMaxEpilogueShare : (cap >= 64 ? 2 : 1);
}

template <int kMode>
cudaError_t launch_gemm(GemmMaps& maps, const GemmParams& params, int sms, cudaStream_t stream) {
  cudaError_t err = cudaFuncSetAttribute(grouped_gemm_kernel<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kGemmSmemBytes));
  if (err != cudaSuccess) return err;
  return launch_chained(grouped_gemm_kernel<kMode>, sms / 2 * 2, 64 + 128 * epilogue_shares(params), 2, kGemmSmemBytes, stream, maps, params);
}

}  // namespace

MoeSizes moe_sizes(long long rows, int topk, int experts, int tile_rows) {
  const long long per_row = topk < experts ? topk : experts;
  const long long entries = rows * per_row;
  MoeSizes sizes;
  sizes.max_tiles = static_cast<int>((entries + tile_rows - 1) / tile_rows + experts);
  sizes.max_sorted_rows = static_cast<long long>(sizes.max_tiles) * tile_rows;
  return sizes;
}

// An expert gets at most one slot of every row (the router chooses without replacement; ids that
// do repeat only cost more tiles), so `rows` bounds the widest useful tile.
int moe_tile_cap(long long rows) {
  int cap = 16;
  while (cap < kMaxTileN && cap < rows) cap *= 2;
  return cap;
}
long long moe_token_tiles(long long max_sorted_rows, int experts) { return max_sorted_rows / 16 + experts; }

cudaError_t launch_moe_align(const long long* local_ids, const float* weights, const int* valid_count, int rows,
                             int topk, int experts, long long max_sorted_rows, int* sorted_row,
                             float* sorted_scale, int* entry_pos, int* tiles, int* counters,
                             int* error_flag, cudaStream_t stream) {
  const long long pairs = static_cast<long long>(rows) * topk;
  if (experts > kMaxLocalExperts || pairs >= (1ll << 30) || max_sorted_rows >= (1ll << 30)) return cudaErrorInvalidValue;
  int cluster = 1;
  while (cluster < kAlignClusterMax && pairs > 2ll * kAlignThreads * cluster) cluster *= 2;
  return launch_chained(moe_align_kernel, cluster, kAlignThreads, cluster, 0, stream, local_ids, weights, valid_count,
                        rows, topk, experts, static_cast<int>(max_sorted_rows), moe_tile_cap(rows), sorted_row, sorted_scale, entry_pos,
                        reinterpret_cast<int4*>(tiles), counters, error_flag);
}

// CTAs of a row mover: one warp per unit, at most eight CTAs of eight warps per SM.
static int mover_ctas(long long rows, int hidden_size) {
  const long long items = rows * ((hidden_size / 8 + kUnitVecs - 1) / kUnitVecs);
  return items < 148 * 8 * 8 ? static_cast<int>((items + 7) / 8) : 148 * 8;
}

cudaError_t launch_moe_scatter(const void* hidden, const int* entry_pos, const int* valid_count, void* sorted_x,
                               int rows, int topk, int hidden_size, cudaStream_t stream) {
  if (hidden_size % 8) return cudaErrorInvalidValue;
  if (rows <= 0) return cudaSuccess;
  return launch_chained(moe_scatter_kernel, mover_ctas(rows, hidden_size), 256, 1, 0, stream,
                        static_cast<const uint4*>(hidden), entry_pos, valid_count, static_cast<uint4*>(sorted_x), rows,
                        topk, hidden_size / 8);
}

cudaError_t launch_moe_gemm_gate_up(const void* sorted_x, const void* w13, void* act, const int* counters,
                                    const int* tiles, int* error_flag, long long rows, long long max_sorted_rows,
                                    int experts, int hidden_size, int inter_size, int sms, cudaStream_t stream,
                                    const int* gather_rows, long long gather_height) {
  if (hidden_size % kTileK || inter_size % kMoeGateUpTile) return cudaErrorInvalidValue;
  if (rows <= 0) return cudaSuccess;     // (no scatter launch stands between this kernel and the align step then)
  if (gather_rows != nullptr && (gather_height <= 0 || gather_height >= (1ll << 31))) return cudaErrorInvalidValue;
  if (encode_tiled() == nullptr) return cudaErrorNotSupported;
  GemmMaps maps{};
  GemmParams params{};
  set_ring(&params, moe_tile_cap(rows));
  bool ok = make_gate_up_map(&maps.a, w13, experts, inter_size, hidden_size);
  if (gather_rows != nullptr) {
    ok = ok && make_map(&maps.b[0], sorted_x, gather_height, hidden_size, 1);   // gather copies take one-row boxes
  } else {
    for (int i = 0; i < kNMaps && (8 << i) <= params.b_rows; ++i)
      ok = ok && make_map(&maps.b[i], sorted_x, max_sorted_rows, hidden_size, 8 << i);
  }
  if (!ok) return cudaErrorInvalidValue;
  params.counters = counters;
  params.tiles = reinterpret_cast<const int4*>(tiles);
  params.out = act;
  params.error_flag = error_flag;
  params.k_steps = hidden_size / kTileK;
  params.m_tiles = inter_size / kMoeGateUpTile;
  params.out_columns = inter_size;
  params.gather_rows = gather_rows;
  params.gather_height = static_cast<int>(gather_height);
  return launch_gemm<0>(maps, params, sms, stream);
}

cudaError_t launch_moe_gemm_down(const void* act, const void* w2, void* y, const float* sorted_scale,
                                 const int* counters, const int* tiles, int* error_flag, long long rows,
                                 long long max_sorted_rows, int experts, int hidden_size, int inter_size, int sms,
                                 cudaStream_t stream) {
  if (inter_size % kTileK || hidden_size % kMoeDownTile) return cudaErrorInvalidValue;
  if (rows <= 0) return cudaSuccess;
  if (encode_tiled() == nullptr) return cudaErrorNotSupported;
  GemmMaps maps{};
  GemmParams params{};
  set_ring(&params, moe_tile_cap(rows));
  bool ok = make_map(&maps.a, w2, static_cast<long long>(experts) * hidden_size, inter_size, 128);
  for (int i = 0; i < kNMaps && (8 << i) <= params.b_rows; ++i)
    ok = ok && make_map(&maps.b[i], act, max_sorted_rows, inter_size, 8 << i);
  if (!ok) return cudaErrorInvalidValue;
  params.counters = counters;
  params.tiles = reinterpret_cast<const int4*>(tiles);
  params.row_scale = sorted_scale;
  params.out = y;
  params.error_flag = error_flag;
  params.k_steps = inter_size / kTileK;
  params.m_tiles = hidden_size / kMoeDownTile;
  params.out_columns = hidden_size;
  return launch_gemm<1>(maps, params, sms, stream);
}

cudaError_t launch_moe_slot_sum(const void* y, const int* entry_pos, const int* valid_count, void* partial,
                                int rows, int topk, int hidden_size, cudaStream_t stream) {
  if (hidden_size % 8) return cudaErrorInvalidValue;
  if (rows <= 0) return cudaSuccess;
  // One wave of warps with one vector per lane, or the streaming form.
  const int vecs = hidden_size / 8;
  const long long small = static_cast<long long>(rows) * ((vecs + 31) / 32);
  if (small <= 148 * 64)
    return launch_chained(moe_slot_sum_kernel<1, 8>, static_cast<int>((small + 7) / 8), 256, 1, 0, stream,
                          static_cast<const uint4*>(y), entry_pos, valid_count, static_cast<uint4*>(partial), rows, topk, vecs);
  return launch_chained(moe_slot_sum_kernel<4, 2>, mover_ctas(rows, hidden_size), 256, 1, 0, stream,
                        static_cast<const uint4*>(y), entry_pos, valid_count, static_cast<uint4*>(partial), rows, topk, vecs);
}

}  // namespace epx
