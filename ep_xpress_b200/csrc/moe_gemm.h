// Host API of the grouped SwiGLU expert runner (plain C++, no torch types).
//
// The stages replace what the reference borrows from its serving framework and patches for a
// device-resident row count: route alignment (ep_xpress/adapters/sglang_valid.py:13-161), the
// grouped GEMMs with SiLU-and-mul in between (sglang_valid.py:233-255 and the act_and_mul patch,
// ep_xpress/adapters/sglang/sglang-v0.5.21.patch:281-330) and the slot-order FP32 sum with one
// BF16 rounding (sglang_valid.py:206-222).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace epx {

constexpr int kMoeTileRows = 128;     // granularity of the workspace bound below
constexpr int kMoeGateUpTile = 128;   // intermediate columns produced by one GEMM-1 tile
constexpr int kMoeDownTile = 256;     // hidden columns produced by one GEMM-2 tile

struct MoeSizes {
  long long max_sorted_rows;   // workspace rows: every local pair, and up to experts + 1 tiles of slack that no kernel needs
  int max_tiles;               // the same in tiles of `tile_rows`
};

// CPU-known bounds for `rows` received rows, `topk` slots per row and `experts` local experts.
MoeSizes moe_sizes(long long rows, int topk, int experts, int tile_rows = kMoeTileRows);
// Entries of the token-tile list for `max_sorted_rows` sorted rows.
long long moe_token_tiles(long long max_sorted_rows, int experts);

// Packs the (row, slot) pairs of this rank's experts by expert (no padding between experts) and
// cuts every expert's rows into token tiles.
//   sorted_row   int32 [max_sorted_rows]  source row of every sorted position
//   sorted_scale f32   [max_sorted_rows]  routing weight of the pair
//   entry_pos    int32 [rows * topk]      sorted position of the pair, -1 when not local (rows below *valid_count)
//   tiles        int32 [moe_token_tiles][4]  {expert, first sorted row, rows, 0}, 16-byte aligned
//   counters     int32 [2]                {tiles in use, sorted rows in use}
//   error_flag   int32 [1]                set to 2 when max_sorted_rows was too small (pairs are dropped)
cudaError_t launch_moe_align(const long long* local_ids, const float* weights, const int* valid_count, int rows,
                             int topk, int experts, long long max_sorted_rows, int* sorted_row, float* sorted_scale,
                             int* entry_pos, int* tiles, int* counters, int* error_flag, cudaStream_t stream);

// sorted_x[entry_pos[row, slot]] = hidden[row] for every local slot of the rows below *valid_count.
cudaError_t launch_moe_scatter(const void* hidden, const int* entry_pos, const int* valid_count, void* sorted_x,
                               int rows, int topk, int hidden_size, cudaStream_t stream);

// GEMM 1: act[pos, :] = silu(x W1_e) * (x W3_e).  w13 is [experts, 2 * inter, hidden] (gate rows
// first, then up rows), K-major. GEMM 2: y[pos, :] = (act W2_e) * sorted_scale[pos], w2 is
// [experts, hidden, inter]. Shapes: hidden % 256 == 0, inter % 128 == 0. `rows` is the same bound
// that was given to the align step. With `gather_rows` (= the align step's sorted_row), `sorted_x`
// is the UNSORTED activation matrix [gather_height, hidden]: the kernel's TMA producer gathers the
// rows of every tile itself (four rows per copy) and no scatter launch or sorted copy is needed.
// Order: without `gather_rows` both GEMMs read `counters` and `tiles` BEFORE they wait for the kernel
// launched before them on the stream. A launch that itself waits for the align step therefore has to
// stand between it and them (the scatter; for the second GEMM, the first); right behind the align step
// they would read a half-written list.
cudaError_t launch_moe_gemm_gate_up(const void* sorted_x, const void* w13, void* act, const int* counters,
                                    const int* tiles, int* error_flag, long long rows, long long max_sorted_rows,
                                    int experts, int hidden_size, int inter_size, int sms, cudaStream_t stream,
                                    const int* gather_rows = nullptr, long long gather_height = 0);
cudaError_t launch_moe_gemm_down(const void* act, const void* w2, void* y, const float* sorted_scale,
                                 const int* counters, const int* tiles, int* error_flag, long long rows,
                                 long long max_sorted_rows, int experts, int hidden_size, int inter_size, int sms,
                                 cudaStream_t stream);

// partial[row] = bf16(sum over slots, in slot order, of float(y[entry_pos[row, slot]])) for rows
// below *valid_count.
cudaError_t launch_moe_slot_sum(const void* y, const int* entry_pos, const int* valid_count, void* partial,
                                int rows, int topk, int hidden_size, cudaStream_t stream);

}  // namespace epx
