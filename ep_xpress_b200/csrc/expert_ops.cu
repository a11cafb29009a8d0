// Small helper kernels around the transport: the synthetic "identity times
// routing weight" expert used for validation and for the communication
// benchmark, and the one-time reset of a fresh slot.
//
// The synthetic expert is the one the reference validates with
// (benchmarks/replay.py:67-71): every received row is scaled by the sum, over
// the slots whose expert lives on this rank, of weight * per-expert factor.
// The scale is accumulated in FP32 in slot order with separately rounded
// multiply and add so that a CPU oracle reproduces it bit for bit.
#include <cuda_bf16.h>
#include "epx_device.cuh"
#include "epx_launch.h"

namespace epx {
namespace {

// Bound by HBM for large batches and by latency for small ones. A warp takes `unit` 16-byte vectors of
// a row: the whole row when there are rows enough to fill the chip, else 2 KB, so that a decode batch
// is spread over the SMs too (128 x 7168: 5.3 us a row per warp). The payload's loads leave before the
// scale is computed.
__global__ void __launch_bounds__(256) scale_rows_kernel(const unsigned short* __restrict__ hidden,
                                                         const long long* __restrict__ local_ids,
                                                         const float* __restrict__ weights,
                                                         const int* __restrict__ valid_count,
                                                         const float* __restrict__ factors, int num_factors,
                                                         unsigned short* __restrict__ partial, int capacity,
                                                         int hidden_size, int topk, int unit, int units) {
  wait_for_previous();
  launch_dependents();
  const int valid = min(*valid_count, capacity);
  const int warps_per_cta = blockDim.x / 32;
  const int lane = threadIdx.x & 31;
  const bool vec = (hidden_size % 8 == 0) && (reinterpret_cast<size_t>(hidden) % 16 == 0) &&
                   (reinterpret_cast<size_t>(partial) % 16 == 0);
  const long long items = static_cast<long long>(valid) * units;
  for (long long item = static_cast<long long>(blockIdx.x) * warps_per_cta + (threadIdx.x >> 5); item < items;
       item += static_cast<long long>(gridDim.x) * warps_per_cta) {
    const long long row = units == 1 ? item : item / units;
    const int first = static_cast<int>(item - row * units) * unit;
    const int last = min(first + unit, (hidden_size + 7) / 8);
    const unsigned short* src = hidden + row * hidden_size;
    unsigned short* dst = partial + row * hidden_size;
    constexpr int kUnroll = 8;   // 128 bytes per lane in flight: the kernel is a pure HBM stream, bound by latency
    uint4 v[kUnroll];
    auto fetch = [&](int base) {
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        if (base + u * 32 < last) v[u] = reinterpret_cast<const uint4*>(src)[base + u * 32];
    };
    if (vec) fetch(first + lane);
    // Lanes fetch the slots in parallel (one memory round trip), then the scale is
    // accumulated in slot order from registers, so the arithmetic stays sequential.
    float scale = 0.f;
    for (int k0 = 0; k0 < topk; k0 += 32) {
      const int k = k0 + lane;
      float term = 0.f;
      bool local = false;
      if (k < topk) {
        const long long id = local_ids[row * topk + k];
        const float weight = weights[row * topk + k];
        if (id >= 0) {
          const float f = factors != nullptr ? factors[id < num_factors ? id : num_factors - 1] : 1.f;
          term = __fmul_rn(weight, f);
          local = true;
        }
      }
      const unsigned votes = __ballot_sync(0xffffffffu, local);
      const int span = min(32, topk - k0);
      for (int j = 0; j < span; ++j) {
        const float t = __shfl_sync(0xffffffffu, term, j);
        if ((votes >> j) & 1u) scale = __fadd_rn(scale, t);
      }
    }
    if (vec) {
      for (int base = first + lane; base < last; base += 32 * kUnroll) {
        if (base != first + lane) fetch(base);
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          if (base + u * 32 >= last) continue;
          unsigned* w = reinterpret_cast<unsigned*>(&v[u]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float lo = __fmul_rn(__uint_as_float(w[q] << 16), scale);
            const float hi = __fmul_rn(__uint_as_float(w[q] & 0xffff0000u), scale);
            w[q] = pack_bf16x2(lo, hi);
          }
          reinterpret_cast<uint4*>(dst)[base + u * 32] = v[u];
        }
      }
    } else {
      for (int i = first * 8 + lane; i < min(last * 8, hidden_size); i += 32)
        dst[i] = float_to_bf16_bits(__fmul_rn(bf16_bits_to_float(src[i]), scale));
    }
  }
}

__global__ void __launch_bounds__(256) slot_reset_kernel(char* slot, SlotLayout l, long long capacity, int hidden,
                                                         int topk) {
  const long long threads = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long me = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  unsigned* hid = reinterpret_cast<unsigned*>(slot + l.hidden);
  unsigned* part = reinterpret_cast<unsigned*>(slot + l.partial);
  const long long words = capacity * hidden / 2;
  for (long long i = me; i < words; i += threads) { hid[i] = 0u; part[i] = 0u; }
  long long* ids = reinterpret_cast<long long*>(slot + l.ids);
  float* w = reinterpret_cast<float*>(slot + l.weights);
  for (long long i = me; i < capacity * topk; i += threads) { ids[i] = -1; w[i] = 0.f; }
  long long* inv = reinterpret_cast<long long*>(slot + l.inverse);
  for (long long i = me; i < capacity * 2; i += threads) inv[i] = -1;
  // Arrival words behind the staging rows must never equal a combine epoch by accident (a
  // re-used heap range holds old payload): the whole plane starts at zero.
  uint4* stage = reinterpret_cast<uint4*>(slot + l.staging);
  const long long stage_vecs = static_cast<long long>(l.partial - l.staging) / 16;
  for (long long i = me; i < stage_vecs; i += threads) stage[i] = make_uint4(0u, 0u, 0u, 0u);
  unsigned* local = reinterpret_cast<unsigned*>(slot + l.mask);
  const long long local_words = static_cast<long long>(l.output - l.mask) / 4;
  for (long long i = me; i < local_words; i += threads) local[i] = 0u;
}

}  // namespace

cudaError_t launch_scale_rows(const void* hidden, const long long* local_ids, const float* weights,
                              const int* valid_count, const float* factors, int num_factors, void* partial,
                              int capacity, int hidden_size, int topk, cudaStream_t stream) {
  if (capacity <= 0) return cudaSuccess;
  const int vecs = (hidden_size + 7) / 8, split = (vecs + 127) / 128;
  const bool whole = capacity >= 148 * 8;      // a row per warp fills the SMs
  const int unit = whole ? vecs : 128, units = whole ? 1 : split;
  const long long items = static_cast<long long>(capacity) * units;
  const int ctas = items < 8 * 148 * 8 ? static_cast<int>((items + 7) / 8) : 148 * 8;
  return launch_chained(scale_rows_kernel, ctas, 256, 1, 0, stream, static_cast<const unsigned short*>(hidden), local_ids,
                        weights, valid_count, factors, num_factors, static_cast<unsigned short*>(partial), capacity,
                        hidden_size, topk, unit, units);
}

cudaError_t launch_slot_reset(char* slot, SlotLayout layout, long long capacity, int hidden, int topk,
                              cudaStream_t stream) {
  slot_reset_kernel<<<148 * 4, 256, 0, stream>>>(slot, layout, capacity, hidden, topk);
  return cudaGetLastError();
}

}  // namespace epx
