// What the two forms of the Gate/Up kernel share: parameters and the walk over work items.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

namespace gg {

// A few integers for a host that polls: the first word arrives last.
struct HostReport {
  const int* values;
  int* words;       // page-locked host memory; null: nothing to report
  int count;
};
// By a warp that has nothing else to do: as a kernel of its own, or in front of other work of one, the
// way over PCIe cost 1.5 us of a decode step.
__device__ __forceinline__ void report_to_polling_host(const HostReport& report, int lane) {
  if (report.words == nullptr || blockIdx.x != 0 || lane != 0) return;
  for (int i = 1; i < report.count; ++i) report.words[i] = report.values[i];
  __threadfence_system();
  *const_cast<volatile int*>(report.words) = report.values[0];
}

struct GateUpParams {
  const float* row_scale;     // gathered: scale_x [T, H/256]; pre-sorted: [S, H/256] by sorted slot
  const long long* order;     // [S] sorted slot -> flattened assignment (gathered mode)
  int top_k;                  // assignment / top_k = token
  const float* silu_table;    // [65536] silu of every value of the output type, by bit pattern
  const float* scale_w;       // [E, H/256, 2I]
  const int* expert_offsets;  // [E+1]
  const int* tile_expert;     // [max_tiles]
  const int* tile_row;        // [max_tiles]
  int8_t* q;                  // [S, I]
  float* s;                   // [S, I/256]
  int hidden, intermediate, max_tiles, interleaved;
  int sw_vectors;             // scale_w starts on a 16-byte boundary
  HostReport report;          // routing statistics for a host that polls
};

// Work item -> (row tile, channel group).  Items of one expert are consecutive and ordered
// channel-group-major: neighbouring CTAs work on different row tiles of the same expert
// against the same 256-channel weight block, so that block is read from DRAM once and served
// from L2 to the other row tiles.  Returns false for items past the last used tile.
__device__ __forceinline__ bool gate_up_item(const GateUpParams& p, int item, int channel_groups,
                                             int& tile, int& jg, int& expert) {
  const int probe = item / channel_groups;
  expert = p.tile_expert[probe];
  if (expert < 0) return false;
  const int begin = p.expert_offsets[expert];
  const int rows = p.expert_offsets[expert + 1] - begin;
  const int first = probe - (p.tile_row[probe] - begin) / 128;
  const int span = (rows + 127) / 128;
  const int local = item - first * channel_groups;
  jg = local / span;
  tile = first + local - jg * span;
  return true;
}

// The two 16-bit floats of a packed pair as FP32 (exact).
template <typename T>
__device__ __forceinline__ float2 unpack_pair(uint32_t packed) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    return make_float2(__uint_as_float(packed << 16), __uint_as_float(packed & 0xffff0000u));
  } else {
    return __half22float2(*reinterpret_cast<const __half2*>(&packed));
  }
}

}  // namespace gg
