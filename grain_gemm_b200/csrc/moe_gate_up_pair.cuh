// Gate/Up for few rows an expert: weight rows on the tensor core's M side, token rows on its N side.
//
// Same operation and same bits as moe_gate_up_tc.cuh, for calls in which most row tiles are far from
// full.  There the 128 lanes of an accumulator are token rows, and a tile with 4 or 30 of them
// pays for 128: operand bytes in shared memory, tensor-core time, promotion.  Here the lanes are weight
// rows, of which there are always enough, and the columns are the tile's tokens: an MMA is
// as wide as there are tokens (in steps of 32), the promotion walks blocks of 32 tokens, and
// a stage of the operand ring spends its room on weights.
//
// A work item (row tile of one expert, 256-channel group) goes to a cluster of two CTAs, 128 channels
// = 256 weight rows each, that exchange the tokens' maxima through distributed shared memory.
//   warp 8    TMA producer: per 128 bytes of K one box of 256 weight rows and one of 16 rows per token block
//   warp 9    MMA issuer of the leader CTA: two cta_group::2 MMAs a K step, each over one M tile (64 channels)
//             of either CTA; a CTA holds half of the token rows.  Two TMEM buffers of 2 x 128 columns.
//   warp 10   scale staging, as in the other kernels
//   warp 11   hands routing statistics to the host where they are asked for
//   warps 0-7 promotion: warp (quarter, half) holds lanes 32 * quarter.. of M tile `half` for all tokens;
//             then SwiGLU, maxima, requantisation.
//
// The tensor map delivers weight rows so that lane 16u + 8j + r of a 32-lane quarter is channel
// 16 * quarter + 2r + j, gate (u = 0) or up (u = 1).  A thread's four rows r, r + 8, r + 16, r + 24 are the
// gate and up values of two neighbouring channels: SwiGLU needs no exchange, the layouts "split" and
// "interleaved" differ in the map's strides only, and a reduction over the eight lanes r that
// halves the tokens a lane holds at every step ends with lane l holding token l of the block.
//
// What bounds it: for few rows the weights' way from HBM.  16 tokens over 8 experts, H = 4096, I = 14336, read
// 0.94 GB in 155 us (6.1 TB/s; token rows on the M side: 185 us, 5.1 TB/s), one token over 8 of 128 experts,
// H = 2048, I = 768, 25 MB in 12.0 us (18): 8000 cycles of K loop, 3000 behind it, the rest before it.  For full
// tiles the epilogue: a group takes the GEMM's 1550 cycles, SwiGLU 4400, the exchange 1200 and the
// requantisation 4700 an item and CTA, more than the single CTA's (gate_up_pairs in abi.cu has both).
#pragma once

#include "gemm_tc.cuh"
#include "moe_gate_up.cuh"
#include "moe_route.cuh"
#include "ptx.cuh"

namespace gg {

struct GateUpPairShape {
  static constexpr int kStages = 4;
  static constexpr int kWeightBytes = 256 * 128;
  static constexpr int kBlockBytes = 16 * 128;             // a CTA's token rows of one block
  static constexpr int kStageBytes = kWeightBytes + 4 * kBlockBytes;
  static constexpr int kRingFloats = 256 + 128;            // weight-row scales, then token scales
  static constexpr int kScaleSlots = 8;
  static constexpr int kScaleChunks = kScaleSlots / kScaleChunkGroups;
  static constexpr int kScaleBytes = kScaleSlots * kRingFloats * 4;
  static constexpr int kSources = 16;                      // promotion warps of both CTAs
  static constexpr int kMaximaBytes = 2 * kSources * 128 * 4;
  static constexpr int kBarriers = 2 * kStages + 4 + 2 * kScaleChunks + 2;
  static constexpr int kSmemBytes =
      1024 + kStages * kStageBytes + kScaleBytes + kMaximaBytes + kBarriers * 8 + 16;
};

// Running state of a promotion warp over its items.
struct GateUpPairState {
  uint32_t group_sequence = 0, scale_chunk = 0, scale_phase = 0;
  uint32_t item_parity = 0, item_phase = 0;
  bool ok = true;
};

struct GateUpPairSmem {
  uint8_t* stages;
  float* ring;
  float* maxima;
  uint64_t *full, *empty, *tmem_full, *tmem_empty, *scale_full, *scale_empty, *exchange;
  uint32_t* tmem_holder;
  volatile int* abort_flag;
};

// max over the eight lanes of equal lane % 4 for eight tokens at a time (token 4k + lane % 4 in
// v[k]); lane l ends with token l.
__device__ __forceinline__ float max_to_token_lane(const float (&v)[8], int lane) {
  const bool b0 = lane & 4, b1 = lane & 8, b2 = lane & 16;
  float a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float other = __shfl_xor_sync(0xffffffffu, b0 ? v[2 * i] : v[2 * i + 1], 4);
    a[i] = fmaxf(b0 ? v[2 * i + 1] : v[2 * i], other);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float other = __shfl_xor_sync(0xffffffffu, b1 ? a[2 * i] : a[2 * i + 1], 8);
    b[i] = fmaxf(b1 ? a[2 * i + 1] : a[2 * i], other);
  }
  const float other = __shfl_xor_sync(0xffffffffu, b2 ? b[0] : b[1], 16);
  return fmaxf(b2 ? b[1] : b[0], other);
}

// The same walk for codes: v[k] holds in its low half the codes of channels 2r, 2r + 1 (r = lane / 4)
// for token 4k + lane % 4; lane l ends with the 16 channels of token l, in order.
__device__ __forceinline__ uint4 codes_to_token_lane(const uint32_t (&v)[8], int lane) {
  const bool b0 = lane & 4, b1 = lane & 8, b2 = lane & 16;
  uint32_t t[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t even = __byte_perm(v[4 * i], v[4 * i + 2], 0x5410);
    const uint32_t odd = __byte_perm(v[4 * i + 1], v[4 * i + 3], 0x5410);
    const uint32_t keep = b0 ? odd : even;
    const uint32_t other = __shfl_xor_sync(0xffffffffu, b0 ? even : odd, 4);
    t[2 * i] = __byte_perm(keep, other, b0 ? 0x1054 : 0x5410);
    t[2 * i + 1] = __byte_perm(keep, other, b0 ? 0x3276 : 0x7632);
  }
  uint32_t s[2][2];   // [token][channels 0..3, 4..7 of the half]
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t keep = b1 ? t[2 * i + 1] : t[2 * i];
    const uint32_t other = __shfl_xor_sync(0xffffffffu, b1 ? t[2 * i] : t[2 * i + 1], 8);
    s[i][0] = b1 ? other : keep;
    s[i][1] = b1 ? keep : other;
  }
  const uint32_t keep0 = b2 ? s[1][0] : s[0][0], keep1 = b2 ? s[1][1] : s[0][1];
  const uint32_t other0 = __shfl_xor_sync(0xffffffffu, b2 ? s[0][0] : s[1][0], 16);
  const uint32_t other1 = __shfl_xor_sync(0xffffffffu, b2 ? s[0][1] : s[1][1], 16);
  return b2 ? make_uint4(other0, other1, keep0, keep1) : make_uint4(keep0, keep1, other0, other1);
}

// One item in a promotion warp: K loop, SwiGLU, exchange of maxima, requantisation.  kBlocks token
// blocks of 32.
template <typename RoundT, int kBlocks>
__device__ __forceinline__ void gate_up_pair_item(const GateUpParams& p, const GateUpPairSmem& m, GateUpPairState& state,
                                                  uint32_t tmem_base, int warp, int lane, uint32_t cta_rank,
                                                  int groups, int row0, int row_end, int channel_group) {
  using Shape = GateUpPairShape;
  const int half = warp >> 2, quarter = warp & 3, fragment_row = lane >> 2, quad = lane & 3;
  float2 acc[4][4 * kBlocks];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int i = 0; i < 4 * kBlocks; ++i) acc[r][i] = make_float2(0.0f, 0.0f);
  }
  for (int g = 0; g < groups; ++g, ++state.group_sequence) {
    const int in_chunk = g & (kScaleChunkGroups - 1);
    if (in_chunk == 0 && state.ok) {
      state.ok = mbar_wait_warp(&m.scale_full[state.scale_chunk], state.scale_phase, kSiteScaleFull, m.abort_flag);
    }
    const float* slot = m.ring + (state.scale_chunk * kScaleChunkGroups + in_chunk) * Shape::kRingFloats;
    // Scales of this thread's rows: gate 2r, gate 2r + 1, up 2r, up 2r + 1; the interleaved layout
    // keeps them as gate 2r, up 2r, gate 2r + 1, up 2r + 1.
    float4 rows = lds_f32x4(smem_u32(slot + (half * 4 + quarter) * 32 + fragment_row * 4));
    if (p.interleaved) {
      const float up = rows.y;
      rows.y = rows.z;
      rows.z = up;
    }
    const float2 scale[4] = {make_float2(rows.x, rows.x), make_float2(rows.y, rows.y),
                             make_float2(rows.z, rows.z), make_float2(rows.w, rows.w)};
    const uint32_t buffer = state.group_sequence & 1u;
    if (state.ok) {
      state.ok = mbar_wait_warp(&m.tmem_full[buffer], (state.group_sequence >> 1) & 1u, kSiteEpilogueTmemFull,
                                m.abort_flag);
    }
    tcgen05_fence_after();
    const uint32_t taddr_low = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buffer * 256 + half * 128;
    const uint32_t taddr_high = taddr_low + (16u << 16);
    uint32_t partial_a[16], partial_b[16];
    float2 tokens[4];
    tmem_ld_16x128b_x8(taddr_low, partial_a);
#pragma unroll
    for (int fragment = 0; fragment < 2 * kBlocks; ++fragment) {
      const int block = fragment >> 1;
      if ((fragment & 1) == 0) load_column_scales(smem_u32(slot + 256 + block * 32 + quad * 8), tokens);
      tmem_ld_wait();
      if (fragment + 1 < 2 * kBlocks) {
        const uint32_t next = ((fragment + 1) & 1 ? taddr_high : taddr_low) + ((fragment + 1) >> 1) * 32;
        if (fragment & 1) tmem_ld_16x128b_x8(next, partial_a);
        else tmem_ld_16x128b_x8(next, partial_b);
      } else {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(&m.tmem_empty[buffer], 0);
      }
      if (fragment & 1) {
        promote_fragment(partial_b, scale[2], scale[3], tokens, &acc[2][block * 4], &acc[3][block * 4]);
      } else {
        promote_fragment(partial_a, scale[0], scale[1], tokens, &acc[0][block * 4], &acc[1][block * 4]);
      }
    }
    if (in_chunk == kScaleChunkGroups - 1 || g == groups - 1) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&m.scale_empty[state.scale_chunk]);
      if (++state.scale_chunk == Shape::kScaleChunks) {
        state.scale_chunk = 0;
        state.scale_phase ^= 1u;
      }
    }
  }

  // SwiGLU on the rounded gate and up values; h of channels 2r, 2r + 1 and token 4k + quad of block b
  // take the place of the gate accumulators: acc[0] and acc[1], pair k / 2, x for even k.
  float* maxima = m.maxima + state.item_parity * (Shape::kSources * 128);
  const int source = static_cast<int>(cta_rank) * 8 + warp;     // 16 channels of the item's 256
#pragma unroll
  for (int b = 0; b < kBlocks; ++b) {
    float largest[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t gate0 = pack_pair<RoundT>(acc[0][b * 4 + i]), gate1 = pack_pair<RoundT>(acc[1][b * 4 + i]);
      const float2 up0 = unpack_pair<RoundT>(pack_pair<RoundT>(acc[2][b * 4 + i]));
      const float2 up1 = unpack_pair<RoundT>(pack_pair<RoundT>(acc[3][b * 4 + i]));
      float2& h0 = acc[0][b * 4 + i];
      float2& h1 = acc[1][b * 4 + i];
      h0.x = __fmul_rn(__ldg(p.silu_table + (gate0 & 0xffffu)), up0.x);
      h0.y = __fmul_rn(__ldg(p.silu_table + (gate0 >> 16)), up0.y);
      h1.x = __fmul_rn(__ldg(p.silu_table + (gate1 & 0xffffu)), up1.x);
      h1.y = __fmul_rn(__ldg(p.silu_table + (gate1 >> 16)), up1.y);
      largest[2 * i] = fmaxf(fabsf(h0.x), fabsf(h1.x));
      largest[2 * i + 1] = fmaxf(fabsf(h0.y), fabsf(h1.y));
    }
    float* mine = maxima + source * 128 + b * 32 + lane;
    const float token_max = max_to_token_lane(largest, lane);
    *mine = token_max;
    store_cluster_f32(mine, cta_rank ^ 1u, token_max);
  }
  // The tokens' maxima from all promotion warps, here and in the peer CTA.  A warp that has failed
  // arrives all the same.  Maxima and barriers alternate between two sets: a warp that arrives
  // for item n + 2 has seen the arrivals for n + 1, which the other warps make after their reads for
  // n, so that neither an arrival nor a store runs ahead into a set still in use.
  uint64_t* exchange = &m.exchange[state.item_parity];
  __syncwarp();
  if (lane == 0) {
    mbar_arrive(exchange);
    mbar_arrive_cluster_release(exchange, cta_rank ^ 1u);
  }
  if (state.ok) state.ok = mbar_wait_warp<true>(exchange, state.item_phase, kSiteDrain, m.abort_flag);

#pragma unroll
  for (int b = 0; b < kBlocks; ++b) {
    float row_max = 0.0f;
#pragma unroll
    for (int s = 0; s < Shape::kSources; ++s) row_max = fmaxf(row_max, maxima[s * 128 + b * 32 + lane]);
    const int row = row0 + b * 32 + lane;          // this lane's token of the block
    const bool row_stored = state.ok && row < row_end;
    const RowQuantizer own(row_max);
    uint32_t code[8];
    // The branch stands outside the loop, so that the eight tokens' chains interleave.
    if (__all_sync(0xffffffffu, own.by_fma)) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float2 h0 = acc[0][b * 4 + (k >> 1)], h1 = acc[1][b * 4 + (k >> 1)];
        // Scale of token 4k + quad, from the lane that holds it.
        const float minus_scale = __shfl_sync(0xffffffffu, own.minus_scale.x, 4 * k + quad);
        const float y = __shfl_sync(0xffffffffu, own.y.x, 4 * k + quad);
        const float2 pair = quantize_pair_by_fma(k & 1 ? make_float2(h0.y, h1.y) : make_float2(h0.x, h1.x),
                                                 make_float2(minus_scale, minus_scale), make_float2(y, y));
        code[k] = __byte_perm(__float_as_uint(pair.x), __float_as_uint(pair.y), 0x0040);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float2 h0 = acc[0][b * 4 + (k >> 1)], h1 = acc[1][b * 4 + (k >> 1)];
        const float scale = __shfl_sync(0xffffffffu, own.scale, 4 * k + quad);
        code[k] = __byte_perm(static_cast<uint32_t>(quantize_value(k & 1 ? h0.y : h0.x, scale)),
                              static_cast<uint32_t>(quantize_value(k & 1 ? h1.y : h1.x, scale)), 0x0040);
      }
    }
    const uint4 channels = codes_to_token_lane(code, lane);
    const int channel0 = channel_group * 256 + source * 16;
    if (row_stored) {
      *reinterpret_cast<uint4*>(p.q + static_cast<long long>(row) * p.intermediate + channel0) = channels;
      if (source == 0) {
        p.s[static_cast<long long>(row) * (p.intermediate / 256) + channel_group] = own.scale;
      }
    }
  }
  state.item_parity ^= 1u;
  if (state.item_parity == 0) state.item_phase ^= 1u;
}

// map_x covers the sorted rows [S, H] in boxes of 16 rows, map_w the weight rows (gate_up_channel_map).
template <typename RoundT>
__device__ __forceinline__ void gate_up_pair_body(const CUtensorMap& map_x, const CUtensorMap& map_w,
                                                  const GateUpParams& p) {
  using Shape = GateUpPairShape;
  constexpr int kStages = Shape::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  GateUpPairSmem m;
  m.stages = smem;
  m.ring = reinterpret_cast<float*>(smem + kStages * Shape::kStageBytes);
  m.maxima = m.ring + Shape::kScaleBytes / 4;
  m.full = reinterpret_cast<uint64_t*>(m.maxima + Shape::kMaximaBytes / 4);
  m.empty = m.full + kStages;
  m.tmem_full = m.empty + kStages;
  m.tmem_empty = m.tmem_full + 2;
  m.scale_full = m.tmem_empty + 2;
  m.scale_empty = m.scale_full + Shape::kScaleChunks;
  m.exchange = m.scale_empty + Shape::kScaleChunks;
  m.tmem_holder = reinterpret_cast<uint32_t*>(m.exchange + 2);
  m.abort_flag = reinterpret_cast<volatile int*>(m.tmem_holder + 1);

  // The same in every lane, and known to be: addresses built from it stay in uniform registers.
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int channel_groups = p.intermediate / 256;
  const int groups = p.hidden / 256;
  const int slabs = p.hidden / 128;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&m.full[i], 1);
      mbar_init(&m.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&m.tmem_full[i], 1);
      mbar_init(&m.tmem_empty[i], 16);   // the promotion warps of both CTAs
      mbar_init(&m.exchange[i], Shape::kSources);
    }
    for (int i = 0; i < Shape::kScaleChunks; ++i) {
      mbar_init(&m.scale_full[i], 32);   // every lane of the scale warp
      mbar_init(&m.scale_empty[i], 8);   // one arrival per promotion warp
    }
    *m.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 8 && lane == 0) {
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_w);
  }
  // The row-tile list has room for the worst case and its used entries come first.
  __shared__ int used_row_tiles;
  if (warp == 1) {
    const int used = used_tiles(p.tile_expert, p.max_tiles, lane);
    if (lane == 0) used_row_tiles = used;
  }
  cluster_sync_all();   // the peer's barriers exist from here on
  if (warp == 9) tmem_alloc<2>(m.tmem_holder, 512);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();   // and so does its tensor memory
  tcgen05_fence_after();
  const uint32_t tmem_base = *m.tmem_holder;
  const int total_items = used_row_tiles * channel_groups;
  const uint32_t cta_rank = cluster_ctarank();
  const int first_item = blockIdx.x / 2, item_step = gridDim.x / 2;

  // Warps 8-11 (producer, MMA issuer, scales, a spare) give registers to the promotion warps.
  if (warp >= 8) {
    setmaxnreg_dec<GG_AUX_REGS>();
    if (warp == 8) {
      // ---------------------------------------------------------- TMA producer
      const bool leader = elect_one();
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int item = first_item; item < total_items && ok; item += item_step) {
        int tile, jg, expert;
        if (!gate_up_item(p, item, channel_groups, tile, jg, expert)) continue;
        const int row0 = p.tile_row[tile];
        const int blocks = (min(128, p.expert_offsets[expert + 1] - row0) + 31) / 32;
        const int first_row = row0 + static_cast<int>(cta_rank) * 16 * blocks;   // this CTA's half of the columns
        const int channel0 = jg * 256 + static_cast<int>(cta_rank) * 128;
        const int row16 = p.interleaved ? (expert * p.intermediate + channel0) / 16
                                        : (expert * 2 * p.intermediate + channel0) / 16;
        for (int slab = 0, x = 0; slab < slabs; ++slab, x += 128) {
          if (!mbar_wait_warp(&m.empty[stage], phase ^ 1u, kSiteProducerEmpty, m.abort_flag)) {
            ok = false;
            break;
          }
          if (leader) {
            uint8_t* weights = m.stages + stage * Shape::kStageBytes;
            uint8_t* tokens = weights + Shape::kWeightBytes;
            if (cta_rank == 0) {
              mbar_expect_tx(&m.full[stage], 2 * (Shape::kWeightBytes + blocks * Shape::kBlockBytes));
            }
            tma_load_channels_pair(weights, &map_w, &m.full[stage], x, row16);
            for (int b = 0; b < blocks; ++b) {
              tma_load_2d_pair(tokens + b * Shape::kBlockBytes, &map_x, &m.full[stage], x, first_row + 16 * b);
            }
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      dependents_may_launch();   // the CTA's last loads are on their way
    } else if (warp == 9) {
      // ---------------------------------------------------------- MMA issuer (of the leader CTA)
      if (cta_rank == 0) {
        const bool leader = elect_one();
        const uint32_t weights_base = smem_desc_low(smem_u32(m.stages));
        uint32_t stage = 0, phase = 0;
        uint32_t buffer = 0, empty_parity = 1;
        bool ok = true;
        for (int item = first_item; item < total_items && ok; item += item_step) {
          int tile, jg, expert;
          if (!gate_up_item(p, item, channel_groups, tile, jg, expert)) continue;
          const int tokens = min(128, p.expert_offsets[expert + 1] - p.tile_row[tile]);
          const uint32_t idesc = make_idesc_i8(256, (tokens + 31) / 32 * 32);
          for (int slab = 0; slab < slabs; ++slab) {
            if (!mbar_wait_warp(&m.full[stage], phase, kSiteMmaFull, m.abort_flag)) {
              ok = false;
              break;
            }
            tcgen05_fence_after();
            const bool group_start = (slab & 1) == 0;
            if (group_start) {
              if (!mbar_wait_warp(&m.tmem_empty[buffer], empty_parity, kSiteMmaTmemEmpty, m.abort_flag)) {
                ok = false;
                break;
              }
              tcgen05_fence_after();
            }
            const uint32_t weights = weights_base + stage * (Shape::kStageBytes >> 4);
            const uint32_t rows = weights + (Shape::kWeightBytes >> 4);
            const uint32_t tmem_d = tmem_base + buffer * 256;
            if (leader) {
#pragma unroll
              for (int t = 0; t < 2; ++t) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  umma_i8<2>(tmem_d + t * 128, weights + t * (128 * 128 >> 4) + 2 * k, rows + 2 * k, idesc,
                             group_start && k == 0 ? 0u : 1u);
                }
              }
              umma_commit_pair(&m.empty[stage], 3);
              if (!group_start) umma_commit_pair(&m.tmem_full[buffer], 3);
            }
            if (!group_start) {
              buffer ^= 1u;
              if (buffer == 0) empty_parity ^= 1u;
            }
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
    } else if (warp == 10) {
      // ---------------------------------------------------------- scale staging
      uint32_t chunk = 0, phase = 0;
      bool ok = true;
      const uint32_t ring_base = smem_u32(m.ring);
      const uint32_t token_position = 1024 + ring_column_bytes(lane);
      for (int item = first_item; item < total_items && ok; item += item_step) {
        int tile, jg, expert;
        if (!gate_up_item(p, item, channel_groups, tile, jg, expert)) continue;
        const int row0 = p.tile_row[tile];
        const int row_end = p.expert_offsets[expert + 1];
        const int channel0 = jg * 256 + static_cast<int>(cta_rank) * 128;
        const float* weight_source = p.scale_w + static_cast<long long>(expert) * groups * 2 * p.intermediate +
                                     (p.interleaved ? 2 * channel0 + 4 * lane : channel0 + 2 * lane);
        const float* token_source = p.row_scale + static_cast<long long>(row0 + lane) * groups;
        for (int g = 0; g < groups; g += kScaleChunkGroups) {
          if (!mbar_wait_warp(&m.scale_empty[chunk], phase ^ 1u, kSiteScaleEmpty, m.abort_flag)) {
            ok = false;
            break;
          }
          const int in_chunk = min(kScaleChunkGroups, groups - g);
          uint32_t destination = ring_base + chunk * (kScaleChunkGroups * Shape::kRingFloats * 4);
          for (int i = 0; i < in_chunk; ++i) {
            // Channel pair `lane` of both M tiles: four scales.
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint32_t to = destination + 16 * lane + 512 * j;
              if (p.interleaved) {
                const float* from = weight_source + 128 * j;
                if (p.sw_vectors) {
                  cp_async_f32x4(to, from, true);
                } else {
#pragma unroll
                  for (int c = 0; c < 4; ++c) cp_async_f32(to + 4 * c, from + c, true);
                }
              } else {
                const float* gate = weight_source + 64 * j;
                const float* up = gate + p.intermediate;
                if (p.sw_vectors) {
                  cp_async_f32x2(to, gate);
                  cp_async_f32x2(to + 8, up);
                } else {
#pragma unroll
                  for (int c = 0; c < 2; ++c) {
                    cp_async_f32(to + 4 * c, gate + c, true);
                    cp_async_f32(to + 8 + 4 * c, up + c, true);
                  }
                }
              }
            }
            weight_source += 2 * p.intermediate;
            // Scales of tokens that do not exist are zero, which keeps their columns at zero.
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              if (32 * b < row_end - row0) {
                cp_async_f32(destination + 128 * b + token_position,
                             token_source + static_cast<long long>(32 * b) * groups + (g + i),
                             32 * b + lane < row_end - row0);
              }
            }
            destination += Shape::kRingFloats * 4;
          }
          cp_async_arrive(&m.scale_full[chunk]);
          if (++chunk == Shape::kScaleChunks) {
            chunk = 0;
            phase ^= 1u;
          }
        }
      }
      cp_async_wait_all();
    } else {
      report_to_polling_host(p.report, lane);
    }
  } else {
    setmaxnreg_inc<GG_PROMO_REGS>();
    GateUpPairState state;
    for (int item = first_item; item < total_items; item += item_step) {
      int tile, jg, expert;
      if (!gate_up_item(p, item, channel_groups, tile, jg, expert)) continue;
      const int row0 = p.tile_row[tile];
      const int row_end = p.expert_offsets[expert + 1];
      const int tokens = min(128, row_end - row0);
      const auto run = [&](auto blocks) {
        gate_up_pair_item<RoundT, decltype(blocks)::value>(p, m, state, tmem_base, warp, lane, cta_rank, groups,
                                                           row0, row_end, jg);
      };
      if (tokens <= 32) run(std::integral_constant<int, 1>());
      else if (tokens <= 64) run(std::integral_constant<int, 2>());
      else if (tokens <= 96) run(std::integral_constant<int, 3>());
      else run(std::integral_constant<int, 4>());
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();   // no CTA leaves while its peer may still write here
  if (warp == 9) tmem_dealloc<2>(tmem_base, 512);
}

}  // namespace gg
