// Shared by the two INT8 paged-attention kernels (warp-level MMA in sb_attention.cu, tcgen05 in
// sb_attention_tc.cu): launch parameters, the exact int8 -> fp16 conversion, and the split merge that both
// kernels end with.
#pragma once
#include "sb_internal.h"
#include "sb_ptx.cuh"

namespace sb {

constexpr int kMaxFused = 128;   // rows x query heads of one KV head

struct AttnParams {
  const uint16_t *queries, *qkv;
  const uint32_t *page_table;
  const uint2 *tree;
  uint16_t *out;
  SbKvLayer cache;
  float *partials;     // [kv_head][split][D / 4][fused][4]: rows next to each other, as both kernels write and the merge reads them
  float *stats;        // [kv_head][split][fused][2]
  uint32_t *counters;  // [kv_head] arrivals, [64 + kv_head] merges done
  uint32_t *status;
  const uint32_t *committed_dev;
  uint32_t rows, q_heads, group, gated, qkv_stride, out_stride, committed, splits, chunks_per_split, fused;
  uint32_t page_table_stride;  // lanes (blockIdx.z): page-table entries between consecutive lanes' tables
};

// Lane blockIdx.z's view of a launch over several lanes: its 16 row slots of the row-indexed buffers, its page table and
// position, its share of the workspace and counters.
__device__ __forceinline__ AttnParams attn_lane_view(AttnParams p) {
  const uint32_t z = blockIdx.z;
  if (z == 0 && gridDim.z == 1) return p;
  const size_t D = p.cache.head_dim;
  p.queries += size_t(16) * z * p.q_heads * D;
  if (p.qkv) p.qkv += size_t(16) * z * p.qkv_stride;
  p.page_table += size_t(z) * p.page_table_stride;
  if (p.tree) p.tree += 16 * z;
  p.out += size_t(16) * z * p.out_stride;
  const size_t per_lane = size_t(p.cache.kv_heads) * p.splits * kMaxFused;
  p.partials += size_t(z) * per_lane * D;
  p.stats += size_t(z) * per_lane * 2;
  p.counters += 128 * z;
  if (p.committed_dev) p.committed_dev += z;
  return p;
}

// 16 int8 (one uint4) -> 16 fp16, exactly: (q ^ 0x80) | 0x6400 is 1024 + q + 128.
__device__ __forceinline__ void int8x16_to_half(const uint4 v, uint4 &lo, uint4 &hi) {
  const uint32_t w[4] = {v.x ^ 0x80808080u, v.y ^ 0x80808080u, v.z ^ 0x80808080u, v.w ^ 0x80808080u};
  uint32_t o[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[2 * i] = hsub2_u32(__byte_perm(w[i], 0x64646464u, 0x4140), 0x64806480u);      // bytes 0, 1
    o[2 * i + 1] = hsub2_u32(__byte_perm(w[i], 0x64646464u, 0x4342), 0x64806480u);  // bytes 2, 3
  }
  lo = make_uint4(o[0], o[1], o[2], o[3]);
  hi = make_uint4(o[4], o[5], o[6], o[7]);
}

// The end of both kernels, called by every thread of the CTA after its split's partials (fp32 O rows and
// (max, sum) in log2 units) are stored. Every split of this KV head publishes its partials, then all of the
// head's CTAs (co-resident: the launch is cooperative and the grid has at most one CTA per SM) share the
// merge: every element's splits are added in split order with weights
// exp2(max_s - max), divides, rounds to bf16 and multiplies by sigmoid(gate)
// (runtime/metal/kernels/common/paged_attention_tile.h:498-535, attention_gate.h:19-45). The wait for the
// other splits is bounded: if they never arrive the kernel sets the status word and leaves.
template <int D>
__device__ __forceinline__ void attention_merge(const AttnParams &p, uint32_t split, uint32_t kvh, uint32_t *s_last) {
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
  const uint32_t F = p.fused, G = p.group;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    atomicAdd(&p.counters[kvh], 1u);
    uint32_t spins = 0;
    while (atomicAdd(&p.counters[kvh], 0u) < p.splits && ++spins < (1u << 22)) __nanosleep(100);
    *s_last = spins < (1u << 22);
    if (!*s_last) atomicExch(p.status, SB_DEV_WAIT_EXPIRED);
  }
  __syncthreads();
  if (!*s_last) return;
  __threadfence();
  // A lane per (fused row, four dimensions), neighbouring lanes neighbouring rows, so a split's share is read in runs of up to 512
  // bytes (32 rows; 4, 8 or 16 where there are no more, and the warp's other lanes take the next dimensions); sixteen splits'
  // loads in flight; the head's CTAs divide the tasks. Every element is summed in split order.
  const uint32_t run = F <= 4 ? 4 : F <= 8 ? 8 : F <= 16 ? 16 : 32, row_groups = (F + run - 1) / run, tasks = D / 4 / (32 / run) * row_groups;
  for (uint32_t task = split + p.splits * warp; task < tasks; task += p.splits * warps) {
    const uint32_t f0 = task % row_groups * run + lane % run, f = min(f0, F - 1), d0 = (task / row_groups * (32 / run) + lane / run) * 4;
    const bool live = f0 < F;
    const float2 *stats = reinterpret_cast<const float2 *>(p.stats) + size_t(kvh) * p.splits * kMaxFused + f;
    const float4 *parts = reinterpret_cast<const float4 *>(p.partials) + (size_t(kvh) * p.splits * (D / 4) + d0 / 4) * kMaxFused + f;
    const uint32_t row = f / G, qh = kvh * G + f % G;
    uint2 g2 = make_uint2(0, 0);
    if (p.gated) g2 = *reinterpret_cast<const uint2 *>(p.qkv + size_t(row) * p.qkv_stride + qh * 2 * D + D + d0);
    float num[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    float den = 0.0f, m = -INFINITY;  // (the largest so far; what is summed is moved to it sixteen splits at a time)
    for (uint32_t s0 = 0; s0 < p.splits; s0 += 16) {
      float2 st[16];
      float4 v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        st[j] = make_float2(-INFINITY, 0.0f), v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (s0 + j >= p.splits) continue;
        st[j] = __ldcg(&stats[size_t(s0 + j) * kMaxFused]);
        v[j] = __ldcg(parts + size_t(s0 + j) * (D / 4) * kMaxFused);
      }
      float most = m;
#pragma unroll
      for (int j = 0; j < 16; ++j) most = fmaxf(most, st[j].x);
      if (most == -INFINITY) continue;
      const float moved = m == -INFINITY ? 0.0f : exp2f(m - most);
#pragma unroll
      for (int i = 0; i < 4; ++i) num[i] *= moved;
      den *= moved, m = most;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (st[j].x == -INFINITY) continue;
        const float w = exp2f(st[j].x - m);
        num[0] += w * v[j].x, num[1] += w * v[j].y, num[2] += w * v[j].z, num[3] += w * v[j].w;
        den += w * st[j].y;
      }
    }
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = round_bf16(den > 0.0f ? num[i] / den : 0.0f);
    if (p.gated) {
      o[0] *= sigmoid_f(bf16_bits_to_float(g2.x & 0xffffu)), o[1] *= sigmoid_f(bf16_bits_to_float(g2.x >> 16));
      o[2] *= sigmoid_f(bf16_bits_to_float(g2.y & 0xffffu)), o[3] *= sigmoid_f(bf16_bits_to_float(g2.y >> 16));
    }
    uint2 packed;
    packed.x = uint32_t(float_to_bf16_bits(o[0])) | (uint32_t(float_to_bf16_bits(o[1])) << 16);
    packed.y = uint32_t(float_to_bf16_bits(o[2])) | (uint32_t(float_to_bf16_bits(o[3])) << 16);
    if (live) *reinterpret_cast<uint2 *>(p.out + size_t(row) * p.out_stride + qh * D + d0) = packed;
  }
  // The last CTA to finish its share returns both counters to zero for the next launch.
  __syncthreads();
  if (tid == 0 && atomicAdd(&p.counters[64 + kvh], 1u) == p.splits - 1) {
    p.counters[kvh] = 0;
    p.counters[64 + kvh] = 0;
  }
}

// The tcgen05 kernel's launcher (sb_attention_tc.cu); `p` comes filled except for the split geometry.
int launch_attention_tc(cudaStream_t stream, AttnParams &p, uint32_t visible, uint32_t lanes);

}  // namespace sb
