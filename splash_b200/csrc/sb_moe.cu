// MoE expert passes. Replaces the expert passes of MoE::addRouted (runtime/ops/MoE.cpp:122-187,260-270; kernels moe_gguf_expert_tile
// of runtime/metal/kernels/common/moe_gguf_expert_tile.h:33-84, the gate/up pass runtime/metal/kernels/shared/moe_gguf.metal:
// 94-160 and moe_combine, runtime/metal/kernels/shared/moe.metal:367-392):
//   intermediate = bf16(bf16(up . x) * silu(bf16(gate . x)))     per route
//   y            = bf16(down . intermediate)                     per route
//   out          = bf16(residual + sum over the row's routes, in slot order, of weight * float(y))
// A lane's block (up to 16 rows, up to 32 routes each): the routes are grouped by expert (up to eight a group, the columns of one
// MMA), so an expert's weights are read once for all the rows that chose it; blocks of small experts take a matrix-vector product a
// route (moe_vector_block). More rows: the groups are tiles of the many-row projection (below).
// A warp takes 16 gate and the 16 up rows (32 down rows) of a group over the whole of K: lane 4 g + t loads rows g and g + 8's sub-blocks
// 2t, 2t + 1 of every super-block straight into registers (two 16-byte loads a row and a header) and feeds them to mma.sync as
// exact integers sc q (sb_q4k.cuh) against the group's activations in fp16 (a power of two a row), the block scales on fp32 sums.
// 16 rows of the 35B-A3B shape, routing included, graph replay: 77 us (185 with a product a route), 180 MB of experts' weights in 45 and
// 24 us of the two passes (ncu, cold: 2.6 TB/s). What bounds them is the L1: a warp's 16-byte loads touch eight rows each, and the
// activations come the same way.
#include <algorithm>

#include "sb_internal.h"
#include "sb_linear_internal.h"
#include "sb_ptx.cuh"
#include "sb_q4k.cuh"

namespace sb {

constexpr uint32_t kMoeFewRows = 16, kMoeFewRoutes = kMoeFewRows * 32;  // rows and routes of a lane's block
constexpr int kMoeThreads = 256, kMoeWarps = kMoeThreads / 32;

// Up to eight routes of one expert.
struct MoeFew {
  uint32_t expert, n, route[8];
};
// The scratch of a call: activations as the expert kernels read them, the intermediate rows, the routes' results, the groups.
struct MoeFewLayout {
  uint64_t counts, groups, x, x_scale, act, act_scale, intermediate, y, bytes;
};
// A converted row of k inputs: per super-block 512 bytes of 16-byte units, then per super-block 32 bytes of sub-block sums.
__host__ __device__ inline uint64_t moe_row_bytes(uint32_t k) { return uint64_t(k) * 2 + k / 8; }
static MoeFewLayout moe_few_layout(uint32_t rows, uint32_t routes, uint32_t hidden, uint32_t inter) {
  MoeFewLayout l{};
  const uint64_t n = uint64_t(rows) * routes;
  uint64_t at = 0;
  auto take = [&](uint64_t bytes) { const uint64_t here = at; at += (bytes + 255) / 256 * 256; return here; };
  l.intermediate = take(n * inter * 2), l.y = take(n * hidden * 2);
  l.counts = take(4), l.groups = take(n * sizeof(MoeFew)), l.x = take(rows * moe_row_bytes(hidden)), l.x_scale = take(rows * 4);
  l.act = take(n * moe_row_bytes(inter)), l.act_scale = take(n * 4);
  l.bytes = at;
  return l;
}

struct MoeParams {
  SbMoeExpertArgs a;
  uint16_t *intermediate;  // bf16 [rows * routes, inter]
  uint16_t *y;             // bf16 [rows * routes, hidden]
  uint32_t *counts;        // [0] groups
  MoeFew *groups;
  uint8_t *x, *act;         // converted rows: [rows], [rows * routes]
  float *x_scale, *act_scale;
};

// A bf16 row in fp16 with a power of two taken out (exact for values down to 2^-26 of the row's largest, smaller ones to within 2^-34
// of it), in the order a lane of
// the expert kernels reads it: unit (i2, p, t) of a super-block holds inputs 32 (2 t + p) + 8 i2 .. + 7 as [0,2,1,3,4,6,5,7] (the
// order the Q4_K nibbles come out in), and lane t's 8 bytes of sums are sub-blocks 2 t, 2 t + 1, each a high and a low half.
__device__ __forceinline__ void moe_convert_row(const uint16_t *src, uint32_t k, uint8_t *dst, float *scale, float *scratch) {
  const uint32_t tid = threadIdx.x, chunks = k / 8;
  const bool wide = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  constexpr int kMost = 8192 / 8 / kMoeThreads;  // chunks a thread keeps
  float v[kMost][8], mx = 0.0f;
#pragma unroll
  for (int i = 0; i < kMost; ++i) {
    const uint32_t c = tid + i * blockDim.x;
    uint32_t u[4] = {0, 0, 0, 0};
    if (c < chunks) {
      if (wide) {
        const uint4 w = *reinterpret_cast<const uint4 *>(src + 8 * c);
        u[0] = w.x, u[1] = w.y, u[2] = w.z, u[3] = w.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) u[j] = uint32_t(src[8 * c + 2 * j]) | (uint32_t(src[8 * c + 2 * j + 1]) << 16);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][2 * j] = bf16_bits_to_float(u[j] & 0xffffu), v[i][2 * j + 1] = bf16_bits_to_float(u[j] >> 16);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(v[i][j]));  // (NaN does not win a max; it stays in the values)
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) scratch[tid >> 5] = mx;
  __syncthreads();
  for (uint32_t w = 0; w < blockDim.x / 32; ++w) mx = fmaxf(mx, scratch[w]);
  const int e = row_exponent(mx);
  const float down = power_of_two(-e);
  if (tid == 0) *scale = power_of_two(e);
#pragma unroll
  for (int i = 0; i < kMost; ++i) {
    const uint32_t c = tid + i * blockDim.x;
    if (c >= chunks) break;  // (whole warps: chunks is a multiple of 32)
    const uint32_t sb = c >> 5, j = (c & 31u) >> 2, q = c & 3u;
    __half h[8];
    float sum = 0.0f;
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) h[jj] = __float2half_rn(v[i][jj] * down), sum += __half2float(h[jj]);
    const __half2 p0 = __halves2half2(h[0], h[2]), p1 = __halves2half2(h[1], h[3]), p2 = __halves2half2(h[4], h[6]), p3 = __halves2half2(h[5], h[7]);
    *reinterpret_cast<uint4 *>(dst + size_t(sb) * 512 + ((q * 2 + (j & 1)) * 4 + (j >> 1)) * 16) =
        make_uint4(*reinterpret_cast<const uint32_t *>(&p0), *reinterpret_cast<const uint32_t *>(&p1), *reinterpret_cast<const uint32_t *>(&p2),
                   *reinterpret_cast<const uint32_t *>(&p3));
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);  // 32 inputs = 4 consecutive lanes
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (q == 0) {
      const __half hi = __float2half_rn(sum), lo = __float2half_rn(sum - __half2float(hi));
      *reinterpret_cast<__half2 *>(dst + size_t(k) * 2 + size_t(sb) * 32 + j * 4) = __halves2half2(hi, lo);
    }
  }
}

// grid (rows + 1): a CTA a row of the input, and one that groups the routes. A route's place among its expert's routes is the
// number of earlier routes of the expert; every eighth of them starts a group, groups in the order they start.
__global__ void __launch_bounds__(kMoeThreads) moe_few_prepare_kernel(const MoeParams p) {
  __shared__ float scratch[kMoeWarps];
  __shared__ uint32_t expert_s[kMoeFewRoutes], rank_s[kMoeFewRoutes], group_s[kMoeFewRoutes], warp_s[2 * kMoeWarps];
  pdl_launch_dependents();
  pdl_wait();
  const SbMoeExpertArgs &a = p.a;
  if (blockIdx.x < a.rows) {
    const uint32_t row = blockIdx.x;
    moe_convert_row(static_cast<const uint16_t *>(a.input) + size_t(row) * a.hidden, a.hidden, p.x + row * moe_row_bytes(a.hidden), p.x_scale + row, scratch);
    return;
  }
  const uint32_t n = a.rows * a.routes, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint32_t i = tid; i < n; i += kMoeThreads) expert_s[i] = min(a.selected[i], a.experts_total - 1);
  __syncthreads();
  // thread t: routes t and t + 256, numbered in that order by warp and lane
  uint32_t rank[2], starts[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t i = tid + k * kMoeThreads;
    rank[k] = 0;
    if (i < n)
      for (uint32_t j = 0; j < i; ++j) rank[k] += expert_s[j] == expert_s[i];
    if (i < n) rank_s[i] = rank[k];
    starts[k] = __ballot_sync(0xffffffffu, i < n && (rank[k] & 7u) == 0);
    if (lane == 0) warp_s[k * kMoeWarps + warp] = uint32_t(__popc(starts[k]));
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t i = tid + k * kMoeThreads;
    uint32_t before = 0;
    for (int w = 0; w < k * kMoeWarps + int(warp); ++w) before += warp_s[w];
    if (i < n && (rank[k] & 7u) == 0) group_s[i] = before + uint32_t(__popc(starts[k] & ((1u << lane) - 1u)));
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t i = tid + k * kMoeThreads;
    if (i >= n) break;
    const uint32_t e = expert_s[i], first = rank[k] & ~7u;
    uint32_t start = i, total = 0;
    for (uint32_t j = 0; j < n; ++j)
      if (expert_s[j] == e) {
        ++total;
        if (rank_s[j] == first) start = j;
      }
    MoeFew &g = p.groups[group_s[start]];
    g.route[rank[k] & 7u] = i;
    if (start == i) g.expert = e, g.n = min(total - first, 8u);
  }
  if (tid == 0) {
    uint32_t groups = 0;
    for (int w = 0; w < 2 * kMoeWarps; ++w) groups += warp_s[w];
    p.counts[0] = groups;
  }
}

// grid (rows * routes): a route's intermediate row.
__global__ void __launch_bounds__(kMoeThreads) moe_few_convert_kernel(const MoeParams p) {
  __shared__ float scratch[kMoeWarps];
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t route = blockIdx.x;
  moe_convert_row(p.intermediate + size_t(route) * p.a.inter, p.a.inter, p.act + route * moe_row_bytes(p.a.inter), p.act_scale + route, scratch);
}

// PAIR: gate and up of the groups' experts over the rows' inputs -> intermediate. Otherwise down over the routes' intermediate
// rows -> y. A warp a (group, column block) in turn; its two 16-row tiles are the gate and the up rows of 16 columns, or the
// down rows of 32.
template <bool PAIR> __global__ void __launch_bounds__(kMoeThreads, 2) moe_few_kernel(const MoeParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const SbMoeExpertArgs &a = p.a;
  const uint32_t lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t k = PAIR ? a.hidden : a.inter, n = PAIR ? a.inter : a.hidden, nsb = k / 256, blocks = n / (PAIR ? 16 : 32);
  const size_t row_bytes = size_t(nsb) * 144, in_bytes = moe_row_bytes(k);
  const uint32_t units = p.counts[0] * blocks, warps = gridDim.x * kMoeWarps;
  // (neighbouring warps of a CTA on neighbouring column blocks of a group: they share its activations in the L1)
  for (uint32_t u = blockIdx.x * kMoeWarps + (threadIdx.x >> 5); u < units; u += warps) {
    const MoeFew &few = p.groups[u / blocks];
    const uint32_t c0 = u % blocks * (PAIR ? 16 : 32), count = few.n;
    const uint32_t mine = few.route[min(g, count - 1)], in_row = PAIR ? mine / a.routes : mine;  // (columns past the group repeat its last)
    const uint8_t *in = (PAIR ? p.x : p.act) + in_row * in_bytes + t * 16, *sums = (PAIR ? p.x : p.act) + in_row * in_bytes + size_t(k) * 2 + t * 8;
    const uint8_t *w[2];
    w[0] = static_cast<const uint8_t *>(PAIR ? a.gate : a.down) + (size_t(few.expert) * n + c0 + g) * row_bytes;
    w[1] = PAIR ? static_cast<const uint8_t *>(a.up) + (size_t(few.expert) * n + c0 + g) * row_bytes : w[0] + 16 * row_bytes;
    float y[2][4] = {};
    for (uint32_t sb = 0; sb < nsb; ++sb) {
      uint4 hdr[2][2], q[2][2][2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint8_t *blk = w[mt] + size_t(8 * r) * row_bytes + size_t(sb) * 144;
          hdr[mt][r] = __ldg(reinterpret_cast<const uint4 *>(blk));
          q[mt][r][0] = __ldg(reinterpret_cast<const uint4 *>(blk + 16 + 32 * t));
          q[mt][r][1] = __ldg(reinterpret_cast<const uint4 *>(blk + 32 + 32 * t));
        }
      Q4Scales sc[2][2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int r = 0; r < 2; ++r) sc[mt][r] = q4_scales(hdr[mt][r], t);
      float aq[2][4] = {};
      const uint32_t kMagic = 0x64006400u;
#pragma unroll
      for (int i2 = 0; i2 < 4; ++i2) {
        const uint4 lo = *reinterpret_cast<const uint4 *>(in + size_t(sb) * 512 + i2 * 128), hi = *reinterpret_cast<const uint4 *>(in + size_t(sb) * 512 + i2 * 128 + 64);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int wi = 0; wi < 2; ++wi) {
            const uint4 q0 = q[mt][0][i2 >> 1], q1 = q[mt][1][i2 >> 1];
            const uint32_t w0 = (i2 & 1) ? (wi ? q0.w : q0.z) : (wi ? q0.y : q0.x), w1 = (i2 & 1) ? (wi ? q1.w : q1.z) : (wi ? q1.y : q1.x);
            const uint32_t w0s = w0 >> 8, w1s = w1 >> 8;
            mma_f16(aq[mt], hfma2_u32(and_or(w0, 0x000f000fu, kMagic), sc[mt][0].mlo, sc[mt][0].blo),
                    hfma2_u32(and_or(w1, 0x000f000fu, kMagic), sc[mt][1].mlo, sc[mt][1].blo),
                    hfma2_u32(and_or(w0s, 0x000f000fu, kMagic), sc[mt][0].mlo, sc[mt][0].blo),
                    hfma2_u32(and_or(w1s, 0x000f000fu, kMagic), sc[mt][1].mlo, sc[mt][1].blo), wi ? lo.z : lo.x, wi ? lo.w : lo.y);
            mma_f16(aq[mt], hfma2_u32(and_or(w0, 0x00f000f0u, kMagic), sc[mt][0].mhi, sc[mt][0].bhi),
                    hfma2_u32(and_or(w1, 0x00f000f0u, kMagic), sc[mt][1].mhi, sc[mt][1].bhi),
                    hfma2_u32(and_or(w0s, 0x00f000f0u, kMagic), sc[mt][0].mhi, sc[mt][0].bhi),
                    hfma2_u32(and_or(w1s, 0x00f000f0u, kMagic), sc[mt][1].mhi, sc[mt][1].bhi), wi ? hi.z : hi.x, wi ? hi.w : hi.y);
          }
      }
      const uint2 s = *reinterpret_cast<const uint2 *>(sums + size_t(sb) * 32);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        float am[4] = {};
        mma_f16(am, sc[mt][0].mn0, sc[mt][1].mn0, sc[mt][0].mn1, sc[mt][1].mn1, s.x, s.y);
#pragma unroll
        for (int c = 0; c < 4; ++c) y[mt][c] = fmaf(sc[mt][c >> 1].ndmin, am[c], fmaf(sc[mt][c >> 1].d, aq[mt][c], y[mt][c]));
      }
    }
    // lane 4 g + t: columns g and g + 8 of the group's routes 2 t, 2 t + 1
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (2 * t + i >= count) continue;
      const uint32_t route = few.route[2 * t + i];
      const float back = PAIR ? p.x_scale[route / a.routes] : p.act_scale[route];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t c = c0 + g + 8 * r;
        if (PAIR) {
          p.intermediate[size_t(route) * a.inter + c] = float_to_bf16_bits(round_bf16(y[1][i + 2 * r] * back) * silu_f(round_bf16(y[0][i + 2 * r] * back)));
        } else {
          p.y[size_t(route) * a.hidden + c] = float_to_bf16_bits(y[0][i + 2 * r] * back);
          p.y[size_t(route) * a.hidden + c + 16] = float_to_bf16_bits(y[1][i + 2 * r] * back);
        }
      }
    }
  }
}

// ---- a few routes of small experts: a matrix-vector product a route ----
// A warp computes eight output columns of a route against the staged row, a lane eight consecutive weights of every super-block: all
// loads of a product in flight, three launches a block. It costs three instructions a weight and route, so it is the better one
// only where the routes are few and the experts small (kMoeVectorWeights below).
constexpr int kMoeColsPair = 8, kMoeColsDown = 8;  // output columns a warp computes (gate/up pass, down pass)
constexpr float kMoeVectorDown = 0x1p-8f;          // on the inputs, taken back by the scales: eight products with codes up to 15 stay finite

// scale and min of sub-block j of a Q4_K super-block from its 12 packed bytes (three words), in registers: bytes 0-3
// hold the low 6 bits of scales 0-3 (and in their top 2 bits the high bits of scales 4-7), bytes 4-7 the same for the mins,
// bytes 8-11 the low nibbles of scales 4-7 (low half) and mins 4-7 (high half).
__device__ __forceinline__ void q4k_scale_min(const uint32_t (&w)[3], uint32_t j, float &sc, float &mn) {
  const uint32_t s8 = 8 * (j & 3);
  uint32_t isc, imn;
  if (j < 4) {
    isc = (w[0] >> s8) & 63u, imn = (w[1] >> s8) & 63u;
  } else {
    isc = ((w[2] >> s8) & 0xFu) | (((w[0] >> (s8 + 6)) & 3u) << 4);
    imn = ((w[2] >> (s8 + 4)) & 0xFu) | (((w[1] >> (s8 + 6)) & 3u) << 4);
  }
  sc = float(isc), mn = float(imn);
}

// acc[m][c] += lane's share of dot(row c of matrix m, x) for NC consecutive Q4_K rows of each of NM matrices; x staged in
// shared memory as floats; lane l takes weights 32 (l / 4) + 8 (l % 4) .. + 7 of every super-block, so the lane's x values
// and their sum are fetched once per super-block for all the rows.
template <int NM, int NC>
__device__ __forceinline__ void q4k_rows_dot(const uint8_t *const (&rows)[NM], size_t row_bytes, const float *x, uint32_t k, uint32_t lane,
                                             float (&acc)[NM][NC]) {
  const uint32_t sub = lane >> 2, t0 = 8 * (lane & 3), shift = (sub & 1) * 4;
#pragma unroll
  for (int m = 0; m < NM; ++m)
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[m][c] = 0.0f;
#pragma unroll 2
  for (uint32_t sb = 0; sb < k / 256; ++sb) {
    const float4 x0 = *reinterpret_cast<const float4 *>(x + 256 * sb + 32 * sub + t0), x1 = *reinterpret_cast<const float4 *>(x + 256 * sb + 32 * sub + t0 + 4);
    const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    const float xsum = ((xs[0] + xs[1]) + (xs[2] + xs[3])) + ((xs[4] + xs[5]) + (xs[6] + xs[7]));
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const uint8_t *blk = rows[m] + size_t(c) * row_bytes + size_t(sb) * 144;
        const uint32_t dm = *reinterpret_cast<const uint32_t *>(blk);
        const float d = __half2float(__ushort_as_half(uint16_t(dm & 0xffffu))) / kMoeVectorDown, dmin = __half2float(__ushort_as_half(uint16_t(dm >> 16))) / kMoeVectorDown;
        const uint32_t sw[3] = {*reinterpret_cast<const uint32_t *>(blk + 4), *reinterpret_cast<const uint32_t *>(blk + 8),
                                *reinterpret_cast<const uint32_t *>(blk + 12)};
        float sc, mn;
        q4k_scale_min(sw, sub, sc, mn);
        const uint2 qs = *reinterpret_cast<const uint2 *>(blk + 16 + 32 * (sub >> 1) + t0);
        float qx = 0.0f;
        const uint32_t n0 = (qs.x >> shift) & 0x0F0F0F0Fu, n1 = (qs.y >> shift) & 0x0F0F0F0Fu;  // the lane's eight codes, a byte each
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          // the code as a float without a conversion instruction (quarter rate): 2^23 + q in the mantissa, minus 2^23
          const float q = __uint_as_float(0x4B000000u | __byte_perm(j < 4 ? n0 : n1, 0, 0x4440 + (j & 3))) - 8388608.0f;
          qx = fmaf(q, xs[j], qx);
        }
        acc[m][c] = fmaf(d * sc, qx, acc[m][c]);
        acc[m][c] = fmaf(-dmin * mn, xsum, acc[m][c]);
      }
  }
#pragma unroll
  for (int m = 0; m < NM; ++m)
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int o = 16; o; o >>= 1) acc[m][c] += __shfl_xor_sync(0xffffffffu, acc[m][c], o);
}

// PAIR: gate and up of the route's expert over the row's input -> intermediate. Otherwise: down over the route's
// intermediate -> y. grid (rows * routes, column blocks).
template <bool PAIR> __global__ void __launch_bounds__(kMoeThreads) moe_expert_kernel(const MoeParams p) {
  constexpr int kMoeColsPerWarp = PAIR ? kMoeColsPair : kMoeColsDown;
  extern __shared__ float xrow[];
  pdl_launch_dependents();
  pdl_wait();
  const SbMoeExpertArgs &a = p.a;
  const uint32_t route = blockIdx.x, row = route / a.routes, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t k = PAIR ? a.hidden : a.inter, n = PAIR ? a.inter : a.hidden;
  const uint32_t expert = min(a.selected[route], a.experts_total - 1);
  const uint16_t *src = PAIR ? static_cast<const uint16_t *>(a.input) + size_t(row) * a.hidden : p.intermediate + size_t(route) * a.inter;
  for (uint32_t i = tid; i < k; i += kMoeThreads) xrow[i] = bf16_bits_to_float(src[i]) * kMoeVectorDown;
  __syncthreads();
  const size_t row_bytes = size_t(k / 256) * 144;
  const uint8_t *w0 = static_cast<const uint8_t *>(PAIR ? a.gate : a.down) + size_t(expert) * n * row_bytes;
  const uint8_t *w1 = PAIR ? static_cast<const uint8_t *>(a.up) + size_t(expert) * n * row_bytes : nullptr;
  const uint32_t c0 = (blockIdx.y * kMoeWarps + warp) * kMoeColsPerWarp;
  if (c0 >= n) return;  // n is a multiple of 256, so a warp's columns are inside or outside together
  if (PAIR) {
    const uint8_t *const rows[2] = {w0 + size_t(c0) * row_bytes, w1 + size_t(c0) * row_bytes};
    float acc[2][kMoeColsPerWarp];
    q4k_rows_dot<2, kMoeColsPerWarp>(rows, row_bytes, xrow, k, lane, acc);
    if (lane < kMoeColsPerWarp) {
      float g = 0.0f, u = 0.0f;
#pragma unroll
      for (int c = 0; c < kMoeColsPerWarp; ++c)
        if (lane == uint32_t(c)) g = acc[0][c], u = acc[1][c];
      p.intermediate[size_t(route) * a.inter + c0 + lane] = float_to_bf16_bits(round_bf16(u) * silu_f(round_bf16(g)));
    }
  } else {
    const uint8_t *const rows[1] = {w0 + size_t(c0) * row_bytes};
    float acc[1][kMoeColsPerWarp];
    q4k_rows_dot<1, kMoeColsPerWarp>(rows, row_bytes, xrow, k, lane, acc);
    if (lane < kMoeColsPerWarp) {
      float v = 0.0f;
#pragma unroll
      for (int c = 0; c < kMoeColsPerWarp; ++c)
        if (lane == uint32_t(c)) v = acc[0][c];
      p.y[size_t(route) * a.hidden + c0 + lane] = float_to_bf16_bits(v);
    }
  }
}

// out = bf16(residual + sum over the row's routes in slot order of weight * float(y)).
__global__ void __launch_bounds__(256) moe_combine_kernel(const MoeParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const SbMoeExpertArgs &a = p.a;
  const uint32_t row = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.hidden) return;
  float acc = 0.0f;
  for (uint32_t s = 0; s < a.routes; ++s)
    acc += a.weights[size_t(row) * a.routes + s] * bf16_bits_to_float(p.y[(size_t(row) * a.routes + s) * a.hidden + c]);
  const float res = a.residual ? bf16_bits_to_float(static_cast<const uint16_t *>(a.residual)[size_t(row) * a.hidden + c]) : 0.0f;
  static_cast<uint16_t *>(a.out)[size_t(row) * a.hidden + c] = float_to_bf16_bits(res + acc);
}

// ---- many rows (the rows of several lanes): routes grouped by expert, the experts' passes on the many-row kernel ----
// (MoE::addRouted's grouping: runtime/metal/kernels/shared/moe.metal:187-287, the row gather :347-365, the expert tiles
// runtime/metal/kernels/common/moe_gguf_expert_tile.h:33-84, the combine moe.metal:367-392.)
constexpr uint32_t kMoeMaxExperts = 512, kMoeMaxRoutes = 16384, kMoeGroupRows = 64, kMoeGroupThreads = 512;
struct MoeGrouping {
  uint32_t *counts;         // [0] groups, [1] row slots
  uint4 *groups;            // {expert, first slot, rows, rows padded to 16}
  uint32_t *slot_of_route;  // [rows * routes]
  uint32_t *slot_src;       // [slots] the input row a slot holds, ~0 for padding
  uint32_t *slot_self;      // [slots] the slot itself, ~0 for padding
  uint32_t *slot_group;     // [slots] group << 8 | row inside the group
};
struct MoeGroupLayout {
  uint64_t counts, groups, slot_of_route, slot_src, slot_self, slot_group, scales1, scales2, prepared1, prepared2, act, y, bytes;
  uint32_t max_groups, max_slots;
};
static MoeGroupLayout moe_group_layout(uint32_t rows, uint32_t routes, uint32_t hidden, uint32_t inter) {
  MoeGroupLayout l{};
  const uint64_t n = uint64_t(rows) * routes;
  l.max_groups = uint32_t(kMoeMaxExperts + n / kMoeGroupRows + 1);
  l.max_slots = uint32_t((n + 15ull * l.max_groups + 15) / 16 * 16);  // every group ends with fewer than 16 padding slots
  uint64_t at = 0;
  auto take = [&](uint64_t bytes) { const uint64_t here = at; at += (bytes + 255) / 256 * 256; return here; };
  l.counts = take(16), l.groups = take(uint64_t(l.max_groups) * 16), l.slot_of_route = take(n * 4);
  l.slot_src = take(uint64_t(l.max_slots) * 4), l.slot_self = take(uint64_t(l.max_slots) * 4), l.slot_group = take(uint64_t(l.max_slots) * 4);
  l.scales1 = take(uint64_t(l.max_slots) * 4), l.scales2 = take(uint64_t(l.max_slots) * 4);
  l.prepared1 = take(uint64_t(l.max_slots) * hidden * 2), l.prepared2 = take(uint64_t(l.max_slots) * inter * 2);
  l.act = take(uint64_t(l.max_slots) * inter * 2), l.y = take(uint64_t(l.max_slots) * hidden * 2);
  l.bytes = at;
  return l;
}

// One CTA of 16 warps: a stable counting sort of the routes by expert. Warp w owns a run of consecutive routes; it counts
// them by expert (a step of 32 routes at a time, equal experts found with a warp match), a thread per expert then adds the
// warps' counts in warp order, one warp lays the experts' groups out one after the other (an expert's routes in groups of
// 64, the last padded to 16 row slots), and the warps walk their runs again to number the routes: a route's place among
// its expert's routes is the earlier warps' count, plus this warp's count so far, plus its rank inside the step.
constexpr uint32_t kMoeGroupWarps = kMoeGroupThreads / 32;
// Which routes a launch takes, and the expert's place in its tensors: all of them (experts0 = 0, local = experts), or a
// rank's share under expert parallelism: experts [expert0, expert0 + local) at 0 .., the shared expert (shared_id) for rows
// [own_row0, own_row0 + own_rows) at `local`.
struct MoeShare {
  uint32_t expert0, local, shared_id, own_row0, own_rows;
};
__global__ void __launch_bounds__(kMoeGroupThreads) moe_group_kernel(const uint32_t *selected, uint32_t n, uint32_t routes, uint32_t experts, MoeGrouping g,
                                                                     uint32_t *status, MoeShare share) {
  __shared__ uint16_t warp_count[kMoeGroupWarps][kMoeMaxExperts];  // then: the place of the warp's next route of the expert
  __shared__ uint32_t count_s[kMoeMaxExperts], slot0_s[kMoeMaxExperts], group0_s[kMoeMaxExperts];
  extern __shared__ uint16_t place_s[];  // [n] the routes' experts' places, kNoPlace for those the launch does not take
  constexpr uint32_t kNoPlace = 0xffffu;
  pdl_launch_dependents();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (uint32_t i = tid; i < kMoeGroupWarps * kMoeMaxExperts; i += kMoeGroupThreads) (&warp_count[0][0])[i] = 0;
  pdl_wait();
  const uint32_t run = ((n + kMoeGroupWarps - 1) / kMoeGroupWarps + 31) / 32 * 32, first = warp * run, last = min(n, first + run);
  const uint32_t lt = (1u << lane) - 1u;
  // Every route's expert once, all threads' loads in flight together.
#pragma unroll 4
  for (uint32_t i = tid; i < n; i += kMoeGroupThreads) {
    const uint32_t e = selected[i];
    uint32_t place = kNoPlace;
    if (e == share.shared_id) {
      const uint32_t row = i / routes;
      if (row >= share.own_row0 && row - share.own_row0 < share.own_rows) place = share.local;
    } else if (e - share.expert0 < share.local) {
      place = e - share.expert0;
    } else if (share.expert0 == 0 && share.shared_id == 0xffffffffu && share.local == experts) {
      atomicCAS(status, 0u, uint32_t(SB_DEV_CONTRACT));  // a whole block: an id outside it breaks the contract
    }  // (else another rank's expert, or a dropped route)
    place_s[i] = uint16_t(place);
  }
  __syncthreads();
  auto expert_at = [&](uint32_t i) -> uint32_t {
    const uint32_t e = i < last ? place_s[i] : kNoPlace;
    return e == kNoPlace ? 0xffffffffu : e;
  };
  for (uint32_t i0 = first; i0 < last; i0 += 32) {
    const uint32_t e = expert_at(i0 + lane);
    const uint32_t same = __match_any_sync(0xffffffffu, e);
    if (e != 0xffffffffu && !(same & lt)) warp_count[warp][e] += uint16_t(__popc(same));
    __syncwarp();
  }
  __syncthreads();
  for (uint32_t e = tid; e < experts; e += kMoeGroupThreads) {
    uint32_t total = 0;
    for (uint32_t w = 0; w < kMoeGroupWarps; ++w) {
      const uint32_t c = warp_count[w][e];
      warp_count[w][e] = uint16_t(total);
      total += c;
    }
    count_s[e] = total;
  }
  __syncthreads();
  if (warp == 0) {
    // 32 experts a round: their group counts and padded slots scanned over the lanes
    uint32_t slot = 0, group = 0;
    for (uint32_t e0 = 0; e0 < experts; e0 += 32) {
      const uint32_t e = e0 + lane, c = e < experts ? count_s[e] : 0;
      const uint32_t groups = (c + kMoeGroupRows - 1) / kMoeGroupRows, slots = (c + 15) / 16 * 16;
      uint32_t gs = groups, ss = slots;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, gs, o), b = __shfl_up_sync(0xffffffffu, ss, o);
        if (lane >= uint32_t(o)) gs += a, ss += b;
      }
      const uint32_t my_group = group + gs - groups, my_slot = slot + ss - slots;
      if (e < experts) slot0_s[e] = my_slot, group0_s[e] = my_group;
      group += __shfl_sync(0xffffffffu, gs, 31), slot += __shfl_sync(0xffffffffu, ss, 31);
    }
    if (lane == 0) g.counts[0] = group, g.counts[1] = slot;
  }
  __syncthreads();
  // A thread per expert: its groups, and the padding slots behind its last route.
  for (uint32_t e = tid; e < experts; e += kMoeGroupThreads) {
    const uint32_t c = count_s[e], groups = (c + kMoeGroupRows - 1) / kMoeGroupRows, slots = (c + 15) / 16 * 16, my_slot = slot0_s[e], my_group = group0_s[e];
    for (uint32_t k = 0; k < groups; ++k) {
      const uint32_t rows = min(c - k * kMoeGroupRows, kMoeGroupRows);
      g.groups[my_group + k] = make_uint4(e, my_slot + k * kMoeGroupRows, rows, (rows + 15) / 16 * 16);
    }
    const uint32_t lastg = my_group + (groups ? groups - 1 : 0);
    for (uint32_t r = c; r < slots; ++r) {
      g.slot_src[my_slot + r] = 0xffffffffu, g.slot_self[my_slot + r] = 0xffffffffu;
      g.slot_group[my_slot + r] = (lastg << 8) | (r - (lastg - my_group) * kMoeGroupRows);
    }
  }
  for (uint32_t i0 = first; i0 < last; i0 += 32) {
    const uint32_t i = i0 + lane, e = expert_at(i);
    const uint32_t same = __match_any_sync(0xffffffffu, e);
    if (e != 0xffffffffu) {
      const uint32_t j = warp_count[warp][e] + __popc(same & lt), slot = slot0_s[e] + j;  // (full groups carry no padding)
      g.slot_of_route[i] = slot;
      g.slot_src[slot] = i / routes, g.slot_self[slot] = slot;
      g.slot_group[slot] = ((group0_s[e] + j / kMoeGroupRows) << 8) | (j % kMoeGroupRows);
    } else if (i < last) {
      g.slot_of_route[i] = 0xffffffffu;
    }
    __syncwarp();
    if (e != 0xffffffffu && !(same & lt)) warp_count[warp][e] += uint16_t(__popc(same));
    __syncwarp();
  }
}

// out = bf16(residual + sum over the row's routes in slot order of weight * float(y)), y at the routes' row slots.
// partial != 0: the routes the launch took only (slot_of_route says which: the others hold ~0), fp32 sums without the residual.
// A thread eight columns, eight routes' values in flight.
__global__ void __launch_bounds__(256) moe_combine_grouped_kernel(const SbMoeExpertArgs a, const uint32_t *slot_of_route, const uint16_t *y, uint32_t partial) {
  __shared__ uint32_t slot_s[32];
  __shared__ float weight_s[32];
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t row = blockIdx.y, c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (threadIdx.x < a.routes) slot_s[threadIdx.x] = slot_of_route[row * a.routes + threadIdx.x], weight_s[threadIdx.x] = a.weights[row * a.routes + threadIdx.x];
  __syncthreads();
  if (c >= a.hidden) return;
  float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  for (uint32_t s0 = 0; s0 < a.routes; s0 += 8) {
    uint4 v[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j)
      if (s0 + j < a.routes && slot_s[s0 + j] != 0xffffffffu) v[j] = *reinterpret_cast<const uint4 *>(y + size_t(slot_s[s0 + j]) * a.hidden + c);
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
      if (s0 + j >= a.routes || slot_s[s0 + j] == 0xffffffffu) continue;  // (not taken by the grouping)
      const float w = weight_s[s0 + j];
      const uint32_t u[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[2 * i] += w * bf16_bits_to_float(u[i] & 0xffffu), acc[2 * i + 1] += w * bf16_bits_to_float(u[i] >> 16);
    }
  }
  if (partial) {
    float *out = static_cast<float *>(a.out) + size_t(row) * a.hidden + c;
    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
      *reinterpret_cast<float4 *>(out) = make_float4(acc[0], acc[1], acc[2], acc[3]), *reinterpret_cast<float4 *>(out + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; i += 2) *reinterpret_cast<float2 *>(out + i) = make_float2(acc[i], acc[i + 1]);
    }
    return;
  }
  // (rows that lie on four bytes only are read and written two values at a time)
  const uint16_t *residual = a.residual ? static_cast<const uint16_t *>(a.residual) + size_t(row) * a.hidden + c : nullptr;
  uint16_t *out = static_cast<uint16_t *>(a.out) + size_t(row) * a.hidden + c;
  uint32_t r[4] = {0, 0, 0, 0};
  if (residual) {
    if ((reinterpret_cast<uintptr_t>(residual) & 15) == 0) {
      const uint4 w = *reinterpret_cast<const uint4 *>(residual);
      r[0] = w.x, r[1] = w.y, r[2] = w.z, r[3] = w.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = reinterpret_cast<const uint32_t *>(residual)[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    r[i] = uint32_t(float_to_bf16_bits(bf16_bits_to_float(r[i] & 0xffffu) + acc[2 * i])) | (uint32_t(float_to_bf16_bits(bf16_bits_to_float(r[i] >> 16) + acc[2 * i + 1])) << 16);
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    *reinterpret_cast<uint4 *>(out) = make_uint4(r[0], r[1], r[2], r[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint32_t *>(out)[i] = r[i];
  }
}

template <class K> static int launch_moe(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const MoeParams &p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = ctx().pdl ? 1 : 0;
  SB_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  return SB_OK;
}

}  // namespace sb

using namespace sb;

extern "C" uint64_t sb_moe_scratch_bytes(uint32_t rows, uint32_t routes, uint32_t hidden, uint32_t inter) {
  return rows > kMoeFewRows ? moe_group_layout(rows, routes, hidden, inter).bytes : moe_few_layout(rows, routes, hidden, inter).bytes;
}

// More than 16 rows: group the routes by expert, gather and convert each group's rows, the experts' one-pass gate/up and
// down on the many-row kernel over the groups, and the combine.
static int moe_experts_grouped(cudaStream_t s, const SbMoeExpertArgs *a, const MoeShare *part = nullptr) {
  const uint64_t n = uint64_t(a->rows) * a->routes;
  SB_REQUIRE(n <= kMoeMaxRoutes && a->experts_total <= kMoeMaxExperts, "sb_moe_experts: %u rows x %u routes over %u experts (up to %u routes, %u experts)",
             a->rows, a->routes, a->experts_total, kMoeMaxRoutes, kMoeMaxExperts);
  SB_REQUIRE(a->inter % 128 == 0 && a->hidden % 256 == 0, "sb_moe_experts: many rows need an intermediate width in 128s and a hidden width in 256s");
  const MoeGroupLayout l = moe_group_layout(a->rows, a->routes, a->hidden, a->inter);
  uint8_t *base = static_cast<uint8_t *>(a->scratch);
  auto at = [&](uint64_t off) { return base + off; };
  MoeGrouping g{reinterpret_cast<uint32_t *>(at(l.counts)), reinterpret_cast<uint4 *>(at(l.groups)), reinterpret_cast<uint32_t *>(at(l.slot_of_route)),
                reinterpret_cast<uint32_t *>(at(l.slot_src)), reinterpret_cast<uint32_t *>(at(l.slot_self)), reinterpret_cast<uint32_t *>(at(l.slot_group))};
  const bool pdl = ctx().pdl;
  {
    cudaLaunchConfig_t cfg = {};
    static std::atomic<uint64_t> allowed;
    const int st = allow_smem(reinterpret_cast<const void *>(moe_group_kernel), kMoeMaxRoutes * sizeof(uint16_t), allowed, ctx().device);
    if (st != SB_OK) return st;
    cfg.gridDim = dim3(1), cfg.blockDim = dim3(kMoeGroupThreads), cfg.dynamicSmemBytes = n * sizeof(uint16_t), cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = pdl ? 1 : 0;
    const MoeShare share = part ? *part : MoeShare{0, a->experts_total, 0xffffffffu, 0, 0};
    SB_CUDA(cudaLaunchKernelEx(&cfg, moe_group_kernel, a->selected, uint32_t(n), a->routes, a->experts_total, g, ctx().status_dev, share));
  }
  WidePrepareGroupedArgs c1{a->input, a->hidden, a->hidden, g.slot_src, g.slot_group, g.counts + 1, l.max_slots, g.groups, at(l.prepared1),
                            reinterpret_cast<float *>(at(l.scales1)), pdl};
  int st = launch_wide_prepare_grouped(s, c1);
  if (st != SB_OK) return st;
  WideGroupedArgs pair{a->gate, a->up, a->experts_total, a->inter, a->hidden, at(l.prepared1), reinterpret_cast<const float *>(at(l.scales1)), g.groups,
                       g.counts, l.max_groups, kMoeGroupRows, at(l.act), a->inter, pdl};
  st = launch_linear_wide_grouped(s, pair);
  if (st != SB_OK) return st;
  WidePrepareGroupedArgs c2{at(l.act), a->inter, a->inter, g.slot_self, g.slot_group, g.counts + 1, l.max_slots, g.groups, at(l.prepared2),
                            reinterpret_cast<float *>(at(l.scales2)), pdl};
  st = launch_wide_prepare_grouped(s, c2);
  if (st != SB_OK) return st;
  WideGroupedArgs down{a->down, nullptr, a->experts_total, a->hidden, a->inter, at(l.prepared2), reinterpret_cast<const float *>(at(l.scales2)), g.groups,
                       g.counts, l.max_groups, kMoeGroupRows, at(l.y), a->hidden, pdl};
  st = launch_linear_wide_grouped(s, down);
  if (st != SB_OK) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a->hidden / 8 + 255) / 256, a->rows), cfg.blockDim = dim3(std::min(256u, a->hidden / 8)), cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = pdl ? 1 : 0;
  SB_CUDA(cudaLaunchKernelEx(&cfg, moe_combine_grouped_kernel, *a, static_cast<const uint32_t *>(g.slot_of_route), reinterpret_cast<const uint16_t *>(at(l.y)),
                             part ? 1u : 0u));
  return SB_OK;
}

static int moe_check(const SbMoeExpertArgs *a, const char *who);

extern "C" int sb_moe_experts_partial(void *stream, const SbMoeExpertArgs *a, uint32_t expert0, uint32_t experts_local, uint32_t shared_id,
                                      uint32_t own_row0, uint32_t own_rows) {
  SB_NEED_DEVICE();
  const int st = moe_check(a, "sb_moe_experts_partial");
  if (st != SB_OK) return st;
  const bool shared = shared_id != 0xffffffffu;
  SB_REQUIRE(experts_local >= 1 && a->experts_total == experts_local + (shared ? 1u : 0u), "sb_moe_experts_partial: %u experts here (+ the shared one) against %u in the tensors",
             experts_local, a->experts_total);
  SB_REQUIRE(!shared || (shared_id >= expert0 + experts_local || shared_id < expert0), "sb_moe_experts_partial: the shared expert's id lies inside the rank's range");
  SB_REQUIRE(own_row0 + own_rows <= a->rows, "sb_moe_experts_partial: own rows [%u, %u) of %u", own_row0, own_row0 + own_rows, a->rows);
  const MoeShare share{expert0, experts_local, shared_id, own_row0, own_rows};
  return moe_experts_grouped(as_stream(stream), a, &share);
}

// Blocks that take a matrix-vector product a route: experts of up to 1024 x 512 and some 4.7 M weights a matrix over all routes.
// 3, 9 and 18 routes of 1024 x 256: 16.0, 16.7 and 17.6 us against 19.2, 19.6 and 20.0 by groups, 27 routes 21.3 against 22.6, 36
// routes 25.4 against 23.8; of 1024 x 512 3 and 6 routes 18.0 and 19.0 against 20.6 and 20.5, 10 routes 25.8 against 21.1; wider
// experts are even at 3 routes (1536 x 512: 22.2 against 22.5) and behind from there. The difference at the small end is two launches.
constexpr uint32_t kMoeVectorHidden = 1024, kMoeVectorInter = 512;
constexpr uint64_t kMoeVectorWeights = 18ull * 1024 * 256;
static bool moe_vector_block(const SbMoeExpertArgs &a) {
  return a.hidden <= kMoeVectorHidden && a.inter <= kMoeVectorInter && uint64_t(a.rows) * a.routes * a.hidden * a.inter <= kMoeVectorWeights;
}

extern "C" int sb_moe_experts(void *stream, const SbMoeExpertArgs *a) {
  SB_NEED_DEVICE();
  const int valid = moe_check(a, "sb_moe_experts");
  if (valid != SB_OK) return valid;
  if (a->rows > kMoeFewRows) return moe_experts_grouped(as_stream(stream), a);
  const MoeFewLayout l = moe_few_layout(a->rows, a->routes, a->hidden, a->inter);
  uint8_t *base = static_cast<uint8_t *>(a->scratch);
  const MoeParams p{*a,
                    reinterpret_cast<uint16_t *>(base + l.intermediate),
                    reinterpret_cast<uint16_t *>(base + l.y),
                    reinterpret_cast<uint32_t *>(base + l.counts),
                    reinterpret_cast<MoeFew *>(base + l.groups),
                    base + l.x,
                    base + l.act,
                    reinterpret_cast<float *>(base + l.x_scale),
                    reinterpret_cast<float *>(base + l.act_scale)};
  cudaStream_t s = as_stream(stream);
  const uint32_t routes = a->rows * a->routes, resident = uint32_t(ctx().sm_count) * 2;
  int st;
  if (moe_vector_block(*a)) {
    constexpr uint32_t kPairBlock = kMoeWarps * kMoeColsPair, kDownBlock = kMoeWarps * kMoeColsDown;
    st = launch_moe(moe_expert_kernel<true>, dim3(routes, (a->inter + kPairBlock - 1) / kPairBlock), dim3(kMoeThreads), size_t(a->hidden) * 4, s, p);
    if (st == SB_OK) st = launch_moe(moe_expert_kernel<false>, dim3(routes, (a->hidden + kDownBlock - 1) / kDownBlock), dim3(kMoeThreads), size_t(a->inter) * 4, s, p);
    if (st != SB_OK) return st;
    return launch_moe(moe_combine_kernel, dim3((a->hidden + 255) / 256, a->rows), dim3(256), 0, s, p);
  }
  st = launch_moe(moe_few_prepare_kernel, dim3(a->rows + 1), dim3(kMoeThreads), 0, s, p);
  if (st == SB_OK) st = launch_moe(moe_few_kernel<true>, dim3(resident), dim3(kMoeThreads), 0, s, p);
  if (st == SB_OK) st = launch_moe(moe_few_convert_kernel, dim3(routes), dim3(std::min(uint32_t(kMoeThreads), a->inter / 8)), 0, s, p);
  if (st == SB_OK) st = launch_moe(moe_few_kernel<false>, dim3(resident), dim3(kMoeThreads), 0, s, p);
  if (st != SB_OK) return st;
  return launch_moe(moe_combine_kernel, dim3((a->hidden + 255) / 256, a->rows), dim3(256), 0, s, p);
}

static int moe_check(const SbMoeExpertArgs *a, const char *who) {
  SB_REQUIRE(a && a->input && a->selected && a->weights && a->gate && a->up && a->down && a->scratch && a->out, "%s: null pointer", who);
  SB_REQUIRE(a->format == SB_FMT_Q4K, "%s: experts in format %u (Q4_K only)", who, a->format);
  SB_REQUIRE(a->rows >= 1 && a->routes >= 1 && a->routes <= 32, "%s: %u rows x %u routes (1..32)", who, a->rows, a->routes);
  SB_REQUIRE(a->hidden && a->hidden % 256 == 0 && a->inter && a->inter % 256 == 0 && a->hidden <= 8192 && a->inter <= 8192,
             "%s: hidden %u and intermediate %u are multiples of 256 up to 8192", who, a->hidden, a->inter);
  SB_REQUIRE(a->experts_total >= 1, "%s: no experts", who);
  SB_REQUIRE(((reinterpret_cast<uintptr_t>(a->gate) | reinterpret_cast<uintptr_t>(a->up) | reinterpret_cast<uintptr_t>(a->down) |
               reinterpret_cast<uintptr_t>(a->scratch)) & 15) == 0,
             "%s: expert tensors and scratch must be 16-byte aligned", who);
  return SB_OK;
}
