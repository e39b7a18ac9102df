// Gated-DeltaNet verify step of one lane and one layer with fp32 state.
//
// Takes the place of the reference's verify_gdn_fused* kernels (runtime/metal/kernels/decode/gdn.metal:
// prologue :139-264, fold :270-298, chain scan :312-415, gate :489-526; primitives
// runtime/metal/kernels/common/gdn_primitives.h:63-106) and of ops::GDN::addDecode / addFold
// (runtime/ops/GDN.cpp:225-328).
//
//   grid     (4, value_heads, lanes): the reference runs one threadgroup per value head (48 on the 27B shape,
//            too few for 148 SMs); a head's 128 state rows (value dimensions) are independent given
//            k, v and the gates, so each CTA takes 32 of them; a head's four CTAs are a cluster and divide what the
//            head's rows share (gate projection, q / k convolution and norms, the rows' inner products, the output norm)
//   steps    (1) conv history = last three input rows before the block (carried rows ++ pending rows);
//            (2) conv + SiLU, q/k RMS norm and scales (2^-7, 128^-1/2), beta and decay per row;
//            (3) fold the pending rows into the state -> committed state stored; (4) the rows' outputs from the
//            committed state; (5) RMS norm over the 128 value dimensions, gate by silu(z), the hidden rows; (6) this step's tape
//
// The delta rule without its serial chain. A row's step S' = d S + u k^T, u = beta (v - d S k) touches the whole state, one row after
// the other. The state after the block is never stored, so it is never formed: with S the committed state, P(t) a row's path from
// the anchor and G(t, j) the product of the decays on it after row j (D_t: of all of them),
//   u_t = beta_t (v_t - D_t (S k_t) - sum over j in P(t), j != t, of G(t, j) (k_j . k_t) u_j)
//   o_t = D_t (S q_t) + sum over j in P(t) of G(t, j) (k_j . q_t) u_j
// that is: the 16 x 128 by 128 products S k_t and S q_t, all rows at once from registers; the rows' inner products; and a
// triangular system of 16 unknowns per state row, one thread each. Chains and trees are the same formulas. The fold is the same
// system over the pending rows, then one update of rank `pending`: S = D S + sum_t G(last, t) u_t k_t^T.
// What bounds it: the prologue's latency (dependent loads, the gate projection), four cluster barriers, and, with many lanes, instruction
// issue (half of the slots) and the shared-memory port. One layer of the 27B shape, 16 rows and 6 to fold, graph replay: 13.8 us (23.7
// with the rows advanced in turn), eight lanes 68 (100), one row and one to fold 10.5 (11.3), eight lanes of those 48.0 (47.7). The
// folded state's error against 64 bits is 5.6e-8 either way, that of the rows' outputs their bf16.
//   CTA      256 threads; warp w owns rows 16 (w & 1).. of the CTA's 32 and key columns 32 (w / 2).. , in fp32 registers laid out as
//            the tensor cores' A operand
//   rollback the state after the block is never stored: the caller passes how many tape rows were accepted
//            (pending_rows, or a device word written by sb_accept) to the next step, which folds them
#include <algorithm>
#include <cooperative_groups.h>
#include <type_traits>

#include "sb_internal.h"
#include "sb_ptx.cuh"
#include "sb_dot.cuh"

namespace sb {

constexpr int kGdnThreads = 256;
constexpr int kGdnRows = 16;      // rows of a verify block
constexpr int kGdnSplit = 4;      // CTAs per value head
constexpr int kGdnVd = 128 / kGdnSplit;  // value dimensions per CTA
constexpr int kD = 128, kTaps = 4;

struct GdnParams {
  SbGdnArgs a;
};

// Lane blockIdx.z's view of a launch over several lanes: its 16 row slots of the row-indexed buffers, its cell, tapes and
// pending words.
__device__ __forceinline__ GdnParams gdn_lane_view(GdnParams p) {
  const uint32_t z = blockIdx.z;
  if (z == 0 && gridDim.z == 1) return p;
  SbGdnArgs &a = p.a;
  const size_t KW = size_t(a.key_heads) * 128, VW = size_t(a.value_heads) * 128, C = 2 * KW + VW, R = 16 * size_t(z);
  auto rows16 = [&](const void *q, size_t stride) { return q ? static_cast<const void *>(static_cast<const uint16_t *>(q) + R * stride) : q; };
  a.qkvz = rows16(a.qkvz, a.qkvz_stride), a.b = rows16(a.b, a.ab_stride), a.a = rows16(a.a, a.ab_stride);
  a.gate_input = rows16(a.gate_input, a.gate_input_stride);
  a.hidden = const_cast<void *>(rows16(a.hidden, a.hidden_stride));
  if (a.tree) a.tree = static_cast<const uint2 *>(a.tree) + R;
  a.conv_state_in = static_cast<const uint16_t *>(a.conv_state_in) + size_t(z) * 3 * C;
  a.conv_state_out = static_cast<uint16_t *>(a.conv_state_out) + size_t(z) * 3 * C;
  a.state_in += size_t(z) * a.value_heads * 128 * 128, a.state_out += size_t(z) * a.value_heads * 128 * 128;
  auto tape = [&](SbGdnTape &t) {
    if (t.inputs) t.inputs = static_cast<uint16_t *>(t.inputs) + R * C;
    if (t.k) t.k = static_cast<uint16_t *>(t.k) + R * KW;
    if (t.v) t.v = static_cast<uint16_t *>(t.v) + R * VW;
    if (t.beta) t.beta = static_cast<uint16_t *>(t.beta) + R * a.value_heads;
    if (t.decay) t.decay += R * a.value_heads;
  };
  tape(a.pending), tape(a.step);
  if (a.pending_rows_dev) a.pending_rows_dev += z;
  if (a.pending_path_dev) a.pending_path_dev += z;
  return p;
}

// Row of the n-th token (from the anchor) of a path mask.
__device__ __forceinline__ uint32_t path_row(uint32_t path, uint32_t n) {
  for (uint32_t i = 0; i < n; ++i) path &= path - 1;
  return path ? uint32_t(__ffs(int(path))) - 1u : 0u;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sixteen values a lane, summed over the warp: lane l ends with value l >> 1 (both lanes of a pair hold it).
__device__ __forceinline__ float sum_scatter16(float (&v)[16], uint32_t lane) {
#pragma unroll
  for (int half = 8; half; half >>= 1) {
    const bool upper = (lane & (2 * half)) != 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i >= half) break;
      const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * half);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

template <int BYTES> __device__ __forceinline__ void copy_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
// Two neighbouring bf16 of a tape whose base need not lie on more than its element's two bytes.
__device__ __forceinline__ uint32_t load_pair(const uint16_t *p) {
  return (reinterpret_cast<uintptr_t>(p) & 3) == 0 ? *reinterpret_cast<const uint32_t *>(p) : uint32_t(p[0]) | (uint32_t(p[1]) << 16);
}
__device__ __forceinline__ void store_pair(uint16_t *p, uint32_t v) {
  if ((reinterpret_cast<uintptr_t>(p) & 3) == 0) *reinterpret_cast<uint32_t *>(p) = v;
  else p[0] = uint16_t(v), p[1] = uint16_t(v >> 16);
}

// Two floats as three bf16 terms each (hi + mid + lo carry the 24 bits of an fp32 significand), packed.
__device__ __forceinline__ void split3(float a, float b, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const float ar = a - __low2float(h), br = b - __high2float(h);
  const __nv_bfloat162 m = __floats2bfloat162_rn(ar, br), l = __floats2bfloat162_rn(ar - __low2float(m), br - __high2float(m));
  hi = *reinterpret_cast<const uint32_t *>(&h), mid = *reinterpret_cast<const uint32_t *>(&m), lo = *reinterpret_cast<const uint32_t *>(&l);
}

constexpr int kKeyPitch = kD + 8, kPendingPitch = kD + 4, kProductPitch = 36, kGramPitch = 20;
constexpr int kLocal = 2 * kD + kGdnVd;  // 288 channels of a CTA: q and k of the key head, 32 value dimensions
struct GdnShared {
  uint16_t x[2][kGdnRows][kKeyPitch];         // bf16 k rows, q rows
  float pk[kGdnRows][kPendingPitch];
  float v[kGdnRows][kGdnVd], pv[kGdnRows][kGdnVd];
  union {
    uint16_t in[kGdnRows + 3][kLocal];                 // convolution inputs, until the tape is written
    float part[4][2 * kGdnRows][kProductPitch];        // then: the four column quarters' shares of S pk_t (pending rows), later of S k_t and S q_t
  };
  float u[kGdnRows][kGdnVd];                  // D_t (S k_t), then the solution: pending rows (scaled for the update), then the block's
  float o[kGdnRows][kGdnVd];                  // D_t (S q_t), this CTA's value dimensions
  float kk[kGdnRows][kGramPitch], kq[kGdnRows][kGramPitch], pkk[kGdnRows][kGramPitch];  // inner products [t][j] and coefficients (see there)
  float out[kGdnRows / kGdnSplit][kD];        // outputs of the rows this CTA normalises
  uint2 w[kLocal];
  float gate[kDotGroups][kGdnRows][2];        // group partial sums of the head's b and a per row (fused gate projection)
  alignas(16) float beta[kGdnRows], decay[kGdnRows], pbeta[kGdnRows], pdecay[kGdnRows];
  alignas(16) float after[kGdnRows];          // products of the pending decays after a row
  float pending_decay;                        // and of all of them
  uint32_t path[kGdnRows];                    // the row's path from the anchor, itself included
  uint8_t tap[kGdnRows][kTaps];               // where in `in` a row's four convolution taps lie (its path's last tokens)
};
static_assert(sizeof(GdnShared) <= 56 * 1024, "four CTAs a SM");
static_assert(kGdnThreads / 32 == kDotGroups && kGdnThreads == kGdnRows * kGdnRows, "a warp a group of the dot product, a thread a coefficient");
static_assert(kGdnRows == 4 * kGdnSplit, "four rows per CTA of the head");

// kTree: the rows may form a tree and the pending path may be any row mask; without it the rows are a chain and the pending
// rows the tape's first, which keeps the tap and path tables out of the usual case.
// kResident: CTAs per SM the registers are held to: two for a launch of one lane (192 CTAs on the 27B shape), four for several.
// Both run the same arithmetic: a lane's bits do not depend on the launch it is in.
template <bool kTree, int kResident = 2>
__global__ void __cluster_dims__(kGdnSplit, 1, 1) __launch_bounds__(kGdnThreads, kResident) gdn_kernel(const GdnParams p_in) {
  const GdnParams p = gdn_lane_view(p_in);  // (one lane: p_in itself)
  const SbGdnArgs &a = p.a;
  extern __shared__ __align__(16) uint8_t gdn_smem[];
  GdnShared &sh = *reinterpret_cast<GdnShared *>(gdn_smem);
  namespace cg = cooperative_groups;
  cg::cluster_group head_ctas = cg::this_cluster();
  auto cluster_arrive = [] { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); };
  auto cluster_wait = [] { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); };
  pdl_launch_dependents();
  cluster_arrive();  // "this CTA runs", waited for before the first store into a peer CTA
  const uint32_t vs = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t KH = a.key_heads, VH = a.value_heads, KW = KH * kD, VW = VH * kD, C = 2 * KW + VW;
  const uint32_t per_key = VH / KH, kh = h / per_key, vd0 = vs * kGdnVd;
  const uint32_t rows = a.rows;
  const bool projects = a.gate_weight && 4 * vs < rows;  // this CTA has rows of the fused gate projection
  const uint16_t *qkvz = static_cast<const uint16_t *>(a.qkvz);
  const uint16_t *conv_w = static_cast<const uint16_t *>(a.conv_w);
  const uint16_t *cs_in = static_cast<const uint16_t *>(a.conv_state_in);
  const uint16_t *pin = static_cast<const uint16_t *>(a.pending.inputs);
  const bool qk_writer = h % per_key == 0 && vs == 0;

  // This warp's share of the state, requested first so the latency hides behind the prologue and, where
  // the caller allows it (below), before the wait for the kernel ahead: in the model's step the cell was written a
  // whole step ago, and this CTA may be resident while the projection before it drains.
  // The share is two 16 x 16 blocks as the tensor cores' A operand has them: rows 16 (warp & 1) + g and + 8 (g = lane / 4), key columns
  // 32 (warp / 2) + 16 b + 2 t, + 1, + 8, + 9 (t = lane % 4) of blocks b = 0, 1; S[8 b + 4 (second row) + 2 (second pair) + i].
  float S[16];
  const uint32_t g4 = lane >> 2, t4 = lane & 3, quarter = warp >> 1, srow = 16 * (warp & 1) + g4, scol = 32 * quarter + 2 * t4;
  const size_t sbase = (size_t(h) * kD + vd0 + srow) * kD + scol;
  auto load_state = [&] {
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int second = 0; second < 2; ++second)
#pragma unroll
        for (int pair = 0; pair < 2; ++pair) {
          const float2 s2 = *reinterpret_cast<const float2 *>(a.state_in + sbase + size_t(8 * second) * kD + 16 * b + 8 * pair);
          S[8 * b + 4 * second + 2 * pair] = s2.x, S[8 * b + 4 * second + 2 * pair + 1] = s2.y;
        }
  };
  // Only a caller that vouches for the cell (SB_GDN_STATE_SETTLED: nothing still running on the stream writes
  // state_in) gets the early load; otherwise the launch ahead may be the one that produced the cell (a fold
  // followed at once by a step on the swapped cells), and the load waits for it like every other read.
  const bool settled = (a.flags & SB_GDN_STATE_SETTLED) != 0;
  if (settled) load_state();
  pdl_wait();
  if (!settled) load_state();
  const float a_scale = a.a_scale[h], dt_bias = bf16_bits_to_float(static_cast<const uint16_t *>(a.dt_bias)[h]);
  // Conv inputs of this CTA's channels (q and k of the key head, 32 value dimensions), in[3 + row][local channel], and their taps'
  // weights: asynchronous copies, on their way while the gate projection runs.
  const uint32_t chan0[3] = {kh * kD, KW + kh * kD, 2 * KW + h * kD + vd0};
  auto global_channel = [&](uint32_t lc) { return lc < kD ? chan0[0] + lc : lc < 2 * kD ? chan0[1] + lc - kD : chan0[2] + lc - 2 * kD; };
  uint32_t pending_path = a.pending_path_dev ? *a.pending_path_dev : a.pending_path;  // (first used below the gate projection)
  uint32_t pending_n = a.pending_rows_dev ? *a.pending_rows_dev : a.pending_rows;
  for (uint32_t i = tid; i < rows * (kLocal / 8); i += kGdnThreads) {
    const uint32_t r = i / (kLocal / 8), lc = (i % (kLocal / 8)) * 8;
    copy_async<16>(&sh.in[3 + r][lc], qkvz + size_t(r) * a.qkvz_stride + global_channel(lc));
  }
  for (uint32_t lc = tid; lc < kLocal; lc += kGdnThreads) copy_async<8>(&sh.w[lc], conv_w + size_t(global_channel(lc)) * kTaps);
  if (tid < kGdnRows) {
    uint32_t path = (2u << tid) - 1u;
    if (kTree && tid < rows) {
      path = (a.tree ? static_cast<const uint2 *>(a.tree)[tid].x & path : path) | (1u << tid);
      const int depth = __popc(path) - 1;
      for (int tap = 0; tap < kTaps; ++tap) {
        const int at = depth - 3 + tap;  // the tap's token, counted from the anchor; before it: the carried history
        sh.tap[tid][tap] = uint8_t(at < 0 ? 3 + at : 3 + int(path_row(path, uint32_t(at))));
      }
    }
    sh.path[tid] = path;
  }
  // Fused gate projection: this CTA takes rows 4 vs .. 4 vs + 3; warp w computes group w's partial sums of those rows x
  // {b, a} over the layer's normalised input and stores them into all four CTAs of the head; the rows' threads add the
  // 8 groups in order below (the order of sb_linear_f32, so the bits agree with the unfused way).
  float gates[4][2];
  if (projects) {
    const float *const wrow[2] = {a.gate_weight + size_t(h) * a.gate_k, a.gate_weight + size_t(VH + h) * a.gate_k};
    const uint16_t *gx = static_cast<const uint16_t *>(a.gate_input);
    const uint16_t *xrow[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) xrow[r] = gx + size_t(min(4 * vs + uint32_t(r), rows - 1)) * a.gate_input_stride;
    lane_dot_group_f32_bf16<2, 4>(wrow, xrow, a.gate_k, lane, warp, gates);
  }
  // The previous step's accepted path in its tape: a row mask, or the tape's first rows.
  if (!a.pending_path_dev && !a.pending_path) pending_path = (1u << min(pending_n, uint32_t(kGdnRows))) - 1u;
  pending_path &= (1u << kGdnRows) - 1u;
  const uint32_t pending = uint32_t(__popc(pending_path));
  auto pending_row = [&](uint32_t n) { return kTree ? path_row(pending_path, n) : n; };
  // History rows -3..-1: row i (0..2, oldest first) is row pending - 3 + i of (carried rows ++ pending rows).
  if (tid < 3 * (kLocal / 8)) {
    const uint32_t r = tid / (kLocal / 8), lc = (tid % (kLocal / 8)) * 8, ch = global_channel(lc);
    const int hsrc = int(pending) - 3 + int(r);
    copy_async<16>(&sh.in[r][lc], hsrc >= 0 ? pin + size_t(pending_row(uint32_t(hsrc))) * C + ch : cs_in + size_t(3 + hsrc) * C + ch);
  }
  // pending rows' keys, values and gates from their tape, requested before the gate projection's lanes are added up and stored
  // after; rows past them are zeros to a whole eight (the products below take eights)
  constexpr int kPkLoads = kGdnRows * kD / 2 / kGdnThreads, kPvLoads = kGdnRows * kGdnVd / kGdnThreads;
  uint32_t pk2[kPkLoads];
  uint16_t pv1[kPvLoads], pbeta1 = 0;
  float pdecay1 = 0.0f;
#pragma unroll
  for (int i = 0; i < kPkLoads; ++i) {
    const uint32_t n = tid / (kD / 2) + i * (kGdnThreads / (kD / 2)), d = 2 * (tid % (kD / 2));
    pk2[i] = n < pending ? load_pair(static_cast<const uint16_t *>(a.pending.k) + size_t(pending_row(n)) * KW + kh * kD + d) : 0u;
  }
#pragma unroll
  for (int i = 0; i < kPvLoads; ++i) {
    const uint32_t n = warp + i * (kGdnThreads / kGdnVd);
    pv1[i] = n < pending ? static_cast<const uint16_t *>(a.pending.v)[size_t(pending_row(n)) * VW + h * kD + vd0 + lane] : uint16_t(0);
  }
  if (tid < pending) {
    const uint32_t trow = pending_row(tid);
    pbeta1 = static_cast<const uint16_t *>(a.pending.beta)[size_t(trow) * VH + h], pdecay1 = a.pending.decay[size_t(trow) * VH + h];
  }
  // The gates' eight sums over the lanes, halved at every exchange: lane l ends with sum l / 4 (row l / 8, b or a). The same
  // additions as a butterfly of each, so the same bits.
  float gate_sum = 0.0f;
  if (projects) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = gates[i >> 1][i & 1];
#pragma unroll
    for (int half = 4; half; half >>= 1) {
      const bool upper = (lane & (4 * half)) != 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i >= half) break;
        const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * half);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    gate_sum = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
  }
#pragma unroll
  for (int i = 0; i < kPkLoads; ++i) {
    const uint32_t n = tid / (kD / 2) + i * (kGdnThreads / (kD / 2));
    if (n >= (pending + 7) / 8 * 8) break;
    *reinterpret_cast<float2 *>(&sh.pk[n][2 * (tid % (kD / 2))]) = make_float2(bf16_bits_to_float(pk2[i] & 0xffffu), bf16_bits_to_float(pk2[i] >> 16));
  }
#pragma unroll
  for (int i = 0; i < kPvLoads; ++i) sh.pv[warp + i * (kGdnThreads / kGdnVd)][lane] = bf16_bits_to_float(pv1[i]);
  if (tid < kGdnRows) sh.pbeta[tid] = bf16_bits_to_float(pbeta1), sh.pdecay[tid] = pdecay1;
  asm volatile("cp.async.wait_all;" ::: "memory");
  // The sixteen inner products of a row with rows of keys, into row t of every CTA's matrix: a warp, four dimensions a lane.
  auto inner_products = [&](auto key, const float4 x4, float (*gram)[kGramPitch], uint32_t t) {
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float4 k4 = key(j);
      v[j] = fmaf(k4.w, x4.w, fmaf(k4.z, x4.z, fmaf(k4.y, x4.y, k4.x * x4.x)));
    }
    const float dot = sum_scatter16(v, lane);
    const uint32_t j = lane >> 1;
    // (the pair's two lanes store to two CTAs each)
#pragma unroll
    for (int half = 0; half < 2; ++half) head_ctas.map_shared_rank(&gram[t][j], int(2 * (lane & 1) + half))[0] = dot;
  };
  auto pending_key = [&](int j) { return *reinterpret_cast<const float4 *>(&sh.pk[j][4 * lane]); };
  auto block_row = [&](int which, int j) {
    const uint2 two = *reinterpret_cast<const uint2 *>(&sh.x[which][j][4 * lane]);
    return make_float4(bf16_bits_to_float(two.x & 0xffffu), bf16_bits_to_float(two.x >> 16), bf16_bits_to_float(two.y & 0xffffu), bf16_bits_to_float(two.y >> 16));
  };
  __syncthreads();  // the CTA's staging is complete
  cluster_wait();   // every CTA of the head runs
  if (projects) head_ctas.map_shared_rank(&sh.gate[warp][4 * vs + (lane >> 3)][(lane >> 2) & 1], int(lane & 3))[0] = gate_sum;
  if (warp >= 4 && 4 * (warp - 4) + vs < pending) inner_products(pending_key, pending_key(4 * (warp - 4) + vs), sh.pkk, 4 * (warp - 4) + vs);
  cluster_arrive();  // (1) the gates' sums and the pending rows' inner products
  // NC neighbouring channels' convolution and SiLU for a row.
  auto conv = [&](uint32_t row, uint32_t lc, auto &out) {
    constexpr int NC = sizeof(out) / sizeof(float);
    uint2 wv[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) wv[c] = sh.w[lc + c];
#pragma unroll
    for (int c = 0; c < NC; ++c) out[c] = 0.0f;
#pragma unroll
    for (int tap = 0; tap < kTaps; ++tap) {
      const uint16_t *x = &sh.in[kTree ? uint32_t(sh.tap[row][tap]) : row + tap][lc];
      uint32_t two[NC / 2];
      if (NC == 4) {
        const uint2 t = *reinterpret_cast<const uint2 *>(x);
        two[0] = t.x, two[NC / 2 - 1] = t.y;
      } else {
        two[0] = *reinterpret_cast<const uint32_t *>(x);
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const uint32_t pair = tap < 2 ? wv[c].x : wv[c].y;
        const float w = bf16_bits_to_float((tap & 1) ? pair >> 16 : pair & 0xffffu);
        out[c] = __fadd_rn(out[c], __fmul_rn(bf16_bits_to_float((c & 1) ? two[c / 2] >> 16 : two[c / 2] & 0xffffu), w));
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) out[c] = round_bf16(silu_f(round_bf16(out[c])));
  };
  // (2) conv outputs: this CTA's 32 value dimensions, and q, k of the key head (128 each) for rows 4 vs .. 4 vs + 3 only:
  // the head's four CTAs divide the rows, normalise their own and store the result into all four. A warp takes q or k of a row,
  // four dimensions a lane, so its convolution, norm and stores need nobody else.
  const uint32_t qk_row = 4 * vs + (warp >> 1);
  if (qk_row < rows) {
    float x[4];
    conv(qk_row, ((warp & 1) ? kD : 0) + 4 * lane, x);
    const float ss = warp_sum((x[0] * x[0] + x[1] * x[1]) + (x[2] * x[2] + x[3] * x[3]));
    const float inv = rsqrtf(ss / float(kD) + 1e-6f);
    const float post = (warp & 1) ? 0.08838834765f : 0.0078125f;
    uint32_t bits[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
      bits[i] = uint32_t(float_to_bf16_bits(round_bf16(x[2 * i] * inv) * post)) | (uint32_t(float_to_bf16_bits(round_bf16(x[2 * i + 1] * inv) * post)) << 16);
    uint16_t *vec = &sh.x[(warp & 1) ? 0 : 1][qk_row][4 * lane];
#pragma unroll
    for (int peer = 0; peer < kGdnSplit; ++peer) *reinterpret_cast<uint2 *>(head_ctas.map_shared_rank(vec, peer)) = make_uint2(bits[0], bits[1]);
  }
  // (rows past the block are zeros to a whole eight: the products take eights, the inner products' of further rows are not used)
  for (uint32_t i = tid; i < ((rows + 7) / 8 * 8 - rows) * (kD / 2); i += kGdnThreads)
    *reinterpret_cast<uint32_t *>(&sh.x[0][rows + i / (kD / 2)][2 * (i % (kD / 2))]) = *reinterpret_cast<uint32_t *>(&sh.x[1][rows + i / (kD / 2)][2 * (i % (kD / 2))]) = 0u;
  // Two values of a row a thread, here and below: row ct, value dimensions 2 cj, + 1.
  const uint32_t ct = tid / kGdnRows, cj = tid % kGdnRows, cv = 2 * cj;
  if (ct >= rows) {
    *reinterpret_cast<float2 *>(&sh.v[ct][cv]) = make_float2(0.0f, 0.0f);  // (and no gate, below: no update)
  } else {
    float v[2];
    conv(ct, 2 * kD + cv, v);
    *reinterpret_cast<float2 *>(&sh.v[ct][cv]) = make_float2(v[0], v[1]);
    store_pair(static_cast<uint16_t *>(a.step.v) + size_t(ct) * VW + h * kD + vd0 + cv, uint32_t(float_to_bf16_bits(v[0])) | (uint32_t(float_to_bf16_bits(v[1])) << 16));
  }
  // (6) this step's tape of inputs and the carried conv rows, from the staged inputs (the value channels, and the key head's in
  // one CTA), eight channels at a time
  {
    uint16_t *tin = static_cast<uint16_t *>(a.step.inputs), *cs_out = static_cast<uint16_t *>(a.conv_state_out);
    const uint32_t lc0 = qk_writer ? 0 : 2 * kD, units = (kLocal - lc0) / 8;
    for (uint32_t i = tid; i < (3 + rows) * units; i += kGdnThreads) {
      const uint32_t r = i / units, lc = lc0 + 8 * (i % units), ch = global_channel(lc);
      uint16_t *dst = r < 3 ? cs_out + size_t(r) * C + ch : tin + size_t(r - 3) * C + ch;
      if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(&sh.in[r][lc]);
      } else {  // (a tape or cell that lies on its element's two bytes only)
#pragma unroll 1
        for (int e = 0; e < 8; ++e) dst[e] = sh.in[r][lc + e];
      }
    }
  }
  cluster_wait();  // (1)
  auto four = [&](const float (&m)[4][2 * kGdnRows][kProductPitch], uint32_t i) {  // the quarters in order
    const float2 p0 = *reinterpret_cast<const float2 *>(&m[0][i][cv]), p1 = *reinterpret_cast<const float2 *>(&m[1][i][cv]);
    const float2 p2 = *reinterpret_cast<const float2 *>(&m[2][i][cv]), p3 = *reinterpret_cast<const float2 *>(&m[3][i][cv]);
    return make_float2(((p0.x + p1.x) + p2.x) + p3.x, ((p0.y + p1.y) + p2.y) + p3.y);
  };
  // Product of the decays of the rows in a mask, in row order.
  auto decays = [&](const float (&d)[kGdnRows], uint32_t mask) {
    float g = 1.0f;
#pragma unroll
    for (int i4 = 0; i4 < kGdnRows; i4 += 4) {
      const float4 d4 = *reinterpret_cast<const float4 *>(&d[i4]);
      g *= (mask >> i4 & 1u) ? d4.x : 1.0f, g *= (mask >> (i4 + 1) & 1u) ? d4.y : 1.0f;
      g *= (mask >> (i4 + 2) & 1u) ? d4.z : 1.0f, g *= (mask >> (i4 + 3) & 1u) ? d4.w : 1.0f;
    }
    return g;
  };
  // The n unknowns of state row `lane`, by one warp: u_t = beta_t (v_t - m_t), m_t = D_t (S k_t) (in sh.u) + sum over j < t of c[j][t] u_j,
  // a finished unknown at a time so that a step waits for three operations only. What the state already holds of v_t is summed by
  // itself: it is small beside v_t, so its roundings are too (with -beta c u_j added to the right-hand side one by one the folded
  // state was 8e-8 off instead of 6e-8). A tree row takes the unknowns on its own path only (not the others times zero: one of them
  // may be no number); in a chain every earlier unknown is on it.
  auto solve = [&](auto tree_rows, uint32_t n, const float (*c)[kGramPitch], const float (&v)[kGdnRows][kGdnVd], const float (&beta)[kGdnRows], float (&u)[kGdnRows]) {
    constexpr bool kPaths = decltype(tree_rows)::value;
    const uint32_t path = kPaths ? sh.path[lane % kGdnRows] : 0u;
#pragma unroll
    for (int t = 0; t < kGdnRows; ++t) u[t] = sh.u[t][lane];
#pragma unroll
    for (int j = 0; j < kGdnRows; ++j) {
      if (uint32_t(j) >= n) break;
      u[j] = beta[j] * (v[j][lane] - u[j]);
      const uint32_t takes = kPaths ? __ballot_sync(0xffffffffu, path >> j & 1u) : 0xffffffffu;  // the rows with j on their path
#pragma unroll
      for (int t4x = (j + 1) / 4 * 4; t4x < kGdnRows; t4x += 4) {
        const float4 c4 = *reinterpret_cast<const float4 *>(&c[j][t4x]);
        if (t4x > j && (takes >> t4x & 1u)) u[t4x] = fmaf(c4.x, u[j], u[t4x]);
        if (t4x + 1 > j && (takes >> (t4x + 1) & 1u)) u[t4x + 1] = fmaf(c4.y, u[j], u[t4x + 1]);
        if (t4x + 2 > j && (takes >> (t4x + 2) & 1u)) u[t4x + 2] = fmaf(c4.z, u[j], u[t4x + 2]);
        if (t4x + 3 > j && (takes >> (t4x + 3) & 1u)) u[t4x + 3] = fmaf(c4.w, u[j], u[t4x + 3]);
      }
    }
  };
  if (pending) {  // (3)
    __syncthreads();  // nobody reads the convolution inputs any more (they have been read since the CTA arrived)
    // S pk_t: eight rows at a time (four where there are no more), a thread its two state rows over its eight columns, summed over
    // the four lanes that share the rows (products halved at every exchange).
    auto products = [&](auto count, uint32_t n0) {
      constexpr int N = decltype(count)::value;
      float v[2 * N];  // [row of the pair][pending row]
#pragma unroll
      for (int n = 0; n < N; ++n) {
        float lo = 0.0f, hi = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // block c / 2, pair c % 2
          const float2 k2 = *reinterpret_cast<const float2 *>(&sh.pk[n0 + n][scol + 16 * (c >> 1) + 8 * (c & 1)]);
          const int at = 8 * (c >> 1) + 2 * (c & 1);
          lo = fmaf(S[at], k2.x, lo), lo = fmaf(S[at + 1], k2.y, lo);
          hi = fmaf(S[at + 4], k2.x, hi), hi = fmaf(S[at + 5], k2.y, hi);
        }
        v[n] = lo, v[N + n] = hi;
      }
#pragma unroll
      for (int half = N; half >= N / 2; half >>= 1) {  // lanes 2 apart divide the pair's rows, lanes 1 apart the products
        const int apart = half == N ? 2 : 1;
        const bool upper = (lane & apart) != 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          if (i >= half) break;
          const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, apart);
        }
      }
#pragma unroll
      for (int i = 0; i < N / 2; ++i) sh.part[quarter][n0 + N / 2 * (lane & 1) + i][srow + ((lane & 2) ? 8 : 0)] = v[i];
    };
    for (uint32_t n0 = 0; n0 < pending; n0 += 8) {
      if (pending - n0 > 4) products(std::integral_constant<int, 8>{}, n0);
      else products(std::integral_constant<int, 4>{}, n0);
    }
    __syncthreads();
    // coefficients [j][t] (into the matrix the block's rows use later) and D_t (S k_t); rows past the pending ones are zeros
    const bool there = ct < pending;
    const uint32_t below = there ? (2u << ct) - 1u : 0u;
    sh.kk[cj][ct] = there && cj < ct ? decays(sh.pdecay, below & ~((2u << cj) - 1u)) * sh.pkk[ct][cj] : 0.0f;
    float2 right = make_float2(0.0f, 0.0f);
    if (there) {
      const float2 sx = four(sh.part, ct);
      const float d = decays(sh.pdecay, below);
      right = make_float2(d * sx.x, d * sx.y);
    }
    *reinterpret_cast<float2 *>(&sh.u[ct][cv]) = right;
    if (there && cj == 0) sh.after[ct] = decays(sh.pdecay, ((1u << pending) - 1u) & ~((2u << ct) - 1u));
    if (tid == 1) sh.pending_decay = decays(sh.pdecay, (1u << pending) - 1u);
    __syncthreads();
    if (warp == 0) {
      float u[kGdnRows];
      solve(std::false_type{}, pending, sh.kk, sh.pv, sh.pbeta, u);
#pragma unroll
      for (int t4x = 0; t4x < kGdnRows; t4x += 4) {
        const float4 g4x = *reinterpret_cast<const float4 *>(&sh.after[t4x]);
        const float g[4] = {g4x.x, g4x.y, g4x.z, g4x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (uint32_t(t4x + i) < pending) sh.u[t4x + i][lane] = g[i] * u[t4x + i];
      }
    }
  }
  if (warp == 1 && lane >= rows && lane < kGdnRows) sh.beta[lane] = 0.0f;
  if (warp == 1 && lane < rows) {  // the rows' gates
    float bb, aa;
    if (a.gate_weight) {
      bb = sh.gate[0][lane][0], aa = sh.gate[0][lane][1];
#pragma unroll
      for (int g = 1; g < kDotGroups; ++g) bb += sh.gate[g][lane][0], aa += sh.gate[g][lane][1];
      bb = round_bf16(bb), aa = round_bf16(aa);
    } else {
      bb = bf16_bits_to_float(static_cast<const uint16_t *>(a.b)[size_t(lane) * a.ab_stride + h]);
      aa = bf16_bits_to_float(static_cast<const uint16_t *>(a.a)[size_t(lane) * a.ab_stride + h]);
    }
    const float be = round_bf16(sigmoid_f(bb));
    const float x = round_bf16(__fadd_rn(aa, dt_bias));
    const float sp = round_bf16(fmaxf(x, 0.0f) + log2f(1.0f + exp2f(-1.44269504089f * fabsf(x))) * 0.69314718056f);
    const float de = expf(a_scale * sp);
    sh.beta[lane] = be;
    sh.decay[lane] = de;
    if (vs == 0) {
      static_cast<uint16_t *>(a.step.beta)[size_t(lane) * VH + h] = float_to_bf16_bits(be);
      a.step.decay[size_t(lane) * VH + h] = de;
    }
  }
  cluster_arrive();
  cluster_wait();  // (2) every row's q and k are in every CTA of the head; this CTA's pending solution and gates
  if (pending) {
    const float d = sh.pending_decay;
#pragma unroll
    for (int i = 0; i < 16; ++i) S[i] *= d;
    for (uint32_t t0 = 0; t0 < pending; t0 += 2) {
#pragma unroll
      for (uint32_t t = t0; t < t0 + 2; ++t) {
        if (t >= pending) break;
        const float u0 = sh.u[t][srow], u1 = sh.u[t][srow + 8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 k2 = *reinterpret_cast<const float2 *>(&sh.pk[t][scol + 16 * (c >> 1) + 8 * (c & 1)]);
          const int at = 8 * (c >> 1) + 2 * (c & 1);
          S[at] = fmaf(u0, k2.x, S[at]), S[at + 1] = fmaf(u0, k2.y, S[at + 1]);
          S[at + 4] = fmaf(u1, k2.x, S[at + 4]), S[at + 5] = fmaf(u1, k2.y, S[at + 5]);
        }
      }
    }
  }
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int second = 0; second < 2; ++second)
#pragma unroll
      for (int pair = 0; pair < 2; ++pair)
        *reinterpret_cast<float2 *>(a.state_out + sbase + size_t(8 * second) * kD + 16 * b + 8 * pair) =
            make_float2(S[8 * b + 4 * second + 2 * pair], S[8 * b + 4 * second + 2 * pair + 1]);
  // (4) the rows' inner products (this CTA: rows vs, vs + 4, ..), and S k_t, S q_t on the tensor cores: the state as three bf16
  // terms, k and q are bf16 as they stand, so every product is exact; the small terms first, a quarter of the columns a warp,
  // the quarters added in fp32.
  {
    const uint32_t t = 4 * (warp >> 1) + vs;
    auto key = [&](int j) { return block_row(0, j); };
    if (t < rows) inner_products(key, block_row(warp & 1, t), (warp & 1) ? sh.kq : sh.kk, t);
  }
  cluster_arrive();  // (3)
  {
    float acc[4][4] = {};
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      uint32_t hi[4], mid[4], lo[4];  // A: (row, pair), (row + 8, pair), (row, second pair), (row + 8, second pair)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int at = 8 * b + 4 * (i & 1) + 2 * (i >> 1);
        split3(S[at], S[at + 1], hi[i], mid[i], lo[i]);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {  // k rows 0-7, 8-15, q rows 0-7, 8-15
        if ((n & 1) && rows <= 8) continue;
        const uint16_t *x = &sh.x[n >> 1][8 * (n & 1) + g4][scol + 16 * b];
        const uint32_t b0 = *reinterpret_cast<const uint32_t *>(x), b1 = *reinterpret_cast<const uint32_t *>(x + 8);
        mma_bf16(acc[n], lo[0], lo[1], lo[2], lo[3], b0, b1);
        mma_bf16(acc[n], mid[0], mid[1], mid[2], mid[3], b0, b1);
        mma_bf16(acc[n], hi[0], hi[1], hi[2], hi[3], b0, b1);
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (!(n & 1) || rows > 8) sh.part[quarter][8 * n + 2 * t4 + (i & 1)][srow + 8 * (i >> 1)] = acc[n][i];
  }
  if (qk_writer)
    for (uint32_t i = tid; i < rows * kD / 2; i += kGdnThreads)
      store_pair(static_cast<uint16_t *>(a.step.k) + size_t(i / (kD / 2)) * KW + kh * kD + 2 * (i % (kD / 2)),
                 *reinterpret_cast<const uint32_t *>(&sh.x[0][i / (kD / 2)][2 * (i % (kD / 2))]));
  // what the gate of the row this warp will finish reads
  const uint32_t out_row = 4 * vs + warp;
  const bool finishes = warp < kGdnRows / kGdnSplit && out_row < rows;
  float z[4], nw[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    z[g] = finishes ? bf16_bits_to_float(qkvz[size_t(out_row) * a.qkvz_stride + C + h * kD + 32 * g + lane]) : 0.0f;
    nw[g] = finishes ? a.norm_w[32 * g + lane] : 0.0f;
  }
  cluster_wait();   // (3) the inner products
  __syncthreads();  // this CTA's products (written since it arrived)
  {
    // Coefficients of the system ([j][t], into the pending rows' matrix) and of the outputs ([t][j]): G(t, j) along row t's path, j
    // on it; D_t (S k_t) and the outputs' first terms. Rows past the block are zeros.
    const bool there = ct < rows, on = there && cj <= ct && (sh.path[ct] >> cj & 1u);
    const uint32_t path = there ? sh.path[ct] : 0u;
    const float g = decays(sh.decay, path & ~((2u << cj) - 1u)), d = decays(sh.decay, path);
    sh.pkk[cj][ct] = on && cj < ct ? g * sh.kk[ct][cj] : 0.0f;
    sh.kq[ct][cj] = on ? g * sh.kq[ct][cj] : 0.0f;
    float2 right = make_float2(0.0f, 0.0f), first = right;
    if (there) {
      const float2 sk = four(sh.part, ct), sq = four(sh.part, kGdnRows + ct);
      right = make_float2(d * sk.x, d * sk.y);
      first = make_float2(d * sq.x, d * sq.y);
    }
    *reinterpret_cast<float2 *>(&sh.u[ct][cv]) = right;
    *reinterpret_cast<float2 *>(&sh.o[ct][cv]) = first;
  }
  __syncthreads();
  if (warp == 0) {
    float u[kGdnRows];
    solve(std::bool_constant<kTree>{}, rows, sh.pkk, sh.v, sh.beta, u);
#pragma unroll
    for (int t = 0; t < kGdnRows; ++t) sh.u[t][lane] = u[t];
  }
  __syncthreads();
  for (uint32_t t = warp; t < rows; t += kGdnThreads / 32) {
    const uint32_t path = sh.path[t];
    float o = sh.o[t][lane];
#pragma unroll
    for (int j4 = 0; j4 < kGdnRows; j4 += 4) {  // the rows on its path (the others may hold no numbers)
      if (uint32_t(j4) > t) break;
      const float4 c4 = *reinterpret_cast<const float4 *>(&sh.kq[t][j4]);
      if (path >> j4 & 1u) o = fmaf(c4.x, sh.u[j4][lane], o);
      if (path >> (j4 + 1) & 1u) o = fmaf(c4.y, sh.u[j4 + 1][lane], o);
      if (path >> (j4 + 2) & 1u) o = fmaf(c4.z, sh.u[j4 + 2][lane], o);
      if (path >> (j4 + 3) & 1u) o = fmaf(c4.w, sh.u[j4 + 3][lane], o);
    }
    head_ctas.map_shared_rank(&sh.out[t % 4][vd0 + lane], int(t / 4))[0] = round_bf16(o);
  }
  head_ctas.sync();  // (4) this CTA's rows, all 128 value dimensions
  // (5) gated RMSNorm: a warp per row, dimensions 32 g + lane, the four partial sums added in order.
  if (!finishes) return;
  const uint32_t out_head = a.tiled ? (h % per_key) * KH + h / per_key : h;
  float val[4], total = 0.0f;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    val[g] = sh.out[warp][32 * g + lane];
    total += warp_sum(val[g] * val[g]);
  }
  const float inv = rsqrtf(total / float(kD) + 1e-6f);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t d = 32 * g + lane;
    const float normalized = round_bf16((val[g] * inv) * nw[g]);
    static_cast<uint16_t *>(a.hidden)[size_t(out_row) * a.hidden_stride + out_head * kD + d] =
        float_to_bf16_bits((normalized * z[g]) / (1.0f + exp2f(-1.44269504089f * z[g])));
  }
}

// Whether the call needs the tree kernel: tree rows, or a pending path that is not known here to be the tape's first rows.
static bool needs_tree_kernel(const SbGdnArgs &a) {
  return a.tree || a.pending_path_dev || (a.pending_path & (a.pending_path + 1u)) != 0;
}

// The limit of sb_gdn_verify_static (its scratch once held this many heads; the kernel needs none now).
constexpr uint32_t kStaticMaxValueHeads = 64;  // the 27B shape has 48

}  // namespace sb

using namespace sb;

namespace sb {
// The argument checks both entry points share; `who` names the caller in the message.
static int gdn_validate(const SbGdnArgs *a, const char *who) {
  SB_REQUIRE(a, "%s: null arguments", who);
  SB_REQUIRE(a->qkvz && ((a->b && a->a) || a->gate_weight) && a->conv_w && a->a_scale && a->dt_bias && a->norm_w && a->conv_state_in &&
                 a->conv_state_out && a->state_in && a->state_out && a->hidden,
             "%s: null pointer", who);
  SB_REQUIRE(a->rows <= kGdnRows && a->pending_rows <= kGdnRows, "%s: rows %u or pending rows %u above %d", who, a->rows, a->pending_rows, kGdnRows);
  SB_REQUIRE(a->key_heads >= 1 && a->value_heads >= 1 && a->value_heads % a->key_heads == 0 && a->value_heads <= 256,
             "%s: %u value heads over %u key heads", who, a->value_heads, a->key_heads);
  const uint32_t C = (2 * a->key_heads + a->value_heads) * kD;
  SB_REQUIRE(a->qkvz_stride >= C + a->value_heads * kD && (a->gate_weight || a->ab_stride >= a->value_heads) && a->hidden_stride >= a->value_heads * kD,
             "%s: a stride is below its row", who);
  SB_REQUIRE(a->rows == 0 || (a->step.inputs && a->step.k && a->step.v && a->step.beta && a->step.decay), "%s: null tape of this step", who);
  SB_REQUIRE((a->pending_rows == 0 && !a->pending_rows_dev && !a->pending_path && !a->pending_path_dev) ||
                 (a->pending.inputs && a->pending.k && a->pending.v && a->pending.beta && a->pending.decay),
             "%s: null pending tape", who);
  SB_REQUIRE(a->pending_path < (1u << kGdnRows), "%s: pending path 0x%x names rows above %d", who, a->pending_path, kGdnRows);
  SB_REQUIRE(a->state_in != a->state_out && a->conv_state_in != a->conv_state_out, "%s: the committed cell is a second cell", who);
  SB_REQUIRE(!a->gate_weight || (a->gate_input && a->gate_k && a->gate_k % 8 == 0 && a->gate_input_stride >= a->gate_k && a->gate_input_stride % 8 == 0 &&
                                 (reinterpret_cast<uintptr_t>(a->gate_weight) & 15) == 0 && (reinterpret_cast<uintptr_t>(a->gate_input) & 15) == 0),
             "%s: fused gate projection needs a 16-byte aligned input and weight, k a multiple of 8 and stride >= k", who);
  SB_REQUIRE((a->flags & ~uint32_t(SB_GDN_STATE_SETTLED)) == 0, "%s: unknown flags 0x%x", who, a->flags);
  SB_REQUIRE(a->lanes <= 64 && size_t(std::max(1u, a->lanes)) * a->value_heads <= kGdnLaunchHeads, "%s: %u lanes of %u value heads exceed a launch", who,
             a->lanes, a->value_heads);
  return SB_OK;
}
}  // namespace sb

static int gdn_launch(void *stream, const SbGdnArgs *a, bool pdl, int device) {
  const GdnParams p{*a};
  const bool tree = needs_tree_kernel(*a), several = a->lanes > 1;
  const auto kernel = several ? (tree ? gdn_kernel<true, 4> : gdn_kernel<false, 4>) : (tree ? gdn_kernel<true, 2> : gdn_kernel<false, 2>);
  static std::atomic<uint64_t> allowed[4];
  const int st = allow_smem(reinterpret_cast<const void *>(kernel), sizeof(GdnShared), allowed[2 * several + tree], device);
  if (st != SB_OK) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kGdnSplit, a->value_heads, std::max(1u, a->lanes));
  cfg.blockDim = dim3(kGdnThreads);
  cfg.dynamicSmemBytes = sizeof(GdnShared);
  cfg.stream = as_stream(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  SB_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  return SB_OK;
}

extern "C" int sb_gdn_verify(void *stream, const SbGdnArgs *a) {
  SB_NEED_DEVICE();
  const int valid = gdn_validate(a, "sb_gdn_verify");
  return valid != SB_OK ? valid : gdn_launch(stream, a, ctx().pdl, ctx().device);
}

extern "C" int sb_gdn_verify_static(void *stream, const SbGdnArgs *a) {
  SB_REQUIRE(a, "sb_gdn_verify_static: null arguments");
  SB_REQUIRE(a->value_heads <= kStaticMaxValueHeads, "sb_gdn_verify_static: %u value heads exceed %u; use sb_gdn_verify", a->value_heads,
             kStaticMaxValueHeads);
  SB_REQUIRE(a->lanes <= 1, "sb_gdn_verify_static: one lane a call");
  const int valid = gdn_validate(a, "sb_gdn_verify_static");
  return valid != SB_OK ? valid : gdn_launch(stream, a, false, -1);  // (no context)
}
