// Selection of one row's next token by a cluster of eight CTAs that holds the row's logits in shared memory
// (launch_selection in sb_ops.cu says which rows come here).
//
// What bounds it: a sampled row needs its weights summed in a fixed order (256 ids at a time in id order, the shards in
// order), so a measurement of the distribution is 256 + shards dependent additions however many threads there are, and the
// ends of the distribution (top-k, top-p) need several. With one block a row, reading the row from the L2 once per bit of a
// 32-bit search key, 128 rows of 151,936 logits at top-k 50 / top-p 0.95 took 5.71 ms. Here
//   - a row is read from memory once; each CTA keeps the keys of an eighth of it (whole shards) in shared memory, and every
//     pass after that runs from there;
//   - a search is two passes instead of 32: a histogram of the logits' distance below the row's largest (counts and
//     approximate masses) names the bin the end lies in, and the bin's tokens, gathered by CTA 0, name the key;
//   - masses that decide anything are still the sums in the fixed order: a key found from approximate masses is taken only if
//     the exact masses at it and above it say so (the exact mass only grows with the set, every weight being >= 0, so the
//     key with that property is the one a bit-by-bit search ends at). Where the nucleus's end lies among so many tokens that the
//     list does not hold them, or that one weighs less than the roundings, the tokens around it are sorted and searched by exact
//     masses. Otherwise, or when a row's largest logit or the temperature makes a weight no number, the search walks the bits.
// The 128 rows above take 268 us, 16 such rows 69 us (5.67 ms), 16 rows without filters 34 us (158), 128 rows at top-p 0.95 and
// temperature 1 without top-k 1.2 ms (3.1). What is left is the passes themselves (a few instructions for each of 152 k tokens a
// pass, 37 rows resident at a time) and the ordered sums.
#pragma once

namespace sb {

constexpr uint32_t kSentinel = 0xFFFFFFFFu;
constexpr uint32_t kShard = 256;
constexpr uint32_t kDrawCandidates = 16, kNoDraw = 0xff;  // a row's draft candidates; "no child drawn" (runtime/metal/abi/ExecutionGeometry.h:63)

constexpr int kSelectCtas = 8, kSelectThreads = 512, kSelectWarps = kSelectThreads / 32;
constexpr uint32_t kSelectShards = 1024, kSelectVocab = kSelectShards * kShard;  // (the filters' limit, and the arrays' below)
constexpr uint32_t kSelectBins = 1024, kSelectList = 1024;
constexpr uint32_t kSparse = 4096;  // tokens up to which a set's masses are summed a warp a shard (151,936 ids: some seven of a shard's 256)
constexpr float kSelectBinScale = 32.0f;  // bins of 1/32 in units of the temperature: the histogram reaches e^-32 of the largest weight
static_assert(kSelectList <= kSelectBins, "the list's weights stand in the histogram");

__device__ __forceinline__ bool selectable(float x) { return !(isnan(x) || x == -INFINITY); }

// ---- the end of a row's distribution: min-p, then top-k, then the top-p nucleus (sampling.metal:604-668) ----
// A token stays iff its key (order-preserving bits of its logit, -0 as +0) is above cut.key, or equal to it with an id
// up to cut.id.
struct RowCut {
  uint32_t key, id;
};
__device__ __forceinline__ uint32_t logit_key(float x) {
  if (x == 0.0f) x = 0.0f;
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_logit(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}
// A token as the cluster keeps it: its key, or 0 if it cannot be selected (every selectable logit's key is above -inf's).
__device__ __forceinline__ uint32_t token_key(float x) { return selectable(x) ? logit_key(x) : 0u; }
__device__ __forceinline__ bool cut_keeps(const RowCut c, uint32_t k, uint32_t v) { return k != 0 && (k > c.key || (k == c.key && v <= c.id)); }
// Greedy order: value descending, id ascending; the sentinel loses.
__device__ __forceinline__ bool better_token(float v1, uint32_t i1, float v2, uint32_t i2) {
  if (i2 == kSentinel) return true;
  if (i1 == kSentinel) return false;
  return v1 > v2 || (v1 == v2 && i1 < i2);
}

// What a cluster's CTAs exchange, the same layout in each (peers write into it).
struct SelectShared {
  float best_v[kSelectWarps];
  uint32_t best_i[kSelectWarps], warp_count[2][kSelectWarps];
  float cta_best_v[kSelectCtas];
  uint32_t cta_best_i[kSelectCtas], cta_count[2][kSelectCtas];
  union {
    struct {
      uint32_t bin_count[kSelectBins];  // this CTA's histogram; CTA 0 then keeps the weights of the list in bin_mass
      float bin_mass[kSelectBins];
      uint32_t row_count[kSelectBins];  // CTA 0: the row's
      float row_mass[kSelectBins];
    };
    float stage[kSelectWarps][kShard];  // between searches: the weights a warp adds up, in id order
  };
  uint32_t list_n, list_key[kSelectList];  // CTA 0: keys of the bin the end lies in
  uint32_t found_bin, found_reach, found_ok, found_key, found_id, outer_bin, list_first, list_last, list_at;
  float total_ge, total_gt, before_mass, outer_mass;
  uint32_t total_n[2], before_count;
  float cand_weight[kDrawCandidates];
  uint32_t pick, pick_state, pick_shard;
  float pick_target;
};
// Dynamic shared memory of a CTA: SelectShared, two arrays of all the row's shards (the sums of the tokens at or above a key and
// of those above it; at the end the sums with and without the drafted child), two of prefixes, the CTA's keys.
__host__ __device__ inline uint32_t select_shards_per_cta(uint32_t vocab) { return ((vocab + kShard - 1) / kShard + kSelectCtas - 1) / kSelectCtas; }
__host__ __device__ inline size_t select_smem_bytes(uint32_t vocab) {
  const size_t shards = size_t(select_shards_per_cta(vocab)) * kSelectCtas;
  return (sizeof(SelectShared) + 15) / 16 * 16 + shards * 4 * 4 + size_t(select_shards_per_cta(vocab)) * kShard * 4;
}

struct SelectRow {
  SelectShared &sh;
  float *mass_ge, *mass_gt;  // [shards]
  uint32_t *slice;           // this CTA's keys, in id order
  const float *l;            // the row in global memory
  uint32_t vocab, shards, per_cta, rank, s0, mine, v0, n_mine;  // mine: shards here; n_mine: tokens here, from v0
  float mx, inv_t, temperature;

  __device__ __forceinline__ float weight_of(float x) const { return expf(__fmul_rn(__fsub_rn(x, mx), inv_t)); }
  __device__ __forceinline__ float key_weight(uint32_t k) const { return weight_of(key_logit(k)); }
  static __device__ __forceinline__ void sync() { cooperative_groups::this_cluster().sync(); }
  template <class T> static __device__ __forceinline__ T *peer(T *p, uint32_t rank) { return cooperative_groups::this_cluster().map_shared_rank(p, rank); }

  // Token i of the slice stands in its shard's 256 places turned by the shard's number: threads that read the same place of
  // different shards, or 32 tokens in a row, meet 32 banks.
  static __device__ __forceinline__ uint32_t slot(uint32_t i) { return (i & ~(kShard - 1)) | ((i + i / kShard) & (kShard - 1)); }

  // f(key, id within the slice) over this CTA's tokens, all threads at it, eight loads in flight; eight tokens a thread whose
  // largest key `worth` turns down in every lane of the warp are passed over. Every lane of a warp makes the same calls (past
  // the end with key 0, which nothing keeps).
  template <class W, class F> __device__ __forceinline__ void each_token(W worth, F f) {
    for (uint32_t i0 = threadIdx.x & ~31u; i0 < n_mine; i0 += 8 * kSelectThreads) {
      uint32_t k[8], most = 0;
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) {
        const uint32_t i = i0 + (threadIdx.x & 31u) + j * kSelectThreads;
        k[j] = i < n_mine ? slice[slot(i)] : 0u;
        most = max(most, k[j]);
      }
      if (!__any_sync(0xffffffffu, worth(most))) continue;
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) f(k[j], i0 + (threadIdx.x & 31u) + j * kSelectThreads);
    }
  }
  // This CTA's shards: the sum in id order of the weights of the kept tokens with at least `key`, and of those above it, into
  // mass_ge and mass_gt of every CTA. Where the set is small a warp takes a shard at a time: all its lanes look for the tokens,
  // lay their weights out one after the other (the others would add nothing), and two lanes add them up, each a sum. Where it
  // is not, a thread takes a shard: a warp's instructions then carry 32 sums.
  __device__ __forceinline__ void sum_shards(RowCut cut, uint32_t key, bool sparse, uint32_t &c_ge, uint32_t &c_gt) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!sparse) {
      if (tid < mine) {
        float a = 0.0f, b = 0.0f;
        for (uint32_t i0 = 0; i0 < kShard; i0 += 8) {
          uint32_t k[8];
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t i = tid * kShard + i0 + j;
            k[j] = i < n_mine ? slice[slot(i)] : 0u;
          }
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) {
            const bool ge = k[j] >= key && cut_keeps(cut, k[j], v0 + tid * kShard + i0 + j), gt = ge && k[j] > key;
            const float w = ge ? key_weight(k[j]) : 0.0f;
            a = __fadd_rn(a, w), b = __fadd_rn(b, gt ? w : 0.0f);
            c_ge += ge, c_gt += gt;
          }
        }
#pragma unroll 1
        for (uint32_t r = 0; r < kSelectCtas; ++r) peer(mass_ge, r)[s0 + tid] = a, peer(mass_gt, r)[s0 + tid] = b;
      }
      return;
    }
    float *stage = sh.stage[warp];
    for (uint32_t s = warp; s < mine; s += kSelectWarps) {
      uint32_t k[8], most = 0;
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) {
        const uint32_t i = s * kShard + 32 * j + lane;
        k[j] = i < n_mine ? slice[slot(i)] : 0u;
        most = max(most, k[j]);
      }
      float ge = 0.0f, gt = 0.0f;
      if (__any_sync(0xffffffffu, most >= key && most >= cut.key)) {
        uint32_t n = 0;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
          const bool keep = k[j] >= key && cut_keeps(cut, k[j], v0 + s * kShard + 32 * j + lane);
          const uint32_t there = __ballot_sync(0xffffffffu, keep);
          if (keep) {
            const float w = key_weight(k[j]);
            stage[n + __popc(there & ((1u << lane) - 1u))] = k[j] == key ? -w : w;  // (the sign marks it; a weight is never negative)
            ++c_ge, c_gt += k[j] > key;
          }
          n += uint32_t(__popc(there));
        }
        __syncwarp();
        if (lane < 2)
          for (uint32_t i = 0; i < n; ++i) {
            const float w = stage[i];
            ge = __fadd_rn(ge, lane == 0 ? fabsf(w) : fmaxf(w, 0.0f));  // (sparse sets have no weight that is no number)
          }
        gt = __shfl_sync(0xffffffffu, ge, 1), ge = __shfl_sync(0xffffffffu, ge, 0);
      }
      if (lane < kSelectCtas) peer(mass_ge, lane)[s0 + s] = ge, peer(mass_gt, lane)[s0 + s] = gt;
      __syncwarp();
    }
  }
  // The sum of the shards in order. (The arrays end with zeros to a whole eight; eight empty shards add nothing.)
  __device__ __forceinline__ float shards_total(const float *m) const {
    float t = 0.0f;
    float4 a = *reinterpret_cast<const float4 *>(m), b = *reinterpret_cast<const float4 *>(m + 4);
    for (uint32_t s = 0; s < shards; s += 8) {
      const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      if (s + 8 < shards) a = *reinterpret_cast<const float4 *>(m + s + 8), b = *reinterpret_cast<const float4 *>(m + s + 12);
#pragma unroll
      for (int j = 0; j < 8; ++j) t = __fadd_rn(t, v[j]);
    }
    return t;
  }
  // Counts and (with want_mass) exact masses of the kept tokens whose key is at least `key`, and of those above it; the same
  // values in every thread of the cluster.
  __device__ void measure(RowCut cut, uint32_t key, bool want_mass, bool sparse, uint32_t &n_ge, uint32_t &n_gt, float &m_ge, float &m_gt) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t c_ge = 0, c_gt = 0;
    if (want_mass)
      sum_shards(cut, key, sparse, c_ge, c_gt);
    else
      each_token([&](uint32_t most) { return most >= key && most >= cut.key; },
                 [&](uint32_t k, uint32_t i) {
                   const bool keep = k >= key && cut_keeps(cut, k, v0 + i);
                   c_ge += keep, c_gt += keep && k > key;
                 });
    exchange_counts(c_ge, c_gt);
    if (tid == 0) {
      uint32_t a = 0, b = 0;
      for (int r = 0; r < kSelectCtas; ++r) a += sh.cta_count[0][r], b += sh.cta_count[1][r];
      sh.total_n[0] = a, sh.total_n[1] = b;
    }
    if (want_mass && lane == 0 && (warp == 1 || warp == 2)) {  // both sums at once
      const float t = shards_total(warp == 1 ? mass_ge : mass_gt);
      if (warp == 1) sh.total_ge = t;
      else sh.total_gt = t;
    }
    sync();  // (the totals, and every CTA has read what the next exchange writes)
    n_ge = sh.total_n[0], n_gt = sh.total_n[1], m_ge = sh.total_ge, m_gt = sh.total_gt;
    __syncthreads();
  }
  // Every CTA's two counts into every CTA's cta_count.
  __device__ void exchange_counts(uint32_t a, uint32_t b) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o), b += __shfl_xor_sync(0xffffffffu, b, o);
    if (lane == 0) sh.warp_count[0][warp] = a, sh.warp_count[1][warp] = b;
    __syncthreads();
    if (tid < kSelectCtas) {
      uint32_t ta = 0, tb = 0;
      for (int w = 0; w < kSelectWarps; ++w) ta += sh.warp_count[0][w], tb += sh.warp_count[1][w];
      peer(&sh.cta_count[0][0], tid)[rank] = ta, peer(&sh.cta_count[1][0], tid)[rank] = tb;
    }
    sync();
  }

  __device__ __forceinline__ uint32_t bin_of(float x) const {
    const float d = __fmul_rn(__fmul_rn(__fsub_rn(mx, x), inv_t), kSelectBinScale);
    return d < float(kSelectBins - 1) ? uint32_t(d) : kSelectBins - 1;
  }
  // The largest key whose kept tokens at or above it number at least `count` (by_mass = false), or weigh more than `nucleus`
  // as far as sums in no particular order say (by_mass); reach: the tokens down to its bin's end. False: the bin does not fit the
  // list, or no such key was seen. Leaves what nucleus_among_many starts from.
  __device__ bool locate(RowCut cut, bool by_mass, uint32_t count, float nucleus, uint32_t &key, uint32_t &reach) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    for (uint32_t i = tid; i < kSelectBins; i += kSelectThreads) sh.bin_count[i] = 0, sh.bin_mass[i] = 0.0f, sh.row_count[i] = 0, sh.row_mass[i] = 0.0f;
    if (tid == 0) sh.list_n = 0;
    sync();
    each_token([&](uint32_t most) { return most >= cut.key; }, [&](uint32_t k, uint32_t i) {
      const bool keep = cut_keeps(cut, k, v0 + i);
      if (!__any_sync(0xffffffffu, keep)) return;
      const uint32_t bin = keep ? bin_of(key_logit(k)) : kSentinel;
      if (!by_mass) {
        if (keep) atomicAdd(&sh.bin_count[bin], 1u);
        return;
      }
      float w = keep ? key_weight(k) : 0.0f;
      if (__all_sync(0xffffffffu, bin == __shfl_sync(0xffffffffu, bin, 0))) {  // (a flat row: one addition a warp instead of 32 on one address)
#pragma unroll
        for (int o = 16; o; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (lane == 0) atomicAdd(&sh.bin_count[bin], 32u), atomicAdd(&sh.bin_mass[bin], w);
      } else if (keep) {
        atomicAdd(&sh.bin_count[bin], 1u), atomicAdd(&sh.bin_mass[bin], w);
      }
    });
    __syncthreads();
    for (uint32_t i = tid; i < kSelectBins; i += kSelectThreads)
      if (sh.bin_count[i]) {
        atomicAdd(peer(&sh.row_count[i], 0), sh.bin_count[i]);
        if (by_mass) atomicAdd(peer(&sh.row_mass[i], 0), sh.bin_mass[i]);
      }
    sync();
    if (rank == 0 && tid < 32) {  // the bin the end lies in: 32 bins a lane, scanned over the lanes
      uint32_t c = 0;
      float m = 0.0f;
      for (uint32_t i = 0; i < kSelectBins / 32; ++i) c += sh.row_count[lane * (kSelectBins / 32) + i], m += sh.row_mass[lane * (kSelectBins / 32) + i];
      uint32_t cs = c;
      float ms = m;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t oc = __shfl_up_sync(0xffffffffu, cs, o);
        const float om = __shfl_up_sync(0xffffffffu, ms, o);
        if (lane >= uint32_t(o)) cs += oc, ms += om;
      }
      const uint32_t there = __ballot_sync(0xffffffffu, by_mass ? ms > nucleus : cs >= count);
      uint32_t bin = kSentinel, n_before = 0;
      float m_before = 0.0f;
      if (there && lane == uint32_t(__ffs(int(there))) - 1u) {
        n_before = cs - c, m_before = ms - m;
        for (bin = lane * (kSelectBins / 32); bin < lane * (kSelectBins / 32) + kSelectBins / 32 - 1; ++bin) {
          if (by_mass ? m_before + sh.row_mass[bin] > nucleus : n_before + sh.row_count[bin] >= count) break;
          n_before += sh.row_count[bin], m_before += sh.row_mass[bin];
        }
        sh.before_count = n_before, sh.before_mass = m_before, sh.outer_mass = bin ? m_before - sh.row_mass[bin - 1] : 0.0f;
        for (uint32_t r = 0; r < kSelectCtas; ++r)
          *peer(&sh.found_bin, r) = sh.row_count[bin] <= kSelectList ? bin : kSentinel, *peer(&sh.found_reach, r) = n_before + sh.row_count[bin], *peer(&sh.outer_bin, r) = bin;
      }
      if (!there && lane < kSelectCtas) *peer(&sh.found_bin, lane) = kSentinel, *peer(&sh.outer_bin, lane) = kSentinel;
    }
    sync();
    const uint32_t want = sh.found_bin;
    if (want == kSentinel) {
      sync();  // (every CTA has read it)
      return false;
    }
    // (a bin never rises with the key, so eight tokens whose largest lies below the bin hold none of it)
    each_token([&](uint32_t most) { return most != 0 && most >= cut.key && bin_of(key_logit(most)) <= want; }, [&](uint32_t k, uint32_t i) {
      if (!cut_keeps(cut, k, v0 + i) || bin_of(key_logit(k)) != want) return;
      const uint32_t place = atomicAdd(peer(&sh.list_n, 0), 1u);
      peer(sh.list_key, 0)[place] = k;
      if (by_mass) peer(sh.bin_mass, 0)[place] = key_weight(k);  // (CTA 0's own histogram is in the row's by now)
    });
    sync();
    if (rank == 0) {
      // A token of the list is the end's if fewer than `count` tokens (no more than the nucleus's mass) lie above it and
      // enough lie at or above it; the largest key of those that qualify.
      if (tid == 0) sh.found_ok = 0, sh.found_key = 0;
      __syncthreads();
      const uint32_t n = sh.list_n;
      for (uint32_t i = tid; i < n; i += kSelectThreads) {
        const uint32_t k = sh.list_key[i];
        uint32_t ge = sh.before_count;
        float w = sh.before_mass;
        for (uint32_t j = 0; j < n; ++j) {
          const uint32_t kj = sh.list_key[j];
          if (kj < k) continue;
          ++ge;
          if (by_mass) w += sh.bin_mass[j];
        }
        if (by_mass ? w > nucleus : ge >= count) sh.found_ok = 1, atomicMax(&sh.found_key, k);
      }
      __syncthreads();
      if (tid < kSelectCtas && tid > 0) *peer(&sh.found_ok, tid) = sh.found_ok, *peer(&sh.found_key, tid) = sh.found_key;
    }
    sync();
    key = sh.found_key, reach = sh.found_reach;
    const bool ok = sh.found_ok != 0;
    sync();
    return ok;
  }
  // The id of the n-th (1-based) kept token whose key equals `key`, in id order.
  __device__ uint32_t nth_tie(RowCut cut, uint32_t key, uint32_t n) {
    const uint32_t tid = threadIdx.x;
    uint32_t c = 0;
    each_token([&](uint32_t most) { return most >= key; }, [&](uint32_t k, uint32_t i) { c += k == key && cut_keeps(cut, k, v0 + i); });
    if (tid == 0) sh.found_id = kSentinel;
    exchange_counts(c, 0);
    uint32_t before = 0;
    for (uint32_t r = 0; r < rank; ++r) before += sh.cta_count[0][r];
    const uint32_t here = sh.cta_count[0][rank];
    if (before < n && n <= before + here && tid < 32) {  // this CTA holds it: a warp walks its tokens
      uint32_t left = n - before;
      for (uint32_t i0 = 0; i0 < n_mine; i0 += 32) {
        const uint32_t i = i0 + tid;
        const uint32_t k = i < n_mine ? slice[slot(i)] : 0u;
        const uint32_t hits = __ballot_sync(0xffffffffu, k == key && cut_keeps(cut, k, v0 + i));
        if (uint32_t(__popc(hits)) < left) {
          left -= uint32_t(__popc(hits));
          continue;
        }
        uint32_t m = hits;
        for (uint32_t t = 1; t < left; ++t) m &= m - 1;
        if (tid < kSelectCtas) *peer(&sh.found_id, tid) = v0 + i0 + uint32_t(__ffs(int(m))) - 1u;
        break;
      }
    }
    sync();
    const uint32_t id = sh.found_id;
    sync();
    return id;
  }
  // The nucleus's end where it lies among so many tokens that a bin does not fit the list, or that one weighs less than the sums'
  // roundings (151,936 logits of standard deviation 1.8 at temperature 1 and top-p 0.95: 1060 tokens a bin, a token 8e-7 of the
  // mass): the four bins around it in 1024 parts, the tokens of as many parts around the crossing as the list holds, sorted, and
  // among them the key with an exact mass above the nucleus and an exact mass above it that is not, by steps that double from the
  // crossing, then halve. 128 such rows take 3.3 ms when every one walks the bits. Not ok: the end is not among them.
  // A call of its own: the rows that do not come here keep their registers.
  struct NucleusEnd {
    uint32_t key, n_ge, n_gt;
    float m_ge, m_gt;
    bool ok;
  };
  static __device__ __noinline__ NucleusEnd nucleus_among_many(SelectRow row, RowCut cut, float nucleus) {
    SelectShared &sh = row.sh;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const float from = float(sh.outer_bin ? sh.outer_bin - 1 : 0u);
    // Parts never rise with the key, as bins do not: every rounding on the way keeps the order. kSentinel: outside the four bins.
    auto part_of = [&](uint32_t k) {
      const float d = __fmul_rn(__fsub_rn(__fmul_rn(__fmul_rn(__fsub_rn(row.mx, key_logit(k)), row.inv_t), kSelectBinScale), from), float(kSelectBins / 4));
      return d >= 0.0f && d < float(kSelectBins) ? uint32_t(d) : kSentinel;
    };
    sync();  // (every CTA has read what locate left)
    for (uint32_t i = tid; i < kSelectBins; i += kSelectThreads) sh.bin_count[i] = 0, sh.bin_mass[i] = 0.0f, sh.row_count[i] = 0, sh.row_mass[i] = 0.0f;
    if (tid == 0) sh.list_n = 0;
    sync();
    row.each_token([&](uint32_t most) { return most != 0 && most >= cut.key; }, [&](uint32_t k, uint32_t i) {
      if (!cut_keeps(cut, k, row.v0 + i)) return;
      const uint32_t part = part_of(k);
      if (part != kSentinel) atomicAdd(&sh.bin_count[part], 1u), atomicAdd(&sh.bin_mass[part], row.key_weight(k));
    });
    __syncthreads();
    for (uint32_t i = tid; i < kSelectBins; i += kSelectThreads)
      if (sh.bin_count[i]) atomicAdd(peer(&sh.row_count[i], 0), sh.bin_count[i]), atomicAdd(peer(&sh.row_mass[i], 0), sh.bin_mass[i]);
    sync();
    if (row.rank == 0 && tid == 0) {
      uint32_t first = 0, n, at;
      float m = sh.outer_mass;
      for (; first < kSelectBins - 1 && !(m + sh.row_mass[first] > nucleus); ++first) m += sh.row_mass[first];
      uint32_t last = first;
      n = sh.row_count[first], at = n / 2;
      for (bool more = n <= kSelectList; more;) {  // a part more either side, while the list holds them
        more = false;
        if (first > 0 && n + sh.row_count[first - 1] <= kSelectList) --first, n += sh.row_count[first], at += sh.row_count[first], more = true;
        if (last < kSelectBins - 1 && n + sh.row_count[last + 1] <= kSelectList) ++last, n += sh.row_count[last], more = true;
      }
      const bool ok = n > 0 && n <= kSelectList;
      for (uint32_t r = 0; r < kSelectCtas; ++r)
        *peer(&sh.found_ok, r) = ok, *peer(&sh.list_first, r) = first, *peer(&sh.list_last, r) = last, *peer(&sh.list_at, r) = at, *peer(&sh.found_reach, r) = n;
    }
    sync();
    NucleusEnd e{};
    if (!sh.found_ok) {
      sync();
      return e;
    }
    const uint32_t first = sh.list_first, last = sh.list_last, n = sh.found_reach;
    row.each_token([&](uint32_t most) { return most != 0 && most >= cut.key; }, [&](uint32_t k, uint32_t i) {
      if (!cut_keeps(cut, k, row.v0 + i)) return;
      const uint32_t part = part_of(k);
      if (part != kSentinel && part >= first && part <= last) peer(sh.list_key, 0)[atomicAdd(peer(&sh.list_n, 0), 1u)] = k;
    });
    sync();
    if (row.rank == 0) {  // sorted, the largest key first
      static_assert(kSelectList <= 2 * kSelectThreads, "two of the list's tokens a thread");
      uint32_t mine[2] = {0, 0}, place[2] = {0, 0};
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t i = tid + h * kSelectThreads;
        if (i >= n) continue;
        mine[h] = sh.list_key[i];
        for (uint32_t j = 0; j < n; ++j) place[h] += sh.list_key[j] > mine[h] || (sh.list_key[j] == mine[h] && j < i);
      }
      __syncthreads();
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h)
        if (tid + h * kSelectThreads < n) sh.list_key[place[h]] = mine[h];
    }
    sync();
    uint32_t above = 0, below = n, step = 1;  // the end's place is >= above and < below
    for (uint32_t at = min(sh.list_at, n - 1); above < below; step *= 2) {
      e.key = peer(sh.list_key, 0)[at];
      row.measure(cut, e.key, true, false, e.n_ge, e.n_gt, e.m_ge, e.m_gt);
      e.ok = e.m_ge > nucleus && !(e.m_gt > nucleus);
      if (e.ok) return e;
      const bool deeper = !(e.m_ge > nucleus);
      if (deeper) above = at + 1;
      else below = at;
      if (above >= below) break;
      if (deeper) at = below < n ? above + (below - above) / 2 : min(at + step, below - 1);
      else at = above > 0 ? above + (below - above) / 2 : at - min(step, at);
    }
    return e;
  }
  // `report`: the caller is told the end, so its id has to be the last kept token's even where every tie stays.
  __device__ RowCut distribution_end(float min_p, uint32_t top_k, float top_p, uint32_t selectable_count, bool report) {
    RowCut cut{0u, kSentinel};
    uint32_t kept_count = selectable_count, n_ge, n_gt, reach = kSentinel;
    float kept_mass = 0.0f, m_ge, m_gt;
    bool mass_known = false;
    const bool nucleus_on = top_p > 0.0f && top_p < 1.0f;
    // (a weight that is no number compares false wherever it stands: such rows walk the bits)
    const bool plain = mx < INFINITY && inv_t < INFINITY;
    if (min_p > 0.0f) {
      const float t = fminf(__fadd_rn(mx, __fmul_rn(temperature, logf(min_p))), mx);
      measure(cut, logit_key(t), false, false, n_ge, n_gt, m_ge, m_gt);
      if (n_ge < kept_count) cut = RowCut{logit_key(t), kSentinel}, kept_count = n_ge;
    }
    if (top_k > 0 && top_k < kept_count) {
      uint32_t key = 0;  // the largest key with at least top_k kept tokens at or above it
      if (!plain || !locate(cut, false, top_k, 0.0f, key, reach)) {
        key = 0, reach = kSentinel;
        for (int bit = 31; bit >= 0; --bit) {
          const uint32_t cand = key | (1u << bit);
          measure(cut, cand, false, false, n_ge, n_gt, m_ge, m_gt);
          if (n_ge >= top_k) key = cand;
        }
      }
      measure(cut, key, nucleus_on, reach <= kSparse, n_ge, n_gt, m_ge, m_gt);
      const uint32_t need = top_k - n_gt;
      cut = RowCut{key, need == n_ge - n_gt && !report ? kSentinel : nth_tie(cut, key, need)};
      kept_count = top_k;
      if (nucleus_on) kept_mass = __fadd_rn(m_gt, __fmul_rn(float(need), weight_of(key_logit(key)))), mass_known = true;
    }
    if (nucleus_on) {
      if (!mass_known) measure(cut, 0u, true, false, n_ge, n_gt, kept_mass, m_gt);
      const float nucleus = __fmul_rn(top_p, kept_mass);
      uint32_t key = 0;  // the largest key whose kept tokens at or above it weigh more than the nucleus
      bool found = plain && locate(cut, true, 0u, nucleus, key, reach);
      if (found) {
        measure(cut, key, true, reach <= kSparse, n_ge, n_gt, m_ge, m_gt);
        found = m_ge > nucleus && !(m_gt > nucleus);
      }
      if (!found && plain && sh.outer_bin != kSentinel) {
        const NucleusEnd e = nucleus_among_many(*this, cut, nucleus);
        found = e.ok, key = e.key, n_ge = e.n_ge, n_gt = e.n_gt, m_ge = e.m_ge, m_gt = e.m_gt;
      }
      if (!found) {
        key = 0;
        for (int bit = 31; bit >= 0; --bit) {
          const uint32_t cand = key | (1u << bit);
          measure(cut, cand, true, false, n_ge, n_gt, m_ge, m_gt);
          if (m_ge > nucleus) key = cand, found = true;
        }
        measure(cut, key, true, false, n_ge, n_gt, m_ge, m_gt);
        found = found || m_ge > nucleus;
      }
      if (found) {  // rounding may leave the nucleus unreached: then everything kept so far stays
        const uint32_t ties = n_ge - n_gt;
        if (ties > 0) {
          const float q = fminf(fmaxf(__fdiv_rn(__fsub_rn(nucleus, m_gt), weight_of(key_logit(key))), 0.0f), float(ties - 1));
          const uint32_t keep = 1u + uint32_t(q);
          cut = RowCut{key, keep == ties && !report ? (key == cut.key ? cut.id : kSentinel) : nth_tie(cut, key, keep)};
        }
      }
    }
    return cut;
  }

  // The weight of token v under the cut, from global memory (the row's logits are not changed by a selection).
  __device__ __forceinline__ float kept_weight(RowCut cut, uint32_t v) const {
    const uint32_t k = token_key(l[v]);
    return cut_keeps(cut, k, v) ? key_weight(k) : 0.0f;
  }
  // CTA 0, all threads: shard s's weights into this CTA's slice (no longer needed as it was).
  __device__ void stage_shard(RowCut cut, uint32_t s) {
    float *w = reinterpret_cast<float *>(slice);
    for (uint32_t i = threadIdx.x; i < kShard; i += kSelectThreads) w[i] = s * kShard + i < vocab ? kept_weight(cut, s * kShard + i) : 0.0f;
    __syncthreads();
  }
};

// Tokens v0 .. v0 + n - 1 from src on, by a CTA of kSelectThreads: the best of them and how many can be selected, a warp's in all
// its lanes; keep(logit, place) sees every one of them.
template <int FLIGHT, class K> __device__ __forceinline__ void best_of(const float *src, uint32_t v0, uint32_t n, float &bv, uint32_t &bi, uint32_t &n_sel, K keep) {
  const uint32_t tid = threadIdx.x;
  bv = -INFINITY, bi = kSentinel, n_sel = 0;
  auto take = [&](float x, uint32_t i) {
    keep(x, i);
    if (!selectable(x)) return;
    ++n_sel;
    if (bi == kSentinel || x > bv) bv = x, bi = v0 + i;  // (ids come in rising order)
  };
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {  // rows that start on 16 bytes: FLIGHT 16-byte loads in flight
    const uint32_t n4 = n / 4;
    for (uint32_t i0 = tid; i0 < n4; i0 += FLIGHT * kSelectThreads) {
      float4 x[FLIGHT];
#pragma unroll
      for (int j = 0; j < FLIGHT; ++j) {
        const uint32_t i = i0 + j * kSelectThreads;
        if (i < n4) x[j] = reinterpret_cast<const float4 *>(src)[i];
      }
#pragma unroll
      for (int j = 0; j < FLIGHT; ++j) {
        const uint32_t i = i0 + j * kSelectThreads;
        if (i < n4) take(x[j].x, 4 * i), take(x[j].y, 4 * i + 1), take(x[j].z, 4 * i + 2), take(x[j].w, 4 * i + 3);
      }
    }
    if (tid < (n & 3u)) take(src[4 * n4 + tid], 4 * n4 + tid);
  } else {
    for (uint32_t i0 = tid; i0 < n; i0 += 8 * kSelectThreads) {
      float x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t i = i0 + j * kSelectThreads;
        if (i < n) x[j] = src[i];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (i0 + j * kSelectThreads < n) take(x[j], i0 + j * kSelectThreads);
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (!better_token(bv, bi, ov, oi)) bv = ov, bi = oi;
    n_sel += __shfl_xor_sync(0xffffffffu, n_sel, o);
  }
}

// A greedy row's selection by one CTA of the cluster (the others have rows of their own).
__device__ __forceinline__ void greedy_row(const SbSampleArgs &a, uint32_t r) {
  __shared__ float best_v[kSelectWarps];
  __shared__ uint32_t best_i[kSelectWarps];
  float bv;
  uint32_t bi, n_sel;
  best_of<8>(a.logits + size_t(r) * a.logit_stride, 0, a.vocab, bv, bi, n_sel, [](float, uint32_t) {});
  if ((threadIdx.x & 31) == 0) best_v[threadIdx.x >> 5] = bv, best_i[threadIdx.x >> 5] = bi;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < kSelectWarps; ++w)
    if (!better_token(bv, bi, best_v[w], best_i[w])) bv = best_v[w], bi = best_i[w];
  a.selected[r] = bi;
}

// One row's selection by the eight CTAs of a cluster; a is the row's lane's view. Thread 0 of CTA 0 writes it.
__device__ __forceinline__ void select_row(const SbSampleArgs &a, uint32_t r, uint8_t *smem) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x % kSelectCtas;
  SelectShared &sh = *reinterpret_cast<SelectShared *>(smem);
  const uint32_t per_cta = select_shards_per_cta(a.vocab), padded = per_cta * kSelectCtas;
  float *arrays = reinterpret_cast<float *>(smem + (sizeof(SelectShared) + 15) / 16 * 16);
  SelectRow row{sh, arrays, arrays + padded, reinterpret_cast<uint32_t *>(arrays + 4 * padded), a.logits + size_t(r) * a.logit_stride, a.vocab, (a.vocab + kShard - 1) / kShard,
                per_cta, rank, rank * per_cta, 0, 0, 0, 0.0f, 0.0f, a.temperature};
  row.mine = row.s0 < row.shards ? min(per_cta, row.shards - row.s0) : 0;
  row.v0 = row.s0 * kShard;
  row.n_mine = row.v0 < a.vocab ? min(a.vocab - row.v0, per_cta * kShard) : 0;
  const bool sampled = a.temperature != 0.0f && a.uniforms;
  if (sampled && tid < 8 && row.shards + tid < padded) row.mass_ge[row.shards + tid] = row.mass_gt[row.shards + tid] = 0.0f;
  // The row's eighth: greedy choice and, for a sampled row, its copy in shared memory.
  float bv;
  uint32_t bi, n_sel;
  best_of<4>(row.l + row.v0, row.v0, row.n_mine, bv, bi, n_sel, [&](float x, uint32_t i) {
    if (sampled) row.slice[SelectRow::slot(i)] = token_key(x);
  });
  if (lane == 0) sh.best_v[warp] = bv, sh.best_i[warp] = bi, sh.warp_count[0][warp] = n_sel;
  __syncthreads();
  if (tid < kSelectCtas) {
    bv = sh.best_v[0], bi = sh.best_i[0], n_sel = sh.warp_count[0][0];
    for (int w = 1; w < kSelectWarps; ++w) {
      if (!better_token(bv, bi, sh.best_v[w], sh.best_i[w])) bv = sh.best_v[w], bi = sh.best_i[w];
      n_sel += sh.warp_count[0][w];
    }
    // (every CTA of the cluster has started: select_kernel's first cluster barrier)
    SelectRow::peer(sh.cta_best_v, tid)[rank] = bv, SelectRow::peer(sh.cta_best_i, tid)[rank] = bi, SelectRow::peer(&sh.cta_count[0][0], tid)[rank] = n_sel;
  }
  SelectRow::sync();
  bv = sh.cta_best_v[0], bi = sh.cta_best_i[0], n_sel = sh.cta_count[0][0];
#pragma unroll
  for (int c = 1; c < kSelectCtas; ++c) {
    if (!better_token(bv, bi, sh.cta_best_v[c], sh.cta_best_i[c])) bv = sh.cta_best_v[c], bi = sh.cta_best_i[c];
    n_sel += sh.cta_count[0][c];
  }
  if (!sampled || bi == kSentinel) {
    if (rank == 0 && tid == 0) a.selected[r] = bi;
    return;
  }
  row.mx = bv, row.inv_t = __fdiv_rn(1.0f, a.temperature);
  SelectRow::sync();  // (every CTA has read the counts: the next exchange may write them)
  const bool has_child = !a.candidate_ids && r + 1 < a.rows;  // (with the draft's candidates given, the children are the rows' draws)
  const uint32_t child = has_child ? a.input_tokens[r + 1] : kSentinel;
  RowCut cut{0u, kSentinel};
  if (a.min_p > 0.0f || (a.top_k > 0 && a.top_k < a.vocab) || (a.top_p > 0.0f && a.top_p < 1.0f))
    cut = row.distribution_end(a.min_p, a.top_k, a.top_p, n_sel, a.cut_out != nullptr);
  if (a.cut_out && rank == 0 && tid == 0) a.cut_out[2 * r] = cut.key, a.cut_out[2 * r + 1] = cut.id;
  // The weights take the keys' place, all threads at it; then a thread a shard sums its 256 in id order, with and without the
  // drafted child, into CTA 0.
  float *shard = row.mass_ge, *shard2 = row.mass_gt, *weights = reinterpret_cast<float *>(row.slice);
  row.each_token([](uint32_t) { return true; }, [&](uint32_t k, uint32_t i) {
    if (i < row.n_mine) weights[SelectRow::slot(i)] = cut_keeps(cut, k, row.v0 + i) ? row.key_weight(k) : 0.0f;
  });
  __syncthreads();
  if (tid < row.mine) {
    float sum = 0.0f, sum2 = 0.0f;
    const uint32_t first = tid * kShard, n = min(kShard, row.n_mine - first), without = child - (row.v0 + first);
    for (uint32_t i0 = 0; i0 < n; i0 += 8) {
      float w[8];
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) w[j] = i0 + j < n ? weights[SelectRow::slot(first + i0 + j)] : 0.0f;
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) sum = __fadd_rn(sum, w[j]), sum2 = __fadd_rn(sum2, i0 + j == without ? 0.0f : w[j]);
    }
    SelectRow::peer(shard, 0)[row.s0 + tid] = sum, SelectRow::peer(shard2, 0)[row.s0 + tid] = sum2;
  }
  SelectRow::sync();
  if (rank != 0) return;  // nothing of this CTA's is read from here on
  const uint32_t shards = row.shards;
  if (a.candidate_ids && tid < kDrawCandidates) {
    const uint32_t id = a.candidate_ids[kDrawCandidates * r + tid];
    sh.cand_weight[tid] = id < a.vocab ? row.kept_weight(cut, id) : 0.0f;
  }
  // The shards in order, every prefix kept (prefix[s]: the sum up to and with shard s); with and without the child side by side.
  float *prefix = arrays + 2 * padded, *prefix2 = arrays + 3 * padded;
  if (lane == 0 && warp < 2) {
    const float *m = warp ? shard2 : shard;
    float *out = warp ? prefix2 : prefix, z = 0.0f;
    float4 x = *reinterpret_cast<const float4 *>(m), y = *reinterpret_cast<const float4 *>(m + 4);
    for (uint32_t s = 0; s < shards; s += 8) {  // (the arrays are whole eights long, zeros after the last shard)
      float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
      if (s + 8 < shards) x = *reinterpret_cast<const float4 *>(m + s + 8), y = *reinterpret_cast<const float4 *>(m + s + 12);
#pragma unroll
      for (int j = 0; j < 8; ++j) z = __fadd_rn(z, v[j]), v[j] = z;
      *reinterpret_cast<float4 *>(out + s) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4 *>(out + s + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  __syncthreads();
  const float z = prefix[shards - 1];
  if (a.candidate_ids) {
    // Recursive rejection sampling without replacement over the children the draft drew for this row
    // (runtime/metal/kernels/decode/sampling.metal:693-885): child i of the row's kDrawCandidates candidates, of
    // probability p_i under the target and q_i under the draft, is taken when u_i q_i < p_i; after a rejection the
    // target becomes its residual max(p - q, 0), renormalised, and the draft loses the rejected child, renormalised; a
    // row that takes none draws from the last residual, its candidates first, then the tokens outside them. A row
    // without drawn children draws from its whole distribution.
    const uint32_t *ids = a.candidate_ids + kDrawCandidates * r;
    if (tid == 0) {
      sh.pick_state = 0;  // 1: selected; 2 | excluding << 2: by the shards below
      const float *cq = a.candidate_q + kDrawCandidates * r;
      const uint8_t *draws = a.draws + 4 * r;
      float target = __fmul_rn(a.uniforms[r], z);
      bool excluding = false, done = false;
      if (draws[0] != kNoDraw && z > 0.0f) {
        float pc[kDrawCandidates], qc[kDrawCandidates];
        for (uint32_t i = 0; i < kDrawCandidates; ++i) {
          const uint32_t id = ids[i];
          const float w = sh.cand_weight[i];
          if (id < a.vocab) shard[id / kShard] = fmaxf(__fsub_rn(shard[id / kShard], w), 0.0f);  // the shards without the candidates
          pc[i] = __fdiv_rn(w, z);
          qc[i] = cq[i];
        }
        float outside_weight = 0.0f;
#pragma unroll 8
        for (uint32_t s = 0; s < shards; ++s) outside_weight = __fadd_rn(outside_weight, shard[s]);
        float outside = __fdiv_rn(outside_weight, z);
        for (uint32_t c = 0; c < 4 && !done; ++c) {
          const uint32_t dc = draws[c];
          if (dc >= kDrawCandidates) break;
          if (__fmul_rn(a.uniforms[16 + 4 * r + c], qc[dc]) < pc[dc]) {
            a.selected[r] = ids[dc];
            done = true;
            break;
          }
          float residual = outside;
          for (uint32_t i = 0; i < kDrawCandidates; ++i) residual = __fadd_rn(residual, fmaxf(__fsub_rn(pc[i], qc[i]), 0.0f));
          if (!(residual > 0.0f)) break;
          for (uint32_t i = 0; i < kDrawCandidates; ++i) pc[i] = __fdiv_rn(fmaxf(__fsub_rn(pc[i], qc[i]), 0.0f), residual);
          outside = __fdiv_rn(outside, residual);
          qc[dc] = 0.0f;
          float rest = 0.0f;
          for (uint32_t i = 0; i < kDrawCandidates; ++i) rest = __fadd_rn(rest, qc[i]);
          for (uint32_t i = 0; rest > 0.0f && i < kDrawCandidates; ++i) qc[i] = __fdiv_rn(qc[i], rest);
        }
        if (!done) {
          float inside = 0.0f;
          for (uint32_t i = 0; i < kDrawCandidates; ++i) inside = __fadd_rn(inside, pc[i]);
          const float point = __fmul_rn(a.uniforms[r], __fadd_rn(inside, outside));
          float cumulative = 0.0f;
          uint32_t last = kDrawCandidates;
          for (uint32_t i = 0; i < kDrawCandidates && !(point < cumulative); ++i)
            if (pc[i] > 0.0f) last = i, cumulative = __fadd_rn(cumulative, pc[i]);
          if (last < kDrawCandidates && (point < cumulative || !(outside > 0.0f))) {
            a.selected[r] = ids[last];
            done = true;
          } else {
            excluding = true;
            target = __fmul_rn(__fdiv_rn(__fsub_rn(point, inside), outside), outside_weight);
          }
        }
      }
      if (done) {
        sh.pick_state = 1;
      } else {
        // By the target's own weights (outside the candidates after rejections): the shard the point falls in (the last one
        // with weight if rounding leaves it unreached), then its ids in order.
        float run = 0.0f, shard_target = 0.0f;
        uint32_t at = kSentinel;
        for (uint32_t s = 0; s < shards; ++s) {
          if (!(shard[s] > 0.0f)) continue;
          at = s, shard_target = __fsub_rn(target, run);
          run = __fadd_rn(run, shard[s]);
          if (run > target) break;
        }
        sh.pick_state = 2u | (excluding ? 4u : 0u), sh.pick_shard = at, sh.pick_target = shard_target;
      }
    }
    __syncthreads();
    if (sh.pick_state == 1) return;
    const bool excluding = (sh.pick_state & 4u) != 0;
    const uint32_t at = sh.pick_shard;
    if (at != kSentinel) {
      row.stage_shard(cut, at);
      if (excluding && tid < kDrawCandidates && ids[tid] / kShard == at) reinterpret_cast<float *>(row.slice)[ids[tid] % kShard] = 0.0f;
      __syncthreads();
    }
    if (tid != 0) return;
    uint32_t pick = kSentinel;
    if (at != kSentinel) {
      float loc = 0.0f;
      const float4 *w4 = reinterpret_cast<const float4 *>(row.slice);  // (zeros past the vocabulary)
      bool over = false;
      for (uint32_t i = 0; i < kShard / 4 && !over; i += 2) {
        const float4 x = w4[i], y = w4[i + 1];
        const float w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
          if (over || !(w[j] > 0.0f)) {
            if (!over) loc = __fadd_rn(loc, w[j]);
            continue;
          }
          pick = at * kShard + 4 * i + j;  // the last id weighed so far: where the walk ends if rounding leaves the target unreached
          loc = __fadd_rn(loc, w[j]);
          over = loc > sh.pick_target;
        }
      }
    }
    a.selected[r] = pick;
    return;
  }
  bool drop = false;
  if (has_child && child < a.vocab) {
    const float u = a.uniforms[16 + 4 * r];
    if (__fmul_rn(u, z) < row.kept_weight(cut, child)) {
      if (tid == 0) a.selected[r] = child;
      return;
    }
    drop = true;
  }
  const float *sums = drop ? prefix2 : prefix;
  const float target = __fmul_rn(a.uniforms[r], sums[shards - 1]);
  // The first shard whose prefix passes the target, then its ids in order; should rounding leave the target unreached inside
  // the shard, the next one that passes it.
  if (tid == 0) sh.pick = kSentinel;
  for (uint32_t from = 0; from < shards;) {
    __syncthreads();  // (the pick, and the last walk is over)
    if (sh.pick != kSentinel) break;
    if (tid == 0) sh.pick_shard = kSentinel;
    __syncthreads();
    for (uint32_t s = from + tid; s < shards; s += kSelectThreads)
      if (sums[s] > target) {
        atomicMin(&sh.pick_shard, s);
        break;
      }
    __syncthreads();
    const uint32_t s = sh.pick_shard;
    if (s == kSentinel) break;
    row.stage_shard(cut, s);
    if (tid == 0) {
      const float run = s ? sums[s - 1] : 0.0f;
      float loc = 0.0f;
      const float4 *w4 = reinterpret_cast<const float4 *>(row.slice);  // (zeros past the vocabulary; none there can pass the target first)
      const uint32_t n = min(kShard, a.vocab - s * kShard), without = drop && child / kShard == s ? child % kShard : kSentinel;
      uint32_t pick = kSentinel;
      for (uint32_t i = 0; i < kShard / 4 && pick == kSentinel; i += 2) {
        const float4 x = w4[i], y = w4[i + 1];
        const float w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
          loc = __fadd_rn(loc, 4 * i + j == without ? 0.0f : w[j]);
          if (pick == kSentinel && 4 * i + j < n && __fadd_rn(run, loc) > target) pick = s * kShard + 4 * i + j;
        }
      }
      sh.pick = pick;
    }
    from = s + 1;
  }
  __syncthreads();
  if (sh.pick == kSentinel) {  // unreached: the last token with weight
    if (tid == 0) sh.pick_shard = 0;
    __syncthreads();
    uint32_t last = 0;  // id + 1
    for (uint32_t v = tid; v < a.vocab; v += kSelectThreads)
      if (row.kept_weight(cut, v) > 0.0f && !(drop && v == child)) last = v + 1;
    if (last) atomicMax(&sh.pick_shard, last);
    __syncthreads();
    if (tid == 0 && sh.pick_shard) sh.pick = sh.pick_shard - 1;
  }
  if (tid == 0) a.selected[r] = sh.pick;
}

}  // namespace sb
