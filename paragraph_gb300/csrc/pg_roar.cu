// pg_roar.cu -- ParaGraph's CPU RoarGraph path (MatchSup rounds, FusionNN) and the final fusion
// (FusionFinal) as GPU kernels (sm_103a).
//
// Reference: tests/test_t2iend.cu, the CPU code its driver runs beside the GPU build --
// compare :31-80, RNGPrune :99-177, MatchSup :365-488, FusionNN :490-537, FusionFinal :539-613.
// Results equal the reference's one-thread run id for id:
//   * distances follow compare()'s AVX-512 FP32 order: 16 FMA lanes over 16-wide chunks, folded
//     8+8, an 8-wide FMA step, folded 4+4, a 4-wide step, then ((s0+s1)+(s2+s3)) -- four lanes of
//     a warp hold four accumulators each and compute one distance;
//   * candidate lists are sorted by (distance, id), SimpleNeighbor's order (:82-91), with one warp
//     bitonic sort of 64-bit keys (ordered distance << 32 | id);
//   * RNGPrune's scan keeps a candidate that no kept entry occludes; here each newly kept entry is
//     tested against every undecided candidate at once, which makes the same decisions.  Its second
//     "double check" scan (:142-165) is not run: every candidate it revisits was kept already or is
//     occluded by the same kept entry as before;
//   * MatchSup's reverse appends keep, per base, the first 128 - M_nn sources in ascending query
//     order (the reference's one-thread order), through the same count/scan/scatter/sort CSR as
//     the link rounds; a merged list too short to be pruned is written in ascending id order (the
//     reference writes std::unordered_set order, which no consumer depends on).
// Most lists are a few ids long and a few fill the capacity, so every stage runs twice: one warp
// per node for lists of up to kShort ids, which also queues the longer ones, and one block per node
// over that queue.  With one warp per node for all lists and candidates tested four at a time, the
// stages waited for the longest lists (about a millisecond each): 200k x 200, six MatchSup rounds
// 33.7 -> 7.8 ms, FusionNN 8.2 -> 1.5, FusionFinal 7.0 -> 1.1.
#include "pg_device.cuh"
#include "pg_kernels.h"

namespace pg {

namespace {

constexpr uint32_t kRoarCap = 256;  // candidates per node
constexpr uint32_t kRoarRes = 128;  // kept entries per node
constexpr uint32_t kShort = 32;     // lists of the one-warp kernels
constexpr uint32_t kWarps = 8;      // warps per block: nodes (one-warp kernels) or one node's team

// Lists of one node.  CAP: candidates.
template <uint32_t CAP>
struct Lists {
  uint32_t cand[CAP];
  uint32_t sid[CAP];
  float sdist[CAP];
  uint32_t res[CAP];
  uint32_t fin[2 * CAP];
  uint16_t und[CAP];  // undecided candidates (places in sid), ascending
  uint8_t occ[CAP];
  uint32_t kept[CAP / 32];  // bits: places that were kept
  uint32_t num[4];
};

// The warps that work on one node: a warp on its own, or the block.
template <int W>
struct Team {
  static_assert(W == 1 || W == kWarps, "a warp or the block");
  static constexpr uint32_t kGroups = 8 * W;  // four lanes per distance
  static constexpr uint32_t kCap = W == 1 ? kShort : kRoarCap;
  static __device__ __forceinline__ uint32_t warp() { return W == 1 ? 0 : threadIdx.x >> 5; }
  static __device__ __forceinline__ bool lead() { return W == 1 || threadIdx.x < 32; }
  static __device__ __forceinline__ void sync() {
    if constexpr (W == 1)
      __syncwarp();
    else
      __syncthreads();
  }
};

__device__ __forceinline__ const float* row_of(const float* base, uint32_t d, uint32_t id) {
  return base + static_cast<uint64_t>(id) * d;
}

__device__ __forceinline__ float4 ld4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ void fma4(float4& s, const float4 x, const float4 y) {
  s.x = fmaf(x.x, y.x, s.x);
  s.y = fmaf(x.y, y.y, s.y);
  s.z = fmaf(x.z, y.z, s.z);
  s.w = fmaf(x.w, y.w, s.w);
}
__device__ __forceinline__ float4 fold4(const float4 s, int o) {  // lane l: its values + lane l+o's
  return make_float4(__shfl_down_sync(kFull, s.x, o, 4) + s.x,
                     __shfl_down_sync(kFull, s.y, o, 4) + s.y,
                     __shfl_down_sync(kFull, s.z, o, 4) + s.z,
                     __shfl_down_sync(kFull, s.w, o, 4) + s.w);
}

// compare() (tests/test_t2iend.cu:31-80), the negated inner product in its exact FP32 order -- 16
// accumulators over 16-wide chunks, folded 8+8, an 8-wide FMA step, folded 4+4, a 4-wide step,
// then ((s0 + s1) + (s2 + s3)) -- of a against each of R rows, by a group of four lanes: lane l
// holds accumulators 4l .. 4l+3 and reads 16 bytes per chunk.  Every lane of the warp calls it (the
// shuffles are warp-wide); the distances are valid in lane 0 of each group.
template <int R>
__device__ __forceinline__ void dist4(const float* __restrict__ a, const float* const (&b)[R],
                                      uint32_t d, float (&out)[R]) {
  const uint32_t l = threadIdx.x & 3u;
  float4 s[R];
#pragma unroll
  for (int r = 0; r < R; r++) s[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  uint32_t i = 0;
#pragma unroll 4
  for (; i + 16 <= d; i += 16) {
    const float4 x = ld4(a + i + 4 * l);
#pragma unroll
    for (int r = 0; r < R; r++) fma4(s[r], x, ld4(b[r] + i + 4 * l));
  }
#pragma unroll
  for (int r = 0; r < R; r++) s[r] = fold4(s[r], 2);
  if (d - i >= 8) {
    if (l < 2) {
      const float4 x = ld4(a + i + 4 * l);
#pragma unroll
      for (int r = 0; r < R; r++) fma4(s[r], x, ld4(b[r] + i + 4 * l));
    }
    i += 8;
  }
#pragma unroll
  for (int r = 0; r < R; r++) s[r] = fold4(s[r], 1);
  if (d - i >= 4 && l == 0) {
    const float4 x = ld4(a + i);
#pragma unroll
    for (int r = 0; r < R; r++) fma4(s[r], x, ld4(b[r] + i));
  }
#pragma unroll
  for (int r = 0; r < R; r++) out[r] = -((s[r].x + s[r].y) + (s[r].z + s[r].w));
}

// use(i, distance of row a to candidate i) once for each i < len, in lane 0 of the group that
// computed it; id_of(i) is the candidate.  Two rows per group and pass while they last.
template <int W, class IdOf, class Use>
__device__ __forceinline__ void team_dists(const float* base, uint32_t d, const float* a,
                                           uint32_t len, IdOf id_of, Use use) {
  constexpr uint32_t G = Team<W>::kGroups;
  const uint32_t w0 = Team<W>::warp() * 8u, g = w0 + (lane_id() >> 2);
  const bool first = (threadIdx.x & 3u) == 0;
  for (uint32_t i0 = 0; i0 + w0 < len; i0 += 2 * G) {  // uniform in the warp
    const uint32_t i = i0 + g, j = i + G;
    const float* ri = row_of(base, d, id_of(min(i, len - 1)));
    if (i0 + G + w0 < len) {
      const float* const rows[2] = {ri, row_of(base, d, id_of(min(j, len - 1)))};
      float dist[2];
      dist4<2>(a, rows, d, dist);
      if (first) {
        if (i < len) use(i, dist[0]);
        if (j < len) use(j, dist[1]);
      }
    } else {
      const float* const rows[1] = {ri};
      float dist[1];
      dist4<1>(a, rows, d, dist);
      if (first && i < len) use(i, dist[0]);
    }
  }
}

// Sorts cand[0 .. len) with the distances sdist[0 .. len) by (distance, id) into sid/sdist, one
// warp; returns their number.  With `unique`, repeats of an id are dropped (they carry the same
// distance, so they sit next to each other after the sort).
template <int E>
__device__ uint32_t sort_by_dist(const uint32_t* cand, uint32_t len, uint32_t* sid, float* sdist,
                                 bool unique) {
  const uint32_t lane = lane_id();
  uint64_t key[E];
  uint32_t val[E];
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    key[s] = ~0ull;
    val[s] = 0;
    if (i < len) {
      const float dist = sdist[i];
      key[s] = (static_cast<uint64_t>(order_key(dist)) << 32) | cand[i];
      val[s] = __float_as_uint(dist);
    }
  }
  __syncwarp();
  warp_sort_kv<E>(key, val);
  uint32_t cnt = 0;
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint64_t up = __shfl_up_sync(kFull, key[s], 1);
    const uint64_t wrap = s > 0 ? __shfl_sync(kFull, key[s > 0 ? s - 1 : 0], 31) : ~0ull;
    const uint64_t prev = lane == 0 ? wrap : up;
    const bool keep = key[s] != ~0ull && !(unique && prev == key[s]);
    const unsigned m = __ballot_sync(kFull, keep);
    if (keep) {
      const uint32_t pos = cnt + __popc(m & ((1u << lane) - 1u));
      sid[pos] = static_cast<uint32_t>(key[s]);
      sdist[pos] = __uint_as_float(val[s]);
    }
    cnt += __popc(m);
  }
  __syncwarp();
  return cnt;
}

template <uint32_t CAP>
__device__ __forceinline__ uint32_t sort_by_dist_any(Lists<CAP>* sm, uint32_t len, bool unique) {
  if (CAP <= 32 || len <= 32) return sort_by_dist<1>(sm->cand, len, sm->sid, sm->sdist, unique);
  if (len <= 64) return sort_by_dist<2>(sm->cand, len, sm->sid, sm->sdist, unique);
  if (len <= 128) return sort_by_dist<4>(sm->cand, len, sm->sid, sm->sdist, unique);
  return sort_by_dist<8>(sm->cand, len, sm->sid, sm->sdist, unique);
}

// Replaces every repeat of an earlier id in cand[0..len) by tomb (first occurrences stay): a sort
// of (id << 32 | position) keys puts the repeats of an id right after its first occurrence.
template <int E>
__device__ void dedupe_first(uint32_t* cand, uint32_t len) {
  const uint32_t lane = lane_id();
  uint64_t key[E];
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    key[s] = i < len ? ((static_cast<uint64_t>(cand[i]) << 32) | i) : ~0ull;
  }
  warp_sort_u64<E>(key);
  __syncwarp();
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint64_t up = __shfl_up_sync(kFull, key[s], 1);
    const uint64_t wrap = s > 0 ? __shfl_sync(kFull, key[s > 0 ? s - 1 : 0], 31) : ~0ull;
    const uint64_t prev = lane == 0 ? wrap : up;
    if (key[s] != ~0ull && prev != ~0ull && (prev >> 32) == (key[s] >> 32))
      cand[static_cast<uint32_t>(key[s])] = kTomb;
  }
  __syncwarp();
}

// The ids of cand[0..len) ascending without repeats, in place; returns their number.  One warp.
template <int E>
__device__ uint32_t sort_unique(uint32_t* cand, uint32_t len) {
  const uint32_t lane = lane_id();
  uint32_t v[E];
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    v[s] = i < len ? cand[i] : kTomb;
  }
  warp_sort_u32<E>(v);
  __syncwarp();
  uint32_t cnt = 0;
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t up = __shfl_up_sync(kFull, v[s], 1);
    const uint32_t wrap = s > 0 ? __shfl_sync(kFull, v[s > 0 ? s - 1 : 0], 31) : kTomb;
    const bool keep = v[s] != kTomb && (lane == 0 ? wrap : up) != v[s];
    const unsigned m = __ballot_sync(kFull, keep);
    if (keep) cand[cnt + __popc(m & ((1u << lane) - 1u))] = v[s];
    cnt += __popc(m);
  }
  __syncwarp();
  return cnt;
}

__device__ __forceinline__ bool warp_contains(const uint32_t* a, uint32_t k, uint32_t x) {
  bool in = false;
  for (uint32_t t = lane_id(); t < k; t += 32) in |= a[t] == x;
  return __ballot_sync(kFull, in) != 0;
}

// Appends to cand[len ..) the ids that lanes hold with `keep`, in lane order; the new length.
__device__ __forceinline__ uint32_t append(uint32_t* cand, uint32_t len, uint32_t x, bool keep) {
  const unsigned m = __ballot_sync(kFull, keep);
  if (keep) cand[len + __popc(m & ((1u << lane_id()) - 1u))] = x;
  return len + __popc(m);
}

// RNGPrune (tests/test_t2iend.cu:99-177) of cand[0 .. len) around node `target`: distances, sort,
// scan; kept ids in res, returns their number (M <= kRoarRes).  cand is visible to the team.
// Not strict: ids must be unique after the sort.
template <int W>
__device__ uint32_t team_prune(const float* base, uint32_t d, uint64_t n, uint32_t M,
                               Lists<Team<W>::kCap>* sm, uint32_t len, uint32_t target,
                               bool unique, bool strict) {
  using T = Team<W>;
  const uint32_t lane = lane_id();
  const unsigned lt_mask = (1u << lane) - 1u;
  team_dists<W>(base, d, row_of(base, d, target), len, [&](uint32_t i) { return sm->cand[i]; },
                [&](uint32_t i, float dist) { sm->sdist[i] = dist; });
  T::sync();
  if (T::lead()) {
    const uint32_t c = sort_by_dist_any(sm, len, unique);
    // the first entry that is not the node is kept; the node itself never is (:133-137)
    uint32_t start = 0, u = 0;
    while (start < c && sm->sid[start] == target) start++;
    for (uint32_t i0 = start + 1; i0 < c; i0 += 32) {
      const uint32_t i = i0 + lane;
      const bool keep = i < c && sm->sid[i] != target;
      const unsigned m = __ballot_sync(kFull, keep);
      if (keep) sm->und[u + __popc(m & lt_mask)] = static_cast<uint16_t>(i);
      u += __popc(m);
    }
    if (lane < T::kCap / 32) sm->kept[lane] = lane == start / 32 ? 1u << (start & 31u) : 0u;
    if (lane == 0) {
      if (start < c) sm->res[0] = sm->sid[start];
      sm->num[0] = u;
      sm->num[1] = start < c;
      sm->num[2] = c;
    }
  }
  T::sync();
  if (!sm->num[1]) {
    T::sync();  // the next node's lists come after everyone has read this one's
    return 0;
  }
  uint32_t k = 1, u = sm->num[0];
  const uint32_t c = sm->num[2];
  while (k < M && u > 0) {
    // the last kept entry against every undecided candidate
    const uint32_t r = sm->res[k - 1];
    team_dists<W>(base, d, row_of(base, d, r), u,
                  [&](uint32_t e) { return sm->sid[sm->und[e]]; },
                  [&](uint32_t e, float dist) {
                    const uint32_t p = sm->und[e];
                    sm->occ[e] = sm->sid[p] == r || dist < sm->sdist[p];
                  });
    T::sync();
    if (T::lead()) {  // the first survivor is kept, the others stay undecided
      uint32_t v = 0;
      for (uint32_t e0 = 0; e0 < u; e0 += 32) {
        const uint32_t e = e0 + lane;
        const bool keep = e < u && !sm->occ[e];
        const uint32_t p = e < u ? sm->und[e] : 0u;
        const unsigned m = __ballot_sync(kFull, keep);
        const uint32_t at = v + __popc(m & lt_mask);
        if (keep && at == 0) {
          sm->res[k] = sm->sid[p];
          sm->kept[p / 32] |= 1u << (p & 31u);
        }
        if (keep && at > 0) sm->und[at - 1] = static_cast<uint16_t>(p);
        v += __popc(m);
        __syncwarp();
      }
      if (lane == 0) {
        sm->num[0] = v ? v - 1 : 0;
        sm->num[1] = v > 0;
      }
    }
    T::sync();
    if (!sm->num[1]) break;
    k++;
    u = sm->num[0];
  }
  if (!strict) {  // :168-176: the others in order, from the second entry on
    T::sync();
    if (T::lead()) {
      for (uint32_t i0 = 0; i0 < c && k < M; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool keep = i >= 1 && i < c && !((sm->kept[i / 32] >> (i & 31u)) & 1u) &&
                          sm->sid[i] < n && sm->sid[i] != target;
        const unsigned m = __ballot_sync(kFull, keep);
        const uint32_t at = k + __popc(m & lt_mask);
        if (keep && at < M) sm->res[at] = sm->sid[i];
        k = min(M, k + __popc(m));
      }
      if (lane == 0) sm->num[3] = k;
    }
    T::sync();
    k = sm->num[3];
  }
  return k;
}

// Nodes of the one-warp kernels and the queue of the others: queue[0] entries, queue[1] taken,
// entries from queue[2] on.
__device__ __forceinline__ uint64_t warp_global() {
  return blockIdx.x * static_cast<uint64_t>(kWarps) + (threadIdx.x >> 5);
}
__device__ __forceinline__ uint64_t warp_count() {
  return static_cast<uint64_t>(gridDim.x) * kWarps;
}
__device__ __forceinline__ void enqueue(uint32_t* queue, uint32_t x) {
  queue[2 + atomicAdd(queue, 1u)] = x;
}
// The block's next queue entry, or tomb; every thread calls it.
__device__ __forceinline__ uint32_t dequeue(uint32_t* queue) {
  __shared__ uint32_t item;
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t i = atomicAdd(queue + 1, 1u);
    item = i < queue[0] ? queue[2 + i] : kTomb;
  }
  __syncthreads();
  return item;
}

// ---- MatchSup (:365-488) ------------------------------------------------------------------

// :378-392: query q claims base gt[q][topn] when no lower query did (the one-thread order).
__global__ void k_sup_claim(const uint32_t* __restrict__ gt, uint64_t q, uint32_t gt_k,
                            uint32_t topn, uint64_t n, uint32_t* __restrict__ claim) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < q;
       i += stride) {
    const uint32_t nn = gt[i * gt_k + topn];
    if (nn < n) atomicMin(claim + nn, static_cast<uint32_t>(i));
  }
}

// Queues the matched queries; the others have no pruned list.
__global__ void k_sup_pick(SupArgs a) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < a.q;
       i += stride) {
    const uint32_t nn = a.gt[i * a.gt_k + a.topn];
    if (nn < a.n && a.claim[nn] == static_cast<uint32_t>(i))
      enqueue(a.queue, static_cast<uint32_t>(i));
    else
      a.pcnt[i] = 0;
  }
}

// :407-441: each matched query prunes its ground-truth list around its base (non-strict).
__global__ void __launch_bounds__(kWarps * 32) k_sup_prune(SupArgs a) {
  __shared__ Lists<kRoarCap> sm_;
  Lists<kRoarCap>* sm = &sm_;
  const uint32_t lane = lane_id();
  for (;;) {
    const uint32_t qi = dequeue(a.queue);
    if (qi == kTomb) break;
    const uint32_t* row = a.gt + static_cast<uint64_t>(qi) * a.gt_k;
    const uint32_t nn = row[a.topn];
    if (threadIdx.x < 32) {  // the row up to its first id >= n, without the base itself
      uint32_t len = 0;
      for (uint32_t c0 = 0; c0 < a.gt_k; c0 += 32) {
        const uint32_t i = c0 + lane;
        const uint32_t x = i < a.gt_k ? row[i] : kTomb;
        const unsigned bad = __ballot_sync(kFull, i < a.gt_k && x >= a.n);
        const unsigned before = bad ? (bad & (0u - bad)) - 1u : kFull;
        len = append(sm->cand, len, x, i < a.gt_k && x != nn && ((before >> lane) & 1u));
        if (bad) break;
      }
      if (lane == 0) sm->num[0] = len;
    }
    __syncthreads();
    const uint32_t len = sm->num[0];
    const uint32_t k = team_prune<kWarps>(a.base, a.d, a.n, a.m_nn, sm, len, nn, true, false);
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
      const uint32_t x = sm->res[i];
      a.plist[static_cast<uint64_t>(qi) * a.m_nn + i] = x;
      atomicAdd(a.indeg + x, 1u);
    }
    if (threadIdx.x == 0) a.pcnt[qi] = k;
  }
}

// :449-475: a base's own pruned list joined with its first 128 - M_nn reverse sources; pruned
// (strict) when longer than M_nn, else ascending.
template <int W>
__device__ __forceinline__ void sup_merge_node(const SupArgs& a, Lists<Team<W>::kCap>* sm,
                                               uint32_t b, uint32_t owner, uint32_t k1,
                                               uint32_t r) {
  using T = Team<W>;
  const uint32_t lane = lane_id(), len = k1 + r;
  if (T::lead()) {
    for (uint32_t i = lane; i < k1; i += 32)
      sm->cand[i] = a.plist[static_cast<uint64_t>(owner) * a.m_nn + i];
    for (uint32_t i = lane; i < r; i += 32) {
      const uint64_t src = a.rev[static_cast<uint64_t>(b) * a.maxdeg + i];
      sm->cand[k1 + i] = a.gt[src * a.gt_k + a.topn];
    }
    __syncwarp();
    const uint32_t u = T::kCap <= 32 || len <= 32 ? sort_unique<1>(sm->cand, len)
                       : len <= 64               ? sort_unique<2>(sm->cand, len)
                                                 : sort_unique<4>(sm->cand, len);
    if (lane == 0) sm->num[0] = u;
  }
  T::sync();
  const uint32_t u = sm->num[0];
  uint32_t* out = a.out + static_cast<uint64_t>(b) * a.m_nn;
  const uint32_t* from = sm->cand;
  uint32_t k = u;
  if (u > a.m_nn) {
    k = team_prune<W>(a.base, a.d, a.n, a.m_nn, sm, u, b, false, true);
    from = sm->res;
  }
  if (T::lead()) {
    for (uint32_t i = lane; i < k; i += 32) out[i] = from[i];
    if (lane == 0) a.cnt[b] = k;
  }
  T::sync();
}

__global__ void __launch_bounds__(kWarps * 32) k_sup_merge(SupArgs a) {
  __shared__ Lists<kShort> sm_all[kWarps];
  Lists<kShort>* sm = sm_all + (threadIdx.x >> 5);
  const uint32_t lane = lane_id();
  for (uint64_t b = warp_global(); b < a.n; b += warp_count()) {
    const uint32_t owner = a.claim[b];
    const uint32_t k1 = owner < a.q ? a.pcnt[owner] : 0u;
    const uint32_t r = a.rnum[b];
    if (k1 + r == 0) {
      if (lane == 0) a.cnt[b] = 0;
    } else if (k1 + r > kShort) {
      if (lane == 0) enqueue(a.queue, static_cast<uint32_t>(b));
    } else {
      sup_merge_node<1>(a, sm, static_cast<uint32_t>(b), owner, k1, r);
    }
  }
}

__global__ void __launch_bounds__(kWarps * 32) k_sup_merge_long(SupArgs a) {
  __shared__ Lists<kRoarCap> sm;
  for (;;) {
    const uint32_t b = dequeue(a.queue);
    if (b == kTomb) break;
    const uint32_t owner = a.claim[b];
    sup_merge_node<kWarps>(a, &sm, b, owner, owner < a.q ? a.pcnt[owner] : 0u, a.rnum[b]);
  }
}

// ---- FusionNN (:490-537) ------------------------------------------------------------------

template <int W>
__device__ __forceinline__ void fusion_nn_node(const FusionArgs& a, Lists<Team<W>::kCap>* sm,
                                               uint32_t b) {
  using T = Team<W>;
  const uint32_t lane = lane_id();
  if (T::lead()) {
    uint32_t len = 0;
    for (uint32_t r = 0; r < a.rounds; r++) {
      const uint64_t rb = static_cast<uint64_t>(r) * a.n + b;
      const uint32_t k = min(a.sup_cnt[rb], a.sup_stride);
      const uint32_t* row = a.sup + rb * a.sup_stride;
      for (uint32_t i0 = 0; i0 < k; i0 += 32) {
        const uint32_t x = i0 + lane < k ? row[i0 + lane] : kTomb;
        len = append(sm->cand, len, x, x < a.n && x != b);
      }
    }
    if (lane == 0) sm->num[0] = len;
  }
  T::sync();
  const uint32_t len = sm->num[0];
  const uint32_t k = team_prune<W>(a.base, a.d, a.n, a.m_out, sm, len, b, true, true);
  if (T::lead()) {
    for (uint32_t i = lane; i < k; i += 32)
      a.out[static_cast<uint64_t>(b) * a.out_stride + i] = sm->res[i];
    if (lane == 0) a.cnt[b] = k;
  }
  T::sync();
}

__global__ void __launch_bounds__(kWarps * 32) k_fusion_nn(FusionArgs a) {
  __shared__ Lists<kShort> sm_all[kWarps];
  Lists<kShort>* sm = sm_all + (threadIdx.x >> 5);
  const uint32_t lane = lane_id();
  for (uint64_t b = warp_global(); b < a.n; b += warp_count()) {
    uint32_t len = 0;
    for (uint32_t r = lane; r < a.rounds; r += 32)
      len += min(a.sup_cnt[static_cast<uint64_t>(r) * a.n + b], a.sup_stride);
    len = __reduce_add_sync(kFull, len);
    if (len == 0) {
      if (lane == 0) a.cnt[b] = 0;
    } else if (len > kShort) {
      if (lane == 0) enqueue(a.queue, static_cast<uint32_t>(b));
    } else {
      fusion_nn_node<1>(a, sm, static_cast<uint32_t>(b));
    }
  }
}

__global__ void __launch_bounds__(kWarps * 32) k_fusion_nn_long(FusionArgs a) {
  __shared__ Lists<kRoarCap> sm;
  for (;;) {
    const uint32_t b = dequeue(a.queue);
    if (b == kTomb) break;
    fusion_nn_node<kWarps>(a, &sm, b);
  }
}

// ---- FusionFinal (:539-613) ---------------------------------------------------------------

struct FinalRow {
  const uint32_t* bip;
  uint32_t blen;
};
__device__ __forceinline__ FinalRow final_row(const FusionArgs& a, uint64_t b) {
  if (a.bip_off)
    return {a.bip + a.bip_off[b], static_cast<uint32_t>(a.bip_off[b + 1] - a.bip_off[b])};
  return {a.bip + b * a.bip_stride, min(a.bip_cnt[b], a.bip_stride)};
}

// The node's candidates, use(id, taken, bipartite) for 32 places at a time: the bipartite ids (not
// the node, < n), then the link ids (< n; the node itself is not skipped, :568-576), then the
// projection ids (not the node, < n).  One warp.
template <class Use>
__device__ __forceinline__ void final_candidates(const FusionArgs& a, const FinalRow& row,
                                                 uint64_t b, Use use) {
  const uint32_t lane = lane_id(), self = static_cast<uint32_t>(b);
  for (uint32_t i0 = 0; i0 < row.blen; i0 += 32) {
    const uint32_t x = i0 + lane < row.blen ? row.bip[i0 + lane] : kTomb;
    use(x, x < a.n && x != self, true);
  }
  for (uint32_t i0 = 0; i0 < a.m_link; i0 += 32) {
    const uint32_t x = i0 + lane < a.m_link ? a.link[b * a.m_link + i0 + lane] : kTomb;
    use(x, x < a.n, false);
  }
  for (uint32_t i0 = 0; i0 < a.m_supply; i0 += 32) {
    const uint32_t x = i0 + lane < a.m_supply ? a.supply[b * a.m_supply + i0 + lane] : kTomb;
    use(x, x < a.n && x != self, false);
  }
}

template <int W>
__device__ __forceinline__ void fusion_final_node(const FusionArgs& a, Lists<Team<W>::kCap>* sm,
                                                  const FinalRow& row, uint32_t b) {
  using T = Team<W>;
  const uint32_t lane = lane_id();
  uint32_t nbip = 0;
  if (T::lead()) {
    uint32_t len = 0, blen = 0;
    final_candidates(a, row, b, [&](uint32_t x, bool take, bool bip) {
      len = append(sm->cand, len, x, take);
      if (bip) blen = len;
    });
    __syncwarp();
    // repeats of any earlier id dropped
    if (T::kCap <= 32 || len <= 32)
      dedupe_first<1>(sm->cand, len);
    else if (len <= 64)
      dedupe_first<2>(sm->cand, len);
    else if (len <= 128)
      dedupe_first<4>(sm->cand, len);
    else
      dedupe_first<8>(sm->cand, len);
    // the final list starts with the surviving bipartite ids, in order
    uint32_t m = 0;
    for (uint32_t i0 = 0; i0 < len; i0 += 32) {
      const uint32_t i = i0 + lane;
      const uint32_t x = i < len ? sm->cand[i] : kTomb;
      __syncwarp();
      nbip = append(sm->fin, nbip, x, i < blen && x != kTomb);
      m = append(sm->cand, m, x, x != kTomb);
      __syncwarp();
    }
    if (lane == 0) sm->num[0] = m;
  }
  T::sync();
  const uint32_t len = sm->num[0];
  const uint32_t k = team_prune<W>(a.base, a.d, a.n, a.m_out, sm, len, b, false, true);
  if (T::lead()) {
    // then the pruned ids not listed yet, up to m_final - nbip of them (an unsigned difference:
    // unlimited when the bipartite ids outnumber m_final, :599-606)
    const uint32_t slots = a.m_out >= nbip ? a.m_out - nbip : 0xFFFFFFFFu;
    uint32_t nf = nbip, added = 0;
    for (uint32_t i = 0; i < k && added < slots; i++) {
      const uint32_t x = sm->res[i];
      if (!warp_contains(sm->fin, nbip, x)) {
        if (lane == 0) sm->fin[nf] = x;
        nf++;
        added++;
      }
    }
    __syncwarp();
    if (nf > a.out_stride) {
      if (lane == 0) {
        raise_error(a.status, kErrCapacity);
        a.cnt[b] = 0;
      }
    } else {
      for (uint32_t i = lane; i < nf; i += 32)
        a.out[static_cast<uint64_t>(b) * a.out_stride + i] = sm->fin[i];
      if (lane == 0) a.cnt[b] = nf;
    }
  }
  T::sync();
}

__global__ void __launch_bounds__(kWarps * 32) k_fusion_final(FusionArgs a) {
  __shared__ Lists<kShort> sm_all[kWarps];
  Lists<kShort>* sm = sm_all + (threadIdx.x >> 5);
  const uint32_t lane = lane_id();
  for (uint64_t b = warp_global(); b < a.n; b += warp_count()) {
    const FinalRow row = final_row(a, b);
    if (row.blen + a.m_link + a.m_supply > kRoarCap) {
      // more candidates than the kernel holds: flag and leave the row empty
      if (lane == 0) {
        raise_error(a.status, kErrCapacity);
        a.cnt[b] = 0;
      }
      continue;
    }
    uint32_t len = 0;
    final_candidates(a, row, b, [&](uint32_t, bool take, bool) {
      len += __popc(__ballot_sync(kFull, take));
    });
    if (len > kShort) {
      if (lane == 0) enqueue(a.queue, static_cast<uint32_t>(b));
    } else {
      fusion_final_node<1>(a, sm, row, static_cast<uint32_t>(b));
    }
  }
}

__global__ void __launch_bounds__(kWarps * 32) k_fusion_final_long(FusionArgs a) {
  __shared__ Lists<kRoarCap> sm;
  for (;;) {
    const uint32_t b = dequeue(a.queue);
    if (b == kTomb) break;
    fusion_final_node<kWarps>(a, &sm, final_row(a, b), b);
  }
}

int roar_grid(uint64_t items, int num_sms) {
  uint64_t blocks = (items + kWarps - 1) / kWarps;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
  if (blocks > cap) blocks = cap;
  return static_cast<int>(blocks ? blocks : 1);
}

// Blocks of a queue kernel: at most 8 per SM, and no more than entries there can be.
int queue_grid(uint64_t items, int num_sms) {
  const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
  return static_cast<int>(items < cap ? (items ? items : 1) : cap);
}

}  // namespace

bool roar_supported(uint32_t d, uint32_t m) { return d > 0 && d % 4 == 0 && m >= 1 && m <= kRoarRes; }

uint32_t roar_capacity() { return kRoarCap; }

cudaError_t launch_sup_claim(const uint32_t* gt, uint64_t q, uint32_t gt_k, uint32_t topn,
                             uint64_t n, uint32_t* claim, int num_sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(claim, 0xFF, n * sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
  uint64_t blocks = (q + 255) / 256;
  if (blocks > static_cast<uint64_t>(num_sms) * 8) blocks = static_cast<uint64_t>(num_sms) * 8;
  k_sup_claim<<<static_cast<unsigned>(blocks ? blocks : 1), 256, 0, st>>>(gt, q, gt_k, topn, n,
                                                                          claim);
  return cudaGetLastError();
}

cudaError_t launch_sup_prune(const SupArgs& a, int num_sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(a.queue, 0, 8, st);
  if (e != cudaSuccess) return e;
  uint64_t blocks = (a.q + 255) / 256;
  if (blocks > static_cast<uint64_t>(num_sms) * 8) blocks = static_cast<uint64_t>(num_sms) * 8;
  k_sup_pick<<<static_cast<unsigned>(blocks ? blocks : 1), 256, 0, st>>>(a);
  k_sup_prune<<<queue_grid(a.q < a.n ? a.q : a.n, num_sms), kWarps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_sup_merge(const SupArgs& a, int num_sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(a.queue, 0, 8, st);
  if (e != cudaSuccess) return e;
  k_sup_merge<<<roar_grid(a.n, num_sms), kWarps * 32, 0, st>>>(a);
  k_sup_merge_long<<<queue_grid(a.n, num_sms), kWarps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fusion_nn(const FusionArgs& a, int num_sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(a.queue, 0, 8, st);
  if (e != cudaSuccess) return e;
  k_fusion_nn<<<roar_grid(a.n, num_sms), kWarps * 32, 0, st>>>(a);
  k_fusion_nn_long<<<queue_grid(a.n, num_sms), kWarps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fusion_final(const FusionArgs& a, int num_sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(a.queue, 0, 8, st);
  if (e != cudaSuccess) return e;
  k_fusion_final<<<roar_grid(a.n, num_sms), kWarps * 32, 0, st>>>(a);
  k_fusion_final_long<<<queue_grid(a.n, num_sms), kWarps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace pg
