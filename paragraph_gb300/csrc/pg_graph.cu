// pg_graph.cu -- projection (K0), prune + reverse edges (K1/K2), reverse lists, merge (K3).
//
// Layout in HBM (all row-major, 64-bit row offsets):
//   base      n x d f32               the vectors (read-only)
//   winner    n u32                   projection winner key per base (K0)
//   pruned    n x P u32 + n counts    RNG-pruned out-lists (K2)
//   indeg     n u32 -> offs n+1       reverse-edge counts -> CSR offsets
//   edges     sum(pruned counts) u32  reverse sources grouped by destination (CSR); 8 bytes each in
//                                     builds, with the edge's distance
//   reverse   n x R u32 + n counts    first R sources per destination, ascending (K2's add_reverse)
//   graph     n x degree u32          merged + pruned out-lists, tomb padded (K3)
// A team of warps sized to the list owns one node in K2 and K3, one thread per candidate; a warp
// finishes a reverse list.  Every distance that decides something is one FMA chain in d order
// (dist_seq), the reference's distance_between, so ids are bit-identical to it.
#include <type_traits>

#include "pg_device.cuh"
#include "pg_kernels.h"

namespace pg {

// ------------------------------------------------------------------ K0: projection winners
// Winner key of query q for its top-1 base: queries whose gt[q][1] is a real id compete by
// lowest id; a query whose gt[q][1] is tomb leaves the CAS slot of match_top1_kernel_v0
// (Gbuilder.cuh:122) at tomb, so a later query overwrites its row: among those the highest id
// is the last writer.  Real-id queries always win over tomb ones.
__device__ __forceinline__ uint32_t winner_key(uint32_t q, bool real_first) {
  return real_first ? q : 0x80000000u + (0x7FFFFFFEu - q);
}
__device__ __forceinline__ uint32_t winner_query(uint32_t key) {
  if (key == kTomb) return kTomb;
  return key < 0x80000000u ? key : 0x7FFFFFFEu - (key - 0x80000000u);
}

__global__ void k_match_winner(const uint32_t* __restrict__ gt, uint64_t q, uint32_t gt_k,
                               uint64_t n, uint32_t* __restrict__ winner, uint32_t* status,
                               const uint64_t* __restrict__ seg_off,
                               const uint64_t* __restrict__ qseg_off, uint32_t seg_count,
                               const uint32_t* __restrict__ place) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t qi = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; qi < q;
       qi += stride) {
    uint64_t off = 0, ns = n;  // the query's sub-index: its ground-truth ids are local to it
    if (seg_count) {
      const uint32_t sg = segment_of(qseg_off, seg_count, qi);
      off = seg_off[sg];
      ns = seg_off[sg + 1] - off;
    }
    const uint32_t bl = gt[qi * gt_k];
    if (bl == kTomb) continue;
    if (bl >= ns) {
      raise_error(status, kErrBadId);
      continue;
    }
    const uint64_t b = place ? place[bl + off] : bl + off;
    const bool real = gt[qi * gt_k + 1] != kTomb;
    atomicMin(winner + b, winner_key(static_cast<uint32_t>(qi), real));
  }
}

// Materialises the n x gt_k projection rows of match_top1_kernel_v0 (stage API only; the build
// reads gt through `winner` directly): row b = gt[w][1..gt_k-2] followed by two tombs.
__global__ void k_match_rows(const uint32_t* __restrict__ gt, uint32_t gt_k, uint64_t n,
                             const uint32_t* __restrict__ winner, uint32_t* __restrict__ out) {
  const uint64_t total = n * gt_k;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total;
       i += stride) {
    const uint64_t b = i / gt_k;
    const uint32_t j = static_cast<uint32_t>(i - b * gt_k);
    const uint32_t w = winner_query(winner[b]);
    out[i] = (w != kTomb && j + 2 < gt_k) ? gt[static_cast<uint64_t>(w) * gt_k + j + 1] : kTomb;
  }
}

// ------------------------------------------------------------------ one node's list
// Lists of up to CAP = 32 W entries and the team of W warps that works on one: thread t holds
// entry t while it is gathered and sorted.
template <int W>
struct NodeLists {
  static constexpr uint32_t kCap = 32u * W;
  uint64_t key[kCap];
  uint32_t id[kCap];    // sorted by (distance, position)
  float dist[kCap];
  // The scans keep at most the list's entries.  The merge's fill (not strict) then takes every entry
  // not yet listed, where a kept id lists its first occurrence only: an id kept k times leaves k - 1 of
  // its entries to be taken, so the two together stay below twice the list.
  uint32_t kept[2 * kCap];
  uint8_t kpos[kCap];   // kept entries' places in the sorted list
  uint8_t own[kCap];    // entries known not to occlude one another (see merge_node)
  uint8_t und[kCap];    // undecided entries' places, ascending
  uint8_t tl[kCap];     // those to test against the newest kept entry
  uint8_t occ[kCap];    // 1: the newest kept entry occludes it
  uint8_t fo[kCap];     // kept index of the first occluder, kNoTest when none was needed
  uint32_t num[4];
};
constexpr uint8_t kNoTest = 0xFF;

template <int W>
struct Team {
  static __device__ __forceinline__ uint32_t tid() {
    return W == 1 ? lane_id() : threadIdx.x;
  }
  static __device__ __forceinline__ bool lead() { return W == 1 || threadIdx.x < 32; }
  static __device__ __forceinline__ void sync() {
    if constexpr (W == 1)
      __syncwarp();
    else
      __syncthreads();
  }
};

// The distance of a kept entry to its node as the prunes store it for the merge: a NaN where the
// list held something else than the FP32 chain (the node itself).
__device__ __forceinline__ float stored_dist(float dist, bool chain) {
  return chain ? dist : __uint_as_float(0x7FFFFFFFu);
}

// Thread t < c holds entry t (id x, distance dist, flag own; an id that stops the scan has tomb):
// sorts the list by (distance, position) -- bubble_sort's order (Gbuilder.cuh:890-902) -- into
// id / dist / own by counting, for every entry, the smaller keys; returns the entry's place.
// num[3] = the first place holding a tomb, or c.  CAP is small enough for counting to beat a
// sorting network: most lists hold a few entries, and the network has no early exit.
template <int W>
__device__ __forceinline__ uint32_t team_sort(NodeLists<W>* sm, uint32_t c, uint32_t x, float dist,
                                              bool own, bool tomb) {
  using T = Team<W>;
  const uint32_t t = T::tid();
  const uint64_t key = pack_key(dist, t);
  if (t < c) sm->key[t] = key;
  if (t == 0) sm->num[3] = c;
  T::sync();
  uint32_t rank = 0;
  for (uint32_t j = 0; j < c; j++) rank += sm->key[j] < key ? 1u : 0u;
  if (t < c) {
    sm->id[rank] = x;
    sm->dist[rank] = dist;
    sm->own[rank] = own;
    if (tomb) atomicMin(&sm->num[3], rank);
  }
  T::sync();
  return rank;
}

// The occlusion scan of fusion_prune_reverse_kernel_v0 (Gbuilder.cuh:1150-1199) and
// fusion_merge_sort_prune_kernel over the sorted entries [1 .. end), entry 0 being kept: in order,
// an entry is kept when no kept entry lies closer to it than the node does, until `limit` are
// kept.  Each newly kept entry is tested against every undecided entry at once (test(tl, T, r)
// sets occ for the T places tl that kept id r occludes); the first undecided entry left is the
// next kept one.  Every entry thus meets the kept entries in kept order up to its first occluder,
// as in the one-at-a-time scan, and kept list and evaluation count (tests up to and including the
// first occluder, entries before the one that fills the list) equal that scan's
// (Gbuilder.cuh:1163-1181).  Ids >= n count as occluded without a test.  Returns the number kept;
// the lead warp's lanes hold parts of the evaluation count in *checks.
template <int W, class Test>
__device__ __forceinline__ uint32_t team_scan(NodeLists<W>* sm, uint64_t n, uint32_t end,
                                              uint32_t limit, Test test, uint32_t* checks) {
  using T = Team<W>;
  const uint32_t lane = lane_id();
  const unsigned lt_mask = (1u << lane) - 1u;
  if (T::lead()) {
    uint32_t u = 0;
    for (uint32_t i0 = 1; i0 < end; i0 += 32) {
      const uint32_t i = i0 + lane;
      const bool in = i < end && sm->id[i] < n;
      const unsigned m = __ballot_sync(kFull, in);
      if (in) sm->und[u + __popc(m & lt_mask)] = static_cast<uint8_t>(i);
      if (i < end) {
        sm->occ[i] = 0;
        sm->fo[i] = kNoTest;
      }
      u += __popc(m);
    }
    if (lane == 0) {
      sm->kept[0] = sm->id[0];
      sm->kpos[0] = 0;
      sm->num[0] = u;
    }
  }
  T::sync();
  uint32_t k = 1, u = sm->num[0];
  while (k < limit && u > 0) {
    if (T::lead()) {  // the undecided entries that may be occluded by the newest kept one
      const bool rown = sm->own[sm->kpos[k - 1]];
      const bool real = sm->kept[k - 1] < n;
      uint32_t tn = 0;
      for (uint32_t e0 = 0; e0 < u; e0 += 32) {
        const uint32_t e = e0 + lane;
        const uint32_t p = e < u ? sm->und[e] : 0u;
        const bool need = e < u && real && !(rown && sm->own[p]);
        const unsigned m = __ballot_sync(kFull, need);
        if (need) sm->tl[tn + __popc(m & lt_mask)] = static_cast<uint8_t>(p);
        tn += __popc(m);
      }
      if (lane == 0) sm->num[1] = tn;
    }
    T::sync();
    const uint32_t tn = sm->num[1];
    if (tn) {
      test(sm->tl, tn, sm->kept[k - 1]);
      T::sync();
    }
    if (T::lead()) {  // the first survivor is kept, the others stay undecided
      uint32_t v = 0;
      for (uint32_t e0 = 0; e0 < u; e0 += 32) {
        const uint32_t e = e0 + lane;
        const uint32_t p = e < u ? sm->und[e] : 0u;
        const bool gone = e < u && sm->occ[p];
        const bool stay = e < u && !gone;
        if (gone) sm->fo[p] = static_cast<uint8_t>(k - 1);
        const unsigned m = __ballot_sync(kFull, stay);
        const uint32_t at = v + __popc(m & lt_mask);
        if (stay && at == 0) {
          sm->kept[k] = sm->id[p];
          sm->kpos[k] = static_cast<uint8_t>(p);
        }
        if (stay && at > 0) sm->und[at - 1] = static_cast<uint8_t>(p);
        v += __popc(m);
        __syncwarp();
      }
      if (lane == 0) {
        sm->num[0] = v ? v - 1 : 0;
        sm->num[2] = v > 0;
      }
    }
    T::sync();
    if (!sm->num[2]) break;
    k++;
    u = sm->num[0];
  }
  if (T::lead()) {
    const uint32_t last = k == limit ? sm->kpos[k - 1] : end;
    uint32_t part = lane == 0 ? k * (k - 1) / 2 : 0;  // the m-th kept entry made m tests
    for (uint32_t i = 1 + lane; i < last; i += 32)
      if (sm->fo[i] != kNoTest) part += sm->fo[i] + 1u;
    *checks += part;
  }
  return k;
}

// occ[p] = the exact chain says that r lies closer to entry p than the node does: one entry per
// thread.
template <int W, bool WIDE>
__device__ __forceinline__ void test_exact(NodeLists<W>* sm, const float* __restrict__ base,
                                           uint32_t d, const uint8_t* tl, uint32_t tn,
                                           uint32_t r) {
  const float* rrow = base + static_cast<uint64_t>(r) * d;
  for (uint32_t e = Team<W>::tid(); e < tn; e += 32u * W) {
    const uint32_t p = tl[e];
    if (dist_seq<WIDE>(base + static_cast<uint64_t>(sm->id[p]) * d, rrow, d) < sm->dist[p])
      sm->occ[p] = 1;
  }
}

// The same decisions from FP32 inner products whose order suits the memory (eight lanes per row,
// two rows per group at a time, 16-byte loads of whole 128-byte lines), the exact chain only
// inside their error bound.  With norms |x|, |y| from launch_screen_norms,
//   |chain(x, y) - xy| <= c_seq |x||y|, c_seq = (D + 2) 2^-23, and
//   |s - xy| <= c_par |x||y|, c_par = (D / 32 + 10) 2^-23 (D / 32 + 6 roundings of 2^-24),
// plus a 2^-20 relative guard on the comparison; an infinite or NaN bound defers to the chain.
// A lane reading whole rows on its own touches 32 cache lines per load.
template <int W>
__device__ __forceinline__ void test_screened(NodeLists<W>* sm, const float* __restrict__ base,
                                              uint32_t d, const float2* __restrict__ norms,
                                              const uint8_t* tl, uint32_t tn, uint32_t r) {
  constexpr uint32_t G = 4u * W;
  const uint32_t g = Team<W>::tid() >> 3, m = threadIdx.x & 7u;
  const uint32_t w0 = (Team<W>::tid() >> 5) * 4u;
  const float* rrow = base + static_cast<uint64_t>(r) * d;
  const float coef = static_cast<float>(d + 2u + d / 32u + 10u) * 1.19209290e-07f;  // 2^-23
  const float nr = __ldg(&norms[r].x);
  for (uint32_t e0 = 0; e0 + w0 < tn; e0 += 2 * G) {  // uniform in the warp
    const uint32_t i = e0 + g, j = i + G;
    const uint32_t pi = tl[min(i, tn - 1)], pj = tl[min(j, tn - 1)];
    const uint32_t xi = sm->id[pi], xj = sm->id[pj];
    const bool up = (m & 4u) != 0;  // lanes with m < 4 finish entry i, the others entry j
    const uint32_t x = up ? xj : xi;
    const float nx = __ldg(&norms[x].x);
    const float* ri = base + static_cast<uint64_t>(xi) * d;
    const float* rj = base + static_cast<uint64_t>(xj) * d;
    float4 si = make_float4(0.f, 0.f, 0.f, 0.f), sj = si;
    auto step = [](float4& s, const float4 u, const float4 v) {
      s.x = fmaf(u.x, v.x, s.x);
      s.y = fmaf(u.y, v.y, s.y);
      s.z = fmaf(u.z, v.z, s.z);
      s.w = fmaf(u.w, v.w, s.w);
    };
    auto ld = [](const float* q) { return __ldg(reinterpret_cast<const float4*>(q)); };
    if (e0 + G + w0 < tn) {
#pragma unroll 4
      for (uint32_t c = 4u * m; c < d; c += 32) {
        const float4 u = ld(rrow + c);
        step(si, u, ld(ri + c));
        step(sj, u, ld(rj + c));
      }
    } else {
#pragma unroll 4
      for (uint32_t c = 4u * m; c < d; c += 32) step(si, ld(rrow + c), ld(ri + c));
    }
    const float a = (si.x + si.y) + (si.z + si.w), b = (sj.x + sj.y) + (sj.z + sj.w);
    float s = (up ? b : a) + __shfl_xor_sync(kFull, up ? a : b, 4);
    s += __shfl_xor_sync(kFull, s, 2);
    s += __shfl_xor_sync(kFull, s, 1);
    if ((m & 3u) == 0 && (up ? j : i) < tn) {
      const uint32_t p = up ? pj : pi;
      const float dp = sm->dist[p], dhat = -s;
      const float bound = coef * nx * nr + fabsf(dhat) * 9.5367431640625e-07f + 1e-30f;
      bool yes = dhat + bound < dp;
      if (!yes && !(dhat - bound >= dp))
        yes = dist_seq<true>(base + static_cast<uint64_t>(x) * d, rrow, d) < dp;
      if (yes) sm->occ[p] = 1;
    }
  }
}

// ------------------------------------------------------------------ K2: prune + reverse
// fusion_prune_reverse_kernel_v0 (Gbuilder.cuh:1093-1244), one block of W warps per node of up to
// 32 W candidates, a thread per candidate.  PHASE1 reads the candidate row of node b straight from
// the winner's ground truth (the K0 row) instead of a materialised graph, and looks for nodes that
// have a winner `look` (at most 32) at a time; in screened builds its tests are decided as the
// merge's are.  Bound by the latency of the chains.  Against one
// warp per node, several candidates per lane and a scan whose window bookkeeping was serial: the
// whole projection of 1000 x 200 0.33 -> 0.12 ms and of 120k x 512 4.2 -> 2.2 ms, both link prunes
// of 120k x 512 (c = 64) 11.9 -> 10.7 ms.
template <int W, bool PHASE1, bool SCREEN, bool WIDE>
__device__ __forceinline__ void prune_node(const PruneArgs& a, NodeLists<W>* sm, uint64_t b,
                                           uint32_t w, uint32_t* ev) {
  using T = Team<W>;
  const uint32_t t = T::tid(), lane = lane_id();
  uint64_t goff = 0, gn = a.n;  // phase 1: ground-truth ids are local to b's sub-index
  if (PHASE1 && a.seg_count) {
    const uint32_t sg = segment_of(a.seg_off, a.seg_count, b);
    goff = a.seg_off[sg];
    gn = a.seg_off[sg + 1] - goff;
  }
  uint32_t x = kTomb;
  if (t < a.c) {
    if (PHASE1) {
      x = (t + 2 < a.gt_k) ? a.gt[static_cast<uint64_t>(w) * a.gt_k + t + 1] : kTomb;
      if (x != kTomb) {
        if (x >= gn) {  // out-of-range input id
          raise_error(a.status, kErrBadId);
          x = kTomb;
        } else {
          x = static_cast<uint32_t>(x + goff);
          if (a.place) x = a.place[x];
        }
      }
    } else {
      x = a.graph[b * a.c + t];
    }
  }
  if (x >= a.n && x != kTomb && x != kMaskedTomb) {  // out-of-range input id
    raise_error(a.status, kErrBadId);
    x = kTomb;
  }
  const bool tomb = x == kTomb || x == kMaskedTomb;
  const bool valid = !tomb && x != static_cast<uint32_t>(b);
  const float dist = valid ? dist_seq<WIDE>(a.base + b * a.d,
                                            a.base + static_cast<uint64_t>(x) * a.d, a.d)
                           : FLT_MAX;
  const uint32_t nv = __popc(__ballot_sync(kFull, valid));
  if (lane == 0) *ev += nv;
  const uint32_t rank = team_sort<W>(sm, a.c, x, dist, false, tomb && t < a.c);
  if (a.sorted && t < a.c) a.sorted[b * a.c + rank] = x;
  const uint32_t end = sm->num[3];
  if (end == 0) {  // the first entry is a tomb: nothing kept
    if (t == 0) a.pruned_num[b] = 0;
    T::sync();
    return;
  }
  uint32_t checks = 0;
  uint32_t k = team_scan<W>(sm, a.n, end, a.p,
                            [&](const uint8_t* tl, uint32_t tn, uint32_t r) {
                              if constexpr (SCREEN)
                                test_screened<W>(sm, a.base, a.d, a.norms, tl, tn, r);
                              else
                                test_exact<W, WIDE>(sm, a.base, a.d, tl, tn, r);
                            },
                            &checks);
  if (T::lead()) {
    *ev += checks;
    // non-strict fill (Gbuilder.cuh:1201-1239), from where the scan stopped
    for (uint32_t j = end; !a.strict && j < a.c && k < a.p; j++) {
      const uint32_t y = sm->id[j];
      if (y == kTomb || y == static_cast<uint32_t>(b) || y == kMaskedTomb) continue;
      bool dup = false;
      for (uint32_t i = lane; i < k; i += 32) dup |= sm->kept[i] == y;
      if (__any_sync(kFull, dup)) continue;
      if (lane == 0) {
        sm->kept[k] = y;
        sm->kpos[k] = static_cast<uint8_t>(j);
      }
      k++;
      __syncwarp();
    }
    if (lane == 0) a.pruned_num[b] = k;
    for (uint32_t i = lane; i < k; i += 32) {
      const uint32_t dst = sm->kept[i];
      a.pruned[b * a.p + i] = dst;
      if (a.pruned_dist)
        a.pruned_dist[b * a.p + i] =
            stored_dist(sm->dist[sm->kpos[i]], dst != static_cast<uint32_t>(b));
      atomicAdd(a.indeg + dst, 1u);
    }
  }
  T::sync();
}

constexpr int kPruneWarps = 24;  // warps per SM (80 registers)

template <int W, bool PHASE1, bool SCREEN, bool WIDE>
__global__ void __launch_bounds__(32 * W, kPruneWarps / W)
k_prune_reverse(PruneArgs a, uint32_t look) {
  __shared__ NodeLists<W> sm;
  uint32_t part = 0;
  uint64_t ev = 0;
  if constexpr (PHASE1) {
    const uint32_t lane = lane_id();
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * look;
    for (uint64_t b0 = blockIdx.x * static_cast<uint64_t>(look); b0 < a.n; b0 += stride) {
      const uint64_t b = b0 + lane;
      const bool in = lane < look && b < a.n;
      const uint32_t w = in ? winner_query(a.winner[b]) : kTomb;
      unsigned todo = __ballot_sync(kFull, w != kTomb);
      if (threadIdx.x < 32 && in && w == kTomb) a.pruned_num[b] = 0;  // nobody's top-1
      for (; todo; todo &= todo - 1u) {
        const int l = __ffs(static_cast<int>(todo)) - 1;
        prune_node<W, true, SCREEN, WIDE>(a, &sm, b0 + l, __shfl_sync(kFull, w, l), &part);
        ev += part;
        part = 0;
      }
    }
  } else {
    for (uint64_t b = blockIdx.x; b < a.n; b += gridDim.x) {
      prune_node<W, false, SCREEN, WIDE>(a, &sm, b, kTomb, &part);
      ev += part;
      part = 0;
    }
  }
  for (int o = 16; o > 0; o >>= 1) ev += __shfl_xor_sync(kFull, ev, o);
  if (lane_id() == 0 && ev) atomicAdd(a.evals, static_cast<unsigned long long>(ev));
}

// The distances of the screened prune's kept edges, which the merge sorts by: one edge per lane,
// the edges of `look` nodes at a time (two or three a node on 1M x 200; at most 32).
template <bool WIDE>
__global__ void __launch_bounds__(256) k_edge_dists(const float* __restrict__ base, uint64_t n,
                                                    uint32_t d,
                                                    const uint32_t* __restrict__ pruned,
                                                    const uint32_t* __restrict__ pruned_num,
                                                    uint32_t p, uint32_t look,
                                                    float* __restrict__ dist) {
  const uint32_t lane = lane_id();
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * 8u * look;
  for (uint64_t b0 = (blockIdx.x * 8ull + (threadIdx.x >> 5)) * look; b0 < n; b0 += stride) {
    const uint32_t cnt = lane < look && b0 + lane < n ? pruned_num[b0 + lane] : 0u;
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += y;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    for (uint32_t e0 = 0; e0 < total; e0 += 32) {
      const uint32_t e = e0 + lane;
      uint32_t l = 0;  // the number of nodes whose edges all come before e: its node
#pragma unroll
      for (uint32_t s = 16; s > 0; s >>= 1)
        if (__shfl_sync(kFull, incl, l + s - 1) <= e) l += s;
      const uint32_t before = __shfl_sync(kFull, incl - cnt, l & 31u);
      if (e < total) {
        const uint64_t b = b0 + l;
        const uint64_t at = b * p + (e - before);
        const uint32_t x = pruned[at];
        const float v = dist_seq<WIDE>(base + b * d, base + static_cast<uint64_t>(x) * d, d);
        dist[at] = stored_dist(v, x != static_cast<uint32_t>(b));
      }
    }
  }
}

// ------------------------------------------------------------------ reverse edges (CSR)
// Exclusive scan of n counts into offs[0..n] (offs[n] = total).  Three passes: per-block sums,
// one block scanning the block sums, per-block scan plus offset.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr uint64_t kScanSmall = 4096;  // counts that one block scans
// callers size the tile-sum buffers by kScanTileElems (pg_kernels.h)
static_assert(kScanTile == kScanTileElems, "scan tile size must match kScanTileElems");

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums,
                                                         uint32_t* total) {
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, o);
    if (lane >= static_cast<uint32_t>(o)) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = (lane < (blockDim.x >> 5)) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, w, o);
      if (lane >= static_cast<uint32_t>(o)) w += y;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  const uint32_t before = (warp ? warp_sums[warp - 1] : 0) + x - v;
  if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const uint32_t* __restrict__ in,
                                                             uint64_t n,
                                                             uint32_t* __restrict__ tile_sums) {
  __shared__ uint32_t ws[32];
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) s += (base + i < n) ? in[base + i] : 0u;
  uint32_t total;
  block_exclusive_scan(s, ws, &total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(uint32_t* __restrict__ sums,
                                                                 uint32_t tiles,
                                                                 uint32_t* __restrict__ total_out) {
  __shared__ uint32_t ws[32];
  uint32_t carry = 0;
  for (uint32_t t0 = 0; t0 < tiles; t0 += kScanThreads) {
    const uint32_t i = t0 + threadIdx.x;
    const uint32_t v = (i < tiles) ? sums[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, ws, &total);
    if (i < tiles) sums[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) *total_out = carry;
}

// Also leaves the counts and the cursors zero, for the next round and the scatter that follows.
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(uint32_t* __restrict__ in, uint64_t n,
                                                             const uint32_t* __restrict__ tile_off,
                                                             uint32_t* __restrict__ out,
                                                             uint32_t* __restrict__ cursor) {
  __shared__ uint32_t ws[32];
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    v[i] = (base + i < n) ? in[base + i] : 0u;
    s += v[i];
  }
  uint32_t run = tile_off[blockIdx.x] + block_exclusive_scan(s, ws, nullptr);
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    if (base + i < n) {
      out[base + i] = run;
      in[base + i] = 0;
      cursor[base + i] = 0;
    }
    run += v[i];
  }
}

// The same in one launch, one block, for small n (three launches cost more than the scan).
__global__ void __launch_bounds__(kScanThreads) k_scan_small(uint32_t* __restrict__ in, uint32_t n,
                                                             uint32_t* __restrict__ out,
                                                             uint32_t* __restrict__ cursor) {
  __shared__ uint32_t ws[32];
  uint32_t carry = 0;
  for (uint32_t t0 = 0; t0 < n; t0 += kScanThreads) {
    const uint32_t i = t0 + threadIdx.x;
    const uint32_t v = i < n ? in[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, ws, &total);
    if (i < n) {
      out[i] = carry + ex;
      in[i] = 0;
      cursor[i] = 0;
    }
    carry += total;
  }
  if (threadIdx.x == 0) out[n] = carry;
}

// Every kept edge b -> p becomes the entry b in p's CSR segment (order fixed later by sorting);
// with distances the entry is (b << 32 | bits of the edge's distance).
template <bool DIST>
__global__ void k_scatter_reverse(const uint32_t* __restrict__ pruned,
                                  const uint32_t* __restrict__ pruned_num,
                                  const float* __restrict__ pruned_dist, uint32_t p_len,
                                  uint64_t rows, const uint32_t* __restrict__ offs,
                                  uint32_t* __restrict__ cursor, uint32_t* __restrict__ edges,
                                  const uint32_t* __restrict__ order) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t b = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; b < rows;
       b += stride) {
    const uint32_t cnt = pruned_num[b];
    const uint32_t src = order ? order[b] : static_cast<uint32_t>(b);
    for (uint32_t t = 0; t < cnt; t++) {
      const uint32_t dst = pruned[b * p_len + t];
      const uint32_t pos = offs[dst] + atomicAdd(cursor + dst, 1u);
      if constexpr (DIST)
        reinterpret_cast<uint64_t*>(edges)[pos] =
            (static_cast<uint64_t>(src) << 32) | __float_as_uint(pruned_dist[b * p_len + t]);
      else
        edges[pos] = src;
    }
  }
}

template <int E>
__device__ __forceinline__ void warp_sort_keys(uint32_t (&key)[E]) {
  warp_sort_u32<E>(key);
}
template <int E>
__device__ __forceinline__ void warp_sort_keys(uint64_t (&key)[E]) {
  warp_sort_u64<E>(key);
}

// The first 32 E entries of a segment of at most 32 E (E < 4), or the 128 smallest of any segment
// (E = 4), ascending, in `best`.
template <int E, class Key>
__device__ __forceinline__ void smallest(const Key* __restrict__ seg, uint32_t deg,
                                         Key (&best)[E]) {
  const uint32_t lane = lane_id();
  for (uint32_t c0 = 0; c0 < deg; c0 += 32 * E) {
    Key chunk[E];
#pragma unroll
    for (int s = 0; s < E; s++) {
      const uint32_t i = c0 + static_cast<uint32_t>(s) * 32u + lane;
      chunk[s] = (i < deg) ? seg[i] : ~Key(0);
    }
    if (c0) {  // nothing below the last of the smallest so far (sources arrive mostly ascending)
      const Key last = __shfl_sync(kFull, best[E - 1], 31);
      bool below = false;
#pragma unroll
      for (int s = 0; s < E; s++) below |= chunk[s] < last;
      if (!__any_sync(kFull, below)) continue;
    }
    warp_sort_keys<E>(chunk);
    if (c0 == 0) {
#pragma unroll
      for (int s = 0; s < E; s++) best[s] = chunk[s];
    } else {
      // best (ascending) against chunk reversed: the element-wise minimum holds the 128
      // smallest as a bitonic sequence, which one merge pass sorts.
#pragma unroll
      for (int s = 0; s < E; s++) {
        const Key rv = __shfl_sync(kFull, chunk[E - 1 - s], 31 - lane);
        best[s] = rv < best[s] ? rv : best[s];
      }
      warp_bitonic_merge<E>(best);
    }
  }
}

// Reverse list of node p: the R smallest sources of its segment in ascending order, which is
// what add_reverse (Gbuilder.cuh:1020-1038) stores when sources run in ascending order; the
// count is min(in-degree, R).  The sort is sized to the segment (most hold a few entries);
// segments longer than 128 keep a running 128-smallest set and pass over chunks that cannot change
// it (a hub of 1M x 200 has about 10^5 sources).
template <bool DIST>
__global__ void __launch_bounds__(256) k_reverse_lists(const uint32_t* __restrict__ offs,
                                                       const uint32_t* __restrict__ edges,
                                                       uint64_t n, uint32_t r,
                                                       uint32_t* __restrict__ rev,
                                                       float* __restrict__ rev_dist,
                                                       uint32_t* __restrict__ rev_num,
                                                       const uint32_t* __restrict__ place) {
  using Key = std::conditional_t<DIST, uint64_t, uint32_t>;
  const uint32_t lane = lane_id();
  const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
  for (uint64_t p = blockIdx.x * static_cast<uint64_t>(blockDim.x >> 5) + (threadIdx.x >> 5);
       p < n; p += nwarps) {
    const uint32_t o0 = offs[p];
    const uint32_t deg = offs[p + 1] - o0;
    const uint32_t cnt = min(deg, r);
    if (lane == 0) rev_num[p] = cnt;
    if (deg == 0) continue;
    const Key* seg = reinterpret_cast<const Key*>(edges) + o0;
    auto put = [&](uint32_t i, Key k) {
      if (i >= cnt) return;
      const uint32_t src = DIST ? static_cast<uint32_t>(static_cast<uint64_t>(k) >> 32)
                                : static_cast<uint32_t>(k);
      rev[p * r + i] = place ? place[src] : src;
      if (DIST) rev_dist[p * r + i] = __uint_as_float(static_cast<uint32_t>(k));
    };
    if (deg <= 32) {
      Key best[1];
      smallest<1>(seg, deg, best);
      put(lane, best[0]);
    } else {
      Key best[4];
      smallest<4>(seg, deg, best);
#pragma unroll
      for (int s = 0; s < 4; s++) put(static_cast<uint32_t>(s) * 32u + lane, best[s]);
    }
  }
}

// ------------------------------------------------------------------ K3: merge + prune
// fusion_merge_sort_prune_kernel (Gbuilder.cuh:1467-1601): merged list = reverse entries then
// pruned entries (pr_sort_list view); sort by distance keeping that order on ties; RNG prune
// into the out row; non-strict fill with first-occurrence marking; tomb padding.
// A build passes the distances that its prune computed for the same edges (the chain is symmetric
// bit for bit), and own_strict when the pruned lists come from a strict scan: two of their entries
// were tested against each other there with the same distances, so neither occludes the other.
// Lists of up to 32 entries take one warp; longer ones are queued for teams of four.  Bound by
// latency (lists, then one round of rows per kept entry).  Rounds 1 + 2 with every distance
// computed again, one warp per node and the window of candidates kept in shared memory:
// 1M x 200: 5.6 + 4.7 ms, 300k x 512 (L = 96): 12.6 + 24.2, 1000 x 200: 0.13 + 0.13; now
// 1.2 + 1.0, 2.4 + 6.2 and 0.065 + 0.065 (screened builds).
template <int W, bool SCREEN, bool WIDE>
__device__ __forceinline__ void merge_node(const MergeArgs& a, NodeLists<W>* sm, uint64_t b,
                                           uint32_t rn, uint32_t nn, uint64_t* ev) {
  using T = Team<W>;
  static_assert(sizeof(sm->kept) >= 2 * 32 * W * sizeof(uint32_t), "kept entries and the fill's");
  const uint32_t t = T::tid(), lane = lane_id();
  const float* brow = a.base + b * a.d;
  uint32_t x = kTomb;
  float dist = FLT_MAX;
  bool own = false;
  if (t < nn) {
    const uint64_t at = t < rn ? b * a.r + t : b * a.p + (t - rn);
    x = t < rn ? a.reverse[at] : a.pruned[at];
    if (x >= a.n) {  // out-of-range input id
      raise_error(a.status, kErrBadId);
      x = kTomb;
    } else {
      bool known = false;
      if (a.pruned_dist) {
        dist = t < rn ? a.reverse_dist[at] : a.pruned_dist[at];
        known = !isnan(dist);
      }
      own = known && a.own_strict && t >= rn;
      if (!known) dist = dist_seq<WIDE>(brow, a.base + static_cast<uint64_t>(x) * a.d, a.d);
    }
  }
  team_sort<W>(sm, nn, x, dist, own, false);
  uint32_t checks = 0;
  uint32_t k = team_scan<W>(sm, a.n, nn, a.degree,
                            [&](const uint8_t* tl, uint32_t tn, uint32_t r) {
                              if constexpr (SCREEN)
                                test_screened<W>(sm, a.base, a.d, a.norms, tl, tn, r);
                              else
                                test_exact<W, WIDE>(sm, a.base, a.d, tl, tn, r);
                            },
                            &checks);
  if (T::lead()) {
    *ev += checks + (lane == 0 ? nn : 0u);
    if (!a.strict && k < a.degree) {
      for (uint32_t i = lane; i < nn; i += 32) sm->occ[i] = 0;  // now: listed already
      __syncwarp();
      for (uint32_t i = 0; i < k; i++) {  // first occurrence of each kept id
        const uint32_t y = sm->kept[i];
        for (uint32_t j0 = 0; j0 < nn; j0 += 32) {
          const uint32_t j = j0 + lane;
          const unsigned m = __ballot_sync(kFull, j < nn && sm->id[j] == y);
          if (m) {
            if (lane == 0) sm->occ[j0 + __ffs(static_cast<int>(m)) - 1] = 1;
            break;
          }
        }
      }
      __syncwarp();
      for (uint32_t i0 = 0; i0 < nn && k < a.degree; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint32_t y = i < nn ? sm->id[i] : kTomb;
        const bool take = i < nn && !sm->occ[i] && y < a.n && y != static_cast<uint32_t>(b);
        const unsigned m = __ballot_sync(kFull, take);
        const uint32_t to = k + __popc(m & ((1u << lane) - 1u));
        if (take && to < a.degree) sm->kept[to] = y;
        k = min(a.degree, k + __popc(m));
      }
      __syncwarp();
    }
    uint32_t* orow = a.out + b * a.degree;
    for (uint32_t i = lane; i < a.degree; i += 32) orow[i] = i < k ? sm->kept[i] : kTomb;
  }
  T::sync();
}

// 24 warps per SM in both kernels (80 registers): 16, 32 and 48 were 0-5% slower or equal on whole
// builds from 1000 x 200 to 300k x 512.
constexpr uint32_t kMergeWarps = 8;  // nodes per block of the one-warp kernel

template <bool SCREEN, bool WIDE>
__global__ void __launch_bounds__(32 * kMergeWarps, 3) k_merge_prune(MergeArgs a) {
  __shared__ NodeLists<1> sm_all[kMergeWarps];
  NodeLists<1>* sm = sm_all + (threadIdx.x >> 5);
  const uint32_t lane = lane_id();
  const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * kMergeWarps;
  uint64_t ev = 0;
  for (uint64_t b = blockIdx.x * static_cast<uint64_t>(kMergeWarps) + (threadIdx.x >> 5); b < a.n;
       b += nwarps) {
    const uint32_t rn = min(a.reverse_num[b], a.r);
    const uint32_t nn = rn + min(a.pruned_num[b], a.p);
    if (nn == 0) {
      for (uint32_t t = lane; t < a.degree; t += 32) a.out[b * a.degree + t] = kTomb;
    } else if (nn > 32) {
      if (lane == 0) a.queue[2 + atomicAdd(a.queue, 1u)] = static_cast<uint32_t>(b);
    } else {
      merge_node<1, SCREEN, WIDE>(a, sm, b, rn, nn, &ev);
    }
  }
  for (int o = 16; o > 0; o >>= 1) ev += __shfl_xor_sync(kFull, ev, o);
  if (lane == 0 && ev) atomicAdd(a.evals, static_cast<unsigned long long>(ev));
}

// The queued nodes: queue[0] of them from queue[2] on, queue[1] taken.
template <bool SCREEN, bool WIDE>
__global__ void __launch_bounds__(128, 6) k_merge_long(MergeArgs a) {
  __shared__ NodeLists<4> sm;
  __shared__ uint32_t item;
  uint64_t ev = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const uint32_t i = atomicAdd(a.queue + 1, 1u);
      item = i < a.queue[0] ? a.queue[2 + i] : kTomb;
    }
    __syncthreads();
    const uint32_t b = item;
    if (b == kTomb) break;
    const uint32_t rn = min(a.reverse_num[b], a.r);
    merge_node<4, SCREEN, WIDE>(a, &sm, b, rn, rn + min(a.pruned_num[b], a.p), &ev);
  }
  for (int o = 16; o > 0; o >>= 1) ev += __shfl_xor_sync(kFull, ev, o);
  if (lane_id() == 0 && ev) atomicAdd(a.evals, static_cast<unsigned long long>(ev));
}

// ------------------------------------------------------------------ launchers
static int grid_for(uint64_t items, int per_block, int num_sms, int max_per_sm) {
  uint64_t blocks = (items + per_block - 1) / per_block;
  uint64_t cap = static_cast<uint64_t>(num_sms) * max_per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks == 0) blocks = 1;
  return static_cast<int>(blocks);
}

cudaError_t launch_match_winner(const uint32_t* gt, uint64_t q, uint32_t gt_k, uint64_t n,
                                uint32_t* winner, uint32_t* status, int num_sms, cudaStream_t st,
                                const uint64_t* seg_off, const uint64_t* qseg_off,
                                uint32_t seg_count, const uint32_t* place) {
  cudaError_t e = cudaMemsetAsync(winner, 0xFF, n * sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
  k_match_winner<<<grid_for(q, 256, num_sms, 8), 256, 0, st>>>(gt, q, gt_k, n, winner, status,
                                                               seg_off, qseg_off, seg_count,
                                                               place);
  return cudaGetLastError();
}

__global__ void k_localize(uint32_t* __restrict__ rows, uint64_t n, uint32_t deg,
                           const uint64_t* __restrict__ seg_off, uint32_t seg_count) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n * deg;
       i += stride) {
    const uint32_t v = rows[i];
    if (v != kTomb) rows[i] = static_cast<uint32_t>(v - seg_off[segment_of(seg_off, seg_count, i / deg)]);
  }
}

cudaError_t launch_localize(uint32_t* rows, uint64_t n, uint32_t deg, const uint64_t* seg_off,
                            uint32_t seg_count, int num_sms, cudaStream_t st) {
  k_localize<<<grid_for(n * deg, 256, num_sms, 8), 256, 0, st>>>(rows, n, deg, seg_off, seg_count);
  return cudaGetLastError();
}

// One thread per output word: a row's words are consecutive threads, so both sides move whole rows.
__global__ void k_restore(const uint32_t* __restrict__ rows, uint64_t n, uint32_t deg,
                          const uint32_t* __restrict__ order, const uint64_t* __restrict__ seg_off,
                          uint32_t seg_count, uint32_t* __restrict__ out) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n * deg;
       i += stride) {
    const uint64_t r = i / deg;
    uint32_t v = rows[i];
    if (v != kTomb) {
      v = order[v];
      if (seg_count) v = static_cast<uint32_t>(v - seg_off[segment_of(seg_off, seg_count, r)]);
    }
    out[static_cast<uint64_t>(order[r]) * deg + (i - r * deg)] = v;
  }
}

cudaError_t launch_restore(const uint32_t* rows, uint64_t n, uint32_t deg, const uint32_t* order,
                           const uint64_t* seg_off, uint32_t seg_count, uint32_t* out, int num_sms,
                           cudaStream_t st) {
  k_restore<<<grid_for(n * deg, 256, num_sms, 8), 256, 0, st>>>(rows, n, deg, order, seg_off,
                                                                seg_count, out);
  return cudaGetLastError();
}

cudaError_t launch_match_rows(const uint32_t* gt, uint32_t gt_k, uint64_t n,
                              const uint32_t* winner, uint32_t* out, int num_sms,
                              cudaStream_t st) {
  k_match_rows<<<grid_for(n * gt_k, 256, num_sms, 8), 256, 0, st>>>(gt, gt_k, n, winner, out);
  return cudaGetLastError();
}

// The 256-bit-load kernels for rows of kWideRowFloats or more on a 32-byte aligned base.
static bool wide_rows(const float* base, uint32_t d) {
  return d >= kWideRowFloats && (d % 8) == 0 && (reinterpret_cast<uintptr_t>(base) % 32) == 0;
}

cudaError_t launch_edge_dists(const float* base, uint64_t n, uint32_t d, const uint32_t* pruned,
                              const uint32_t* pruned_num, uint32_t p, float* dist, int num_sms,
                              cudaStream_t st) {
  auto kern = wide_rows(base, d) ? k_edge_dists<true> : k_edge_dists<false>;
  uint64_t look = n / (static_cast<uint64_t>(num_sms) * 64);  // one round of 64 warps per SM
  look = look < 1 ? 1 : look > 32 ? 32 : look;
  kern<<<grid_for(n, static_cast<int>(8 * look), num_sms, 8), 256, 0, st>>>(
      base, n, d, pruned, pruned_num, p, static_cast<uint32_t>(look), dist);
  return cudaGetLastError();
}

template <int W, bool P1>
static cudaError_t launch_prune_w(const PruneArgs& a, int num_sms, cudaStream_t st) {
  // phase 1: few nodes have a winner, so a block looks at up to 32, fewer when they are few enough
  // for every block to get some
  const int per_sm = kPruneWarps / W;
  uint64_t look = P1 ? a.n / (static_cast<uint64_t>(num_sms) * per_sm) : 1;
  look = look < 1 ? 1 : look > 32 ? 32 : look;
  const unsigned grid = grid_for(a.n, static_cast<int>(look), num_sms, per_sm);
  auto kern = wide_rows(a.base, a.d) ? k_prune_reverse<W, P1, false, true>
                                     : k_prune_reverse<W, P1, false, false>;
  if constexpr (P1)
    if (a.norms) kern = k_prune_reverse<W, P1, true, true>;
  kern<<<grid, 32 * W, 0, st>>>(a, static_cast<uint32_t>(look));
  return cudaGetLastError();
}

cudaError_t launch_prune_reverse(const PruneArgs& a, bool phase1, int num_sms, cudaStream_t st) {
  if (a.c <= 32) return phase1 ? launch_prune_w<1, true>(a, num_sms, st)
                               : launch_prune_w<1, false>(a, num_sms, st);
  if (a.c <= 64) return phase1 ? launch_prune_w<2, true>(a, num_sms, st)
                               : launch_prune_w<2, false>(a, num_sms, st);
  return phase1 ? launch_prune_w<4, true>(a, num_sms, st)
                : launch_prune_w<4, false>(a, num_sms, st);
}

cudaError_t launch_reverse_csr(const uint32_t* pruned, const uint32_t* pruned_num, uint32_t p_len,
                               uint64_t n, uint32_t* indeg, uint32_t* offs,
                               uint32_t* tile_sums, uint32_t* cursor, uint32_t* edges,
                               int num_sms, cudaStream_t st, uint64_t rows,
                               const uint32_t* order, const float* pruned_dist) {
  if (rows == 0) rows = n;
  if (n <= kScanSmall) {
    k_scan_small<<<1, kScanThreads, 0, st>>>(indeg, static_cast<uint32_t>(n), offs, cursor);
  } else {
    const uint32_t tiles = static_cast<uint32_t>((n + kScanTile - 1) / kScanTile);
    k_scan_tiles<<<tiles, kScanThreads, 0, st>>>(indeg, n, tile_sums);
    k_scan_tile_sums<<<1, kScanThreads, 0, st>>>(tile_sums, tiles, offs + n);
    k_scan_apply<<<tiles, kScanThreads, 0, st>>>(indeg, n, tile_sums, offs, cursor);
  }
  auto scatter = pruned_dist ? k_scatter_reverse<true> : k_scatter_reverse<false>;
  scatter<<<grid_for(rows, 256, num_sms, 8), 256, 0, st>>>(pruned, pruned_num, pruned_dist, p_len,
                                                           rows, offs, cursor, edges, order);
  return cudaGetLastError();
}

cudaError_t launch_reverse_lists(const uint32_t* offs, const uint32_t* edges, uint64_t n,
                                 uint32_t r, uint32_t* rev, uint32_t* rev_num, int num_sms,
                                 cudaStream_t st, const uint32_t* place, float* rev_dist) {
  auto lists = rev_dist ? k_reverse_lists<true> : k_reverse_lists<false>;
  lists<<<grid_for(n, 8, num_sms, 8), 256, 0, st>>>(offs, edges, n, r, rev, rev_dist, rev_num,
                                                    place);
  return cudaGetLastError();
}

// 16-byte words from src to dst by the SMs (host memory mapped into the device address space
// on one side): each thread moves four words per pass, so that every SM keeps many requests in
// flight over the CPU-GPU link.
__global__ void __launch_bounds__(256) k_copy16(uint4* __restrict__ dst,
                                                const uint4* __restrict__ src, uint64_t words) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < words; i += 4 * stride) {
    const uint4 v0 = src[i], v1 = src[i + stride], v2 = src[i + 2 * stride],
                v3 = src[i + 3 * stride];
    dst[i] = v0;
    dst[i + stride] = v1;
    dst[i + 2 * stride] = v2;
    dst[i + 3 * stride] = v3;
  }
  for (; i < words; i += stride) dst[i] = src[i];
}

cudaError_t launch_copy16(void* dst, const void* src, uint64_t bytes, int num_sms,
                          cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  if ((bytes % 16) != 0 || (reinterpret_cast<uintptr_t>(dst) % 16) != 0 ||
      (reinterpret_cast<uintptr_t>(src) % 16) != 0)
    return cudaErrorInvalidValue;
  k_copy16<<<static_cast<unsigned>(num_sms) * 4, 256, 0, st>>>(
      static_cast<uint4*>(dst), static_cast<const uint4*>(src), bytes / 16);
  return cudaGetLastError();
}

template <bool SCREEN, bool WIDE>
static cudaError_t launch_merge(const MergeArgs& a, int num_sms, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(a.queue, 0, 8, st);
  if (e != cudaSuccess) return e;
  k_merge_prune<SCREEN, WIDE>
      <<<grid_for(a.n, kMergeWarps, num_sms, 8), 32 * kMergeWarps, 0, st>>>(a);
  if (a.r + a.p > 32)
    k_merge_long<SCREEN, WIDE><<<grid_for(a.n, 1, num_sms, 16), 128, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_merge_prune(const MergeArgs& a, int num_sms, cudaStream_t st) {
  if (a.norms) return launch_merge<true, true>(a, num_sms, st);
  return wide_rows(a.base, a.d) ? launch_merge<false, true>(a, num_sms, st)
                                : launch_merge<false, false>(a, num_sms, st);
}

}  // namespace pg
