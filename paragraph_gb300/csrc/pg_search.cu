// pg_search.cu -- beam search with every base point as the query (K4/K8).
//
// Semantics of link_process_v0_store_base_data (Gsearcher.cuh:890-1066): list of L = Km + Kp*Kd
// (distance, id); seeds (seed_base + i) % n in slots Km.., Km slots at FLT_MAX; sort; visited set
// = the top Km; loop { pick the first Kp unexplored of the top Km (collect_top_p_normal,
// Gsearcher.cuh:75-106) and mark them; read their first Kd graph neighbours; score each new id
// (visited or repeated ids get FLT_MAX); sort; every reset_iter iterations rebuild the visited set
// from the top Km }.  Output: all L ids with the parent bit cleared.
//
// GB300 design, one warp per query, persistent warps pulling queries from a work counter:
//   * the sorted top Km lives in registers (Km/32 slots, element i = lane i%32, slot i/32) as
//     32-bit ordered distances and ids; new candidates are merged into it by rank (ballot/popc),
//     which gives the stable order of the reference, ties going to the lower list position;
//   * the visited set is an exact open-addressing table in shared memory (Ghashtable semantics);
//   * the rows of the new candidates are read straight from global memory: eight lanes cover one
//     row with 16-byte loads, four rows per warp-wide load, up to eight rows in flight;
//   * distances keep the reference's FP32 order exactly: residue r = i mod 32 accumulates
//     q[i]*x[i] in i order, then the shuffle-down tree 16,8,4,2,1.  Lane m of a group owns
//     residues 4m..4m+3, and a transposed butterfly (xor 4, 2, 1 + two in-register adds) forms
//     exactly that tree.
#include "pg_device.cuh"
#include "pg_kernels.h"

namespace pg {

namespace {

__device__ __forceinline__ uint32_t hslot(uint32_t key, uint32_t mask) {
  uint32_t h = key * 0x9E3779B1u;
  h ^= h >> 16;
  return h & mask;
}

__device__ __forceinline__ void hash_insert(uint32_t* t, uint32_t mask, uint32_t key) {
  uint32_t s = hslot(key, mask);
  for (uint32_t probe = 0; probe <= mask; probe++) {
    const uint32_t old = atomicCAS(t + s, 0u, key + 1);
    if (old == 0 || old == key + 1) return;
    s = (s + 1) & mask;
  }
}

// Inserts key unless present, in one probe sequence; true when it was absent
// (warp_level_test_and_set, Ghashtable.cuh:39-64).  The lanes of a warp insert distinct keys, so
// a concurrent claim of a slot by another lane only moves the probe on.
__device__ __forceinline__ bool hash_test_and_set(uint32_t* t, uint32_t mask, uint32_t key) {
  uint32_t s = hslot(key, mask);
  for (uint32_t probe = 0; probe <= mask; probe++) {
    const uint32_t old = atomicCAS(t + s, 0u, key + 1);
    if (old == 0) return true;
    if (old == key + 1) return false;
    s = (s + 1) & mask;
  }
  return false;  // cannot happen: the table has at least 1.6 times the slots of the ids it ever holds
}

__device__ __forceinline__ void hash_clear(uint32_t* t, uint32_t slots) {
  uint4* t4 = reinterpret_cast<uint4*>(t);
  for (uint32_t i = lane_id(); i < (slots >> 2); i += 32) t4[i] = make_uint4(0, 0, 0, 0);
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// What bounds the search: issue slots and the latency of each iteration's chain (list -> graph row
// -> visited set -> candidate rows -> merge), with L2 behind the row loads (DRAM where a large base is
// not relocated, and for queries not asked before).  Hence few instructions per iteration and many
// resident warps:
//   * rows come by plain coalesced loads.  One cp.async.bulk per row into shared memory (the
//     earlier scheme) is issued lane by lane and held 6-16 KB of shared memory per warp;
//   * 32-bit keys, one pass over the entering candidates only, and the same ranks for the output
//     instead of two 64-element sorting networks per query;
//   * registers held to about 80 (20-24 warps per SM) where there are queries for that many; for rows
//     over 256 floats the query stays in shared memory.
// Both rounds on the caller's rows, 1M x 200, Km = 32: 25.5 + 22.5 -> 18.2 + 15.1 ms; 400k x 512,
// Km = 32: 6.6 + 10.6 -> 1.4 + 5.8 ms; 200k x 128, Km = 96: 16 + 12.6 -> 10.2 + 7.8 ms; 300k x 512,
// Km = 64: 38 + 59.4 -> 23.3 + 58.5 ms (DRAM-bound; on relocated rows 16.9 + 27.7).
namespace {

// The query row of the lane's residues, in registers (KSTEPS <= 8) or in shared memory
// (kQueryShared): lane m = lane % 8 of every group reads float4 32k + 4m.
template <int KSTEPS>
constexpr bool kQueryShared = KSTEPS > 8;

template <int KSTEPS>
struct Query {
  float4 v[kQueryShared<KSTEPS> ? 1 : KSTEPS];
  const float4* s;  // kQueryShared: KSTEPS x 8 float4
  __device__ __forceinline__ float4 at(int k, uint32_t m) const {
    if constexpr (kQueryShared<KSTEPS>)
      return s[8 * k + m];
    else
      return v[k];
  }
  __device__ __forceinline__ void load(const float* qrow, uint32_t d, float4* smem) {
    const uint32_t lane = lane_id(), m = lane & 7u;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (kQueryShared<KSTEPS>) {
      s = smem;
#pragma unroll
      for (int i = 0; i < (KSTEPS + 3) / 4; i++) {
        const uint32_t at = 32u * i + lane;
        smem[at] = 4u * at < d ? __ldg(reinterpret_cast<const float4*>(qrow) + at) : zero;
      }
      __syncwarp();
    } else {
#pragma unroll
      for (int k = 0; k < KSTEPS; k++) {
        const uint32_t off = 32u * k + 4u * m;
        v[k] = off < d ? __ldg(reinterpret_cast<const float4*>(qrow + off)) : zero;
      }
    }
  }
};

// How many queries a launch has for each SM, which decides how many registers a warp may take for
// rows in flight.  A call with few queries lasts as long as its longest chain of row reads, so a warp
// that shares its SM with few others takes more of them.
enum class Load : int { kMany, kMid, kMidLong, kFew };

// Rows per pass.  kMany: eight short rows (up to 256 floats) whole in flight, four long ones with
// half of each in flight, or four where eight would spill (short rows past 224 floats, Km > 32: 3745
// -> 2711 us for 39k queries, Km = 64).  Long rows, eight at a time with a quarter in flight: 4864
// queries x 512, Km = 64: 1518 -> 1054 us, and 300k x 512 builds' searches 19.7 + 30.9 -> 16.9 + 27.7
// ms.  kFew: 16 short or 8 long rows whole in flight (608 queries x 512, Km = 64: 601 -> 411 us).
// Between them eight: whole, or long ones halved where sixteen warps share an SM.
constexpr int search_rows(int km_s, int ksteps, Load load) {
  if (load == Load::kFew) return ksteps > 8 ? 8 : 16;
  if (load != Load::kMany) return 8;
  return ksteps > 8 || (ksteps == 8 && km_s > 1) ? 4 : 8;
}

// Steps of 32 floats whose loads are in flight together.
constexpr int load_steps(int ksteps, Load load) {
  return ksteps > 8 && (load == Load::kMany || load == Load::kMid) ? 8 : ksteps;
}

// Warps per SM that the registers are allocated for.  kMany: the fastest of 16..32; one more or less
// costs 1-3%, 16 or 32 cost 10-30% (too few warps, or spills).  The others hold one resident round of
// the launches that take them.
constexpr int search_warps(int km_s, int ksteps, Load load) {
  if (load == Load::kFew) return 8;
  if (load == Load::kMidLong) return 12;
  if (load == Load::kMid) return 16;
  return ksteps > 8 ? 24 : km_s == 1 ? 23 : ksteps == 8 ? 20 : 21;
}

// The lines of a row to L2, without waiting for them.
__device__ __forceinline__ void prefetch_l2(const float* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Scores rows list[c0 .. c0 + 4R) (R rounds of four rows, one per 8-lane group; entries past the
// last repeat it).  Lane (g, m) accumulates residues 4m..4m+3 of rows c0 + 4r + g (the
// reference's lane-strided FMA chains), straight from global memory: one warp-wide load reads
// four 128-byte row segments.  The first log2(R) butterfly levels are transposed (each lane keeps
// one row), the others plain xor reductions.  Row c0 + 4r + g ends up in lane 8g + m(r).
template <int KSTEPS, int R, Load LOAD, class Ahead>
__device__ __forceinline__ float score_rows(const float* __restrict__ base, uint32_t d,
                                            const Query<KSTEPS>& q, const uint32_t* list,
                                            uint32_t c0, uint32_t last, Ahead ahead) {
  const uint32_t lane = lane_id(), g = lane >> 3, m = lane & 7u;
  const float* row[R];
#pragma unroll
  for (int r = 0; r < R; r++)
    row[r] = base + static_cast<uint64_t>(list[min(c0 + 4u * r + g, last)]) * d + 4u * m;
  float p[R][4];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int i = 0; i < 4; i++) p[r][i] = 0.0f;
  constexpr int KB = load_steps(KSTEPS, LOAD);
#pragma unroll
  for (int k0 = 0; k0 < KSTEPS; k0 += KB) {
    float4 x[R][KB];
#pragma unroll
    for (int k = 0; k < KB && k0 + k < KSTEPS; k++)
#pragma unroll
      for (int r = 0; r < R; r++)
        x[r][k] = 32u * (k0 + k) + 4u * m < d
                      ? __ldg(reinterpret_cast<const float4*>(row[r] + 32 * (k0 + k)))
                      : make_float4(0.f, 0.f, 0.f, 0.f);
    if (k0 == 0) ahead();
#pragma unroll
    for (int k = 0; k < KB && k0 + k < KSTEPS; k++) {
      if (32u * (k0 + k) + 4u * m < d) {
        const float4 u = q.at(k0 + k, m);
#pragma unroll
        for (int r = 0; r < R; r++) {
          p[r][0] = fmaf(u.x, x[r][k].x, p[r][0]);
          p[r][1] = fmaf(u.y, x[r][k].y, p[r][1]);
          p[r][2] = fmaf(u.z, x[r][k].z, p[r][2]);
          p[r][3] = fmaf(u.w, x[r][k].w, p[r][3]);
        }
      }
    }
  }
  const bool bA = (m & 4u) != 0, bB = (m & 2u) != 0;
  float v[4];
  // levels xor 4, 2, 1 add residues +16, +8, +4
  if constexpr (R == 1) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float t = p[0][j];
      t = t + __shfl_xor_sync(kFull, t, 4);
      t = t + __shfl_xor_sync(kFull, t, 2);
      v[j] = t + __shfl_xor_sync(kFull, t, 1);
    }
  } else {
    float w[R / 2][4];
#pragma unroll
    for (int i = 0; i < R / 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float send = bA ? p[i][j] : p[i + R / 2][j];
        const float keep = bA ? p[i + R / 2][j] : p[i][j];
        w[i][j] = keep + __shfl_xor_sync(kFull, send, 4);
      }
    if constexpr (R == 2) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float t = w[0][j];
        t = t + __shfl_xor_sync(kFull, t, 2);
        v[j] = t + __shfl_xor_sync(kFull, t, 1);
      }
    } else {
      static_assert(R == 4, "1, 2 or 4 rounds");
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float send = bB ? w[0][j] : w[1][j];
        const float keep = bB ? w[1][j] : w[0][j];
        const float t = keep + __shfl_xor_sync(kFull, send, 2);
        v[j] = t + __shfl_xor_sync(kFull, t, 1);
      }
    }
  }
  return (v[0] + v[2]) + (v[1] + v[3]);
}

// Distances of the lanes whose `newc` is set (FLT_MAX elsewhere), up to ROWS rows per pass.
template <int KSTEPS, int ROWS, Load LOAD>
__device__ __forceinline__ float score_new(const SearchArgs& a, const Query<KSTEPS>& q,
                                           uint32_t node, bool newc, uint32_t* list) {
  const uint32_t lane = lane_id();
  const unsigned newmask = __ballot_sync(kFull, newc);
  const uint32_t nnew = __popc(newmask);
  const uint32_t ci = __popc(newmask & ((1u << lane) - 1u));
  if (newc) list[ci] = node;
  __syncwarp();
  float result = FLT_MAX;
  for (uint32_t c0 = 0; c0 < nnew; c0 += ROWS) {
    const uint32_t left = nnew - c0;
    // The rows of the next pass to L2 while this one's are on their way.  The branch also keeps the
    // compiler from moving loads between the FMAs, to save registers that these kernels have: without it
    // 2432 queries x 512, Km = 32, took 745 instead of 334 us.
    auto ahead = [&]() {
      if constexpr (LOAD != Load::kMany && KSTEPS > 8) {
        constexpr uint32_t T = 32 / ROWS;  // lanes per row
        const uint32_t c = c0 + ROWS + lane / T;
        if (a.prefetch && c < nnew) {
          const float* row = a.base + static_cast<uint64_t>(list[c]) * a.d;
          for (uint32_t i = 32u * (lane % T); i < a.d; i += 32u * T) prefetch_l2(row + i);
          if (lane % T == T - 1) prefetch_l2(row + a.d - 1);  // a row that starts inside a line
        }
      }
    };
    const uint32_t lc = ci - c0, r = lc >> 2;
    float total = 0.0f;
    uint32_t src = (lc & 3u) << 3;
    if (ROWS == 4 || left <= 4) {
      total = score_rows<KSTEPS, 1, LOAD>(a.base, a.d, q, list, c0, nnew - 1, ahead);
    } else if (ROWS <= 8 || left <= 8) {
      total = score_rows<KSTEPS, 2, LOAD>(a.base, a.d, q, list, c0, nnew - 1, ahead);
      src |= (r & 1u) << 2;
    } else if constexpr (ROWS == 16) {
      total = score_rows<KSTEPS, 4, LOAD>(a.base, a.d, q, list, c0, nnew - 1, ahead);
      src |= ((r >> 1) & 1u) << 2 | (r & 1u) << 1;
    }
    const float dd = __shfl_sync(kFull, total, src & 31u);
    if (newc && ci >= c0 && lc < ROWS) result = -dd;
  }
  __syncwarp();  // the list is rewritten by the next call
  return result;
}

}  // namespace

template <int KM_S, int KSTEPS, Load LOAD>
__device__ __forceinline__ void search_queries(const SearchArgs& a) {
  constexpr uint32_t KM = 32u * KM_S;
  constexpr int ROWS = search_rows(KM_S, KSTEPS, LOAD);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t lane = lane_id();
  uint2* merged = reinterpret_cast<uint2*>(smem_raw);                // KM (key, id)
  uint32_t* list = reinterpret_cast<uint32_t*>(smem_raw + 8 * KM);   // 32 new candidates
  uint32_t* hash = reinterpret_cast<uint32_t*>(smem_raw + 8 * KM + 128);
  float4* qs = reinterpret_cast<float4*>(smem_raw + 8 * KM + 128 + 4u * a.hash_slots);
  const uint32_t hmask = a.hash_slots - 1u;
  const uint32_t kp = a.kp, kd = a.kd;
  const uint32_t e_of_lane = lane / kd, nb_of_lane = lane % kd;
  const unsigned lt_mask = (1u << lane) - 1u;
  const uint32_t kmax = order_key(FLT_MAX);
  unsigned long long ev = 0, it_all = 0;

  for (;;) {
    uint32_t qi = 0;
    if (lane == 0) qi = atomicAdd(a.work, 1u);
    qi = __shfl_sync(kFull, qi, 0);
    if (qi >= (a.queries ? a.nq : a.n)) break;
    const uint32_t qid = qi;
    const float* qrow = (a.queries ? a.queries : a.base) + static_cast<uint64_t>(qid) * a.d;
    Query<KSTEPS> q;
    q.load(qrow, a.d, qs);
    // The list is the sorted top (keys ascending, entry i = 32 s + lane) before the last merge,
    // then the last candidates in lane order: keys are order_key(distance), ties go to the lower
    // position, so a retained entry precedes a candidate of the same distance.
    uint32_t top_key[KM_S], top_id[KM_S], cur_key[KM_S], cur_id[KM_S];
#pragma unroll
    for (int s = 0; s < KM_S; s++) {
      top_key[s] = kmax;
      top_id[s] = kTomb;
    }
    uint32_t cand_key, cand_id;
    bool newc = true;
    {  // seeds: every slot is scored (Gsearcher.cuh:958-976 has no visited test)
      uint64_t soff = 0, sn = a.n;  // entry points are drawn inside the query's sub-index
      if (a.seg_count) {
        const uint32_t sg = segment_of(a.seg_off, a.seg_count, qid);
        soff = a.seg_off[sg];
        sn = a.seg_off[sg + 1] - soff;
      }
      cand_id = static_cast<uint32_t>((a.seed_base + static_cast<uint64_t>(lane)) % sn + soff);
      if (a.place) cand_id = a.place[cand_id];
      // scored for every query at once by k_seed_dists, or here
      const float dist = a.seed_dist ? a.seed_dist[static_cast<uint64_t>(qid) * 32u + lane]
                                     : score_new<KSTEPS, ROWS, LOAD>(a, q, cand_id, true, list);
      cand_key = order_key(dist);
      ev += (lane == 0) ? 32u : 0u;
    }
    {  // the first top: the seeds below FLT_MAX in (distance, lane) order, then empty slots
      uint64_t k1[1] = {(static_cast<uint64_t>(cand_key) << 32) | lane};
      uint32_t i1[1] = {cand_id};
      warp_sort_kv<1>(k1, i1);
      const uint32_t k = static_cast<uint32_t>(k1[0] >> 32);
      cur_key[0] = k < kmax ? k : kmax;
      cur_id[0] = k < kmax ? i1[0] : kTomb;
#pragma unroll
      for (int s = 1; s < KM_S; s++) {
        cur_key[s] = kmax;
        cur_id[s] = kTomb;
      }
    }
    hash_clear(hash, a.hash_slots);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < KM_S; s++) hash_insert(hash, hmask, cur_id[s] & kMaskedTomb);
    __syncwarp();

    uint32_t iter = 0, total = 0;
    for (;;) {
      // collect_top_p_normal: the first kp unexplored of the top, marked explored; lane l reads
      // neighbour l % kd of the (l / kd)-th of them
      uint32_t ex = kTomb, before = 0;
#pragma unroll
      for (int s = 0; s < KM_S; s++) {
        const bool unexp = (cur_id[s] & kParent) == 0;
        const unsigned um = __ballot_sync(kFull, unexp);
        unsigned mm = e_of_lane >= before ? um : 0u;
        for (uint32_t i = before; i < e_of_lane; i++) mm &= mm - 1u;
        const uint32_t v =
            __shfl_sync(kFull, cur_id[s], mm ? __ffs(static_cast<int>(mm)) - 1 : 0);
        if (mm) ex = v;
        if (unexp && before + __popc(um & lt_mask) < kp) cur_id[s] |= kParent;
        before += __popc(um);
      }
      if (before == 0) break;
      if (++total > a.max_iters) {
        if (lane == 0) raise_error(a.status, kErrIterCap);
        break;  // the output is the list of the last completed merge
      }
      uint32_t node = kTomb;
      if (ex < a.n)
        node = a.graph[static_cast<uint64_t>(ex) * a.graph_degree + nb_of_lane];
      else if (ex != kTomb)
        raise_error(a.status, kErrCapacity);
      if (node >= a.n && node != kTomb) {
        raise_error(a.status, kErrBadId);
        node = kTomb;
      }
      const unsigned same = __match_any_sync(kFull, node);
      newc = node != kTomb && (same & lt_mask) == 0 && hash_test_and_set(hash, hmask, node);
      __syncwarp();
      const float dist = score_new<KSTEPS, ROWS, LOAD>(a, q, node, newc, list);
      const unsigned scored = __ballot_sync(kFull, newc);
      ev += (lane == 0) ? __popc(scored) : 0u;
#pragma unroll
      for (int s = 0; s < KM_S; s++) {
        top_key[s] = cur_key[s];
        top_id[s] = cur_id[s];
      }
      cand_key = newc ? order_key(dist) : kmax;
      cand_id = node;
      // merge by rank: only scored candidates below the current last key enter the top (one above
      // it displaces nothing and lands past the end, and every candidate below an entering one
      // enters too)
      const uint32_t worst = __shfl_sync(kFull, cur_key[KM_S - 1], 31);
      const bool enters = newc && cand_key < worst;
      const unsigned entering = __ballot_sync(kFull, enters);
      if (entering) {
        uint32_t shift[KM_S], cpos = 0;
#pragma unroll
        for (int s = 0; s < KM_S; s++) shift[s] = 0;
        for (unsigned rem = entering; rem; rem &= rem - 1u) {
          const uint32_t c = static_cast<uint32_t>(__ffs(static_cast<int>(rem)) - 1);
          const uint32_t kc = __shfl_sync(kFull, cand_key, c);
          uint32_t below = 0;
#pragma unroll
          for (int s = 0; s < KM_S; s++) {
            const bool after = top_key[s] > kc;
            below += __popc(__ballot_sync(kFull, !after));
            shift[s] += after ? 1u : 0u;
          }
          cpos += (lane == c) ? below : (kc < cand_key || (kc == cand_key && c < lane)) ? 1u : 0u;
        }
#pragma unroll
        for (int s = 0; s < KM_S; s++) {
          const uint32_t tpos = static_cast<uint32_t>(s) * 32u + lane + shift[s];
          if (tpos < KM) merged[tpos] = make_uint2(top_key[s], top_id[s]);
        }
        if (enters && cpos < KM) merged[cpos] = make_uint2(cand_key, cand_id);
        __syncwarp();
#pragma unroll
        for (int s = 0; s < KM_S; s++) {
          const uint2 e = merged[static_cast<uint32_t>(s) * 32u + lane];
          cur_key[s] = e.x;
          cur_id[s] = e.y;
        }
        __syncwarp();
      }
      if (++iter == a.reset_iter) {
        hash_clear(hash, a.hash_slots);
        __syncwarp();
#pragma unroll
        for (int s = 0; s < KM_S; s++) hash_insert(hash, hmask, cur_id[s] & kMaskedTomb);
        __syncwarp();
        iter = 0;
      }
    }
    it_all += (lane == 0) ? total : 0u;
    // The output is the whole list sorted: the same ranks over all scored candidates.  The others
    // hold FLT_MAX, at or after every retained entry, and follow in lane order -- unless a scored
    // distance is not below FLT_MAX, when every candidate is ranked.
    unsigned ranked = __ballot_sync(kFull, newc);
    if (__any_sync(kFull, newc && cand_key >= kmax)) ranked = kFull;
    const bool mine = (ranked >> lane) & 1u;
    uint32_t shift[KM_S];
    uint32_t cpos = mine ? 0u : KM + __popc(ranked) + __popc(~ranked & lt_mask);
#pragma unroll
    for (int s = 0; s < KM_S; s++) shift[s] = 0;
    for (unsigned rem = ranked; rem; rem &= rem - 1u) {
      const uint32_t c = static_cast<uint32_t>(__ffs(static_cast<int>(rem)) - 1);
      const uint32_t kc = __shfl_sync(kFull, cand_key, c);
      uint32_t below = 0;
#pragma unroll
      for (int s = 0; s < KM_S; s++) {
        const bool after = top_key[s] > kc;
        below += __popc(__ballot_sync(kFull, !after));
        shift[s] += after ? 1u : 0u;
      }
      if (mine)
        cpos += (lane == c) ? below : (kc < cand_key || (kc == cand_key && c < lane)) ? 1u : 0u;
    }
    uint32_t* orow = a.out + static_cast<uint64_t>(qid) * a.out_width;
#pragma unroll
    for (int s = 0; s < KM_S; s++) {
      const uint32_t tpos = static_cast<uint32_t>(s) * 32u + lane + shift[s];
      if (tpos < a.out_width) orow[tpos] = top_id[s] & kMaskedTomb;
    }
    if (cpos < a.out_width) orow[cpos] = cand_id & kMaskedTomb;
    if (a.out_key) {  // for launch_list_dists: only stores here, since more code in this place made
                      // the search loop's registers spill (300k x 512: 27.7 -> 32.5 ms)
      uint32_t* krow = a.out_key + static_cast<uint64_t>(qid) * a.out_width;
#pragma unroll
      for (int s = 0; s < KM_S; s++) {
        const uint32_t tpos = static_cast<uint32_t>(s) * 32u + lane + shift[s];
        if (tpos < a.out_width) krow[tpos] = top_key[s];
      }
      if (cpos < a.out_width) krow[cpos] = newc ? cand_key : kNoKey;
    }
  }
  if (lane == 0) {
    if (ev) atomicAdd(a.evals, ev);
    if (it_all) atomicAdd(a.iters, it_all);
  }
}

template <int KSTEPS, Load LOAD>
__global__ void __launch_bounds__(32, search_warps(1, KSTEPS, LOAD)) k_search_m32(SearchArgs a) {
  search_queries<1, KSTEPS, LOAD>(a);
}

// Km = 64, 96
template <int KM_S, int KSTEPS, Load LOAD>
__global__ void __launch_bounds__(32, search_warps(KM_S, KSTEPS, LOAD)) k_search_mk(SearchArgs a) {
  search_queries<KM_S, KSTEPS, LOAD>(a);
}

// Per warp: the merge buffer, the list of new candidates, the visited set and, for long rows, the
// query.
size_t search_smem(uint32_t km, uint32_t hash_slots, int ksteps, bool qshared) {
  return 8 * static_cast<size_t>(km) + 128 + 4 * static_cast<size_t>(hash_slots) +
         (qshared ? static_cast<size_t>((ksteps + 3) / 4 * 4) * 128 : 0);
}

template <int KM_S, int KS, Load LOAD>
static cudaError_t launch_search_k(const SearchArgs& a, int num_sms, size_t smem_optin,
                                   cudaStream_t st) {
  const size_t smem = search_smem(32u * KM_S, a.hash_slots, KS, kQueryShared<KS>);
  if (smem > smem_optin) return cudaErrorInvalidValue;
  void (*kern)(SearchArgs);
  if constexpr (KM_S == 1)
    kern = k_search_m32<KS, LOAD>;
  else
    kern = k_search_mk<KM_S, KS, LOAD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32, smem);
  if (e != cudaSuccess) return e;
  if (a.max_blocks_per_sm && per_sm > static_cast<int>(a.max_blocks_per_sm))
    per_sm = static_cast<int>(a.max_blocks_per_sm);
  if (per_sm < 1) per_sm = 1;
  uint64_t blocks = static_cast<uint64_t>(num_sms) * per_sm;
  const uint64_t nq = a.queries ? a.nq : a.n;
  if (blocks > nq) blocks = nq;
  kern<<<static_cast<unsigned>(blocks), 32, smem, st>>>(a);
  return cudaGetLastError();
}

// The distances of every query to its 32 seeds ((seed_base + s) % n_sub + offset), in the
// search's FP32 order (Gsearcher.cuh:958-976): residue r = i mod 32 accumulates q[i]*x[i] in i
// order, then the shuffle-down tree 16, 8, 4, 2, 1.  Lane s holds seed s's 32 residue chains of
// kSeedQ queries in registers and folds them in the tree's pairs.  The seeds of one (sub-)index
// are the same 32 rows for every query: a block stages them in shared memory (row stride an odd
// number of float4, so the 32 lanes read their rows without bank conflicts) and keeps them for
// its whole range of queries, whose rows stream through two shared tiles filled one tile ahead.
// Per float4 step a warp takes one shared load of seeds (four wavefronts) and kSeedQ broadcast
// loads for 4 kSeedQ FMAs.
constexpr int kSeedQ = 4;
constexpr uint32_t kSeedWarps = 8;
constexpr uint32_t kSeedTile = kSeedWarps * kSeedQ;  // queries per tile

__host__ __device__ __forceinline__ uint32_t seed_stride4(uint32_t d) { return (d / 4) | 1u; }

__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

template <bool KEYS>
__global__ void __launch_bounds__(32 * kSeedWarps) k_seed_dists(SearchArgs a,
                                                                float* __restrict__ out,
                                                                uint32_t* __restrict__ keys,
                                                                uint32_t* __restrict__ bins,
                                                                uint32_t seg_keys) {
  extern __shared__ __align__(16) float4 seeds4[];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint64_t nq = a.queries ? a.nq : a.n;
  const uint32_t d = a.d, d4 = d / 4, stride = seed_stride4(d);
  float4* tiles = seeds4 + 32u * stride;  // two tiles of kSeedTile rows
  const float4* rows = reinterpret_cast<const float4*>(a.queries ? a.queries : a.base);
  const uint64_t tiles_all = (nq + kSeedTile - 1) / kSeedTile;
  const uint64_t per = (tiles_all + gridDim.x - 1) / gridDim.x * kSeedTile;
  const uint64_t end = min(nq, per * (blockIdx.x + 1));
  for (uint64_t q0 = per * blockIdx.x; q0 < end;) {
    uint64_t soff = 0, sn = a.n, stop = end;  // this block's queries of one sub-index
    uint32_t sg = 0;
    if (a.seg_count) {
      sg = segment_of(a.seg_off, a.seg_count, q0);
      soff = a.seg_off[sg];
      sn = a.seg_off[sg + 1] - soff;
      stop = min(end, soff + sn);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 32u * d4; i += blockDim.x) {
      const uint32_t r = i / d4, c = i - r * d4;
      const uint64_t node = (a.seed_base + static_cast<uint64_t>(r)) % sn + soff;
      seeds4[r * stride + c] = __ldg(reinterpret_cast<const float4*>(a.base + node * d) + c);
    }
    auto fill = [&](uint64_t t0, uint32_t buf) {  // a tile is one contiguous range
      if (t0 < stop) {
        const uint32_t words = static_cast<uint32_t>(min(stop - t0, uint64_t(kSeedTile))) * d4;
        float4* dst = tiles + buf * kSeedTile * d4;
        const float4* src = rows + t0 * d4;
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) cp16(dst + i, src + i);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint32_t buf = 0;
    fill(q0, 0);
    const float4* x4 = seeds4 + lane * stride;
    for (uint64_t t0 = q0; t0 < stop; t0 += kSeedTile, buf ^= 1u) {
      fill(t0 + kSeedTile, buf ^ 1u);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      const float4* q4 = tiles + (buf * kSeedTile + warp * kSeedQ) * d4;
      const uint64_t qb = t0 + warp * kSeedQ;
      if (qb < stop) {
        float s[kSeedQ][32];  // rows past the end hold an earlier tile's or no data: not written
#pragma unroll
        for (int t = 0; t < kSeedQ; t++)
#pragma unroll
          for (int r = 0; r < 32; r++) s[t][r] = 0.f;
        auto step = [&](uint32_t b, uint32_t j) {
          const float4 x = x4[b + j];
#pragma unroll
          for (int t = 0; t < kSeedQ; t++) {
            const float4 q = q4[t * d4 + b + j];
            s[t][4 * j] = fmaf(q.x, x.x, s[t][4 * j]);
            s[t][4 * j + 1] = fmaf(q.y, x.y, s[t][4 * j + 1]);
            s[t][4 * j + 2] = fmaf(q.z, x.z, s[t][4 * j + 2]);
            s[t][4 * j + 3] = fmaf(q.w, x.w, s[t][4 * j + 3]);
          }
        };
        uint32_t b = 0;
#pragma unroll 1
        for (; b + 8 <= d4; b += 8) {
#pragma unroll
          for (uint32_t j = 0; j < 8; j++) step(b, j);
        }
#pragma unroll
        for (uint32_t j = 0; j < 8; j++)
          if (b + j < d4) step(b, j);
#pragma unroll
        for (int t = 0; t < kSeedQ; t++) {
#pragma unroll
          for (int w = 16; w >= 1; w >>= 1)
#pragma unroll
            for (int r = 0; r < w; r++) s[t][r] = s[t][r] + s[t][r + w];
          if (qb + t >= stop) continue;
          const float dist = -s[t][0];
          out[(qb + t) * 32u + lane] = dist;
          if (KEYS) {  // nearest and second nearest seed
            const uint32_t k = order_key(dist);
            const uint32_t first = __reduce_min_sync(kFull, k);
            const uint32_t l1 = __ffs(static_cast<int>(__ballot_sync(kFull, k == first))) - 1;
            const uint32_t k2 = lane == l1 ? 0xFFFFFFFFu : k;
            const uint32_t second = __reduce_min_sync(kFull, k2);
            const uint32_t l2 = __ffs(static_cast<int>(__ballot_sync(kFull, k2 == second))) - 1;
            if (lane == 0) {
              const uint32_t key = sg * seg_keys + (seg_keys == 32 ? l1 : l1 * 32u + l2);
              keys[qb + t] = key;
              atomicAdd(bins + key, 1u);
            }
          }
        }
      }
      __syncthreads();  // the tile is overwritten two fills later
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    q0 = stop;
  }
}

// Keys per sub-index: nearest and second nearest seed, or the nearest alone when many sub-indexes
// would make the table of counts large.
static uint32_t keys_per_segment(uint32_t seg_count) { return seg_count <= 64 ? 1024u : 32u; }

cudaError_t launch_seed_dists(const SearchArgs& a, float* out, uint32_t* keys, uint32_t* bins,
                              int num_sms, size_t smem_optin, cudaStream_t st) {
  if (a.d == 0 || (a.d % 4) != 0 || !out) return cudaErrorInvalidValue;
  const uint64_t nq = a.queries ? a.nq : a.n;
  if (nq == 0) return cudaSuccess;
  const size_t smem = 32 * static_cast<size_t>(seed_stride4(a.d)) * 16 +
                      2 * kSeedTile * static_cast<size_t>(a.d) * 4;
  if (smem > smem_optin) return cudaErrorInvalidValue;
  auto kern = keys ? k_seed_dists<true> : k_seed_dists<false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kSeedWarps, smem);
  if (e != cudaSuccess) return e;
  uint64_t blocks = (nq + kSeedTile - 1) / kSeedTile;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * (per_sm < 1 ? 1 : per_sm);
  if (blocks > cap) blocks = cap;
  kern<<<static_cast<unsigned>(blocks), 32 * kSeedWarps, smem, st>>>(
      a, out, keys, bins, keys_per_segment(a.seg_count));
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Relocation.  A point's lists hold points near it, and points near each other share their nearest
// seeds.  Working on a copy of the base sorted by (nearest, second nearest seed) puts the rows that
// neighbouring warps gather next to each other: fewer DRAM rows, fewer address translations, more
// cache hits.  Nothing in the search or the prunes depends on the numbering (ties go by position);
// the reverse lists, which keep the first sources by id, are sorted by original id.
// Whole builds on the caller's rows -> relocated: 1M x 512 cosine (L = 96) 758 -> 491 ms,
// 300k x 512 199 -> 147, 1M x 200 72.3 -> 69.5, 100k x 200 8.80 -> 8.53, 50k x 200 4.97 -> 4.81,
// 20k x 200 2.53 -> 2.57, 10k x 512 4.33 -> 4.53: below 32 MB the base stays in L2 and the extra
// passes cost more than they give.  The copy doubles the base's memory, so it stops at 32 GB (and
// where the workspace cannot be allocated).
uint32_t reloc_keys(uint64_t n, uint32_t d, uint32_t seg_count) {
  constexpr uint64_t kMin = 32ull << 20, kMax = 32ull << 30;  // bytes of the base
  if (n * d * 4 < kMin || n * d * 4 > kMax || seg_count > 2048) return 0;
  const uint32_t k = (seg_count ? seg_count : 1u) * keys_per_segment(seg_count);
  return (k + 1023u) / 1024u * 1024u;
}

// Counts -> starting places, in place (one block; count a multiple of 1024).
__global__ void __launch_bounds__(1024) k_reloc_starts(uint32_t* __restrict__ bins,
                                                       uint32_t count) {
  __shared__ uint32_t ws[32];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < count; b0 += 1024) {
    const uint32_t v = bins[b0 + threadIdx.x];
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, o);
      if (lane >= static_cast<uint32_t>(o)) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    const uint32_t w = ws[lane];
    uint32_t all = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, all, o);
      if (lane >= static_cast<uint32_t>(o)) all += y;
    }
    const uint32_t before = __shfl_sync(kFull, all - w, static_cast<int>(warp));
    bins[b0 + threadIdx.x] = carry + before + x - v;
    carry += __shfl_sync(kFull, all, 31);
    __syncthreads();
  }
}

__global__ void k_reloc_place(const uint32_t* __restrict__ keys, uint64_t n,
                              uint32_t* __restrict__ cursor, uint32_t* __restrict__ order,
                              uint32_t* __restrict__ place) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    const uint32_t at = atomicAdd(cursor + keys[i], 1u);
    order[at] = static_cast<uint32_t>(i);
    place[i] = at;
  }
}

// One warp per row: d / 4 + 8 float4 copies, coalesced on both sides.
__global__ void __launch_bounds__(256) k_reloc_rows(const float4* __restrict__ base, uint64_t n,
                                                    uint32_t d4, const float4* __restrict__ seeds,
                                                    const uint32_t* __restrict__ order,
                                                    float4* __restrict__ out_base,
                                                    float4* __restrict__ out_seeds) {
  const uint32_t lane = lane_id();
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * 8;
  for (uint64_t i = blockIdx.x * 8ull + (threadIdx.x >> 5); i < n; i += nw) {
    const uint64_t o = order[i];
#pragma unroll 4
    for (uint32_t c = lane; c < d4; c += 32) out_base[i * d4 + c] = __ldg(base + o * d4 + c);
    if (lane < 8) out_seeds[i * 8 + lane] = __ldg(seeds + o * 8 + lane);
  }
}

cudaError_t launch_reloc_order(const uint32_t* keys, uint64_t n, uint32_t* bins, uint32_t nkeys,
                               uint32_t* order, uint32_t* place, int num_sms, cudaStream_t st) {
  k_reloc_starts<<<1, 1024, 0, st>>>(bins, nkeys);
  uint64_t blocks = (n + 255) / 256;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
  if (blocks > cap) blocks = cap;
  k_reloc_place<<<static_cast<unsigned>(blocks), 256, 0, st>>>(keys, n, bins, order, place);
  return cudaGetLastError();
}

cudaError_t launch_reloc_rows(const float* base, uint64_t n, uint32_t d, const float* seeds,
                              const uint32_t* order, float* out_base, float* out_seeds,
                              int num_sms, cudaStream_t st) {
  uint64_t blocks = (n + 7) / 8;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
  if (blocks > cap) blocks = cap;
  k_reloc_rows<<<static_cast<unsigned>(blocks), 256, 0, st>>>(
      reinterpret_cast<const float4*>(base), n, d / 4, reinterpret_cast<const float4*>(seeds),
      order, reinterpret_cast<float4*>(out_base), reinterpret_cast<float4*>(out_seeds));
  return cudaGetLastError();
}

bool search_supported(uint32_t d, uint32_t km, uint32_t kp, uint32_t kd) {
  return d > 0 && d <= 512 && (d % 4) == 0 && kp * kd == 32 && kp >= 1 && km >= 32 &&
         km <= 96 && (km % 32) == 0;
}

template <int KM_S, int KS>
static cudaError_t launch_search_load(const SearchArgs& a, Load load, int num_sms,
                                      size_t smem_optin, cudaStream_t st) {
  if (load == Load::kFew) return launch_search_k<KM_S, KS, Load::kFew>(a, num_sms, smem_optin, st);
  if constexpr (KS > 8)
    if (load == Load::kMidLong)
      return launch_search_k<KM_S, KS, Load::kMidLong>(a, num_sms, smem_optin, st);
  if (load != Load::kMany) return launch_search_k<KM_S, KS, Load::kMid>(a, num_sms, smem_optin, st);
  return launch_search_k<KM_S, KS, Load::kMany>(a, num_sms, smem_optin, st);
}

template <int KM_S>
static cudaError_t launch_search_d(const SearchArgs& a, Load load, int num_sms, size_t smem_optin,
                                   cudaStream_t st) {
  if (a.d <= 224) return launch_search_load<KM_S, 7>(a, load, num_sms, smem_optin, st);
  if (a.d <= 256) return launch_search_load<KM_S, 8>(a, load, num_sms, smem_optin, st);
  return launch_search_load<KM_S, 16>(a, load, num_sms, smem_optin, st);
}

cudaError_t launch_search(const SearchArgs& a, int num_sms, size_t smem_optin, cudaStream_t st) {
  if (!search_supported(a.d, a.km, a.kp, a.kd)) return cudaErrorInvalidValue;
  if (a.rows != 0 && a.rows != 8 && a.rows != 16) return cudaErrorInvalidValue;
  // The kernels that hold all the queries in one resident round, up to 16 per SM: a second round of few
  // queries lasts as long as the first.  Queries never asked before, by class (kFew, kMidLong, kMid,
  // kMany; us):
  //   1000 x 200, Km = 32:  119,   -, 125, 162      2432 x 200, Km = 32:  160,   -, 124, 149
  //   1300 x 512, Km = 32:  312, 312, 347, 469      2432 x 512, Km = 32:  376, 335, 358, 473
  //   1300 x 384, Km = 96:    -, 556, 559, 650      2432 x 384, Km = 96:    -, 737, 608, 694
  // Rows of up to 64 floats leave the registers of kMid unused (1300 x 64: 129, 124).  Past 16 per SM
  // kMany is faster on most graphs (3000 x 320, Km = 32: 309, 288; 400k points, 3000 x 512: 212, 185) but
  // not on all (200k points with one long chain, 3000 x 512: 360, 481).
  const uint64_t nq = a.queries ? a.nq : a.n, sms = static_cast<uint64_t>(num_sms);
  const Load load = nq <= sms * 8 || (a.rows == 16 && a.km == 32) ? Load::kFew
                    : nq > sms * 16 || a.d <= 64                 ? Load::kMany
                    : nq <= sms * 12                             ? Load::kMidLong
                                                                 : Load::kMid;
  // Few long rows: the passes of an iteration wait for each other, so rows that lie in DRAM (queries
  // not asked before) cost one DRAM latency per pass unless they are sent to L2 a pass ahead.  Km = 32,
  // new queries and the same again: 16 x 512 297 -> 277 and 232 -> 231 us, 300 x 384 228 -> 224 and 186
  // -> 194.  Up to 320 floats it cost as much as it gave, and with more than two queries per SM other
  // queries hide the latency.
  SearchArgs b = a;
  b.prefetch = a.d > 320 && nq <= sms * 2;
  switch (a.km / 32) {
    case 1: return launch_search_d<1>(b, load, num_sms, smem_optin, st);
    case 2: return launch_search_d<2>(b, load, num_sms, smem_optin, st);
    default: return launch_search_d<3>(b, load, num_sms, smem_optin, st);
  }
}

}  // namespace pg
