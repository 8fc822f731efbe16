// pg_prune_tc.cu -- screened prune + reverse (K6/K10) with the candidate Gram on the tcgen05
// tensor cores.
//
// Same result as k_prune_reverse (strict rounds), bit for bit: the RNG occlusion scan of
// fusion_prune_reverse_kernel_v0 (Gbuilder.cuh:1093-1244, scan at :1150-1199).  Every decision --
// which candidate is the nearest undecided one, whether dist(p, r) < d_p -- is taken from values
// whose distance from the reference's FP32 chain is bounded, and from the exact chain where the
// bound leaves it open.
//
// One CTA works on tiles of 128 candidate rows -- two nodes of up to 64 candidates (c <= 64) or
// one node of up to 128 -- with one thread per tile row (four warps):
//   1. the rows' 16-bit copies (launch_screen_norms) stream into a ring of S chunk stages, 64
//      columns per chunk, by 16-byte cp.async copies, eight lanes per 128-byte row segment, laid
//      out as the MMA reads them (128-byte swizzle): the data never pass through registers;
//   2. one thread issues tcgen05.mma (M = N = 128, K = 16 per instruction, FP32 accumulation)
//      for the chunk: the Gram G = A A^T of the tile's 16-bit rows accumulates in 128 TMEM
//      columns, and each node's block of G lies in the node's own TMEM lanes and columns;
//   3. the distance of each candidate to the node comes from the search, which computed it in
//      another FP32 order (launch_list_dists fills in the few it has not); the nearest undecided
//      candidate is the one whose interval lies below the others', or the exact minimum
//      (distance, slot) of those whose intervals overlap;
//   4. for each kept entry r every undecided candidate p reads G[p][r] from its own TMEM lane (one
//      tcgen05.ld column) and decides dist(p, r) < d_p from it outside the bound, or by exact
//      chains.  A candidate's recorded occluder is thus the first kept entry, in kept order, that
//      occludes it, and the kept list equals the reference's one-candidate-at-a-time scan.
// Error bounds (x, y = FP32 rows, x^ = the 16-bit x, e_x = x - x^, Cauchy-Schwarz throughout;
// the two norms per point come from launch_screen_norms, once per build):
//   |sum x^y^ - sum xy| <= |e_x|(|y| + |e_y|) + |x||e_y|
//   |MMA(x^, y^) - sum x^y^| <= c_acc (|x| + |e_x|)(|y| + |e_y|)   (FP32 accumulation of Dp terms)
//   |chain(x, y) - sum xy| <= c_seq |x||y|                          (the reference's FP32 chain)
//   |search(x, y) - sum xy| <= c_par |x||y|                         (the search's FP32 order)
// with c_acc = (Dp + 32) 2^-21 (eight times the sequential-summation bound, covering the tensor
// core's accumulation), c_seq = (D + 2) 2^-23 and c_par = (D / 32 + 10) 2^-23 (the search's
// D / 32 + 6 roundings of 2^-24), plus a 2^-20 relative guard on each comparison.
// Values beyond FP16's range give infinite norms, which send every test of that node to the
// exact chain.  Every mbarrier wait is bounded (one second); a thread that gives up makes the
// whole CTA stop at its next barrier and raises kErrWait.
// Bound by the latency of a tile's steps (copies, MMAs, then two exchanges per kept entry) and the
// L2 gathers.  Streaming the FP32 rows instead, with the exact chain and the rounding of every
// candidate done by its thread, and exact chains for every test inside the 16-bit margin, took
// 10.6 + 10.7 ms at 1M x 200 and 22 + 31 ms at 300k x 512, L = 96.  Now 7.1 + 7.6 ms, with 0.5 ms
// each for launch_list_dists and launch_edge_dists, and 15.8 + 26.9 ms with them.  Two or four
// stages are 2-4% slower than three.  Putting a doubtful test off until its candidate may be kept
// gained nothing (1M x 200 56.1 -> 57.6 ms, 1M x 512 335 -> 361): the next kept entry is usually
// among the doubtful.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "pg_device.cuh"
#include "pg_kernels.h"
#include "pg_tc.cuh"

namespace pg {

namespace {

using namespace tcu;

constexpr uint32_t kTile = 128;                 // tile rows = MMA M = N = TMEM columns = threads
constexpr uint32_t kWarps = kTile / 32;
constexpr uint32_t kCk = 64;                    // 16-bit columns per chunk: 128 bytes of a row
constexpr uint32_t kStageBytes = kTile * 128;
constexpr uint32_t kBarAll = 1, kBarNode = 2;   // named barriers: all threads; node 0 (+ node)
constexpr uint32_t kNone = 0xFFFFFFFFu;

struct TcShape {
  uint32_t cap;    // candidate slots per node: 64 (two nodes per tile) or 128 (one)
  uint32_t dp;     // 16-bit row length: D rounded up to 16
  uint32_t nk;     // chunks per row
  uint64_t tiles;  // ceil(n / nodes per tile)
};

// Shared-memory layout, offsets from a 1024-byte aligned base.
struct Layout {
  uint32_t stage, id, nrm, err, last, xch, bars, words, total;
};
__host__ __device__ constexpr Layout layout(uint32_t stages) {
  Layout l{};
  l.stage = 0;
  l.id = stages * kStageBytes;
  l.nrm = l.id + kTile * 4;
  l.err = l.nrm + kTile * 4;
  l.last = l.err + kTile * 4;       // per node: the last kept entry's distance and bound
  l.xch = l.last + 2 * 8;
  l.bars = l.xch + 2 * kWarps * 4;  // free[stages], acc, drained
  l.words = l.bars + (stages + 2) * 8;  // TMEM address
  l.total = l.words + 16;
  return l;
}
constexpr uint32_t kMinStages = 2, kMaxStages = 4;
size_t smem_bytes(uint32_t stages) { return layout(stages).total + 1024; }

// 16 bytes global -> shared, cached in L2 only, completing with the thread's copy groups.
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <uint32_t N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Bounded wait (one second) on the phase of parity `parity`, sleeping between tries: try_wait
// with a suspend-time hint returns as soon as the phase completes.
__device__ __forceinline__ bool bar_wait_hint(uint64_t* b, uint32_t parity) {
  constexpr uint32_t kHintNs = 100000;
  const uint64_t t0 = now_ns();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(saddr(b)), "r"(parity), "r"(kHintNs)
        : "memory");
    if (ok) return true;
    if (now_ns() - t0 > 1000000000ull) return false;
  }
}

__device__ __forceinline__ void named_sync(uint32_t id, uint32_t threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Named barrier that also returns the AND of `v` over the participating threads.
__device__ __forceinline__ bool named_and(uint32_t id, uint32_t threads, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\t"
      "bar.red.and.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"(v ? 1u : 0u)
      : "memory");
  return r != 0;
}

// The threads of one node: warps col0 / 32 .. + nw - 1, named barrier `bar`.  Every thread of the
// node makes the same sequence of exchanges, numbered by q.
struct Node {
  uint32_t* xch;
  uint32_t w0, nw, bar, threads;
  uint32_t q;
  // One word per warp of the node, seen by all its threads.
  __device__ __forceinline__ const uint32_t* exchange(uint32_t v) {
    uint32_t* xb = xch + (q & 1u) * kWarps;
    q++;
    if ((threadIdx.x & 31u) == 0) xb[threadIdx.x >> 5] = v;
    __syncwarp();
    named_sync(bar, threads);
    return xb + w0;
  }
  __device__ __forceinline__ uint32_t min(uint32_t v) {
    const uint32_t* x = exchange(__reduce_min_sync(kFull, v));
    uint32_t m = kNone;
    for (uint32_t w = 0; w < nw; w++) m = ::min(m, x[w]);
    return m;
  }
  // How many threads hold f, and the lowest slot that does (kNone: none).
  __device__ __forceinline__ uint32_t count(bool f, uint32_t& first) {
    const uint32_t* x = exchange(__ballot_sync(kFull, f));
    uint32_t c = 0;
    first = kNone;
    for (uint32_t w = 0; w < nw; w++) {
      const uint32_t m = x[w];
      if (m && first == kNone)
        first = 32u * w + static_cast<uint32_t>(__ffs(static_cast<int>(m)) - 1);
      c += __popc(m);
    }
    return c;
  }
};

// order_key with the largest value left free to mean "none".
__device__ __forceinline__ uint32_t dist_key(float f) { return min(order_key(f), kNone - 1u); }

// This thread's candidate id in tile t, or kNone when the slot holds no row to stage (past the
// end, a tomb, an out-of-range id or the node itself).
__device__ __forceinline__ uint32_t cand_id(const PruneArgs& a, uint64_t t, uint32_t P,
                                            uint32_t node, uint32_t slot) {
  const uint64_t b = t * P + node;
  if (b >= a.n || slot >= a.c) return kNone;
  const uint32_t x = a.graph[b * a.c + slot];
  return (x >= a.n || x == static_cast<uint32_t>(b)) ? kNone : x;
}

// The copy stream of one thread: the chunks of its warp's rows in the CTA's tile order, one
// cp.async group per chunk (empty past the last tile).
struct Feed {
  uint64_t t;   // tile of the next chunk to issue
  uint32_t kc;  // the chunk
  uint32_t x;   // this thread's candidate id in tile t (kNone: nothing to stage)
};

// Issues chunk f.kc of tile f.t into `st`.  The warp copies its 32 rows four at a time: eight lanes
// per row, one 16-byte piece each, so that each copy instruction reads whole row segments, swizzled
// as the MMA's descriptors expect (piece j of row r at j ^ (r mod 8) of its 128 bytes).
__device__ __forceinline__ void feed_issue(Feed& f, const PruneArgs& a, const TcShape& sh,
                                           uint8_t* st, uint32_t P, uint32_t node, uint32_t slot) {
  const uint32_t R = threadIdx.x, lane = R & 31u;
  if (f.t < sh.tiles) {
    const uint32_t pieces = min(kCk, sh.dp - f.kc * kCk) / 8;
    const uint32_t j = lane & 7u;
    const uint8_t* src = static_cast<const uint8_t*>(a.rows16) + f.kc * 128u + 16u * j;
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
      const uint32_t rr = (R & ~31u) + 4u * i + (lane >> 3);  // tile row copied by this lane
      const uint32_t xr = __shfl_sync(kFull, f.x, 4u * i + (lane >> 3));
      if (xr != kNone && j < pieces)
        cp16(st + rr * 128u + ((j ^ (rr & 7u)) << 4),
             src + static_cast<uint64_t>(xr) * (2u * sh.dp));
    }
    if (++f.kc == sh.nk) {
      f.kc = 0;
      f.t += gridDim.x;
      f.x = f.t < sh.tiles ? cand_id(a, f.t, P, node, slot) : kNone;
    }
  }
  cp_commit();
}

__device__ __forceinline__ float4 ldg4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ void fma4(float4& s, const float4 u, const float4 v) {
  s.x = fmaf(u.x, v.x, s.x);
  s.y = fmaf(u.y, v.y, s.y);
  s.z = fmaf(u.z, v.z, s.z);
  s.w = fmaf(u.w, v.w, s.w);
}
__device__ __forceinline__ float sum4(const float4 s) { return (s.x + s.y) + (s.z + s.w); }

// FP32 inner products of row r with the rows x of the lanes that `want` one, each valid in its
// lane.  Loads are whole 128-byte lines.  Four rows at a time, eight lanes each; with WHOLE the
// last one or two take the whole warp, which holds a row of 512 floats in one round of loads.  That
// is the usual case in the prune, whose scan waits for it: round 2 of 1M x 512 96.7 -> 87.7 ms, but
// of 1M x 200 9.0 -> 9.5 (the larger kernel), hence only for rows over 256 floats.
template <bool WHOLE>
__device__ __forceinline__ float warp_dots(const float* __restrict__ base, uint32_t d, uint32_t r,
                                           uint32_t x, bool want) {
  const uint32_t lane = threadIdx.x & 31u, g = lane >> 3, m = lane & 7u;
  unsigned todo = __ballot_sync(kFull, want);
  const float* rrow = base + static_cast<uint64_t>(r) * d;
  float mine = 0.f;
  constexpr uint32_t few = WHOLE ? 2 : 0;
  while (__popc(todo) > few) {
    unsigned t = todo;
    for (uint32_t i = 0; i < g; i++) t &= t - 1u;  // group g takes the g-th lane, or repeats one
    const int src = __ffs(static_cast<int>(t ? t : todo)) - 1;
    const float* xrow = base + static_cast<uint64_t>(__shfl_sync(kFull, x, src)) * d;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (uint32_t c = 4u * m; c < d; c += 32) fma4(s, ldg4(rrow + c), ldg4(xrow + c));
    float v = sum4(s);
    v += __shfl_xor_sync(kFull, v, 4);
    v += __shfl_xor_sync(kFull, v, 2);
    v += __shfl_xor_sync(kFull, v, 1);
    const uint32_t rank = __popc(todo & ((1u << lane) - 1u));
    const float got = __shfl_sync(kFull, v, static_cast<int>((rank & 3u) << 3));
    if (((todo >> lane) & 1u) && rank < 4) mine = got;
    for (uint32_t i = 0; i < 4; i++) todo &= todo - 1u;  // 0 stays 0
  }
  if (WHOLE && todo) {
    const int l0 = __ffs(static_cast<int>(todo)) - 1;
    const int l1 = 31 - __clz(static_cast<int>(todo));
    const float* x0 = base + static_cast<uint64_t>(__shfl_sync(kFull, x, l0)) * d;
    const float* x1 = base + static_cast<uint64_t>(__shfl_sync(kFull, x, l1)) * d;
    float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
#pragma unroll 4
    for (uint32_t c = 4u * lane; c < d; c += 128) {
      const float4 u = ldg4(rrow + c);
      fma4(s0, u, ldg4(x0 + c));
      fma4(s1, u, ldg4(x1 + c));
    }
    // the lower half of the warp finishes the first, the upper half the second
    const float a = sum4(s0), b = sum4(s1);
    const bool up = lane >= 16;
    float v = (up ? b : a) + __shfl_xor_sync(kFull, up ? a : b, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    const float v0 = __shfl_sync(kFull, v, 0), v1 = __shfl_sync(kFull, v, 16);
    if (static_cast<int>(lane) == l0) mine = v0;
    if (static_cast<int>(lane) == l1) mine = l0 == l1 ? v0 : v1;
  }
  return mine;
}

// One warp per list of 32 E entries: the distances that its search does not know belong to ids that
// it had visited before its last step.  Such an id may stand elsewhere in the list; the others are
// scored.
template <int E>
__global__ void __launch_bounds__(256) k_list_dists(const float* __restrict__ base, uint64_t n,
                                                    uint32_t d, const uint32_t* __restrict__ lists,
                                                    uint32_t* __restrict__ keys) {
  constexpr uint32_t C = 32u * E;
  __shared__ uint4 ids_all[8][C / 4];
  __shared__ uint32_t key_all[8][C];
  uint4* ids = ids_all[threadIdx.x >> 5];
  uint32_t* ks = key_all[threadIdx.x >> 5];
  const uint32_t lane = lane_id();
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * 8;
  for (uint64_t b = blockIdx.x * 8ull + (threadIdx.x >> 5); b < n; b += nw) {
    uint32_t id[E], key[E];
    bool any = false;
#pragma unroll
    for (int e = 0; e < E; e++) {
      id[e] = lists[b * C + 32 * e + lane];
      key[e] = keys[b * C + 32 * e + lane];
      if (id[e] >= n) key[e] = order_key(FLT_MAX);
      if (key[e] == kNoKey && id[e] == static_cast<uint32_t>(b)) key[e] = order_key(FLT_MAX);
      any |= key[e] == kNoKey;
    }
    if (__any_sync(kFull, any)) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        reinterpret_cast<uint32_t*>(ids)[32 * e + lane] = id[e];
        ks[32 * e + lane] = key[e];
      }
      __syncwarp();
#pragma unroll
      for (int e = 0; e < E; e++) {
        if (!__any_sync(kFull, key[e] == kNoKey)) continue;
        uint32_t at = 32u * e + lane;  // another entry of the same id whose distance is known
#pragma unroll 4
        for (uint32_t j = 0; j < C / 4; j++) {
          const uint4 v = ids[j];
          if (v.x == id[e] && ks[4 * j] != kNoKey) at = 4 * j;
          if (v.y == id[e] && ks[4 * j + 1] != kNoKey) at = 4 * j + 1;
          if (v.z == id[e] && ks[4 * j + 2] != kNoKey) at = 4 * j + 2;
          if (v.w == id[e] && ks[4 * j + 3] != kNoKey) at = 4 * j + 3;
        }
        if (key[e] == kNoKey) key[e] = ks[at];
        const bool want = key[e] == kNoKey;
        const float s32 = warp_dots<false>(base, d, static_cast<uint32_t>(b), id[e], want);
        if (want) key[e] = order_key(-s32);
      }
    }
#pragma unroll
    for (int e = 0; e < E; e++) keys[b * C + 32 * e + lane] = __float_as_uint(key_dist(key[e]));
    __syncwarp();
  }
}

template <bool HALF, bool LONG, uint32_t S>
__global__ void __launch_bounds__(kTile, S <= 3 ? 4 : 3) k_prune_tc(const PruneArgs a,
                                                                   const TcShape sh) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* sm = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
  constexpr Layout L = layout(S);
  uint8_t* stage = sm + L.stage;
  uint32_t* sid = reinterpret_cast<uint32_t*>(sm + L.id);
  float* snrm = reinterpret_cast<float*>(sm + L.nrm);
  float* serr = reinterpret_cast<float*>(sm + L.err);
  float2* slast = reinterpret_cast<float2*>(sm + L.last);
  uint64_t* sfree = reinterpret_cast<uint64_t*>(sm + L.bars);  // [S]
  uint64_t* accfull = sfree + S;
  uint64_t* drained = accfull + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L.words);

  const uint32_t R = threadIdx.x, warp = R >> 5, lane = R & 31u;
  const uint32_t cap = sh.cap, P = kTile / cap;
  const uint32_t node = R / cap, slot = R - node * cap, col0 = node * cap;
  Node nd{reinterpret_cast<uint32_t*>(sm + L.xch), col0 / 32u, cap / 32u, kBarNode + node, cap, 0};

  if (R == 0) {
    for (uint32_t i = 0; i < S; i++) bar_init(sfree + i, 1);
    bar_init(accfull, 1);
    bar_init(drained, 1);
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, kTile);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t taddr = tmem + ((warp * 32u) << 16);

  const uint32_t d = a.d;
  const float c_acc = static_cast<float>(sh.dp + 32u) * 4.76837158e-07f;  // 2^-21
  const float c_seq = static_cast<float>(d + 2u) * 1.19209290e-07f;       // 2^-23
  const float c_par = static_cast<float>(d / 32u + 10u) * 1.19209290e-07f;
  constexpr float kGuard = 9.5367431640625e-07f;                         // 2^-20
  const uint32_t kmax = order_key(FLT_MAX);
  // A and B FP16 (format 0) or BF16 (format 1, bits 7-9 and 10-12)
  constexpr uint32_t kIdesc = idesc_f16(kTile, kTile) | (HALF ? 0u : ((1u << 7) | (1u << 10)));
  uint64_t ev = 0, resc = 0;
  uint32_t g = 0, it = 0;
  bool ok = true, w = true;

  Feed f{blockIdx.x, 0, kNone};
  if (f.t < sh.tiles) f.x = cand_id(a, f.t, P, node, slot);
  for (uint32_t i = 0; i + 1 < S; i++)
    feed_issue(f, a, sh, stage + i * kStageBytes, P, node, slot);
  // the scan's inputs are read a tile ahead: ids and distances, then the norms that hang on them
  uint32_t x_next = kTomb;
  float dist_next = FLT_MAX;
  auto fetch = [&](uint64_t t) {
    const uint64_t b = t * P + node;
    const bool in = t < sh.tiles && b < a.n && slot < a.c;
    x_next = in ? a.graph[b * a.c + slot] : kTomb;
    dist_next = in ? a.cand_dist[b * a.c + slot] : FLT_MAX;
  };
  fetch(blockIdx.x);

  uint64_t t = blockIdx.x;
  for (; t < sh.tiles; t += gridDim.x, it++) {
    const uint64_t b = t * P + node;
    const bool bval = b < a.n;
    uint32_t x = x_next;
    float dist = dist_next;  // of the candidate to the node: within `bound` of the exact chain's
    if (x >= a.n && x != kTomb && x != kMaskedTomb) {
      raise_error(a.status, kErrBadId);
      x = kTomb;
    }
    const bool in = bval && slot < a.c;
    const bool tomb = in && (x == kTomb || x == kMaskedTomb);
    const bool valid = in && !tomb && x != static_cast<uint32_t>(b);
    const float2 ne = valid ? __ldg(a.norms + x) : make_float2(0.f, 0.f);
    const float nb = bval ? __ldg(&a.norms[b].x) : 0.f;
    fetch(t + gridDim.x);
    for (uint32_t kc = 0; kc < sh.nk; kc++, g++) {
      cp_wait<S - 2>();  // this thread's copies of chunk g have landed
      fence_proxy_async();
      ok = named_and(kBarAll, kTile, w);  // and everyone's
      if (!ok) break;
      if (R == 0) {
        fence_after();
        const uint32_t a0 = saddr(stage + (g % S) * kStageBytes);
        const uint32_t steps = min(kCk, sh.dp - kc * kCk) / 16u;
        for (uint32_t k = 0; k < steps; k++) {
          const uint64_t dsc = sw128_desc(a0 + 32u * k);
          mma_f16(tmem, dsc, dsc, kIdesc, (kc | k) != 0);
        }
        commit(sfree + g % S);  // the stage is free once these MMAs have read it
        if (kc + 1 == sh.nk) commit(accfull);
      }
      // the next chunk of the stream goes where chunk g - 1 was
      const uint32_t at = (g + S - 1) % S;
      if (g >= 1) w = __all_sync(kFull, bar_wait_hint(sfree + at, ((g - 1) / S) & 1u));
      if (w)
        feed_issue(f, a, sh, stage + at * kStageBytes, P, node, slot);
      else
        cp_commit();
    }
    if (!ok) break;
    sid[R] = x;
    snrm[R] = ne.x;
    serr[R] = ne.y;
    __syncwarp();
    ok = named_and(kBarAll, kTile, w && bar_wait_hint(accfull, it & 1u));
    if (!ok) break;
    fence_after();

    // ---- the node's scan
    const float* brow = a.base + (bval ? b : 0) * d;
    const float* xrow = a.base + static_cast<uint64_t>(valid ? x : 0u) * d;
    float bound = 0.f;  // 0: dist is the exact chain's (or FLT_MAX)
    auto exact = [&]() {  // a settlement holds up the scan: 256-bit loads whatever the row length
      dist = dist_seq<true>(brow, xrow, d);
      bound = 0.f;
    };
    if (valid) {
      bound = 0.5f * (c_seq + c_par) * nb * ne.x + fabsf(dist) * 2.4e-7f + 1e-30f;
      if (!(fabsf(dist) < 1e37f && bound < 1e37f)) exact();
    } else {
      dist = FLT_MAX;
    }
    const uint32_t nv = __popc(__ballot_sync(kFull, valid));
    if (lane == 0) ev += nv;
    // undecided: candidates that come before the first tomb in (distance, slot) order
    uint32_t first_tomb;
    const uint32_t tombs = nd.count(tomb, first_tomb);
    bool open = in && !tomb;
    if (open && tombs) {
      const uint32_t key = dist_key(dist);
      open = key < kmax || (key == kmax && slot < first_tomb);
    }
    // The undecided candidate that comes first: the one whose interval may hold the smallest
    // distance, or, among several, the exact minimum.
    auto next = [&]() -> uint32_t {
      for (uint32_t pass = 0;; pass++) {
        const uint32_t m = nd.min(open ? dist_key(dist + bound) : kNone);
        if (m == kNone) return kNone;
        const bool may = open && dist_key(dist - bound) <= m;
        uint32_t s;
        if (nd.count(may, s) == 1 || pass) return s;
        if (may && bound > 0.f) exact();
      }
    };
    uint32_t K = 0, my_kept = kNone, fo = kNone;
    bool full = false;
    uint32_t ro = next();
    while (ro != kNone) {
      if (slot == ro) {
        my_kept = K;
        open = false;
      }
      const uint32_t t_k = K++;
      if (K == a.p) {
        full = true;
        break;
      }
      const uint32_t ri = sid[col0 + ro];
      const float nr = snrm[col0 + ro], er = serr[col0 + ro];
      const float gv = __uint_as_float(tmem_ld1(taddr + col0 + ro));
      tmem_wait_ld();
      bool yes = false, sure = !open;
      const bool other = ri != static_cast<uint32_t>(b);  // the node itself has no row in the tile
      if (open && other) {
        if (valid) {
          const float dhat = -gv;
          const float e = ne.y * (nr + er) + ne.x * er + c_acc * (ne.x + ne.y) * (nr + er) +
                          c_seq * ne.x * nr + fabsf(dhat) * kGuard + 1e-30f + bound;
          yes = dhat + e < dist;
          sure = yes || dhat - e >= dist;
        } else if (nb * nr < 1e37f) {  // the node: at FLT_MAX, past any chain this bounds
          yes = sure = true;
        }
      }
      const uint32_t nun = __popc(__ballot_sync(kFull, !sure));
      if (nun) {  // inside the 16-bit margin: FP32 products, exact chains inside theirs (or NaN)
        const float s32 = warp_dots<LONG>(a.base, d, ri, x, !sure && valid && other);
        if (!sure) {
          if (valid && other) {
            const float dhat = -s32;
            const float e = (c_seq + c_par) * ne.x * nr + fabsf(dhat) * kGuard + 1e-30f + bound;
            yes = dhat + e < dist;
            sure = yes || dhat - e >= dist;
          }
          if (!sure) {
            if (bound > 0.f) exact();
            yes = dist_seq<true>(a.base + static_cast<uint64_t>(x) * d,
                                 a.base + static_cast<uint64_t>(ri) * d, d) < dist;
          }
        }
        if (lane == 0) resc += nun;
      }
      if (open && yes) {
        fo = t_k;
        open = false;
      }
      ro = next();
    }
    // evaluations: the occluded candidates that come before the entry that filled the list
    bool counted = fo != kNone;
    if (full) {
      auto tell = [&]() {
        if (my_kept == K - 1) slast[node] = make_float2(dist, bound);
        __syncwarp();
        named_sync(nd.bar, nd.threads);
        return slast[node];
      };
      float2 l = tell();
      bool unsure = counted && !(dist_key(dist + bound) < dist_key(l.x - l.y)) &&
                    !(dist_key(dist - bound) > dist_key(l.x + l.y));
      uint32_t s;
      if (nd.count(unsure, s)) {  // also separates the two uses of slast
        if ((unsure || my_kept == K - 1) && bound > 0.f) exact();
        l = tell();
      }
      if (counted) {
        const uint32_t key = dist_key(dist - bound), lkey = dist_key(l.x + l.y);
        counted = unsure ? dist_key(dist) < dist_key(l.x) ||
                               (dist_key(dist) == dist_key(l.x) && slot < ro)
                         : !(key > lkey);
      }
      __syncwarp();
      named_sync(nd.bar, nd.threads);  // slast is written again by the next tile
    }
    const uint32_t chs = __reduce_add_sync(kFull, counted ? fo + 1u : 0u);
    if (lane == 0) ev += chs;
    if (bval) {
      if (R == col0) {
        a.pruned_num[b] = K;
        if (K > 1) ev += static_cast<uint64_t>(K) * (K - 1) / 2;  // kept entry m made m tests
      }
      if (my_kept != kNone) {
        a.pruned[b * a.p + my_kept] = x;
        atomicAdd(a.indeg + x, 1u);
      }
    }
    fence_before();  // the TMEM reads above precede the next tile's first MMA
  }
  // After a wait that gave up, the nodes not reached keep nothing: the kernels that follow read counts.
  if (!ok)
    for (; t < sh.tiles; t += gridDim.x)
      if (slot == 0 && t * P + node < a.n) a.pruned_num[t * P + node] = 0;
  cp_wait<0>();  // no copy lands after the CTA exits
  if (lane == 0) {
    if (ev) atomicAdd(a.evals, static_cast<unsigned long long>(ev));
    if (resc && a.rescored) atomicAdd(a.rescored, static_cast<unsigned long long>(resc));
  }
  if (R == 0) {
    if (!ok) raise_error(a.status, kErrWait);
    commit(drained);  // arrives once every MMA issued above has completed
    bar_wait(drained, 0, nullptr);
  }
  fence_before();
  __syncthreads();
  if (warp == 0) {
    fence_after();
    tmem_dealloc(tmem, kTile);
  }
}

}  // namespace

template <bool HALF, bool LONG, uint32_t S>
cudaError_t launch_s(const PruneArgs& a, const TcShape& sh, int num_sms, cudaStream_t st) {
  const size_t smem = smem_bytes(S);
  auto kern = k_prune_tc<HALF, LONG, S>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  // the largest shared-memory carveout, so that several CTAs fit on an SM (the driver otherwise
  // picks the smallest carveout that holds one)
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return e;
  // CTAs per SM from the kernel's registers and shared memory (at most 4: 4 x 128 TMEM columns)
  cudaFuncAttributes fa{};
  e = cudaFuncGetAttributes(&fa, kern);
  if (e != cudaSuccess) return e;
  int dev = 0, smem_sm = 0, regs_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) !=
      cudaSuccess)
    return e;
  if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) !=
      cudaSuccess)
    return e;
  const int regs_cta = ((fa.numRegs + 7) / 8 * 8) * static_cast<int>(kTile);
  int per_sm = smem_sm / static_cast<int>(smem + fa.sharedSizeBytes + 1024);  // + reserved 1 KB
  if (regs_cta > 0 && regs_sm / regs_cta < per_sm) per_sm = regs_sm / regs_cta;
  if (per_sm < 1) per_sm = 1;
  if (per_sm > 4) per_sm = 4;
  uint64_t blocks = static_cast<uint64_t>(num_sms) * per_sm;
  if (blocks > sh.tiles) blocks = sh.tiles;
  kern<<<static_cast<unsigned>(blocks), kTile, smem, st>>>(a, sh);
  return cudaGetLastError();
}

template <uint32_t S>
cudaError_t launch_half(const PruneArgs& a, const TcShape& sh, bool half, bool rows512, int num_sms,
                        cudaStream_t st) {
  if (rows512)
    return half ? launch_s<true, true, S>(a, sh, num_sms, st)
                : launch_s<false, true, S>(a, sh, num_sms, st);
  return half ? launch_s<true, false, S>(a, sh, num_sms, st)
              : launch_s<false, false, S>(a, sh, num_sms, st);
}

cudaError_t launch_list_dists(const float* base, uint64_t n, uint32_t d, const uint32_t* lists,
                              uint32_t c, uint32_t* keys, int num_sms, cudaStream_t st) {
  uint64_t blocks = (n + 7) / 8;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
  if (blocks > cap) blocks = cap;
  auto kern = c == 64 ? k_list_dists<2> : c == 96 ? k_list_dists<3> : k_list_dists<4>;
  if (c != 64 && c != 96 && c != 128) return cudaErrorInvalidValue;
  kern<<<static_cast<unsigned>(blocks), 256, 0, st>>>(base, n, d, lists, keys);
  return cudaGetLastError();
}

cudaError_t launch_prune_screen(const PruneArgs& a, int num_sms, size_t smem_optin,
                                cudaStream_t st) {
  if (!screen_supported(a.c, a.d, a.strict) || !a.norms || !a.rows16 || !a.cand_dist ||
      (reinterpret_cast<uintptr_t>(a.base) % 16) != 0 ||
      (reinterpret_cast<uintptr_t>(a.rows16) % 16) != 0)
    return cudaErrorInvalidValue;
  if (a.n == 0) return cudaSuccess;
  if (a.n > 0x7FFFFFFFull) return cudaErrorInvalidValue;
  TcShape sh{};
  sh.cap = a.c <= 64 ? 64u : 128u;
  sh.dp = screen_row(a.d);
  sh.nk = (sh.dp + kCk - 1) / kCk;
  const uint32_t per_tile = kTile / sh.cap;
  sh.tiles = (a.n + per_tile - 1) / per_tile;
  uint32_t s = a.stages ? a.stages : kPruneStages;
  if (s < kMinStages) s = kMinStages;
  if (s > kMaxStages) s = kMaxStages;
  while (s > kMinStages && smem_bytes(s) > smem_optin) s--;
  if (smem_bytes(s) > smem_optin) return cudaErrorInvalidValue;
  const bool half = a.screen_half != 0, rows512 = a.d > 256;
  switch (s) {
    case 2: return launch_half<2>(a, sh, half, rows512, num_sms, st);
    case 3: return launch_half<3>(a, sh, half, rows512, num_sms, st);
    default: return launch_half<4>(a, sh, half, rows512, num_sms, st);
  }
}

}  // namespace pg
