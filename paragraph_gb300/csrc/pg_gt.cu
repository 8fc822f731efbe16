// pg_gt.cu -- exact inner-product top-k ground truth on the GPU (sm_103a).
//
// The reference's build reads each training query's top-128 base ids from a file made outside it
// (README.md:25-31, notebooks); here they are computed on the GPU.  Result: for every query q the
// k base ids with the largest FP64 inner product q.x, ties to the lower id -- exact, whatever the
// arithmetic used to find them.
//
//   1. FP16 copies of base and queries, rows zero-padded to a multiple of 16 elements, with
//      per-row norms |x^| and |x - x^| (k_half_rows);
//   2. screening scores s^ = q^.x^ on the tensor cores: k_gt_tc, a persistent tcgen05 GEMM
//      (TMA-loaded 128-byte-swizzled tiles, FP32 accumulators in TMEM) whose epilogue consumes
//      each tile of scores in registers -- no score matrix is ever stored;
//   3. a rigorous bound: |q.x - s^| <= E_q = (|q^| + |e_q|) max|e_x| + |e_q| max|x^|
//      + g (|q^| max|x^|), with g covering the FP32 accumulation (d' * 2^-22, four times the
//      IEEE unit roundoff, for the tensor core's accumulation);
//   4. pass 1 (k_gt_tc<kMax>): the maximum screened score of every group of base rows per query
//      (disjoint groups, about 4096 or more of them), over a sample of the base tiles where it is
//      large; the k-th largest group maximum theta_q is the score of k distinct base rows, so
//      theta_q <= t_k, the k-th largest screened score of the row (k_gt_theta);
//   5. pass 2 (k_gt_tc<kFilter>): every base row with s^ >= theta_q - 2 E_q is a candidate --
//      a superset of {s^ >= t_k - 2 E_q}, which holds the true top k (a true top-k member has
//      s^ >= s_k - E_q and s_k >= t_k - E_q);
//   6. k_gt_final: the candidates with s^ >= t_k - 2 E_q, exact FP64 inner products, sorted by
//      (score desc, id asc).
// With groups many enough that the top k fall in nearly distinct groups, theta_q sits just
// below t_k and a query keeps about 1.1 k candidates.  From a sample of every step-th tile it keeps
// about 1.1 k step, which k_gt_narrow brings back to 1.1 k; pass 1 then costs 1 / step of pass 2.
// A query whose sampled threshold lets through more than its list holds (near rows that miss the
// sample, as in a base stored cluster by cluster) is filtered again, up to twice: the k-th best of the
// candidates that its list did hold is a higher threshold.  300k x 200 in the order of 1000 clusters,
// 100k queries near them, k = 10: 47 ms (66 ms when one such query had the whole call done again with
// every tile); shuffled 14.5 ms.  Where there is nothing to do the two passes
// cost some 10 us.
#include <cuda.h>
#include <cuda_fp16.h>

#include <cmath>

#include "pg_device.cuh"
#include "pg_kernels.h"
#include "pg_tc.cuh"

namespace pg {

namespace {

constexpr uint32_t kGtCap = 1024;          // candidates per query
constexpr uint32_t kGtTile = 128;          // queries per tile of the GEMM passes
constexpr int kGtAgain = 2;                // further filter passes after a sampled threshold
constexpr uint32_t kGtErrRange = 1u << 4;  // a value beyond the FP16 range
constexpr uint32_t kGtErrFinal = 1u << 6;  // a query kept more candidates than kGtCap
constexpr uint32_t kGtShort = 256;         // lists of the final pass's common kernel

__device__ __forceinline__ float key_value(uint64_t key) {  // inverse of desc_key's value part
  const uint32_t o = ~static_cast<uint32_t>(key >> 32);
  const uint32_t u = (o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o;
  return __uint_as_float(u);
}

// descending value, then ascending id, as an ascending 64-bit key
__device__ __forceinline__ uint64_t desc_key(float v, uint32_t id) {
  return (static_cast<uint64_t>(~order_key(v)) << 32) | id;
}

// FP16 copy of rows x d FP32 values with row stride dp >= d (zeros in the padding), and per row
// upper bounds of |x^| and |x - x^|: FP32 sums of squares with every operation rounded up (the
// difference x - x^ is exact).  FP64 sums took 2.1 ms for 550k rows of 200 floats, the FP64 units
// being the limit.
__global__ void k_half_rows(const float* __restrict__ x, uint64_t rows, uint32_t d, uint32_t dp,
                            __half* __restrict__ h, float* __restrict__ nrm,
                            float* __restrict__ enrm, uint32_t* __restrict__ status) {
  const uint32_t lane = lane_id();
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
  for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x >> 5) + (threadIdx.x >> 5);
       r < rows; r += nw) {
    float a = 0.0f, e = 0.0f;
    bool big = false;
    for (uint32_t i = lane; i < dp; i += 32) {
      if (i >= d) {
        h[r * dp + i] = __float2half_rn(0.0f);
        continue;
      }
      const float v = x[r * d + i];
      big |= !(fabsf(v) <= 65000.0f);  // beyond FP16 range (or NaN)
      const __half hv = __float2half_rn(v);
      h[r * dp + i] = hv;
      const float fv = __half2float(hv);
      a = __fmaf_ru(fv, fv, a);
      const float ev = v - fv;
      e = __fmaf_ru(ev, ev, e);
    }
    for (int o = 16; o > 0; o >>= 1) {
      a = __fadd_ru(a, __shfl_xor_sync(kFull, a, o));
      e = __fadd_ru(e, __shfl_xor_sync(kFull, e, o));
    }
    if (__any_sync(kFull, big) && lane == 0) raise_error(status, kGtErrRange);
    if (lane == 0) {
      nrm[r] = __fsqrt_ru(a);
      enrm[r] = __fsqrt_ru(e);
    }
  }
}

__global__ void k_max2(const float* __restrict__ a, const float* __restrict__ b, uint64_t n,
                       uint32_t* __restrict__ out) {  // out[0] = max a, out[1] = max b (>= 0)
  float ma = 0.0f, mb = 0.0f;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    ma = fmaxf(ma, a[i]);
    mb = fmaxf(mb, b[i]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    ma = fmaxf(ma, __shfl_xor_sync(kFull, ma, o));
    mb = fmaxf(mb, __shfl_xor_sync(kFull, mb, o));
  }
  if (lane_id() == 0) {  // non-negative floats order like their bit patterns
    atomicMax(out, __float_as_uint(ma));
    atomicMax(out + 1, __float_as_uint(mb));
  }
}

// Per query of the chunk: 2 E_q plus a relative slack for the FP32 arithmetic of the threshold.
// The tensor core accumulates over dp (d plus zero padding) products.
__global__ void k_gt_band(const float* __restrict__ qn, const float* __restrict__ qe,
                          const uint32_t* __restrict__ xmax, uint32_t rows, uint32_t dp,
                          float* __restrict__ band) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const double xn = __uint_as_float(xmax[0]), xe = __uint_as_float(xmax[1]);
  const double dd = dp + 16.0, u = 1.0 / 4194304.0;  // 2^-22
  const double g = dd * u / (1.0 - dd * u);
  const double q = qn[r], e = qe[r];
  const double E = (q + e) * xe + e * xn + g * q * xn;
  band[r] = __double2float_ru(2.0 * E * (1.0 + 1e-6) + 1e-30);
}

// ---------------------------------------------------------------- selection helpers

// Sorts buf[0 .. cnt) (desc value, asc id) and keeps the prefix with value >= the k-th largest
// value - band (all of it when cnt < k); cnt updated.
template <int E>
__device__ void compact_sorted(uint64_t* buf, uint32_t& cnt, uint32_t k, float band) {
  const uint32_t lane = lane_id();
  uint64_t key[E];
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    key[s] = i < cnt ? buf[i] : ~0ull;
  }
  __syncwarp();
  warp_sort_u64<E>(key);
  float theta = -INFINITY;
  if (cnt >= k) {
    const int s = static_cast<int>((k - 1) / 32);
    uint64_t kk = 0;
#pragma unroll
    for (int t = 0; t < E; t++)
      if (t == s) kk = __shfl_sync(kFull, key[t], (k - 1) & 31u);
    theta = key_value(kk);
  }
  const float lo = theta - band;
  uint32_t keep = 0;
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    const bool ok = i < cnt && key_value(key[s]) >= lo;
    keep += __popc(__ballot_sync(kFull, ok));
    if (ok) buf[i] = key[s];
  }
  __syncwarp();
  cnt = keep;
}

template <uint32_t CAP>
__device__ void compact_any(uint64_t* buf, uint32_t& cnt, uint32_t k, float band) {
  if (cnt <= 128)
    compact_sorted<4>(buf, cnt, k, band);
  else if (CAP <= 256 || cnt <= 256)
    compact_sorted<8>(buf, cnt, k, band);
  else if (cnt <= 512)
    compact_sorted<16>(buf, cnt, k, band);
  else
    compact_sorted<32>(buf, cnt, k, band);
}

struct GtArgs {
  const float* base;     // n x d (FP32)
  const float* queries;  // rows x d (FP32, this chunk)
  uint32_t d, k;
  uint32_t rows;
  const uint64_t* cand;      // rows x kGtCap keys (desc_key), two halves of kGtCap / 2
  const uint32_t* cand_cnt;  // rows x 2
  const float* band;         // rows
  const float *qn, *qe;      // rows: upper bounds of |q^| and |q - q^|
  const uint32_t* xmax;      // bits of max |x^| and max |x - x^|
  uint32_t* out;             // rows x k
};

template <bool VEC>
__device__ __forceinline__ float4 load4(const float* p) {
  if constexpr (VEC) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// FP32 inner products of the query (shared memory) with the rows of ids buf[0 .. cnt) (low words):
// eight lanes per row, four rows per load, two loads in flight per step.  Lane m of a group sums
// elements 32 k + 4 m + j in four chains, so a score carries at most d / 32 + 6 roundings.  The
// keys are replaced by (score descending, id).
template <bool VEC>
__device__ __forceinline__ void score_candidates(const float* __restrict__ base, uint32_t d,
                                                 const float* q_s, uint64_t* buf, uint32_t cnt) {
  const uint32_t lane = lane_id(), g = lane >> 3, m = lane & 7u;
  for (uint32_t c0 = 0; c0 < cnt; c0 += 8) {
    const uint32_t i0 = min(c0 + g, cnt - 1), i1 = min(c0 + 4 + g, cnt - 1);
    const uint32_t id0 = static_cast<uint32_t>(buf[i0]), id1 = static_cast<uint32_t>(buf[i1]);
    const float* r0 = base + static_cast<uint64_t>(id0) * d;
    const float* r1 = base + static_cast<uint64_t>(id1) * d;
    float p0[4] = {0.f, 0.f, 0.f, 0.f}, p1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (uint32_t c = 4u * m; c < d; c += 32) {
      const float4 x = load4<VEC>(r0 + c), y = load4<VEC>(r1 + c);
      const float4 u = *reinterpret_cast<const float4*>(q_s + c);
      p0[0] = fmaf(u.x, x.x, p0[0]);
      p0[1] = fmaf(u.y, x.y, p0[1]);
      p0[2] = fmaf(u.z, x.z, p0[2]);
      p0[3] = fmaf(u.w, x.w, p0[3]);
      p1[0] = fmaf(u.x, y.x, p1[0]);
      p1[1] = fmaf(u.y, y.y, p1[1]);
      p1[2] = fmaf(u.z, y.z, p1[2]);
      p1[3] = fmaf(u.w, y.w, p1[3]);
    }
    // lanes with m < 4 reduce the first row, the others the second
    const float s0 = (p0[0] + p0[1]) + (p0[2] + p0[3]), s1 = (p1[0] + p1[1]) + (p1[2] + p1[3]);
    const bool up = (m & 4u) != 0;
    float t = (up ? s1 : s0) + __shfl_xor_sync(kFull, up ? s0 : s1, 4);
    t += __shfl_xor_sync(kFull, t, 2);
    t += __shfl_xor_sync(kFull, t, 1);
    __syncwarp();
    if (m == 0 && c0 + g < cnt) buf[c0 + g] = desc_key(t, id0);
    if (m == 4 && c0 + 4 + g < cnt) buf[c0 + 4 + g] = desc_key(t, id1);
    __syncwarp();
  }
}

template <int E>
__device__ __forceinline__ void sort_keys(uint64_t* buf, uint32_t cnt) {
  const uint32_t lane = lane_id();
  uint64_t key[E];
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    key[s] = i < cnt ? buf[i] : ~0ull;
  }
  __syncwarp();
  warp_sort_u64<E>(key);
#pragma unroll
  for (int s = 0; s < E; s++) {
    const uint32_t i = static_cast<uint32_t>(s) * 32u + lane;
    if (i < cnt) buf[i] = key[s];
  }
  __syncwarp();
}

template <uint32_t CAP>
__device__ void sort_any(uint64_t* buf, uint32_t cnt) {
  if (cnt <= 32)
    sort_keys<1>(buf, cnt);
  else if (cnt <= 64)
    sort_keys<2>(buf, cnt);
  else if (cnt <= 128)
    sort_keys<4>(buf, cnt);
  else if (CAP <= 256 || cnt <= 256)
    sort_keys<8>(buf, cnt);
  else if (cnt <= 512)
    sort_keys<16>(buf, cnt);
  else
    sort_keys<32>(buf, cnt);
}

// Warps (queries in flight) per block of the final pass, and its shared memory: per warp the keys,
// FP64 scores, link bits and the query, then the block's list of runs to settle.
template <bool LONG>
struct Final {
  static constexpr uint32_t kCap = LONG ? kGtCap : kGtShort;
  static constexpr uint32_t kWarps = LONG ? 4 : 8;
  static constexpr uint32_t kWarpBytes = kCap * 16 + kCap / 8;
  static size_t smem(uint32_t d) { return kWarps * (kWarpBytes + 4ull * d + kCap * 2); }
};

// One warp per query with at most kGtShort candidates (LONG: with more): the candidates, which hold
// the true top k, in the order of their FP64 inner products.  An FP32 score s is within E32 of the
// exact product and of its FP64 chain, E32 = (d / 32 + 9) 2^-24 |q| max|x|; candidates sorted by s
// whose neighbours lie farther than 2 E32 away are thereby in place.  Runs of closer ones that
// begin before place k are scored by the FP64 chain (ascending element order) and ordered by
// (score desc, id asc) inside their run.
// About three candidates of 140 are in such runs.  A warp-wide FP64 instruction occupies the FP64
// units equally long for three lanes as for 32, so the block's warps pool their runs and one lane
// takes one candidate.  250k queries of 200 floats, k = 128: 47 ms with an FP64 chain for every
// candidate, 17 ms with each warp settling its own runs, and 5.4 ms this way (row gathers and the
// sort).
template <bool LONG, bool VEC>
__global__ void __launch_bounds__(Final<LONG>::kWarps * 32) k_gt_final(GtArgs a) {
  extern __shared__ __align__(16) unsigned char final_smem[];
  using F = Final<LONG>;
  constexpr uint32_t CAP = F::kCap;
  __shared__ uint32_t listed;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t stride = F::kWarpBytes + 4 * a.d;
  unsigned char* mine = final_smem + warp * stride;
  uint64_t* buf = reinterpret_cast<uint64_t*>(mine);
  double* exact = reinterpret_cast<double*>(mine + CAP * 8);
  uint32_t* links = reinterpret_cast<uint32_t*>(mine + CAP * 16);
  float* q_s = reinterpret_cast<float*>(mine + F::kWarpBytes);
  uint16_t* list = reinterpret_cast<uint16_t*>(final_smem + F::kWarps * stride);  // warp, place
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * F::kWarps;
  const float xm = __fadd_ru(__uint_as_float(a.xmax[0]), __uint_as_float(a.xmax[1]));
  const float coef = static_cast<float>(a.d / 32u + 10u) * 5.9604645e-08f;  // one spare rounding
  if (threadIdx.x == 0) listed = 0;
  for (uint64_t row0 = blockIdx.x * static_cast<uint64_t>(F::kWarps); row0 < a.rows; row0 += nw) {
    const uint64_t row = row0 + warp;
    // the row's list is two halves of kGtCap / 2, one per half of the columns
    uint32_t c0 = 0, c1 = 0;
    if (row < a.rows) {
      c0 = min(a.cand_cnt[2 * row], kGtCap / 2);
      c1 = min(a.cand_cnt[2 * row + 1], kGtCap / 2);
    }
    uint32_t cnt = c0 + c1;
    const bool active = row < a.rows && (cnt > kGtShort) == LONG;
    if (!__syncthreads_or(active)) continue;
    auto linked = [&](uint32_t i) { return (links[i / 32] >> (i & 31u)) & 1u; };
    auto in_run = [&](uint32_t i) { return linked(i) || (i > 0 && linked(i - 1)); };
    auto run_start = [&](uint32_t i) {
      while (i > 0 && linked(i - 1)) i--;
      return i;
    };
    bool any = false;
    if (active) {
      const uint64_t* src = a.cand + row * kGtCap;
      const float* q = a.queries + row * a.d;
      for (uint32_t i = lane; i < c0; i += 32) buf[i] = src[i];
      for (uint32_t i = lane; i < c1; i += 32) buf[c0 + i] = src[kGtCap / 2 + i];
      for (uint32_t i = lane; i < a.d; i += 32) q_s[i] = q[i];
      __syncwarp();
      if (cnt > 2 * a.k) compact_any<CAP>(buf, cnt, a.k, a.band[row]);  // those >= t_k - band
      if (cnt) score_candidates<VEC>(a.base, a.d, q_s, buf, cnt);
      sort_any<CAP>(buf, cnt);
      const float gap = __fmul_ru(__fmul_ru(2.0f * coef, xm), __fadd_ru(a.qn[row], a.qe[row])) +
                        1e-37f;
      for (uint32_t i0 = 0; i0 < cnt; i0 += 32) {  // bit i: candidates i and i + 1 are too close
        const uint32_t i = i0 + lane;
        const bool l = i + 1 < cnt && !(key_value(buf[i]) - key_value(buf[i + 1]) > gap);
        const unsigned w = __ballot_sync(kFull, l);
        if (lane == 0) links[i0 / 32] = w;
        any |= w != 0;
      }
      __syncwarp();
      if (any)
        for (uint32_t i = lane; i < cnt; i += 32)
          if (in_run(i) && run_start(i) < a.k)
            list[atomicAdd(&listed, 1u)] = static_cast<uint16_t>(warp * CAP + i);
    }
    __syncthreads();
    const uint32_t total = listed;
    for (uint32_t t = threadIdx.x; t < total; t += blockDim.x) {
      const uint32_t w = list[t] / CAP, i = list[t] % CAP;
      unsigned char* its = final_smem + w * stride;
      const uint32_t id = static_cast<uint32_t>(reinterpret_cast<const uint64_t*>(its)[i]);
      const float* xr = a.base + static_cast<uint64_t>(id) * a.d;
      const float* qr = reinterpret_cast<const float*>(its + F::kWarpBytes);
      double acc = 0.0;
#pragma unroll 2
      for (uint32_t j = 0; j < a.d; j += 4) {
        const float4 x = load4<VEC>(xr + j);
        const float4 u = *reinterpret_cast<const float4*>(qr + j);
        acc = fma(static_cast<double>(u.x), static_cast<double>(x.x), acc);
        acc = fma(static_cast<double>(u.y), static_cast<double>(x.y), acc);
        acc = fma(static_cast<double>(u.z), static_cast<double>(x.z), acc);
        acc = fma(static_cast<double>(u.w), static_cast<double>(x.w), acc);
      }
      reinterpret_cast<double*>(its + CAP * 8)[i] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) listed = 0;  // the next use follows the loop's first barrier
    if (!active) continue;
    uint32_t* o = a.out + row * a.k;
    for (uint32_t i = lane; i < cnt; i += 32) {
      const uint32_t id = static_cast<uint32_t>(buf[i]);
      uint32_t pos = i;
      if (any && in_run(i)) {
        pos = run_start(i);
        if (pos < a.k) {
          const double mv = exact[i];
          for (uint32_t j = pos;; j++) {
            const double v = exact[j];
            if (v > mv || (v == mv && static_cast<uint32_t>(buf[j]) < id)) pos++;
            if (!linked(j)) break;
          }
        }
      }
      if (pos < a.k) o[pos] = id;
    }
    for (uint32_t i = cnt + lane; i < a.k; i += 32) o[i] = kTomb;
    __syncwarp();
  }
}

template <bool LONG>
cudaError_t launch_final(const GtArgs& f, int num_sms, cudaStream_t st) {
  using F = Final<LONG>;
  const bool vec = (reinterpret_cast<uintptr_t>(f.base) & 15u) == 0;
  auto kern = vec ? k_gt_final<LONG, true> : k_gt_final<LONG, false>;
  const size_t smem = F::smem(f.d);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, F::kWarps * 32, smem);
  if (e != cudaSuccess) return e;
  uint64_t blocks = (f.rows + F::kWarps - 1) / F::kWarps;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * (per_sm < 1 ? 1 : per_sm);
  if (blocks > cap) blocks = cap;
  kern<<<static_cast<unsigned>(blocks), F::kWarps * 32, smem, st>>>(f);
  return cudaGetLastError();
}

// The k-th largest of the values that `each` visits, given the smallest (mn) and largest (mx) of
// them and at least k of them; one warp.  A histogram of kThetaBins equal steps between the two finds
// the step that holds it; that step's few values are then gathered and ranked.  A step with more
// than kThetaBins of them (an outlier far above the rest) is divided again.  The values spread over
// the steps, so the shared-memory counters see few collisions, and three passes over them mostly
// do.
constexpr uint32_t kThetaBins = 512;
template <class Each>
__device__ float kth_largest(Each each, float mn, float mx, uint32_t k, uint32_t* hist,
                             uint32_t* fill) {
  const uint32_t lane = lane_id();
  uint32_t need = k;  // its rank among the values in [mn, mx]
  for (;;) {
    const float scale = static_cast<float>(kThetaBins - 1) / (mx - mn);
    // equal, or not divisible (a value out of range, which raised its error): all count
    if (!(mx > mn) || !(scale > 0.0f && scale < INFINITY)) break;
    const float low = mn, high = mx;
    auto bin = [&](float v) {  // non-decreasing in v
      return min(static_cast<uint32_t>((v - low) * scale), kThetaBins - 1);
    };
    for (uint32_t b = lane; b < kThetaBins; b += 32) hist[b] = 0;
    __syncwarp();
    each([&](float v) {
      if (v >= low && v <= high) atomicAdd(hist + bin(v), 1u);
    });
    __syncwarp();
    // lane l sums bins from the top: kThetaBins - 1 - 16 l downwards
    constexpr uint32_t kPer = kThetaBins / 32;
    uint32_t sum = 0;
    for (uint32_t t = 0; t < kPer; t++) sum += hist[kThetaBins - 1 - (lane * kPer + t)];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += y;
    }
    const uint32_t excl = incl - sum;
    const unsigned owner = __ballot_sync(kFull, excl < need && need <= incl);
    const int src = __ffs(static_cast<int>(owner)) - 1;
    uint32_t at = 0, above = 0, held = 0;
    if (static_cast<int>(lane) == src) {
      above = excl;
      for (uint32_t t = 0; t < kPer; t++) {
        at = kThetaBins - 1 - (lane * kPer + t);
        held = hist[at];
        if (above + held >= need) break;
        above += held;
      }
    }
    at = __shfl_sync(kFull, at, src);
    above = __shfl_sync(kFull, above, src);
    held = __shfl_sync(kFull, held, src);
    need -= above;
    __syncwarp();
    if (held <= kThetaBins) {  // its values in the counters' place; the need-th largest of them
      float* vals = reinterpret_cast<float*>(hist);
      if (lane == 0) *fill = 0;
      __syncwarp();
      each([&](float v) {
        if (v >= low && v <= high && bin(v) == at) vals[atomicAdd(fill, 1u)] = v;
      });
      __syncwarp();
      mn = INFINITY;
      for (uint32_t i = lane; i < held; i += 32) {
        const float v = vals[i];
        uint32_t gt = 0, eq = 0;
        for (uint32_t j = 0; j < held; j++) {
          gt += vals[j] > v ? 1u : 0u;
          eq += vals[j] == v ? 1u : 0u;
        }
        if (gt < need && need <= gt + eq) mn = v;
      }
      for (int o = 16; o > 0; o >>= 1) mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      __syncwarp();
      break;
    }
    mn = INFINITY;
    mx = -INFINITY;
    each([&](float v) {
      if (v >= low && v <= high && bin(v) == at) {
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
      }
    });
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
  }
  return mn;
}

// One warp per query: lo = theta - 2 E_q, theta the k-th largest of the row's group maxima (-inf
// when there are fewer than k groups: every base row is then a candidate).  3.4 -> 1.6 ms for 250k
// rows of 4700 maxima against a radix select, whose first of four histograms collides on the sign and
// exponent.
template <bool PAIRS>  // an even number of groups: rows start on 8 bytes
__global__ void __launch_bounds__(256) k_gt_theta(const float* __restrict__ maxima,
                                                  uint32_t rows, uint32_t groups, uint32_t k,
                                                  const float* __restrict__ band,
                                                  float* __restrict__ lo) {
  __shared__ uint32_t hist_all[8][kThetaBins];
  __shared__ uint32_t fill_all[8];
  uint32_t* hist = hist_all[threadIdx.x >> 5];
  uint32_t* fill = fill_all + (threadIdx.x >> 5);
  const uint32_t lane = lane_id();
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * 8;
  for (uint64_t row = blockIdx.x * 8ull + (threadIdx.x >> 5); row < rows; row += nw) {
    const float* m = maxima + row * groups;
    auto each = [&](auto&& use) {  // every maximum once, eight loads in flight per lane
      if constexpr (PAIRS) {
        const float2* m2 = reinterpret_cast<const float2*>(m);
#pragma unroll 8
        for (uint32_t i = lane; i < groups / 2; i += 32) {
          const float2 v = m2[i];
          use(v.x);
          use(v.y);
        }
      } else {
#pragma unroll 8
        for (uint32_t i = lane; i < groups; i += 32) use(m[i]);
      }
    };
    // the finite maxima's range and number (a group past the base's end is -inf)
    float mn = INFINITY, mx = -INFINITY;
    uint32_t have = 0;
    each([&](float v) {
      if (v > -INFINITY) {
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
        have++;
      }
    });
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
    have = __reduce_add_sync(kFull, have);
    if (have < k) {
      if (lane == 0) lo[row] = -INFINITY;
      continue;
    }
    const float theta = kth_largest(each, mn, mx, k, hist, fill);
    if (lane == 0) lo[row] = theta - band[row];
  }
}

// After a sampled threshold: one warp per query keeps, of its candidates, those within 2 E_q of the
// k-th largest screened score (all of them when there are no more than k), in the list's first half
// and then its second.  A query with more candidates than its list holds takes that bound, from those
// it does hold, as its threshold of another filter pass (`again` marks its tile of 128 queries); the
// others' thresholds become infinite, so that pass leaves them alone.  first: of the passes; the later
// ones look at the queries that were filtered again.  again == NULL: no pass follows.
__global__ void __launch_bounds__(128) k_gt_narrow(uint64_t* __restrict__ cand,
                                                   uint32_t* __restrict__ cand_cnt, uint32_t rows,
                                                   uint32_t k, const float* __restrict__ band,
                                                   float* __restrict__ lo,
                                                   uint32_t* __restrict__ again, bool first) {
  __shared__ uint64_t buf_all[4][kGtCap];
  __shared__ uint32_t hist_all[4][kThetaBins];
  __shared__ uint32_t fill_all[4];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint64_t* buf = buf_all[warp];
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * 4;
  for (uint64_t row = blockIdx.x * 4ull + warp; row < rows; row += nw) {
    if (!first && !(lo[row] < INFINITY)) continue;
    const uint32_t n0 = cand_cnt[2 * row], n1 = cand_cnt[2 * row + 1];
    const uint32_t c0 = min(n0, kGtCap / 2), c1 = min(n1, kGtCap / 2);
    const uint32_t cnt = c0 + c1;
    const bool more = again && cnt < n0 + n1;
    if (!more && lane == 0) lo[row] = INFINITY;
    if (cnt <= k) continue;
    uint64_t* list = cand + row * kGtCap;
    float mn = INFINITY, mx = -INFINITY;
    for (uint32_t i = lane; i < cnt; i += 32) {
      const uint64_t key = list[i < c0 ? i : kGtCap / 2 + (i - c0)];
      buf[i] = key;
      const float v = key_value(key);
      mn = fminf(mn, v);
      mx = fmaxf(mx, v);
    }
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
    __syncwarp();
    auto each = [&](auto&& use) {
      for (uint32_t i = lane; i < cnt; i += 32) use(key_value(buf[i]));
    };
    const float low = kth_largest(each, mn, mx, k, hist_all[warp], fill_all + warp) - band[row];
    if (more) {
      if (lane == 0) {
        lo[row] = fmaxf(lo[row], low);
        again[row / kGtTile] = 1;
      }
      __syncwarp();
      continue;
    }
    uint32_t kept = 0;
    for (uint32_t i0 = 0; i0 < cnt; i0 += 32) {
      const uint32_t i = i0 + lane;
      const uint64_t key = i < cnt ? buf[i] : 0;
      const bool keep = i < cnt && key_value(key) >= low;
      const unsigned m = __ballot_sync(kFull, keep);
      if (keep) list[kept + __popc(m & ((1u << lane) - 1u))] = key;
      kept += __popc(m);
    }
    if (lane == 0) {
      cand_cnt[2 * row] = min(kept, kGtCap / 2);
      cand_cnt[2 * row + 1] = kept - min(kept, kGtCap / 2);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- tcgen05 screening GEMM
//
// D (128 queries x BN base rows, FP32 in TMEM) = A (queries, FP16, K-major) . B (base rows,
// FP16, K-major)^T, K = dp in boxes of 64 elements (one 128-byte swizzled row per box row; the
// last box's columns past dp are read as zeros and its MMA K steps past dp are not issued).
// One CTA per SM, persistent over query tiles of 128 * MT rows (MT = 256 / BN M tiles sharing
// each B tile); for each query tile it sweeps every base tile in order:
//   warp 0      TMA producer: A tiles once per query tile, B boxes through a ring of stages;
//   warp 1      TMEM owner and MMA issuer (one thread): 4 MMAs (K = 16) per K box per M tile,
//               into one of two accumulator buffers per M tile;
//   warps 2..9  epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (one thread per query row)
//               and half of each tile's columns; each thread takes 128 scores per tile (4 chunks
//               of 32) with one TMEM wait, does the mode's work in straight-line code, then
//               releases the buffer.
// Every wait is bounded (1 s); a wait that gives up raises kErrWait, the CTA's roles stop, the
// issued MMAs are drained and the TMEM is freed before the CTA exits.
namespace tc {

using namespace tcu;

constexpr uint32_t kRows = 128;  // rows of an A tile (queries) and of a TMA box
constexpr uint32_t kChunk = 64;  // K elements per TMA box
constexpr uint32_t kBox = kRows * kChunk * 2;  // 16 KB
constexpr uint32_t kEpiWarps = 8;
constexpr uint32_t kThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kMaxKc = 8;  // dp <= 512
constexpr uint32_t kMinStages = 3, kMaxStages = 6;
constexpr uint32_t kHalfCap = kGtCap / 2;  // candidates per (query row, half of the columns)

// kind::f16 instruction descriptor: FP32 accumulator (bits 4-5 = 1), A and B FP16 (0), both
// K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
template <uint32_t BN>
constexpr uint32_t idesc() {
  return (1u << 4) | ((BN >> 3) << 17) | ((kRows >> 4) << 24);
}

enum Mode : int { kMax = 0, kFilter = 1, kDump = 2 };

struct Args {
  uint32_t q0;      // first row of this chunk in the query tensor map
  uint32_t nq;      // query rows of this chunk
  uint32_t n;       // base rows
  uint32_t kc;      // K boxes per row: ceil(dp / 64)
  uint32_t klast;   // MMA K steps (of 16) in the last box: 1 .. 4
  uint32_t stages;  // B ring stages
  // kMax: groups of base rows whose maxima are stored (groups per query row).  span > 0: a
  // group is `span` consecutive 32-column chunks of one thread (one half of each tile); span
  // == 0: a group is gs consecutive columns (gs < 32, for small n).
  uint32_t span, gs, groups;
  uint32_t step;    // kMax: every step-th base tile is swept (1 in the other modes)
  float* maxima;    // kMax: nq x groups
  const float* lo;  // kFilter: nq thresholds
  uint64_t* cand;   // kFilter: nq x kGtCap keys, two halves of kGtCap / 2
  uint32_t* cand_cnt;  // kFilter: nq x 2 (hits per half, also those past the list's end)
  // kFilter: the second pass after a sampled threshold sweeps the query tiles marked here, for their
  // rows with a finite threshold; NULL: every tile and row
  const uint32_t* again;
  bool refuse;  // kFilter: no pass follows that could bring a list past its end back
  float* dump;      // kDump: nq x n scores
  uint32_t* status;
};

template <uint32_t BN>
__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t acc) {
  mma_f16(d_tmem, a, b, idesc<BN>(), acc);
}

__device__ __forceinline__ float max32(const uint32_t* v) {  // pairwise tree, 31 FMNMX
  float m[16];
#pragma unroll
  for (int j = 0; j < 16; j++) m[j] = fmaxf(__uint_as_float(v[j]), __uint_as_float(v[j + 16]));
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1)
#pragma unroll
    for (int j = 0; j < w; j++) m[j] = fmaxf(m[j], m[j + w]);
  return m[0];
}

// Bits j of the 32 columns col0 + j that are < n.
__device__ __forceinline__ uint32_t in_range(uint32_t col0, uint32_t n) {
  if (col0 + 32 <= n) return 0xFFFFFFFFu;
  return col0 >= n ? 0u : ((1u << (n - col0)) - 1u);
}

template <uint32_t BN>
size_t smem_bytes(uint32_t kc, uint32_t stages) {
  constexpr uint32_t MT = 256 / BN;
  return 1024 + static_cast<size_t>(MT) * kc * kBox + static_cast<size_t>(stages) * BN * 128 + 256;
}

template <int MODE, uint32_t BN>
__global__ void __launch_bounds__(kThreads, 1)
    k_gt_tc(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
            const Args a) {
  constexpr uint32_t MT = 256 / BN;           // M tiles per query tile
  constexpr uint32_t kStageBytes = BN * 128;  // BN rows x 64 K x 2 bytes
  constexpr uint32_t kHalf = BN / 2;          // columns per epilogue thread per tile
  constexpr uint32_t kCpt = kHalf / 32;       // chunks per thread per tile and M tile
  static_assert(MT * kCpt == 4, "four 32-column chunks per thread per tile");
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* sm = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
  uint8_t* sA = sm;                                       // MT x kc boxes
  uint8_t* sB = sA + static_cast<size_t>(MT) * a.kc * kBox;  // stages x (BN rows x 128 bytes)
  uint64_t* full = reinterpret_cast<uint64_t*>(sB + static_cast<size_t>(a.stages) * kStageBytes);
  uint64_t* empty = full + a.stages;
  uint64_t* a_full = empty + a.stages;
  uint64_t* a_empty = a_full + 1;
  uint64_t* t_full = a_empty + 1;   // [2]
  uint64_t* t_empty = t_full + 2;   // [2]
  uint64_t* drained = t_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  volatile uint32_t* stop = tmem_slot + 1;

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  constexpr uint32_t rows_per_tile = kRows * MT;
  const uint32_t q_tiles = (a.nq + rows_per_tile - 1) / rows_per_tile;
  const uint32_t n_tiles = ((a.n + BN - 1) / BN + a.step - 1) / a.step;  // tiles swept
  constexpr uint32_t ncols = 2 * BN * MT;  // two accumulator buffers per M tile (512)
  auto swept = [&](uint32_t st) { return MODE != kFilter || !a.again || a.again[st] != 0; };
  if (MODE == kFilter && a.again) {  // mostly nothing to do
    bool any = false;
    for (uint32_t st = blockIdx.x; st < q_tiles; st += gridDim.x) any |= swept(st);
    if (!any) return;
  }

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < a.stages; s++) {
      bar_init(full + s, 1);
      bar_init(empty + s, 1);
    }
    bar_init(a_full, 1);
    bar_init(a_empty, 1);
    for (int b = 0; b < 2; b++) {
      bar_init(t_full + b, 1);
      bar_init(t_empty + b, 32 * kEpiWarps);
    }
    bar_init(drained, 1);
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     saddr(tmem_slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---- TMA producer
    if (lane == 0) {
      bool ok = true;
      uint32_t it = 0, sti = 0;
      for (uint32_t st = blockIdx.x; ok && st < q_tiles; st += gridDim.x) {
        if (!swept(st)) continue;
        const uint32_t sp = sti++ & 1u;
        if (!bar_wait(a_empty, sp ^ 1u, stop)) {
          ok = false;
          break;
        }
        bar_expect_tx(a_full, MT * a.kc * kBox);
        for (uint32_t m = 0; m < MT; m++)
          for (uint32_t c = 0; c < a.kc; c++)
            tma_load(sA + (m * a.kc + c) * kBox, &ta, c * kChunk,
                     a.q0 + st * rows_per_tile + m * kRows, a_full);
        for (uint32_t bt = 0; ok && bt < n_tiles; bt++)
          for (uint32_t c = 0; c < a.kc; c++, it++) {
            const uint32_t s = it % a.stages, ph = (it / a.stages) & 1u;
            if (!bar_wait(empty + s, ph ^ 1u, stop)) {
              ok = false;
              break;
            }
            bar_expect_tx(full + s, kStageBytes);
#pragma unroll
            for (uint32_t r = 0; r < BN / kRows; r++)
              tma_load(sB + s * kStageBytes + r * kBox, &tb, c * kChunk, bt * a.step * BN + r * kRows,
                       full + s);
          }
      }
      if (!ok) {
        raise_error(a.status, kErrWait);
        *stop = 1;
      }
      // the loads still in flight land before the CTA exits: each stage's last issued load
      for (uint32_t j = 0; j < a.stages && j < it; j++) {
        const uint32_t i = it - 1 - j;
        bar_wait(full + (i % a.stages), (i / a.stages) & 1u, nullptr);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer
    if (lane == 0) {
      bool ok = true;
      uint32_t it = 0, t = 0, sti = 0;
      const uint32_t a0 = saddr(sA), b0 = saddr(sB);
      for (uint32_t st = blockIdx.x; ok && st < q_tiles; st += gridDim.x) {
        if (!swept(st)) continue;
        const uint32_t sp = sti++ & 1u;
        if (!bar_wait(a_full, sp, stop)) {
          ok = false;
          break;
        }
        fence_after();
        for (uint32_t bt = 0; ok && bt < n_tiles; bt++, t++) {
          const uint32_t buf = t & 1u, use = t >> 1;
          if (!bar_wait(t_empty + buf, (use & 1u) ^ 1u, stop)) {
            ok = false;
            break;
          }
          fence_after();
          for (uint32_t c = 0; c < a.kc; c++, it++) {
            const uint32_t s = it % a.stages, ph = (it / a.stages) & 1u;
            if (!bar_wait(full + s, ph, stop)) {
              ok = false;
              break;
            }
            fence_after();
            const uint32_t ks = c + 1 == a.kc ? a.klast : 4u;  // zero columns past dp skipped
#pragma unroll
            for (uint32_t m = 0; m < MT; m++)
#pragma unroll
              for (uint32_t k = 0; k < 4; k++)
                if (k < ks)
                  mma<BN>(tmem + (m * 2 + buf) * BN,
                          sw128_desc(a0 + (m * a.kc + c) * kBox + k * 32),
                          sw128_desc(b0 + s * kStageBytes + k * 32), (c | k) != 0);
            commit(empty + s);  // the stage is free once these MMAs have read it
          }
          if (ok) commit(t_full + buf);
        }
        if (ok) commit(a_empty);
      }
      if (!ok) {
        raise_error(a.status, kErrWait);
        *stop = 1;
      }
      if (sti) {
        commit(drained);  // arrives when every MMA issued above has completed
        bar_wait(drained, 0, nullptr);
      }
    }
  } else {
    // ---- epilogue: one thread per (query row, half of the tile's columns)
    const uint32_t quarter = warp & 3u;
    const uint32_t half = (warp - 2) >> 2;
    const uint32_t row = quarter * 32u + lane;
    const uint32_t lane_base = (quarter * 32u) << 16;
    bool ok = true;
    uint32_t t = 0;
    const uint32_t chunks = n_tiles * kCpt;  // this thread's 32-column chunks per M tile
    uint32_t st = blockIdx.x;
    for (; st < q_tiles; st += gridDim.x) {
      if (!swept(st)) continue;
      uint32_t qrow[MT], cnt[MT];
      bool valid[MT];
      float lo[MT], run[MT];
#pragma unroll
      for (uint32_t m = 0; m < MT; m++) {
        qrow[m] = st * rows_per_tile + m * kRows + row;
        valid[m] = qrow[m] < a.nq;
        lo[m] = (MODE == kFilter && valid[m]) ? a.lo[qrow[m]] : INFINITY;
        if (MODE == kFilter && a.again) valid[m] = lo[m] < INFINITY;
        run[m] = -INFINITY;
        cnt[m] = 0;
      }
      for (uint32_t bt = 0; bt < n_tiles; bt++, t++) {
        const uint32_t buf = t & 1u, use = t >> 1;
        ok = __all_sync(kFull, bar_wait(t_full + buf, use & 1u, stop));
        if (!ok) break;
        fence_after();
        uint32_t v[4][32];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
          const uint32_t m = i / kCpt, ch = i % kCpt;
          tmem_ld32(tmem + lane_base + (m * 2 + buf) * BN + half * kHalf + ch * 32, v[i]);
        }
        tmem_wait_ld();
        fence_before();
        bar_arrive(t_empty + buf);  // the scores are in registers: the buffer is free
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
          const uint32_t m = i / kCpt, ch = i % kCpt;
          if (!valid[m]) continue;
          const uint32_t col0 = bt * a.step * BN + half * kHalf + ch * 32;
          const uint32_t inr = in_range(col0, a.n);
          if (MODE == kMax) {
            if (a.span) {
              float mx = max32(v[i]);
              if (inr != 0xFFFFFFFFu) {  // the last tile: only columns < n count
                mx = -INFINITY;
#pragma unroll
                for (uint32_t j = 0; j < 32; j++)
                  if ((inr >> j) & 1u) mx = fmaxf(mx, __uint_as_float(v[i][j]));
              }
              run[m] = fmaxf(run[m], mx);
              const uint32_t u = bt * kCpt + ch;  // this thread's chunk index
              if (((u + 1) & (a.span - 1)) == 0 || u + 1 == chunks) {
                a.maxima[static_cast<uint64_t>(qrow[m]) * a.groups + (u / a.span) * 2 + half] =
                    run[m];
                run[m] = -INFINITY;
              }
            } else {  // small n: groups of gs < 32 columns
#pragma unroll
              for (uint32_t j = 0; j < 32; j++) {
                const uint32_t c = col0 + j;
                if ((inr >> j) & 1u) {
                  run[m] = fmaxf(run[m], __uint_as_float(v[i][j]));
                  if (((c + 1) & (a.gs - 1)) == 0 || c + 1 == a.n) {
                    a.maxima[static_cast<uint64_t>(qrow[m]) * a.groups + c / a.gs] = run[m];
                    run[m] = -INFINITY;
                  }
                }
              }
            }
          } else if (MODE == kFilter) {
            uint32_t hit = 0;
#pragma unroll
            for (uint32_t j = 0; j < 32; j++)
              hit |= (__uint_as_float(v[i][j]) >= lo[m]) ? (1u << j) : 0u;
            hit &= inr;
            if (hit) {  // rare (about 1.1 k hits per row): a short loop over a local copy, so the
                        // unrolled common path stays small in the instruction cache
              float tmp[32];
#pragma unroll
              for (uint32_t j = 0; j < 32; j++) tmp[j] = __uint_as_float(v[i][j]);
              uint64_t* dst = a.cand + static_cast<uint64_t>(qrow[m]) * kGtCap + half * kHalfCap;
#pragma unroll 1
              while (hit) {
                const uint32_t j = static_cast<uint32_t>(__ffs(static_cast<int>(hit)) - 1);
                const uint32_t c = cnt[m];
                uint32_t at = c, pop = 1;
                if (c < kHalfCap) {
                  hit &= hit - 1u;
                } else {  // past its end the list stays a sample of the hits, whose k-th best is then
                          // worth most as the next threshold: one of these may take a place
                  pop = __popc(hit);
                  at = __umulhi(c * 0x9E3779B1u, c + pop) / pop;
                  hit = 0;
                }
                if (at < kHalfCap) dst[at] = desc_key(tmp[j], col0 + j);
                cnt[m] = c + pop;
              }
            }
          } else {
            float* o = a.dump + static_cast<uint64_t>(qrow[m]) * a.n;
#pragma unroll
            for (uint32_t j = 0; j < 32; j++)
              if ((inr >> j) & 1u) o[col0 + j] = __uint_as_float(v[i][j]);
          }
        }
      }
      if (!ok) break;
      if (MODE == kFilter) {
        // each half of a row keeps its candidates in its own half of the row's list
#pragma unroll
        for (uint32_t m = 0; m < MT; m++)
          if (valid[m]) {
            a.cand_cnt[static_cast<uint64_t>(qrow[m]) * 2 + half] = cnt[m];
            if (cnt[m] > kHalfCap && a.refuse) raise_error(a.status, kGtErrFinal);
          }
      }
    }
    if (!ok) {
      if (lane == 0) {
        raise_error(a.status, kErrWait);
        *stop = 1;
      }
      // the queries not reached have no candidates: the kernels that follow read rows by id
      if (MODE == kFilter)
        for (; st < q_tiles; st += gridDim.x)
#pragma unroll
          for (uint32_t m = 0; m < MT; m++) {
            const uint32_t r = st * rows_per_tile + m * kRows + row;
            if (r < a.nq) a.cand_cnt[static_cast<uint64_t>(r) * 2 + half] = 0;
          }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(ncols)
                 : "memory");
  }
}

// A rows x dp FP16 matrix (row stride dp * 2 bytes, a multiple of 32) as TMA boxes of
// 64 x 128 with 128-byte swizzling; rows and columns past the end read as zeros.
bool make_map(CUtensorMap* m, const __half* p, uint64_t rows, uint32_t dp) {
  EncodeTiled enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {dp, rows};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(dp) * 2};
  const cuuint32_t box[2] = {kChunk, kRows};
  const cuuint32_t elem[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(p), dims, strides, box,
             elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <uint32_t BN>
uint32_t stages_for(uint32_t kc, size_t smem_optin) {
  uint32_t s = kMaxStages;
  while (s > kMinStages && smem_bytes<BN>(kc, s) > smem_optin) s--;
  return smem_bytes<BN>(kc, s) <= smem_optin ? s : 0;
}

template <int MODE, uint32_t BN>
cudaError_t launch_bn(const CUtensorMap& ta, const CUtensorMap& tb, const Args& a, int num_sms,
                      cudaStream_t st) {
  const size_t smem = smem_bytes<BN>(a.kc, a.stages);
  auto kern = k_gt_tc<MODE, BN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  constexpr uint32_t rows_per_tile = kRows * (256 / BN);
  const uint32_t q_tiles = (a.nq + rows_per_tile - 1) / rows_per_tile;
  const uint32_t grid = q_tiles < static_cast<uint32_t>(num_sms) ? q_tiles
                                                                  : static_cast<uint32_t>(num_sms);
  kern<<<grid ? grid : 1, kThreads, smem, st>>>(ta, tb, a);
  return cudaGetLastError();
}

// The launched shape: 256 base rows per tile against one 128-row query tile (measured faster
// than 128 base rows against two query tiles: 1.12 s against 1.28 s for 1M x 1M x 200).
constexpr uint32_t kBN = 256;
static_assert(kRows * (256 / kBN) == kGtTile, "query rows per tile");

template <int MODE>
cudaError_t launch(const CUtensorMap& ta, const CUtensorMap& tb, const Args& a, int num_sms,
                   cudaStream_t st) {
  return launch_bn<MODE, kBN>(ta, tb, a, num_sms, st);
}

}  // namespace tc

int blocks_for(uint64_t warps, int per_block, int num_sms, int per_sm) {
  uint64_t b = (warps + per_block - 1) / per_block;
  const uint64_t cap = static_cast<uint64_t>(num_sms) * per_sm;
  if (b > cap) b = cap;
  return static_cast<int>(b ? b : 1);
}

// FP16 rows are zero-padded to a multiple of 16 elements (one MMA K step); TMA reads the last
// 64-element box past the row end as zeros.
uint32_t padded_dim(uint32_t d) { return (d + 15) / 16 * 16; }
uint32_t k_boxes(uint32_t dp) { return (dp + tc::kChunk - 1) / tc::kChunk; }
uint32_t k_last(uint32_t dp) { return (dp - (k_boxes(dp) - 1) * tc::kChunk) / 16; }

}  // namespace

uint32_t gt_max_k() { return 256; }

uint32_t gt_max_dim() { return tc::kChunk * tc::kMaxKc; }

GtPlan gt_plan(uint64_t n, uint64_t nq, uint32_t d, uint32_t k, bool sampled, int num_sms,
               size_t smem_optin) {
  GtPlan p{};
  p.dp = padded_dim(d);
  p.kc = k_boxes(p.dp);
  p.bn = tc::kBN;
  p.stages = tc::stages_for<tc::kBN>(p.kc, smem_optin);
  // groups of base rows for the threshold pass, about 4096 or more per query where n allows:
  // each epilogue thread's chunks (32 columns of one half of each tile), `span` at a time, or
  // for small n groups of gs < 32 columns
  const uint64_t n_tiles = (n + p.bn - 1) / p.bn;
  const uint64_t chunks = n_tiles * (p.bn / 64);  // per thread
  // A sample of the base, every step-th tile, gives a threshold too: the k-th largest of its group
  // maxima is the score of k distinct rows.  Then about k step rows pass the filter, so step keeps
  // them well inside the selection's room, and the sample keeps 16 k groups.
  p.step = 1;
  if (sampled && 2 * chunks >= 4096)
    while (p.step < 8 && 2ull * p.step * k <= 560 && chunks / p.step >= 16ull * k) p.step *= 2;
  const uint64_t swept = (n_tiles + p.step - 1) / p.step * (p.bn / 64);
  if (2 * chunks >= 4096) {
    p.span = 1;
    while (2 * ((swept + 2 * p.span - 1) / (2 * p.span)) >= 4096) p.span *= 2;
    p.gs = 0;
    p.groups = static_cast<uint32_t>(2 * ((swept + p.span - 1) / p.span));
  } else {
    p.span = 0;
    p.gs = 1;
    while (p.gs < 16 && n / (2ull * p.gs) >= 4096) p.gs *= 2;
    p.groups = static_cast<uint32_t>((n + p.gs - 1) / p.gs);
  }
  // queries per chunk: whole waves of query tiles, the chunk's maxima and candidate lists
  // within 4 GB
  const uint64_t wave = 256ull * static_cast<uint64_t>(num_sms);
  const uint64_t per_q = static_cast<uint64_t>(p.groups) * 4 + kGtCap * 8 + 16;
  uint64_t cq = (4ull << 30) / per_q / wave * wave;
  if (cq < 256) cq = 256;
  if (cq > nq) cq = nq;
  p.cq = cq;
  return p;
}

size_t gt_workspace_bytes(const GtPlan& p, uint64_t n, uint64_t nq) {
  auto al = [](uint64_t b) { return (b + 1023) & ~1023ull; };
  return al(n * p.dp * 2) + al(nq * p.dp * 2) + 2 * al(n * 4) + 2 * al(nq * 4) + al(8) +
         2 * al(p.cq * 4) + al(p.cq * p.groups * 4) + al(p.cq * kGtCap * 8) + al(p.cq * 8) +
         al(kGtAgain * ((p.cq + kGtTile - 1) / kGtTile) * 4);
}

int ground_truth(const GtPlan& plan, const float* base, uint64_t n, uint32_t d,
                 const float* queries, uint64_t nq, uint32_t k, uint32_t* out, char* ws,
                 uint32_t* status, int num_sms, cudaStream_t st, float* diag) {
  const uint32_t dp = plan.dp;
  const uint64_t cq = plan.cq;
  auto al = [](uint64_t b) { return (b + 1023) & ~1023ull; };
  char* p = ws;
  auto take = [&](uint64_t bytes) {
    char* r = p;
    p += al(bytes);
    return r;
  };
  __half* b16 = reinterpret_cast<__half*>(take(n * dp * 2));
  __half* q16 = reinterpret_cast<__half*>(take(nq * dp * 2));
  float* bn = reinterpret_cast<float*>(take(n * 4));
  float* be = reinterpret_cast<float*>(take(n * 4));
  float* qn = reinterpret_cast<float*>(take(nq * 4));
  float* qe = reinterpret_cast<float*>(take(nq * 4));
  uint32_t* xmax = reinterpret_cast<uint32_t*>(take(8));
  float* band = reinterpret_cast<float*>(take(cq * 4));
  float* lo = reinterpret_cast<float*>(take(cq * 4));
  float* maxima = reinterpret_cast<float*>(take(cq * plan.groups * 4));
  uint64_t* cand = reinterpret_cast<uint64_t*>(take(cq * kGtCap * 8));
  uint32_t* cand_cnt = reinterpret_cast<uint32_t*>(take(cq * 8));
  const uint64_t again_words = (cq + kGtTile - 1) / kGtTile;
  uint32_t* again = reinterpret_cast<uint32_t*>(take(kGtAgain * again_words * 4));

  cudaError_t e;
  k_half_rows<<<blocks_for(n, 8, num_sms, 8), 256, 0, st>>>(base, n, d, dp, b16, bn, be, status);
  k_half_rows<<<blocks_for(nq, 8, num_sms, 8), 256, 0, st>>>(queries, nq, d, dp, q16, qn, qe,
                                                               status);
  if ((e = cudaMemsetAsync(xmax, 0, 8, st)) != cudaSuccess) return -static_cast<int>(e);
  {
    uint64_t g = (n + 255) / 256;
    if (g > static_cast<uint64_t>(num_sms) * 4) g = static_cast<uint64_t>(num_sms) * 4;
    k_max2<<<static_cast<unsigned>(g ? g : 1), 256, 0, st>>>(bn, be, n, xmax);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return -static_cast<int>(e);
  CUtensorMap ta, tb;
  if (!tc::make_map(&ta, q16, nq, dp) || !tc::make_map(&tb, b16, n, dp)) return 1;
  for (uint64_t q0 = 0; q0 < nq; q0 += cq) {
    const uint32_t rows = static_cast<uint32_t>(min(cq, nq - q0));
    k_gt_band<<<(rows + 255) / 256, 256, 0, st>>>(qn + q0, qe + q0, xmax, rows, dp, band);
    tc::Args a{};
    a.q0 = static_cast<uint32_t>(q0);
    a.nq = rows;
    a.n = static_cast<uint32_t>(n);
    a.kc = plan.kc;
    a.klast = k_last(dp);
    a.stages = plan.stages;
    a.span = plan.span;
    a.gs = plan.gs;
    a.groups = plan.groups;
    a.step = plan.step;
    a.maxima = maxima;
    a.lo = lo;
    a.cand = cand;
    a.cand_cnt = cand_cnt;
    a.status = status;
    if ((e = tc::launch<tc::kMax>(ta, tb, a, num_sms, st)) != cudaSuccess)
      return -static_cast<int>(e);
    auto theta = plan.groups % 2 ? k_gt_theta<false> : k_gt_theta<true>;
    theta<<<blocks_for(rows, 8, num_sms, 8), 256, 0, st>>>(maxima, rows, plan.groups, k, band, lo);
    a.step = 1;
    a.refuse = plan.step == 1;
    if ((e = tc::launch<tc::kFilter>(ta, tb, a, num_sms, st)) != cudaSuccess)
      return -static_cast<int>(e);
    if (plan.step > 1) {
      const int blocks = blocks_for(rows, 4, num_sms, 12);
      if ((e = cudaMemsetAsync(again, 0, kGtAgain * again_words * 4, st)) != cudaSuccess)
        return -static_cast<int>(e);
      for (int pass = 0; pass < kGtAgain; pass++) {
        uint32_t* marks = again + pass * again_words;
        k_gt_narrow<<<blocks, 128, 0, st>>>(cand, cand_cnt, rows, k, band, lo, marks, pass == 0);
        a.again = marks;
        a.refuse = pass + 1 == kGtAgain;
        if ((e = tc::launch<tc::kFilter>(ta, tb, a, num_sms, st)) != cudaSuccess)
          return -static_cast<int>(e);
      }
      k_gt_narrow<<<blocks, 128, 0, st>>>(cand, cand_cnt, rows, k, band, lo, nullptr, false);
    }
    GtArgs f{};
    f.base = base;
    f.queries = queries + q0 * d;
    f.d = d;
    f.k = k;
    f.rows = rows;
    f.cand = cand;
    f.cand_cnt = cand_cnt;
    f.band = band;
    f.qn = qn + q0;
    f.qe = qe + q0;
    f.xmax = xmax;
    f.out = out + q0 * k;
    // most lists are short; the long ones take a kernel with room for them
    if ((e = launch_final<false>(f, num_sms, st)) != cudaSuccess) return -static_cast<int>(e);
    if ((e = launch_final<true>(f, num_sms, st)) != cudaSuccess)
      return -static_cast<int>(e);
    if (diag && q0 == 0) {  // the first query's margin and the base's largest norms
      if ((e = cudaMemcpyAsync(diag, band, 4, cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
        return -static_cast<int>(e);
      if ((e = cudaMemcpyAsync(diag + 1, xmax, 8, cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
        return -static_cast<int>(e);
    }
  }
  return 0;
}

size_t screen_scores_workspace(uint64_t na, uint64_t nb, uint32_t d) {
  auto al = [](uint64_t b) { return (b + 1023) & ~1023ull; };
  const uint32_t dp = padded_dim(d);
  return al(na * dp * 2) + al(nb * dp * 2) + 2 * al(na * 4) + 2 * al(nb * 4);
}

int screen_scores(const float* a, uint64_t na, const float* b, uint64_t nb, uint32_t d,
                  float* out, char* ws, uint32_t* status, int num_sms, size_t smem_optin,
                  cudaStream_t st) {
  const uint32_t dp = padded_dim(d);
  auto al = [](uint64_t x) { return (x + 1023) & ~1023ull; };
  char* p = ws;
  auto take = [&](uint64_t bytes) {
    char* r = p;
    p += al(bytes);
    return r;
  };
  __half* a16 = reinterpret_cast<__half*>(take(na * dp * 2));
  __half* b16 = reinterpret_cast<__half*>(take(nb * dp * 2));
  float* an = reinterpret_cast<float*>(take(na * 4));
  float* ae = reinterpret_cast<float*>(take(na * 4));
  float* bn = reinterpret_cast<float*>(take(nb * 4));
  float* be = reinterpret_cast<float*>(take(nb * 4));
  k_half_rows<<<blocks_for(na, 8, num_sms, 8), 256, 0, st>>>(a, na, d, dp, a16, an, ae, status);
  k_half_rows<<<blocks_for(nb, 8, num_sms, 8), 256, 0, st>>>(b, nb, d, dp, b16, bn, be, status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return -static_cast<int>(e);
  CUtensorMap ta, tb;
  if (!tc::make_map(&ta, a16, na, dp) || !tc::make_map(&tb, b16, nb, dp)) return 1;
  tc::Args x{};
  x.q0 = 0;
  x.nq = static_cast<uint32_t>(na);
  x.n = static_cast<uint32_t>(nb);
  x.kc = k_boxes(dp);
  x.klast = k_last(dp);
  x.stages = tc::stages_for<tc::kBN>(x.kc, smem_optin);
  x.span = 1;
  x.groups = 1;
  x.step = 1;
  x.dump = out;
  x.status = status;
  e = tc::launch<tc::kDump>(ta, tb, x, num_sms, st);
  return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

}  // namespace pg
