// Hash-probe intersection kernels: triangle counting, set-similarity search,
// the raw two-set intersection, and conjunctive retrieval.
//
// Reference kernels: dynamic_triangle_count (triangle-count/TC.cu:128-190),
// set_similarity_search_kernel (set-similarity-search/sss.cu:93-154),
// intersection_kernel (set_size/intersection.cu:154-181), ir_kernel
// (information-retrieval/ir.cu:94-176).  All share the probe rule of
// search_in_hashtable (TC.cu:11-31): walk the slots of the home bucket, then
// the next bucket; a hit is an equal slot, a miss an empty (-1) slot.
//
// Scheduling (B200): the reference gives every pair a whole warp, so a warp
// probing a 3-element set idles 29 lanes.  Here a warp takes 32 pairs (one
// per lane), loads each pair's two packed 16-byte set descriptors, and
// flattens the probes of all 32 pairs: round r gives lane i the probe with
// flat index 32r+i, found by a 5-step shuffle binary search over the pairs'
// prefix sums.  Tiny intersections thus run at thread granularity, medium
// ones spread over the warp, and hub x hub pairs over as many rounds as
// they need; the grid is persistent and walks 32-pair chunks grid-stride.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "probe_common.cuh"

namespace rst {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kIrSlice = 512;  // candidates per IR work item
constexpr int64_t kOwnerEdges = 1 << 19;  // edges from which they are grouped by owner

// ----------------------------------------------------------------- TC ----

// desc, kcols: the key rows; off, cols, chunk_row: the edges (u, v), whose rows
// are intersected.  OWN: every edge's hits are also added to owner_hits[u].
template <bool HIER, int ROUNDS, bool LEAN, bool OWN = false>
__global__ void __launch_bounds__(kThreads, 4)
    tc_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ kcols,
              const int32_t* __restrict__ off, const int32_t* __restrict__ cols,
              const int32_t* __restrict__ chunk_row, int32_t n, int64_t m,
              const int32_t* __restrict__ table, int64_t bn, int b, int lg_max,
              unsigned long long* __restrict__ count,
              unsigned long long* __restrict__ owner_hits,
              unsigned long long* __restrict__ cursor, int lg_grab, int warp_pair_min,
              int32_t* __restrict__ status) {
  __shared__ int s_qx[kWarps][32 * ROUNDS], s_qh[kWarps][32 * ROUNDS];
  __shared__ int s_own[OWN ? kWarps : 1][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // edges past off[n] have no row: never read them (nor their chunk rows)
  const int64_t me = min(m, (int64_t)__ldg(off + n));
  const int grab = 1 << lg_grab;  // edges a warp takes at a time, at most 32
  const int64_t n_grabs = (me + grab - 1) >> lg_grab;
  unsigned long long hits = 0;
  // dynamic schedule: a warp takes the next edges when it is done
  for (;;) {
    unsigned long long cc = 0;
    if (lane == 0) cc = atomicAdd(cursor, 1ull);
    const int64_t c = (int64_t)__shfl_sync(kFull, cc, 0);
    if (c >= n_grabs) break;
    const int64_t e0 = c << lg_grab, e64 = e0 + lane;
    const bool valid = lane < grab && e64 < me;
    const int e = (int)min(e0 + min(lane, grab - 1), me - 1);
    int u0 = __ldg(chunk_row + (e0 >> 5));
    if ((unsigned)u0 >= (unsigned)n) u0 = 0;
    int u = row_of_edge(off, n, u0, e);
    int v = __ldg(cols + e);
    bool ok = valid;
    if ((unsigned)u >= (unsigned)n || (unsigned)v >= (unsigned)n) {
      if (valid) atomicOr(status, kErrBadId);
      ok = false;
      u = v = 0;
    }
    const int4 du = __ldg(desc + u);
    const int4 dv = __ldg(desc + v);
    // TC.cu:148-157: the larger set's table is probed (ties: u probes v).
    const bool sw = du.y > dv.y;
    const int4 A = sw ? dv : du;
    const int4 B = sw ? du : dv;
    const int s = ok ? A.y : 0;
    // pairs with a warp's worth of keys get the whole warp, one at a time;
    // the rest are flattened across the lanes
    const bool big = s >= warp_pair_min;
    unsigned bigm = __ballot_sync(kFull, big);
    const int64_t bt = desc_toff(B);
    const int blg = desc_lg(B);
    if (OWN) {
      s_own[warp][lane] = 0;
      __syncwarp();
    }
    while (bigm) {
      const int k = __ffs(bigm) - 1;
      bigm &= bigm - 1;
      const int ks = __shfl_sync(kFull, s, k);
      const int ka = __shfl_sync(kFull, A.x, k);
      const int klg = __shfl_sync(kFull, blg, k);
      const int64_t kt = __shfl_sync(kFull, bt, k);
      int h;
      if (LEAN)
        h = warp_probe_pair_lean<HIER, ROUNDS>(kcols + ka, ks, table + kt, klg, lg_max, bn, b,
                                               status, s_qx[warp], s_qh[warp]);
      else
        h = warp_probe_pair<HIER, ROUNDS>(kcols + ka, ks, table + kt, klg, lg_max, bn, b, status,
                                          s_qx[warp], s_qh[warp]);
      hits += h;
      if (OWN) {
        h = __reduce_add_sync(kFull, h);
        if (lane == 0) s_own[warp][k] = h;
      }
    }
    hits += flat_probe<HIER>(kcols, table, big ? 0 : s, A.x, bt, blg, lg_max, bn, b, status,
                             [&](int k) {
                               if (OWN) atomicAdd(&s_own[warp][k], 1);
                             });
    if (OWN) {
      __syncwarp();
      if (s_own[warp][lane])
        atomicAdd(owner_hits + u, (unsigned long long)(unsigned)s_own[warp][lane]);
      __syncwarp();
    }
  }
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(count, hits);
}

// ---------------------------------------------------------------- SSS ----

// Decisions only, for runs of pairs that share their first set (a join's): a
// bitmap of the shared set's hashed keys in the warp's shared memory, past
// which the other sets' first keys stream with full lines, where probing
// reads a sector or two of HBM per key (and is bound by them).  It can only
// take keys for common that are not, so a pair with more misses than its
// decision allows is settled; the few others are decided by the tables.
// 5.4 M candidate pairs of sets of up to 1024 keys: 2.87 ms without the
// bitmap, 1.84 with it.  Pairs in no order never fill one.
//
// It is taken where it is likely to settle its pairs and costs less than the
// lookups that it spares, and given up where the keys streamed show that the
// sets share too much.  us a call, no bitmap / every run / by this rule:
// 400,000 pairs of one set, at 1/100 with 100 keys and 5000 a set 302 / 5060 /
// 311; 2000 keys a set that share a third, at 7/10 873 / 1358 / 899, at 1/10
// 1461 / 3598 / 1491; 2000 keys that share 2%, at 1/10 4330 / 2063 / 2127.
constexpr int kFilterBits = 16384;
constexpr int kFilterWords = kFilterBits / 32;
constexpr int kFilterMax = 4096;  // keys of the shared set: a quarter of the bits, past
                                  // which too many unlike keys are taken for common
constexpr int kFilterRun = 3;     // a run that pays for clearing and filling the bitmap
constexpr int kFilterLook = 512;  // keys after which a stream is first looked at
constexpr int kFilterStream = 1 << 25;  // keys streamed for a pair: 32 of them fit an int

__device__ __forceinline__ unsigned filter_hash(int x) { return (unsigned)x * 0x9E3779B1u; }

// Enters the keys of a row; false if they do not ascend (repeated keys count
// as often as they occur, which the bitmap does not tell).
__device__ __forceinline__ bool filter_fill(const int32_t* __restrict__ row, int n,
                                            uint32_t* bits) {
  const int lane = threadIdx.x & 31;
  for (int i = lane; i < kFilterWords / 4; i += 32)
    reinterpret_cast<int4*>(bits)[i] = make_int4(0, 0, 0, 0);
  __syncwarp();
  bool ok = true;
#pragma unroll 4
  for (int j = lane; j < n; j += 32) {
    const int x = __ldg(row + j);
    ok = ok && (j == 0 || __ldg(row + j - 1) < x);
    const unsigned h = filter_hash(x);
    atomicOr(bits + (h >> 23), 1u << (h >> 18 & 31));
  }
  __syncwarp();
  return __all_sync(kFull, ok);
}

// The first n <= kFilterStream keys of every lane's row (start in elems)
// looked up in the bitmap, flattened across the lanes; counts into hits[lane].
// Given up (false) where clearly more than `most` of the keys so far are held.
__device__ __forceinline__ bool filter_stream(const int32_t* __restrict__ elems, int start, int n,
                                              float most, const uint32_t* bits, int* hits) {
  constexpr int R = 4;
  const int lane = threadIdx.x & 31;
  int total, look = kFilterLook;
  const int P = warp_excl_scan(n, &total);
  const int src = start - P;
  for (int base = 0; base < total; base += 32 * R) {
    if (base == look) {  // (a look at 512, 1024, ... keys; three standard deviations)
      const float mean = most * (float)base;
      if ((float)__reduce_add_sync(kFull, hits[lane]) > mean + 3.f * sqrtf(mean)) return false;
      if (look <= kFilterStream) look *= 2;
    }
    int x[R], k[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int f = base + r * 32 + lane;
      k[r] = owner_lane(P, f);
      const int at = __shfl_sync(kFull, src, k[r]) + f;
      x[r] = f < total ? __ldg(elems + at) : 0;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned h = filter_hash(x[r]);
      const bool hit = base + r * 32 + lane < total && (bits[h >> 23] >> (h >> 18 & 31) & 1u);
      const int k0 = __shfl_sync(kFull, k[r], 0);
      if (__all_sync(kFull, k[r] == k0)) {
        const int c = __popc(__ballot_sync(kFull, hit));
        if (lane == 0) hits[k0] += c;
      } else if (hit) {
        atomicAdd(hits + k[r], 1);
      }
      __syncwarp();
    }
  }
  return true;
}

template <bool HIER, bool FLOAT_RULE, int ROUNDS, bool LEAN, bool EARLY = false>
__global__ void __launch_bounds__(kThreads, 4)
    sss_kernel(const int4* __restrict__ desc, int32_t n,
               const int32_t* __restrict__ elems,
               const int32_t* __restrict__ pa, const int32_t* __restrict__ pb,
               int64_t np, const int64_t* __restrict__ np_dev,
               unsigned long long* __restrict__ cursor, int lg_grab,
               const int32_t* __restrict__ table, int64_t bn, int b,
               int lg_max, int num, int den, float thr, int warp_pair_min,
               uint8_t* __restrict__ flags, int32_t* __restrict__ inter,
               int32_t* __restrict__ status) {
  __shared__ int s_hits[kWarps][32];
  // a warp's queue of open probes, and between probes the bitmap of a run: 16 KB
  // more of shared memory are 16 KB less of L1, which whole rows of sorted keys
  // need (400,000 pairs of 4000 keys at 1/100: 18.2 ms with both, 15.4 this way)
  __shared__ __align__(16) int s_queue[kWarps][64 * ROUNDS];
  static_assert(!EARLY || 64 * ROUNDS >= kFilterWords, "the bitmap lies in the queue");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* const qx = s_queue[warp];
  int* const qh = qx + 32 * ROUNDS;
  int pause = 0;  // 1: the last bitmap settled nothing; more: runs to leave out
  if (np_dev) np = *np_dev;  // pair count set on the device (captured graphs)
  const int grab = 1 << lg_grab;  // pairs a warp takes at a time, at most 32
  const int64_t n_chunks = (np + grab - 1) >> lg_grab;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t it = 0;; ++it) {
    int64_t c;
    if (cursor) {  // dynamic schedule: next chunk of 32 pairs
      unsigned long long cc = 0;
      if (lane == 0) cc = atomicAdd(cursor, 1ull);
      c = (int64_t)__shfl_sync(kFull, cc, 0);
    } else {
      c = gw + it * nw;
    }
    if (c >= n_chunks) break;
    const int64_t p = (c << lg_grab) + lane;
    const bool valid = lane < grab && p < np;
    int a = valid ? __ldg(pa + p) : 0;
    int q = valid ? __ldg(pb + p) : 0;
    bool ok = valid;
    if ((unsigned)a >= (unsigned)n || (unsigned)q >= (unsigned)n) {
      if (valid) atomicOr(status, kErrBadId);
      ok = false;
      a = q = 0;
    }
    const int4 da = __ldg(desc + a);
    const int4 dq = __ldg(desc + q);
    const bool sw = da.y > dq.y;  // sss.cu:108-115
    const int4 A = sw ? dq : da;
    const int4 B = sw ? da : dq;
    const int s = ok ? A.y : 0;
    const int64_t bt = desc_toff(B);
    const int blg = desc_lg(B);
    s_hits[warp][lane] = 0;
    __syncwarp();
    // Looks up n keys of A from the j0-th on, counted in s_hits: pairs with a
    // warp's worth of keys by the whole warp, one pair at a time (with EARLY
    // stopped when need hits are reached or more than miss keys missed), the
    // rest flattened across the lanes.
    auto look_up = [&](int j0, int n, int need, int miss) {
      const bool big = n >= warp_pair_min;
      for (unsigned bigm = __ballot_sync(kFull, big); bigm; bigm &= bigm - 1) {
        const int k = __ffs(bigm) - 1;
        const int ks = __shfl_sync(kFull, n, k);
        const int32_t* kr = elems + __shfl_sync(kFull, A.x + j0, k);
        const int klg = __shfl_sync(kFull, blg, k);
        const int32_t* kt = table + __shfl_sync(kFull, bt, k);
        int h;
        if (EARLY) {
          h = warp_probe_pair_lean<HIER, ROUNDS, true>(
              kr, ks, kt, klg, lg_max, bn, b, status, qx, qh,
              __shfl_sync(kFull, need, k), __shfl_sync(kFull, miss, k));
        } else if (LEAN) {
          h = warp_probe_pair_lean<HIER, ROUNDS>(kr, ks, kt, klg, lg_max, bn, b, status, qx, qh);
        } else {
          h = warp_probe_pair<HIER, ROUNDS>(kr, ks, kt, klg, lg_max, bn, b, status, qx, qh);
        }
        h = __reduce_add_sync(kFull, h);
        if (lane == 0) s_hits[warp][k] += h;
        __syncwarp();
      }
      flat_probe<HIER>(elems, table, big ? 0 : n, A.x + j0, bt, blg, lg_max, bn, b, status,
                       [&](int k) { atomicAdd(&s_hits[warp][k], 1); });
      __syncwarp();
    };
    if (EARLY) {
      // decisions only: the rule holds from `need` hits on, so it fails as
      // soon as more than s - need keys have missed.  Most pairs share little:
      // as many keys and a quarter settle them, a quarter of the keys at
      // threshold 7/10 and equal sizes, none where the sizes differ too much.
      // A pair still open goes on by as many keys as settle it if the rest are
      // like these, then by the rest: three steps at most, and none where a
      // step is a batch of the whole warp or more, which stops by itself.  By
      // the misses left each time, equal sets took a step per 8 keys at 1/1.
      // 1 M random pairs: 354 us with all keys at once, 113 this way; 40,000
      // pairs of 5000 keys that differ in 20, at 99/100: 2.84 and 2.73 ms (3.9
      // by the misses left).  Slower than all at once by up to 1.6x are sets of
      // 250 to 500 keys that share about as many as the rule asks for.
      const int64_t parts = (int64_t)num + den;
      const int64_t need64 = ((int64_t)num * (da.y + dq.y) + parts - 1) / parts;
      const int need = (int)min(need64, (int64_t)INT_MAX);
      // runs of pairs with the same first set: most are settled by its bitmap
      int allowed = s - need;  // keys that may miss; negative: settled
      const int before = __shfl_up_sync(kFull, a, 1);
      const unsigned runs = __ballot_sync(kFull, ok && lane > 0 && before == a);
      if (__popc(runs) >= kFilterRun - 1 &&
          __popc(__ballot_sync(kFull, allowed >= 0 && need > 0)) >= kFilterRun) {
        uint32_t* const bits = reinterpret_cast<uint32_t*>(qx);
        for (unsigned heads = ~runs; heads; heads &= heads - 1) {
          const int k = __ffs(heads) - 1;
          // lanes k .. z - 1 follow k
          const unsigned after = heads & (heads - 1);
          const int z = after ? __ffs(after) - 1 : 32;
          const int na = __shfl_sync(kFull, da.y, k);
          if (z - k < kFilterRun || na > kFilterMax) continue;
          // the keys of the other set that settle the pair, where they are
          // likely to, and the lookups that they would spare
          const int64_t miss = (int64_t)dq.y - need;
          int n = 0, spared = 0;
          if (lane >= k && lane < z && allowed >= 0 && need > 0) {
            n = (int)min((int64_t)dq.y, miss + 8 + (miss >> 2));
            spared = (int)min((int64_t)min(s, kFilterStream), (int64_t)allowed + 8 + (allowed >> 2));
            // (as many are held by chance as bits are set; 1 in 20 and one more allowed for)
            if ((float)n * (0.95f - (float)na / kFilterBits) <= (float)(miss + 1)) n = spared = 0;
          }
          if (__any_sync(kFull, n > kFilterStream)) continue;  // (left to the lookups)
          const int streamed = __reduce_add_sync(kFull, n);
          const int looked_up = __reduce_add_sync(kFull, spared);
          // a lookup costs about five keys entered or streamed
          if ((int64_t)streamed + na + 256 >= (int64_t)5 * looked_up) continue;
          if (pause > 1) {
            --pause;
            continue;
          }
          const int row = __shfl_sync(kFull, da.x, k);
          const float misses = (float)__reduce_add_sync(kFull, n > 0 ? (int)miss : 0);
          const bool settles =
              filter_fill(elems + row, na, bits) &&
              filter_stream(elems, dq.x, n, 1.f - misses / (float)streamed, bits, s_hits[warp]);
          __syncwarp();
          if (settles && n > 0 && n - s_hits[warp][lane] > miss) allowed = -1;
          pause = settles ? 0 : pause ? 9 : 1;
          __syncwarp();
          s_hits[warp][lane] = 0;
          __syncwarp();
        }
      }
      for (int step = 0, j = 0, I = 0; step < 3; ++step) {
        const int miss = I < need ? allowed - (j - I) : -1;  // that may still miss
        const int rest = miss < 0 ? 0 : s - j;
        if (!__any_sync(kFull, rest > 0)) break;
        float likely = (float)miss + 8.f + (float)(miss >> 2);
        if (step == 1)
          likely = 8.f + 1.25f * (float)j * fminf((float)(miss + 1) / (float)max(j - I, 1),
                                                  (float)(need - I) / (float)max(I, 1));
        const int n = rest == 0 || step == 2 || likely >= 32.f * ROUNDS
                          ? rest : min(rest, (int)likely);
        look_up(j, n, need - I, miss);
        j += n;
        I = s_hits[warp][lane];
      }
    } else {
      look_up(0, s, 0, 0);
    }
    const int I = s_hits[warp][lane];
    __syncwarp();
    if (ok) {
      const int U = da.y + dq.y - I;
      bool f;
      if (FLOAT_RULE) {
        f = ((float)I / (float)U) >= thr;  // sss.cu:139-140
      } else {
        f = U > 0 && (int64_t)den * I >= (int64_t)num * U;
      }
      flags[p] = (uint8_t)f;
      if (inter) inter[p] = I;
    } else if (valid) {
      flags[p] = 0;
      if (inter) inter[p] = 0;
    }
  }
}

// ----------------------------------------------------------- raw pair ----
//
// |A ∩ B| with A's multiplicity needs membership in B only, so B goes into a
// hash set of its own (linear probing, at most half full) and not into the
// reference's table: the order of insertion does not matter, no size has to
// be read back, and nothing can fail on the device.  Up to kPairSmem keys of B
// every CTA builds the set in its shared memory and looks up its share of A:
// one launch.  Larger sets lie in HBM (L2): one launch to insert, one to look
// up (at 16384 keys 46 us a call against 73 in every CTA's shared memory).
// Latency-bound.  A call through Python, us, by a table build / now: 1000 x
// 1500 keys 140 / 41, 300 x 100000 353 / 58, 2^20 x 2^20 1162 / 79.
constexpr int kPairThreads = 512;
constexpr int kPairSmem = 4096;  // keys (a set of up to 64 KB)

struct PairSet {  // 1 << lg slots at S (lg 1..32), -1 = empty
  int32_t* S;
  int lg;
  __device__ __forceinline__ unsigned home(int x) const {
    return ((unsigned)x * 0x9E3779B1u) >> (32 - lg);
  }
  __device__ __forceinline__ unsigned next(unsigned h) const {
    return (h + 1) & (0xFFFFFFFFu >> (32 - lg));
  }
  __device__ __forceinline__ void insert(int x) const {
    for (unsigned h = home(x);; h = next(h)) {
      const int old = atomicCAS(S + h, -1, x);
      if (old == -1 || old == x) return;
    }
  }
  __device__ __forceinline__ bool holds(int x) const {
    for (unsigned h = home(x);; h = next(h)) {
      const int s = S[h];
      if (s == x) return true;
      if (s == -1) return false;
    }
  }
};

__global__ void __launch_bounds__(kPairThreads)
    pair_smem_kernel(const int32_t* __restrict__ a, int64_t na, const int32_t* __restrict__ b,
                     int nb, int lg, unsigned long long* __restrict__ count) {
  extern __shared__ __align__(16) int32_t pair_sm[];
  __shared__ unsigned long long s_sum[kPairThreads / 32];
  const PairSet set{pair_sm, lg};
  const int tid = threadIdx.x;
  for (int i = tid; i < (1 << lg) / 4; i += kPairThreads)
    reinterpret_cast<int4*>(pair_sm)[i] = make_int4(-1, -1, -1, -1);
  __syncthreads();
  for (int i = tid; i < nb; i += kPairThreads) set.insert(__ldg(b + i));
  __syncthreads();
  unsigned long long hits = 0;
  const int64_t step = (int64_t)gridDim.x * kPairThreads;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * kPairThreads + tid; i < na; i += step)
    hits += set.holds(__ldg(a + i));
  hits = warp_sum_u64(hits);
  if ((tid & 31) == 0) s_sum[tid >> 5] = hits;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kPairThreads / 32; ++w) hits += s_sum[w];
    if (gridDim.x == 1) *count = hits;  // (else zeroed before the launch)
    else if (hits) atomicAdd(count, hits);
  }
}

__global__ void __launch_bounds__(kThreads)
    pair_insert_kernel(const int32_t* __restrict__ b, int64_t nb, int32_t* __restrict__ slots,
                       int lg) {
  const PairSet set{slots, lg};
  for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < nb;
       i += (int64_t)gridDim.x * kThreads)
    set.insert(__ldg(b + i));
}

__global__ void __launch_bounds__(kThreads)
    pair_lookup_kernel(const int32_t* __restrict__ a, int64_t na, int32_t* __restrict__ slots,
                       int lg, unsigned long long* __restrict__ count) {
  const PairSet set{slots, lg};
  unsigned long long hits = 0;
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < na;
       i += (int64_t)gridDim.x * kThreads)
    hits += set.holds(__ldg(a + i));
  hits = warp_sum_u64(hits);
  if ((threadIdx.x & 31) == 0 && hits) atomicAdd(count, hits);
}

// ----------------------------------------------------------------- IR ----

__global__ void ir_plan_kernel(const int4* __restrict__ desc, int32_t n,
                               const int32_t* __restrict__ query,
                               const int32_t* __restrict__ qoff, int32_t nq,
                               int64_t* __restrict__ sl_off,
                               int32_t* __restrict__ status) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nq;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int qs = qoff[q], ql = qoff[q + 1] - qs;
    int64_t ns = 0;
    if (ql > 0) {
      const int t0 = query[qs];
      if ((unsigned)t0 < (unsigned)n) {
        const int df = desc[t0].y;
        ns = (df + kIrSlice - 1) / kIrSlice;
      } else {
        atomicOr(status, kErrBadId);
      }
    }
    sl_off[q] = ns;
  }
}

__global__ void ir_total_kernel(const int64_t* __restrict__ ns_excl,
                                int64_t* __restrict__ sl_off, int32_t nq,
                                int64_t* __restrict__ total) {
  // sl_off holds the exclusive scan of the slice counts for q < nq; the
  // count of the last query is recomputed by the caller into ns_excl[0].
  int64_t t = nq > 0 ? sl_off[nq - 1] + ns_excl[0] : 0;
  sl_off[nq] = t;
  *total = t;
}

// Looks the keys x[r] whose bit r of `pend` is set up in one table; the bits
// of those found.  All start at slot 0 of their buckets and step together, so
// the slot is one for the warp and each step has R independent loads per lane.
template <bool HIER, int R>
__device__ __forceinline__ unsigned probe_keys(const int (&x)[R], unsigned pend,
                                               const int32_t* __restrict__ tb, int lg,
                                               int lg_max, int64_t bn, int b, int32_t* status) {
  const int l = 1 << lg;
  const int64_t cap = (int64_t)l * b;
  int h[R];
#pragma unroll
  for (int r = 0; r < R; ++r) h[r] = home_bucket<HIER>(x[r], lg, lg_max);
  unsigned hits = 0;
  const int32_t* plane = tb;
  int k = 0;
  for (int64_t t = 0; t < cap && __any_sync(kFull, pend); ++t) {
    int s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = pend >> r & 1u ? __ldg(plane + h[r]) : -1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (s[r] == x[r]) hits |= pend & 1u << r;
      if (s[r] == x[r] || s[r] == -1) pend &= ~(1u << r);
    }
    plane += bn;
    if (++k == b) {
      k = 0;
      plane = tb;
#pragma unroll
      for (int r = 0; r < R; ++r) h[r] = (h[r] + 1) & (l - 1);
    }
  }
  if (pend) atomicOr(status, kErrProbeLimit);
  return hits;
}

// One warp per slice of kIrSlice candidates of the first term's list:
// every candidate is checked against all further terms, survivors are
// compacted with ballot/popc to the front of the slice's own region
// stage[slice * kIrSlice ...], in first-term order, and their number goes to
// sl_cnt[slice].  Bound by random sectors of HBM (a miss reads every filled
// slot of its bucket), so kIrKeys candidates per lane are looked up at a time
// and the terms' descriptors are read once per slice.  512 queries, 37 M
// candidates, an index of 77 M documents: 467 us with one candidate per lane
// (49% of the DRAM's rate), 358 with 4, 320 with 8 (5.7 TB/s).
constexpr int kIrKeys = 8;

template <bool HIER>
__global__ void __launch_bounds__(kThreads, 3)
    ir_slice_kernel(const int4* __restrict__ desc, int32_t n,
                    const int32_t* __restrict__ docs,
                    const int32_t* __restrict__ query,
                    const int32_t* __restrict__ qoff, int32_t nq,
                    const int64_t* __restrict__ sl_off,
                    int32_t* __restrict__ stage, int32_t* __restrict__ sl_cnt,
                    const int32_t* __restrict__ table, int64_t bn, int b,
                    int lg_max, int32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  const int64_t total = sl_off[nq];
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t sidx = gw; sidx < total; sidx += nw) {
    // query owning this slice: largest q with sl_off[q] <= sidx
    int lo = 0, hi = nq - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (sl_off[mid] <= sidx) lo = mid; else hi = mid - 1;
    }
    const int q = lo;
    const int qs = qoff[q], ql = qoff[q + 1] - qs;
    const int4 d0 = desc[query[qs]];
    // lane k: further term k + 1 (id -1: not a set), of the first 32
    int term = -1;
    int4 dt = make_int4(0, 0, 0, 0);
    if (lane + 1 < ql) {
      term = __ldg(query + qs + 1 + lane);
      if ((unsigned)term < (unsigned)n) dt = __ldg(desc + term);
    }
    const int64_t j0 = (sidx - sl_off[q]) * kIrSlice;
    const int64_t j1 = min((int64_t)d0.y, j0 + kIrSlice);
    int32_t* out = stage + sidx * kIrSlice;
    int w = 0;
    for (int64_t jb = j0; jb < j1; jb += 32 * kIrKeys) {
      int x[kIrKeys];
      unsigned ok = 0;
#pragma unroll
      for (int r = 0; r < kIrKeys; ++r) {
        const int64_t j = jb + r * 32 + lane;
        x[r] = j < j1 ? __ldg(docs + d0.x + j) : 0;
        ok |= (unsigned)(j < j1) << r;
      }
      for (int i = 1; i < ql; ++i) {  // ir.cu:131-161, all terms per candidate
        if (!__any_sync(kFull, ok)) break;
        int t = __shfl_sync(kFull, term, (i - 1) & 31);
        int4 d;
        d.z = __shfl_sync(kFull, dt.z, (i - 1) & 31);
        d.w = __shfl_sync(kFull, dt.w, (i - 1) & 31);
        if (i > 32) t = __ldg(query + qs + i);
        if ((unsigned)t >= (unsigned)n) {
          if (ok) atomicOr(status, kErrBadId);
          ok = 0;
          break;
        }
        if (i > 32) d = __ldg(desc + t);
        ok = probe_keys<HIER>(x, ok, table + desc_toff(d), desc_lg(d), lg_max, bn, b, status);
      }
#pragma unroll
      for (int r = 0; r < kIrKeys; ++r) {
        const unsigned msk = __ballot_sync(kFull, ok >> r & 1u);
        if (ok >> r & 1u) out[w + __popc(msk & lt)] = x[r];
        w += __popc(msk);
      }
    }
    if (lane == 0) sl_cnt[sidx] = w;
  }
}

// Exclusive scan of per-slice survivor counts: pos[s] = survivors before slice
// s, pos[ns] = all survivors.  A block per kScanBlock counts; each sums the
// counts before its own anew, which costs less than a second launch and needs
// no scratch.  72,000 slices: 76 us in one block with a count per thread and
// pass, 61 with kScanItems of them, 10 this way.
constexpr int kScanItems = 16;
constexpr int kScanBlock = 1024 * kScanItems;

__global__ void __launch_bounds__(1024)
    slice_scan_kernel(const int32_t* __restrict__ cnt, int64_t ns, int64_t* __restrict__ pos) {
  __shared__ int64_t s_part[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = (int64_t)blockIdx.x * kScanBlock;
  int64_t carry = 0;
  if (base) {
#pragma unroll 16
    for (int64_t i = tid; i < base; i += 1024) carry += cnt[i];
    carry = (int64_t)warp_sum_u64((unsigned long long)carry);
    if (lane == 0) s_part[warp] = carry;
    __syncthreads();
    carry = s_part[lane];
#pragma unroll
    for (int o = 16; o; o >>= 1) carry += __shfl_xor_sync(kFull, carry, o);
  }
  // rows of 32 counts: warp w has rows w * kScanItems ..., a lane one of each
  const int64_t at = base + warp * 32 * kScanItems + lane;
  int v[kScanItems], row[kScanItems];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) v[k] = at + k * 32 < ns ? cnt[at + k * 32] : 0;
  int64_t sum = 0;  // of this warp's rows (a count is at most kIrSlice)
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int incl = v[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    row[k] = (int)sum + incl - v[k];
    sum += __shfl_sync(kFull, incl, 31);
  }
  __syncthreads();  // (the sums above are read)
  if (lane == 0) s_part[warp] = sum;
  __syncthreads();
  const int64_t part = s_part[lane];
  int64_t incl = part;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  const int64_t before = carry + __shfl_sync(kFull, incl - part, warp);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (at + k * 32 < ns) pos[at + k * 32] = before + row[k];
  carry += __shfl_sync(kFull, incl, 31);
  if (tid == 0 && ns - base <= kScanBlock) pos[ns] = carry;
}

// One warp per kGatherSlices slices: copies their survivors out of the stage,
// out of place, so all slices move in parallel; the lanes search for the
// slices' queries at the same time (12.7 M survivors: 45 us with a slice per
// warp and time, 24 this way).  Query q's survivors land at
//   res + res_off[q] + (pos[s] - pos[sl_off[q]])   (res_off given), or
//   res + pos[s]                                    (packed, res_off NULL).
constexpr int kGatherSlices = 8;

__global__ void __launch_bounds__(kThreads)
    ir_gather_kernel(const int64_t* __restrict__ sl_off, int32_t nq,
                     const int32_t* __restrict__ sl_cnt,
                     const int64_t* __restrict__ pos,
                     const int32_t* __restrict__ stage,
                     const int64_t* __restrict__ res_off,
                     int32_t* __restrict__ res) {
  const int lane = threadIdx.x & 31;
  const int64_t total = sl_off[nq];
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t s0 = gw * kGatherSlices; s0 < total; s0 += nw * kGatherSlices) {
    const int64_t s = s0 + lane;  // a lane looks a slice's place up
    int c = 0;
    int64_t dst = 0;
    if (lane < kGatherSlices && s < total) {
      c = sl_cnt[s];
      dst = pos[s];
      if (res_off && c) {
        int lo = 0, hi = nq - 1;  // query owning slice s
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (sl_off[mid] <= s) lo = mid; else hi = mid - 1;
        }
        dst = res_off[lo] + (dst - pos[sl_off[lo]]);
      }
    }
    for (unsigned left = __ballot_sync(kFull, c > 0); left; left &= left - 1) {
      const int k = __ffs(left) - 1;
      const int ck = __shfl_sync(kFull, c, k);
      const int32_t* src = stage + (s0 + k) * kIrSlice;
      int32_t* to = res + __shfl_sync(kFull, dst, k);
#pragma unroll 4
      for (int j = lane; j < ck; j += 32) to[j] = src[j];
    }
  }
}

// Per query: its count, and (packed mode) where its survivors start.
__global__ void ir_counts_kernel(const int64_t* __restrict__ sl_off, int32_t nq,
                                 const int64_t* __restrict__ pos,
                                 int32_t* __restrict__ cnt,
                                 int64_t* __restrict__ packed_off) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nq;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = pos[sl_off[q]], b = pos[sl_off[q + 1]];
    cnt[q] = (int32_t)(b - a);
    if (packed_off) {
      packed_off[q] = a;
      if (q == nq - 1) packed_off[nq] = b;
    }
  }
}

// Launches the slice, scan, gather and count kernels for a planned batch.
template <bool HIER>
reset_status ir_run(const reset_table* t, const int4* desc, const int32_t* docs,
                    const int32_t* query, const int32_t* qoff, int32_t nq,
                    const int64_t* sl_off, int64_t total_slices,
                    const int64_t* res_off, int32_t* res, int32_t* stage,
                    int32_t* sl_cnt, int64_t* pos, int32_t* cnt,
                    int64_t* packed_off, cudaStream_t st, bool yield);

int persistent_grid(const void* kernel) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0);
  if (per_sm < 1) per_sm = 1;
  return sm_count() * per_sm;
}

int64_t clamp_grid(int64_t want, int cap) {
  if (want < 1) want = 1;
  return want < cap ? want : cap;
}

template <bool HIER>
reset_status ir_run(const reset_table* t, const int4* desc, const int32_t* docs,
                    const int32_t* query, const int32_t* qoff, int32_t nq,
                    const int64_t* sl_off, int64_t total_slices,
                    const int64_t* res_off, int32_t* res, int32_t* stage,
                    int32_t* sl_cnt, int64_t* pos, int32_t* cnt,
                    int64_t* packed_off, cudaStream_t st, bool yield) {
  // yield: a warp per slice (or kGatherSlices of them) and no persistent grid,
  // so the blocks retire as they finish and the block scheduler can interleave
  // other streams' (higher-priority) work; otherwise a persistent grid walks
  // the slices
  auto blocks = [&](int64_t slices, const void* kernel) {
    const int64_t want = std::min<int64_t>((total_slices + slices - 1) / slices, INT32_MAX);
    return yield ? want : clamp_grid(want, persistent_grid(kernel));
  };
  if (total_slices > 0) {
    const int64_t g = blocks(kWarps, (const void*)ir_slice_kernel<HIER>);
    note_launch();
    ir_slice_kernel<HIER><<<(int)g, kThreads, 0, st>>>(
        desc, t->n, docs, query, qoff, nq, sl_off, stage, sl_cnt, t->d_table,
        t->bucket_num, t->bucket, t->lg_max, t->d_status);
    RST_CUDA(cudaGetLastError());
  }
  note_launch();
  slice_scan_kernel<<<(int)std::max<int64_t>(1, (total_slices + kScanBlock - 1) / kScanBlock), 1024,
                      0, st>>>(sl_cnt, total_slices, pos);
  RST_CUDA(cudaGetLastError());
  if (total_slices > 0) {
    const int64_t g = blocks(kWarps * kGatherSlices, (const void*)ir_gather_kernel);
    note_launch();
    ir_gather_kernel<<<(int)g, kThreads, 0, st>>>(sl_off, nq, sl_cnt, pos, stage, res_off,
                                                   res);
    RST_CUDA(cudaGetLastError());
  }
  note_launch();
  ir_counts_kernel<<<(int)clamp_grid((nq + 255) / 256, sm_count() * 8), 256, 0, st>>>(
      sl_off, nq, pos, cnt, packed_off);
  RST_CUDA(cudaGetLastError());
  return RESET_OK;
}

// Resolves the descriptor array for a probe call: the table's own when the
// caller passes the offsets the table was built on, else a fresh one.
struct DescScope {
  const int4* desc = nullptr;
  int4* owned = nullptr;
  cudaStream_t st = nullptr;
  ~DescScope() {
    if (owned) cudaFreeAsync(owned, st);
  }
};

reset_status resolve_desc(const reset_table* t, const int32_t* d_off,
                          cudaStream_t st, DescScope* ds) {
  ds->st = st;
  if (!d_off || d_off == t->build_off) {
    ds->desc = t->d_desc;
    return RESET_OK;
  }
  RST_CHECK(make_desc(t, d_off, &ds->owned, st));
  ds->desc = ds->owned;
  return RESET_OK;
}

}  // namespace

// Edges of a graph without long rows have few keys to look up: the groups'
// passes take longer than the lookups, edge by edge, do.  The bound on the
// longest row is alpha times its table's slots, so it moves in steps of two.
// Measured, us, methods 1 / 3: a grid of 4 M vertices 465 / 990; random graphs of
// 2 M vertices, bound 64 with 10 edges each 1349 / 2691, with 14 2310 / 3318, bound
// 128 with 20 4154 / 4211, with 28 7550 / 5474.  Past it hubs decide: 96 R-MAT
// graphs of scales 8 to 12, bound 128, 269 / 249; scale 19 with 4 a vertex, bound
// 256, 443 / 347.
bool tc_sparse(const reset_table* t) {
  return (double)t->alpha * t->bucket * t->max_len < 96;
}

reset_status tc_edges(const reset_table* t, const int4* kdesc, const int32_t* kcols,
                      const int32_t* eoff, const int32_t* ecols, const int32_t* echunk_rows,
                      int64_t me, unsigned long long* count, cudaStream_t st,
                      unsigned long long* owner_hits) {
  unsigned long long* cursor = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&cursor), sizeof(*cursor), st));
  cudaError_t e = cudaMemsetAsync(cursor, 0, sizeof(*cursor), st);
  const reset_tuning tun = tuning();
#define TC_LAUNCH(...)                                                         \
  do {                                                                         \
    const int most = persistent_grid((const void*)tc_kernel<__VA_ARGS__>);     \
    /* 32 edges at a time, fewer where that leaves warps idle (at least 4) */  \
    int lg_grab = 5;                                                           \
    while (lg_grab > 2 && (me >> lg_grab) < (int64_t)most * kWarps) --lg_grab; \
    const int64_t g = clamp_grid(((me >> lg_grab) + kWarps) / kWarps, most);   \
    note_launch();                                                             \
    tc_kernel<__VA_ARGS__><<<(int)g, kThreads, 0, st>>>(                       \
        kdesc, kcols, eoff, ecols, echunk_rows, t->n, me, t->d_table,          \
        t->bucket_num, t->bucket, t->lg_max, count, owner_hits, cursor,        \
        lg_grab, tun.warp_pair_min, t->d_status);                              \
  } while (0)
#define TC_VARIANT(H)                                                          \
  do {                                                                         \
    if (owner_hits) TC_LAUNCH(H, 4, false, true);                              \
    else if (tun.probe_variant == 1 && tun.probe_rounds == 2) TC_LAUNCH(H, 2, true); \
    else if (tun.probe_variant == 1 && tun.probe_rounds == 8) TC_LAUNCH(H, 8, true); \
    else if (tun.probe_variant == 1) TC_LAUNCH(H, 4, true);                    \
    else if (tun.probe_rounds == 2) TC_LAUNCH(H, 2, false);                    \
    else TC_LAUNCH(H, 4, false);                                               \
  } while (0)
  if (e == cudaSuccess) {
    if (t->hier) TC_VARIANT(true); else TC_VARIANT(false);
    e = cudaGetLastError();
  }
#undef TC_VARIANT
#undef TC_LAUNCH
  cudaFreeAsync(cursor, st);
  if (e != cudaSuccess) return cuda_fail(e, "tc_kernel launch", __FILE__, __LINE__);
  return RESET_OK;
}

// Persistent pair kernel for the batched form: pair count read on the device
// (np_dev), dynamic 32-pair chunks (cursor, zeroed by the caller), exact
// rule.  No allocation and no synchronisation, so it can be captured.
reset_status sss_launch_persistent(const reset_table* t, const int32_t* elems,
                                   const int32_t* pa, const int32_t* pb,
                                   const int64_t* np_dev,
                                   unsigned long long* cursor, int64_t capacity,
                                   int32_t num, int32_t den, uint8_t* flags,
                                   int32_t* inter, bool decisions_only,
                                   cudaStream_t st) {
  const reset_tuning tun = tuning();
  const int wpm = tun.warp_pair_min;
#define SSS_P(H, R, LN, E)                                                     \
  do {                                                                         \
    const int64_t g = clamp_grid(((capacity + 31) / 32 + kWarps - 1) / kWarps, \
                                 persistent_grid((const void*)sss_kernel<H, false, R, LN, E>)); \
    note_launch();                                                             \
    sss_kernel<H, false, R, LN, E><<<(int)g, kThreads, 0, st>>>(               \
        t->d_desc, t->n, elems, pa, pb, capacity, np_dev, cursor, 5,           \
        t->d_table, t->bucket_num, t->bucket, t->lg_max, num, den, 0.f, wpm,   \
        flags, E ? nullptr : inter, t->d_status);                              \
  } while (0)
  if (decisions_only) {
    if (t->hier) SSS_P(true, 8, true, true); else SSS_P(false, 8, true, true);
  } else if (tun.probe_variant == 1) {
    if (t->hier) SSS_P(true, 8, true, false); else SSS_P(false, 8, true, false);
  } else {
    if (t->hier) SSS_P(true, 4, false, false); else SSS_P(false, 4, false, false);
  }
#undef SSS_P
  RST_CUDA(cudaGetLastError());
  return RESET_OK;
}

int ir_slice_size() { return kIrSlice; }

// Conjunctive retrieval for a batch whose slice plan is on the device:
// sl_off[q] = sum over earlier queries of ceil(df(first term) / kIrSlice),
// sl_off[nq] = total_slices.  Scratch: stage (total_slices * kIrSlice ints),
// sl_cnt (total_slices ints), pos (total_slices + 1 int64).  Results go to
// res at res_off[q] (as reset_ir) or, with res_off NULL, packed query after
// query with packed_off[q] (nq + 1 int64) giving where each starts.  Uses
// the table's own descriptors.  No allocation, no synchronisation.
reset_status ir_launch_planned(const reset_table* t, const int32_t* docs,
                               const int32_t* query, const int32_t* qoff,
                               int32_t nq, const int64_t* sl_off,
                               int64_t total_slices, const int64_t* res_off,
                               int32_t* res, int32_t* stage, int32_t* sl_cnt,
                               int64_t* pos, int32_t* cnt, int64_t* packed_off,
                               cudaStream_t st, bool yield) {
  if (nq <= 0) return RESET_OK;
  if (t->hier)
    return ir_run<true>(t, t->d_desc, docs, query, qoff, nq, sl_off, total_slices, res_off,
                        res, stage, sl_cnt, pos, cnt, packed_off, st, yield);
  return ir_run<false>(t, t->d_desc, docs, query, qoff, nq, sl_off, total_slices, res_off,
                       res, stage, sl_cnt, pos, cnt, packed_off, st, yield);
}

}  // namespace rst

using namespace rst;

extern "C" {

reset_status reset_tc_count_ex(const reset_table* t, const int32_t* d_off,
                               const int32_t* d_cols, int64_t m, int32_t method,
                               uint64_t* d_count, reset_stream_t stream) {
  if (!t || !d_count) return arg_fail("NULL table or count");
  if (m < 0 || m > INT32_MAX) return arg_fail("m out of range");
  if (m > 0 && (!d_cols || !d_off)) return arg_fail("NULL offsets or cols");
  if (method < 0 || method > 3) return arg_fail("method must be 0, 1, 2 or 3");
  const bool cols16 = (reinterpret_cast<uintptr_t>(d_cols) & 15) == 0;
  if (method == 3 && !cols16)
    return arg_fail("method 3 needs a 16-byte aligned column array");
  // Up to half a million edges the edge-flattened count, whose tables then lie
  // in L2, is done by the time that grouping takes.  Measured (R-MAT, methods
  // 1 / 3): 10k edges 36 / 92 us, 213k 93 / 109, 441k 149 / 148, 909k 288 / 197.
  if (method == 0)
    method = cols16 && m >= kOwnerEdges && m <= INT32_MAX - 16 && t->n < INT32_MAX &&
                     !tc_sparse(t) ? 3 : 1;
  cudaStream_t st = as_stream(stream);
  RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), st));
  if (m == 0 || t->n == 0) return RESET_OK;
  DescScope ds;
  RST_CHECK(resolve_desc(t, d_off, st, &ds));
  unsigned long long* cnt = reinterpret_cast<unsigned long long*>(d_count);
  if (method == 2) return tc_staged(t, ds.desc, d_cols, m, cnt, st);
  const int32_t* rows = t->d_chunk_row;
  int32_t* owned_rows = nullptr;
  if (d_off != t->build_off || m != t->m) {
    RST_CHECK(make_chunk_rows(d_off, t->n, m, &owned_rows, st));
    rows = owned_rows;
  }
  reset_status s = RESET_ERR_OOM;
  if (method == 3) {
    s = tc_owner(t, ds.desc, d_off, d_cols, m, d_off, d_cols, rows, m, cnt, st);
    if (s == RESET_ERR_OOM) {  // no memory for the groups
      cudaGetLastError();
      RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), st));
    }
  }
  if (s == RESET_ERR_OOM)
    s = tc_edges(t, ds.desc, d_cols, d_off, d_cols, rows, m, cnt, st);
  if (owned_rows) cudaFreeAsync(owned_rows, st);
  return s;
}

reset_status reset_tc_count(const reset_table* t, const int32_t* d_off,
                            const int32_t* d_cols, int64_t m,
                            uint64_t* d_count, reset_stream_t stream) {
  return reset_tc_count_ex(t, d_off, d_cols, m, 0, d_count, stream);
}

static reset_status sss_common(const reset_table* t, const int32_t* d_off,
                               const int32_t* d_elems, const int32_t* d_pa,
                               const int32_t* d_pb, int64_t np, bool float_rule,
                               int32_t num, int32_t den, float thr,
                               uint8_t* d_flags, int32_t* d_inter,
                               reset_stream_t stream) {
  if (!t) return arg_fail("NULL table");
  if (np < 0) return arg_fail("negative pair count");
  if (np == 0) return RESET_OK;
  if (!d_elems || !d_pa || !d_pb || !d_flags) return arg_fail("NULL pointer");
  if (!float_rule && (den <= 0 || num < 0)) return arg_fail("threshold num/den");
  cudaStream_t st = as_stream(stream);
  DescScope ds;
  RST_CHECK(resolve_desc(t, d_off, st, &ds));
  const reset_tuning tun = tuning();
  const bool el16 = (reinterpret_cast<uintptr_t>(d_elems) & 15) == 0;
  if (tun.pair_method == 2 && !el16)
    return arg_fail("pair_method 2 needs a 16-byte aligned element array");
  // default: the pair-flattened kernel (measured faster or equal on B200 for
  // graph pairs and self-join candidates, and it stops deciding pairs early)
  if (tun.pair_method == 2 && el16 && np <= INT32_MAX && t->m <= INT32_MAX - 4)
    return sss_owner(t, ds.desc, d_elems, t->m, d_pa, d_pb, np, float_rule, num, den, thr,
                     d_flags, d_inter, st);
#define SSS_LAUNCH(H, F, R, LN, ...)                                         \
  do {                                                                       \
    const int most = persistent_grid((const void*)sss_kernel<H, F, R, LN, ##__VA_ARGS__>); \
    /* 32 pairs at a time, fewer where that leaves warps idle */             \
    int lg_grab = 5;                                                         \
    while (lg_grab > 0 && (np >> lg_grab) < (int64_t)most * kWarps) --lg_grab; \
    const int64_t g = clamp_grid(((np >> lg_grab) + kWarps) / kWarps, most); \
    note_launch(); sss_kernel<H, F, R, LN, ##__VA_ARGS__><<<(int)g, kThreads, 0, st>>>( \
        ds.desc, t->n, d_elems, d_pa, d_pb, np, nullptr, nullptr, lg_grab,   \
        t->d_table, t->bucket_num, t->bucket, t->lg_max, num, den, thr,       \
        tun.warp_pair_min, d_flags, d_inter, t->d_status);                    \
  } while (0)
#define SSS_V(H, F)                                                          \
  do {                                                                       \
    if (tun.probe_variant == 1) SSS_LAUNCH(H, F, 8, true);                   \
    else SSS_LAUNCH(H, F, 4, false);                                         \
  } while (0)
  if (!float_rule && !d_inter) {
    // decisions only: pairs stop as soon as the rule is settled
    if (t->hier) SSS_LAUNCH(true, false, 8, true, true);
    else SSS_LAUNCH(false, false, 8, true, true);
  } else if (t->hier) {
    if (float_rule) SSS_V(true, true); else SSS_V(true, false);
  } else {
    if (float_rule) SSS_V(false, true); else SSS_V(false, false);
  }
#undef SSS_V
#undef SSS_LAUNCH
  RST_CUDA(cudaGetLastError());
  return RESET_OK;
}

reset_status reset_sss(const reset_table* t, const int32_t* d_off,
                       const int32_t* d_elems, const int32_t* d_pair_a,
                       const int32_t* d_pair_b, int64_t npairs, int32_t num,
                       int32_t den, uint8_t* d_flags, int32_t* d_inter,
                       reset_stream_t stream) {
  return sss_common(t, d_off, d_elems, d_pair_a, d_pair_b, npairs, false, num,
                    den, 0.f, d_flags, d_inter, stream);
}

reset_status reset_sss_float(const reset_table* t, const int32_t* d_off,
                             const int32_t* d_elems, const int32_t* d_pair_a,
                             const int32_t* d_pair_b, int64_t npairs,
                             float thr, uint8_t* d_flags, int32_t* d_inter,
                             reset_stream_t stream) {
  return sss_common(t, d_off, d_elems, d_pair_a, d_pair_b, npairs, true, 0, 1,
                    thr, d_flags, d_inter, stream);
}

reset_status reset_intersect_count(const int32_t* d_a, int64_t na,
                                   const int32_t* d_b, int64_t nb,
                                   const reset_params* params,
                                   int64_t* d_count, reset_stream_t stream) {
  if (!d_count) return arg_fail("NULL count");
  if (na < 0 || nb < 0 || nb > INT32_MAX) return arg_fail("sizes out of range");
  if ((na > 0 && !d_a) || (nb > 0 && !d_b)) return arg_fail("NULL set");
  reset_params p;
  reset_params_default(&p);
  if (params) p = *params;
  if (na > 0 && nb > 0) {  // what a table with these parameters refuses
    if (!(p.alpha > 0.f && p.alpha <= 1.f)) return arg_fail("alpha must be in (0, 1]");
    if (p.bucket < 1 || p.bucket > 16) return arg_fail("bucket must be in 1..16");
    // (lengths of 2^31 buckets wrap around to 8, calculate_length)
    const float q = (float)nb / p.alpha;
    if ((q >= 2147483648.f ? INT32_MAX : (int)q) / p.bucket >= (1 << 30) && nb > 8 * p.bucket) {
      set_error("a set did not fit its table (or a CSR row had negative length)");
      return RESET_ERR_TABLE_FULL;
    }
  }
  cudaStream_t st = as_stream(stream);
  unsigned long long* count = reinterpret_cast<unsigned long long*>(d_count);
  int lg = 6;
  while (((int64_t)1 << lg) < 2 * nb) ++lg;
  if (na > 0 && nb > 0 && nb <= kPairSmem) {
    ++lg;  // (at most a quarter full)
    const int smem = (int)sizeof(int32_t) << lg;
    // (the same for every size: other threads may be between here and a launch)
    RST_CUDA(cudaFuncSetAttribute(pair_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(int32_t) * 4 * kPairSmem));
    // a CTA looks up about as many keys as it inserts, all CTAs that fit at once
    // (one per SM left the chip half empty: 2^26 x 3000 keys 602 us, 250 this way)
    const int64_t share = std::max<int64_t>(4 * kPairThreads, nb);
    const int per_sm = std::min(2048 / kPairThreads, (200 << 10) / std::max(smem, 1 << 10));
    const int grid = (int)clamp_grid((na + share - 1) / share, sm_count() * per_sm);
    if (grid > 1) RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int64_t), st));
    note_launch();
    pair_smem_kernel<<<grid, kPairThreads, smem, st>>>(d_a, na, d_b, (int)nb, lg, count);
    RST_CUDA(cudaGetLastError());
    return RESET_OK;
  }
  RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int64_t), st));
  if (na == 0 || nb == 0) return RESET_OK;
  int32_t* slots = nullptr;
  const size_t bytes = sizeof(int32_t) << lg;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&slots), bytes, st));
  cudaError_t e = cudaMemsetAsync(slots, 0xFF, bytes, st);
  if (e == cudaSuccess) {
    const int cap = sm_count() * 8;
    note_launch(2);
    pair_insert_kernel<<<(int)clamp_grid((nb + kThreads - 1) / kThreads, cap), kThreads, 0, st>>>(
        d_b, nb, slots, lg);
    pair_lookup_kernel<<<(int)clamp_grid((na + kThreads - 1) / kThreads, cap), kThreads, 0, st>>>(
        d_a, na, slots, lg, count);
    e = cudaGetLastError();
  }
  cudaFreeAsync(slots, st);
  if (e != cudaSuccess) return cuda_fail(e, "raw pair kernels", __FILE__, __LINE__);
  return RESET_OK;
}

reset_status reset_ir(const reset_table* t, const int32_t* d_toff,
                      const int32_t* d_docs, const int32_t* d_query,
                      const int32_t* d_qoff, int32_t nq,
                      const int64_t* d_res_off, int32_t* d_res,
                      int32_t* d_cnt, reset_stream_t stream) {
  if (!t) return arg_fail("NULL table");
  if (nq < 0) return arg_fail("negative query count");
  if (nq == 0) return RESET_OK;
  if (!d_docs || !d_query || !d_qoff || !d_res_off || !d_res || !d_cnt)
    return arg_fail("NULL pointer");
  cudaStream_t st = as_stream(stream);
  DescScope ds;
  RST_CHECK(resolve_desc(t, d_toff, st, &ds));
  int64_t* d_sl = nullptr;
  int64_t* d_tot = nullptr;
  int32_t* d_slc = nullptr;
  int64_t* d_pos = nullptr;
  int32_t* d_stage = nullptr;
  void* d_tmp = nullptr;
  reset_status rs = RESET_OK;
  auto cleanup = [&]() {
    if (d_pos) cudaFreeAsync(d_pos, st);
    if (d_stage) cudaFreeAsync(d_stage, st);
    if (d_sl) cudaFreeAsync(d_sl, st);
    if (d_tot) cudaFreeAsync(d_tot, st);
    if (d_slc) cudaFreeAsync(d_slc, st);
    if (d_tmp) cudaFreeAsync(d_tmp, st);
  };
#define IR_CUDA(call)                                                       \
  do {                                                                      \
    cudaError_t _e = (call);                                                \
    if (_e != cudaSuccess) {                                                \
      rs = cuda_fail(_e, #call, __FILE__, __LINE__);                        \
      cleanup();                                                            \
      return rs;                                                            \
    }                                                                       \
  } while (0)
  IR_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_sl), sizeof(int64_t) * (nq + 1), st));
  IR_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_tot), sizeof(int64_t) * 2, st));
  note_launch(); ir_plan_kernel<<<(int)clamp_grid((nq + 255) / 256, sm_count() * 8), 256, 0, st>>>(
      ds.desc, t->n, d_query, d_qoff, nq, d_sl, t->d_status);
  IR_CUDA(cudaGetLastError());
  // keep the last count, then scan in place
  IR_CUDA(cudaMemcpyAsync(d_tot + 1, d_sl + (nq - 1), sizeof(int64_t), cudaMemcpyDeviceToDevice, st));
  size_t tb = 0;
  IR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, d_sl, d_sl, nq, st));
  IR_CUDA(scratch_malloc(&d_tmp, tb, st));
  IR_CUDA(cub::DeviceScan::ExclusiveSum(d_tmp, tb, d_sl, d_sl, nq, st));
  note_launch(); ir_total_kernel<<<1, 1, 0, st>>>(d_tot + 1, d_sl, nq, d_tot);
  IR_CUDA(cudaGetLastError());
  int64_t total = 0;
  IR_CUDA(cudaMemcpyAsync(&total, d_tot, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  IR_CUDA(cudaStreamSynchronize(st));
  IR_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_slc), sizeof(int32_t) * (total > 0 ? total : 1), st));
  IR_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_pos), sizeof(int64_t) * (total + 1), st));
  IR_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_stage),
                          sizeof(int32_t) * (size_t)(total > 0 ? total : 1) * kIrSlice, st));
  rs = t->hier ? ir_run<true>(t, ds.desc, d_docs, d_query, d_qoff, nq, d_sl, total, d_res_off,
                              d_res, d_stage, d_slc, d_pos, d_cnt, nullptr, st, false)
               : ir_run<false>(t, ds.desc, d_docs, d_query, d_qoff, nq, d_sl, total, d_res_off,
                               d_res, d_stage, d_slc, d_pos, d_cnt, nullptr, st, false);
  if (rs != RESET_OK) {
    cleanup();
    return rs;
  }
#undef IR_CUDA
  cleanup();
  return RESET_OK;
}

}  // extern "C"
