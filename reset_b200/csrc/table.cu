// Table build: the per-set bucketed hash tables of the reference, built
// deterministically on sm_100a.
//
// Reference: triangle-count/hashtable.cu:21-183 (calculate_length,
// calculate_hash_length, scan, build_hash_table_normal/_hierarchical) and
// baseline/common/hash_table.cu:69-192.  The reference inserts with one
// thread per element and atomicCAS, so slot placement depends on timing.
// Here every set is inserted in CSR order with the same rule (home bucket,
// first empty slot, next bucket when full), so the table is a pure function
// of the input and equals the CPU restatement byte for byte.
//
// Layout of the work:
//  * meta:   len[u] = calc_len(deg u), max_len, and the list of "long" sets
//            whose table does not fit a shared-memory tile.
//  * layout: off[u] = sum_{w<u} len[w] (64-bit), off[n] = bucket_num; packed
//            16-byte per-set descriptors for the probe kernels, the row of
//            every 32-edge chunk, and the first set of every tile.
//  * tile build: one CTA per tile of ~T consecutive buckets.  The tile's
//            b slot planes live in shared memory; small sets (deg <= 8) are
//            inserted by one thread each, larger ones by a warp that
//            inserts 32 keys per round with __match_any_sync, committing
//            the longest prefix of lanes whose placement cannot depend on a
//            later lane (so the result is the sequential one).  The planes
//            are then written to HBM with cp.async.bulk (the TMA engine's
//            1-D bulk copy) -- every table byte is written exactly once and
//            no separate memset pass runs.
//  * long sets: all of them together, key- and bucket-parallel (see
//            long_insert_kernel), straight in HBM.
#include <cub/cub.cuh>

#include <cstring>
#include <memory>
#include <mutex>
#include <new>

#include "common.cuh"
#include "probe_common.cuh"

namespace rst {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTileThreads = 512;  // threads of a tile-build CTA (3 CTAs, 48 warps per SM)
constexpr int kTileWarps = kTileThreads / 32;
constexpr bool kTileDynamic = true;  // warps take a tile's larger sets from a cursor
constexpr int kThreadSetMax = 8;      // sets with deg <= this: thread per set
constexpr int kTileSmemBudget = 72 * 1024;  // (a multiple of 16, as g.smem is)
constexpr int kBigFillSmemMax = 64 * 1024;  // buckets whose fill bytes fit smem
constexpr int kHugeKeys = 1 << 16;  // crowded sets this long are built by build_huge

struct Geom {
  int R_max;  // buckets per shared-memory tile (stride of a slot plane)
  int T;      // buckets assigned per CTA
  int LT;     // largest table length built in a tile
  size_t smem;
};

Geom tile_geom(int b) {
  Geom g;
  int per = 4 * b + 1;
  g.R_max = (kTileSmemBudget / per) & ~7;
  g.LT = 8;
  while (g.LT * 2 <= g.R_max / 3) g.LT *= 2;
  g.T = (g.R_max - g.LT) & ~7;
  g.smem = (size_t)g.R_max * 4 * b + (size_t)g.R_max;
  g.smem = (g.smem + 15) & ~(size_t)15;
  return g;
}

// ------------------------------------------------------------- PTX bits --

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_store(void* gdst, const void* ssrc,
                                           unsigned bytes) {
  unsigned s = (unsigned)__cvta_generic_to_shared(ssrc);
  asm volatile(
      "cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
          gdst),
      "r"(s), "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read_all() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ------------------------------------------------------------ meta pass --

// What the host reads back to size the table.
struct BuildInfo {
  int32_t max_len;
  int32_t n_long;   // sets whose table does not fit a tile
  int32_t n_huge;   // ... of kHugeKeys keys or more
  unsigned long long long_keys, long_buckets;
  int64_t bucket_num;
  unsigned long long keys_lg[16];  // keys of the long sets of 2^i .. 2^(i+1) - 1 keys
};

// Sets [bid * per, (bid + 1) * per) of block bid.
__global__ void __launch_bounds__(kThreads)
    meta_kernel(const int32_t* __restrict__ off, int32_t n, int64_t per, float alpha, int b,
                int LT, int32_t* __restrict__ len, int64_t* __restrict__ blk_sum,
                int32_t* __restrict__ long_list, int64_t long_cap, BuildInfo* __restrict__ info,
                int32_t* __restrict__ status) {
  __shared__ int64_t s_sum[kWarps];
  const int64_t u1 = min((int64_t)n, (blockIdx.x + 1) * per);
  int mx = 0;
  int64_t sum = 0;
  for (int64_t u = blockIdx.x * per + threadIdx.x; u < u1; u += kThreads) {
    int d = off[u + 1] - off[u];
    if (d < 0) {
      atomicOr(status, kErrTableFull);
      d = 0;
    }
    const int l = calc_len(d, alpha, b);
    len[u] = l;
    sum += l;
    mx = max(mx, l);
    if (l > LT) {
      const int at = atomicAdd(&info->n_long, 1);
      if (at < long_cap) long_list[at] = (int32_t)u;
      if (d >= kHugeKeys) atomicAdd(&info->n_huge, 1);
      else atomicAdd(&info->keys_lg[31 - __clz(max(d, 1))], (unsigned long long)d);
      atomicAdd(&info->long_keys, (unsigned long long)d);
      atomicAdd(&info->long_buckets, (unsigned long long)l);
    }
  }
  mx = __reduce_max_sync(kFull, mx);
  sum = (int64_t)warp_sum_u64((unsigned long long)sum);
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = sum;
    if (mx > 0) atomicMax(&info->max_len, mx);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w) sum += s_sum[w];
    blk_sum[blockIdx.x] = sum;
  }
}

// v (rows that start in 32-edge chunk c, or the first set of tile c) written
// to out[c0 .. c1) by every lane of the warp: short runs by their own lane,
// long ones (a hub's row, a large table) by all lanes.
__device__ __forceinline__ void fill_runs(int32_t* __restrict__ out, int64_t c0, int64_t c1,
                                          int32_t v) {
  const int lane = threadIdx.x & 31;
  const bool wide = c1 - c0 > 8;
  if (!wide)
    for (int64_t c = c0; c < c1; ++c) out[c] = v;
  for (unsigned m = __ballot_sync(kFull, wide); m; m &= m - 1) {
    const int k = __ffs(m) - 1;
    const int64_t a = __shfl_sync(kFull, c0, k), z = __shfl_sync(kFull, c1, k);
    const int32_t x = __shfl_sync(kFull, v, k);
    for (int64_t c = a + lane; c < z; c += 32) out[c] = x;
  }
}

// The row of every 32-edge chunk of a CSR.
__global__ void __launch_bounds__(kThreads)
    chunk_rows_kernel(const int32_t* __restrict__ off, int32_t n, int64_t n_chunks,
                      int32_t* __restrict__ chunk_row) {
  for (int64_t base = (int64_t)blockIdx.x * kThreads; base < n;
       base += (int64_t)gridDim.x * kThreads) {
    const int64_t u = base + threadIdx.x;
    const bool in = u < n;
    const int s = in ? off[u] : 0, e = in ? off[u + 1] : 0;
    fill_runs(chunk_row, ((int64_t)s + 31) >> 5, in ? min(((int64_t)e + 31) >> 5, n_chunks) : 0,
              (int32_t)u);
  }
}

// Offsets, descriptors, chunk rows and the first set of every tile, over
// meta_kernel's blocks of sets.
__global__ void __launch_bounds__(kThreads)
    layout_kernel(const int32_t* __restrict__ off, const int32_t* __restrict__ len, int32_t n,
                  int64_t per, const int64_t* __restrict__ blk_sum, int64_t* __restrict__ off64,
                  int4* __restrict__ desc, int64_t n_chunks, int32_t* __restrict__ chunk_row,
                  int32_t* __restrict__ tile_first, int64_t tile_cap, int T,
                  BuildInfo* __restrict__ info) {
  using Reduce = cub::BlockReduce<int64_t, kThreads>;
  using Scan = cub::BlockScan<int64_t, kThreads>;
  __shared__ union {
    typename Reduce::TempStorage reduce;
    typename Scan::TempStorage scan;
  } tmp;
  __shared__ int64_t s_carry;
  int64_t part = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += kThreads) part += blk_sum[i];
  part = Reduce(tmp.reduce).Sum(part);
  if (threadIdx.x == 0) s_carry = part;
  __syncthreads();
  int64_t carry = s_carry;
  const int64_t u1 = min((int64_t)n, (blockIdx.x + 1) * per);
  for (int64_t base = blockIdx.x * per; base < u1; base += kThreads) {
    const int64_t u = base + threadIdx.x;
    const bool in = u < u1;
    const int l = in ? len[u] : 0;
    int64_t toff, total;
    __syncthreads();  // tmp is used again
    Scan(tmp.scan).ExclusiveSum((int64_t)l, toff, total);
    toff += carry;
    carry += total;
    const int s = in ? off[u] : 0, e = in ? off[u + 1] : 0;
    if (in) {
      const int lg = 31 - __clz(l);
      off64[u] = toff;
      desc[u] = make_int4(s, e - s, (int)(uint32_t)toff,
                          (int)(((toff >> 32) & 0xFFFFFF) | ((int64_t)lg << 24)));
      if (u == n - 1) {
        off64[n] = toff + l;
        info->bucket_num = toff + l;
        const int64_t end = (toff + l + T - 1) / T;
        if (end < tile_cap) tile_first[end] = n;
      }
    }
    fill_runs(chunk_row, ((int64_t)s + 31) >> 5, in ? min(((int64_t)e + 31) >> 5, n_chunks) : 0,
              (int32_t)u);
    // tile c's first set is the first one at or after bucket c * T: the one
    // after the set that bucket c * T lies in, beyond its first bucket
    fill_runs(tile_first, in ? toff / T + 1 : 0, in ? min((toff + l) / T + 1, tile_cap) : 0,
              (int32_t)u + 1);
    if (in && u == 0) tile_first[0] = 0;
  }
}

// ------------------------------------------------------- slot storages --

// Shared-memory tile: plane k of the tile at S + k*stride; per-bucket fill
// counts in bytes.
struct SmemSlots {
  int32_t* S;
  int stride;
  unsigned char* fill;
  int base;  // first bucket of the set inside the tile
  __device__ __forceinline__ int get_fill(int bb) const {
    return fill[base + bb];
  }
  __device__ __forceinline__ void set_fill(int bb, int f) const {
    fill[base + bb] = (unsigned char)f;
  }
  __device__ __forceinline__ void put(int bb, int k, int x) const {
    S[k * stride + base + bb] = x;
  }
};

// HBM slots of one set, fill counts in shared memory.
struct GlobalSlotsSmemFill {
  int32_t* G;  // table + off[u]
  int64_t bn;
  unsigned char* fill;
  __device__ __forceinline__ int get_fill(int bb) const { return fill[bb]; }
  __device__ __forceinline__ void set_fill(int bb, int f) const {
    fill[bb] = (unsigned char)f;
  }
  __device__ __forceinline__ void put(int bb, int k, int x) const {
    G[bb + (int64_t)k * bn] = x;
  }
};

// HBM slots of one set; the fill count is re-read from the slots (slots of
// a bucket fill in order, so it is the index of the first -1).
struct GlobalSlotsScan {
  int32_t* G;
  int64_t bn;
  int b;
  __device__ __forceinline__ int get_fill(int bb) const {
    int k = 0;
    while (k < b && __ldcg(G + bb + (int64_t)k * bn) != -1) ++k;
    return k;
  }
  __device__ __forceinline__ void set_fill(int, int) const {}
  __device__ __forceinline__ void put(int bb, int k, int x) const {
    __stcg(G + bb + (int64_t)k * bn, x);
  }
};

// One thread inserts one set sequentially (triangle-count/hashtable.cu:65-74
// rule, CSR order).
template <bool HIER, class Slots>
__device__ void insert_set_thread(const int32_t* __restrict__ keys, int d,
                                  int lg, int lg_max, int b, const Slots& sl,
                                  int32_t* status) {
  const int l = 1 << lg;
  for (int j = 0; j < d; ++j) {
    int x = keys[j];
    int bb = home_bucket<HIER>(x, lg, lg_max);
    int f = sl.get_fill(bb);
    int guard = 0;
    while (f >= b && guard < l) {
      bb = (bb + 1) & (l - 1);
      f = sl.get_fill(bb);
      ++guard;
    }
    if (guard >= l) {
      atomicOr(status, kErrTableFull);
      continue;
    }
    sl.put(bb, f, x);
    sl.set_fill(bb, f + 1);
  }
}

// A warp inserts one set, 32 keys per batch, with the result of sequential
// CSR-order insertion.  Per round, every pending lane finds the first
// non-full bucket B from its current bucket and the fill k0 there; lanes
// aiming at the same bucket are ranked by lane order (match_any).  Lanes
// below the first lane that would overflow its bucket are committed: none of
// them lands outside its bucket, so none can change another's placement.
// The lowest pending lane never overflows, so every round makes progress.
template <bool HIER, class Slots>
__device__ void insert_set_warp(const int32_t* __restrict__ keys, int d,
                                int lg, int lg_max, int b, const Slots& sl,
                                int32_t* status) {
  const int lane = threadIdx.x & 31;
  const int l = 1 << lg;
  const unsigned lt = lanemask_lt(), gt = lanemask_gt();
  // the next round's keys are loaded before this round is inserted, so the
  // load latency overlaps the insertion (long sets take many rounds)
  int xn = lane < d ? __ldg(keys + lane) : 0;
  for (int j0 = 0; j0 < d; j0 += 32) {
    const int j = j0 + lane;
    const bool valid = j < d;
    const int x = xn;
    if (j + 32 < d) xn = __ldg(keys + j + 32);
    int h = valid ? home_bucket<HIER>(x, lg, lg_max) : 0;
    unsigned pending = __ballot_sync(kFull, valid);
    while (pending) {
      const bool me = (pending >> lane) & 1u;
      int B = -1 - lane;  // unique for lanes not in this round
      int k0 = 0;
      bool dropped = false;
      if (me) {
        int f = sl.get_fill(h);
        int guard = 0;
        while (f >= b && guard < l) {
          h = (h + 1) & (l - 1);
          f = sl.get_fill(h);
          ++guard;
        }
        if (guard >= l) {
          atomicOr(status, kErrTableFull);
          dropped = true;
          B = -100 - lane;
        } else {
          B = h;
          k0 = f;
        }
      }
      const unsigned grp = __match_any_sync(kFull, B);
      const int rank = __popc(grp & pending & lt);
      const bool over = me && !dropped && (k0 + rank >= b);
      const unsigned ov = __ballot_sync(kFull, over);
      const unsigned below = ov ? ((1u << (__ffs(ov) - 1)) - 1u) : kFull;
      const bool commit = me && ((below >> lane) & 1u);
      const unsigned cm = __ballot_sync(kFull, commit);
      if (commit && !dropped) {
        sl.put(B, k0 + rank, x);
        if ((grp & cm & gt) == 0) sl.set_fill(B, k0 + rank + 1);
      }
      __syncwarp();
      pending &= ~cm;
    }
  }
}

// Reads one set's slots back in bucket order (slot-major within the set)
// and appends the non-empty ones to out (baseline/common/utils.cu:105-131).
template <class Get>
__device__ void extract_set_warp(int l, int b, int32_t* __restrict__ out,
                                 const Get& get) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  int w = 0;
  const int total = l * b;
  for (int i0 = 0; i0 < total; i0 += 32) {
    int i = i0 + lane;
    int v = -1;
    if (i < total) v = get(i / b, i % b);
    unsigned msk = __ballot_sync(kFull, v != -1);
    if (v != -1) out[w + __popc(msk & lt)] = v;
    w += __popc(msk);
  }
}

// ----------------------------------------------------------- tile build --

template <bool HIER>
__global__ void __launch_bounds__(kTileThreads)
    tile_build_kernel(const int32_t* __restrict__ off,
                      const int32_t* __restrict__ elems,
                      const int32_t* __restrict__ len,
                      const int64_t* __restrict__ off64,
                      const int32_t* __restrict__ tile_first,
                      int64_t bucket_num, int b, int lg_max, int R_max, int LT,
                      int32_t* __restrict__ table,
                      int32_t* __restrict__ hash_out,
                      int32_t* __restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem[];
  int32_t* S = reinterpret_cast<int32_t*>(smem);
  unsigned char* fill = smem + (size_t)R_max * 4 * b;
  __shared__ int s_span[kTileWarps];
  __shared__ int s_wnext;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int s0 = tile_first[blockIdx.x], s1 = tile_first[blockIdx.x + 1];
  int u = s0;
  while (u < s1) {
    // Next segment: long sets are skipped (built after the tiles); a run is
    // the maximal span of consecutive tile-sized sets.  Every warp finds it
    // (the same answer, from L1-cached lengths), so no barrier waits for one
    // warp's scan.
    int r = u;
    if (len[u] > LT) {
      r = -(u + 1);
    } else {
      for (;;) {
        int idx = r + lane;
        bool stop = idx >= s1 || len[idx] > LT;
        unsigned msk = __ballot_sync(kFull, stop);
        if (msk) {
          r += __ffs(msk) - 1;
          break;
        }
        r += 32;
      }
    }
    if (r < 0) {  // a long set
      u = -r;
      continue;
    }
    const int64_t RA = off64[u];
    const int R = (int)(off64[r] - RA);  // multiple of 8, <= R_max

    // 1. clear the tile: b planes of R slots to -1, R fill bytes to 0.
    {
      const int4 neg = make_int4(-1, -1, -1, -1);
      const int q = R >> 2;
      for (int k = 0; k < b; ++k) {
        int4* P = reinterpret_cast<int4*>(S + (size_t)k * R_max);
        for (int i = tid; i < q; i += kTileThreads) P[i] = neg;
      }
      int32_t* F = reinterpret_cast<int32_t*>(fill);
      for (int i = tid; i < q; i += kTileThreads) F[i] = 0;
      if (tid == 0) s_wnext = 0;
    }
    __syncthreads();

    // 2a. small sets, one thread each.
    for (int s = u + tid; s < r; s += kTileThreads) {
      int rs = off[s], d = off[s + 1] - rs;
      if (d > kThreadSetMax || d == 0) continue;
      int lg = 31 - __clz(len[s]);
      SmemSlots sl{S, R_max, fill, (int)(off64[s] - RA)};
      insert_set_thread<HIER>(elems + rs, d, lg, lg_max, b, sl, status);
    }
    // 2b. larger sets, one warp each, taken from a shared cursor (a fixed
    // round-robin left warps with one long set waiting at the barrier)
    for (int wround = 0;; ++wround) {
      int s = 0;
      if (kTileDynamic) {
        if (lane == 0) s = u + atomicAdd(&s_wnext, 1);
        s = __shfl_sync(kFull, s, 0);
      } else {
        s = u + warp + kTileWarps * wround;
      }
      if (s >= r) break;
      int rs = off[s], d = off[s + 1] - rs;
      if (d <= kThreadSetMax) continue;
      int lg = 31 - __clz(len[s]);
      SmemSlots sl{S, R_max, fill, (int)(off64[s] - RA)};
      insert_set_warp<HIER>(elems + rs, d, lg, lg_max, b, sl, status);
    }
    fence_proxy_async_smem();
    __syncthreads();

    // 3. planes -> HBM through the bulk-copy engine.
    if (tid == 0) {
      for (int k = 0; k < b; ++k)
        bulk_store(table + (int64_t)k * bucket_num + RA, S + (size_t)k * R_max,
                   (unsigned)R * 4u);
      bulk_commit();
    }
    // 4. optional: rows in bucket order, read from the tile.  The run's sets
    // are consecutive in the tile and their rows consecutive in the CSR, so
    // the rows in bucket order are the tile's non-empty slots in (bucket,
    // slot) order, compacted into hash_out[off[u] .. off[r]): each warp
    // counts a contiguous span of buckets, then writes its keys after the
    // spans before it.  A lane takes a bucket, not a slot: with 5 slots to a
    // bucket most are empty (R-MAT scale 22, build with rows: 3.24 -> 2.33 ms).
    if (hash_out) {
      const int span = (((R + kTileWarps - 1) / kTileWarps) + 31) & ~31;
      const int h_lo = min(R, warp * span), h_hi = min(R, h_lo + span);
      auto keys_of = [&](int h) {  // a bucket's keys (its slots fill in order)
        int f = 0;
        if (h < h_hi)
          while (f < b && S[f * R_max + h] != -1) ++f;
        return f;
      };
      int c = 0;
      for (int h = h_lo + lane; h < h_hi; h += 32) c += b == 1 ? S[h] != -1 : keys_of(h);
      c = __reduce_add_sync(kFull, c);
      if (lane == 0) s_span[warp] = c;
      __syncthreads();
      int w = off[u];
      for (int k = 0; k < warp; ++k) w += s_span[k];
      const unsigned lt = lanemask_lt();
      if (b == 1) {
        for (int h0 = h_lo; h0 < h_hi; h0 += 32) {
          const int h = h0 + lane, v = h < h_hi ? S[h] : -1;
          const unsigned m = __ballot_sync(kFull, v != -1);
          if (v != -1) hash_out[w + __popc(m & lt)] = v;
          w += __popc(m);
        }
      } else for (int h0 = h_lo; h0 < h_hi; h0 += 32) {
        const int h = h0 + lane, f = keys_of(h);
        // keys before this bucket's: at most b ballots, usually one or two
        int before = 0, all = 0;
        for (int k = 0; k < b; ++k) {
          const unsigned m = __ballot_sync(kFull, f > k);
          if (!m) break;
          before += __popc(m & lt);
          all += __popc(m);
        }
        for (int k = 0; k < f; ++k) hash_out[w + before + k] = S[k * R_max + h];
        w += all;
      }
    }
    if (tid == 0) bulk_wait_read_all();
    __syncthreads();
    u = r;
  }
  if (tid == 0) bulk_wait_all();
}

// ------------------------------------------------------------ long sets --
//
// Sets whose table does not fit a tile, all of them together, with exactly
// the slots of sequential CSR-order insertion.  Which slots are occupied does
// not depend on the insertion order, only which key lies where, so:
//  1. long_insert: every key, in parallel, puts its INDEX in the row into the
//     first free slot at or after its home bucket (a compare-and-swap on the
//     slots themselves).  The occupied slots are then the final ones.
//  2. long_fix: a run is a maximal stretch of full buckets and the bucket
//     after it.  A key never leaves its home's run, so the run's slots hold
//     exactly the indices of the run's keys: one thread per run sorts them
//     and replays the sequential rule, writing the keys.
// Runs are a few buckets long at the loads in use.  A set with a walk of
// kWalkMax buckets or a run of more than kRunMax keys is "crowded" (a key
// repeated many times, a full table): one warp inserts it sequentially, or
// build_huge builds it if it is long.  Sets that their load makes likely to be
// (crowded_by_load) are so from the start: insert and fix would come on top.
// Builds with rows, us, one warp per set / all through insert and fix / by
// load: 60 sets of 30,000 keys, 16 slots a bucket, load 0.92 1030 / 4340 / 680;
// 400 of 5000, one slot, load 0.61 343 / 618 / 265; 10 of 200,000, 5 slots,
// load 0.61 2200 / 613 / 608 (a long set is likely by its own keys: build_huge takes
// one set, while a sequential one holds all up).
// Bound by the latency of the scattered slot accesses.  Index of 2M documents
// and 100k terms (8M postings, ~100 long sets), build with rows, b = 5 / b = 1:
// one warp per set, and 20 launches per set of 2^16 keys, 7.9 / 31 ms; all
// sets together 0.57 / 1.07 ms; 20M documents, 1M terms 36.7 / 59 -> 4.5 / 8.2.
constexpr int kKeyItem = 2048;     // keys per CTA of long_insert
constexpr int kBucketItem = 2048;  // buckets per CTA of long_fix / long_rows
constexpr int kWalkMax = 256;
constexpr int kRunMax = 96;

struct LongSet {
  int32_t crowded;  // from the start: a warp inserts it, or build_huge
  int32_t rs, d, lg;
  int64_t toff;
  // its first items: keys, buckets, and buckets of sets that are not crowded
  // from the start (which have no items of keys either)
  int32_t key_item, bucket_item, work_item;
};

// Whether runs of more than kRunMax keys are likely among `keys` keys at this
// load.  Their number falls as exp(-kRunMax * (load - 1 - ln load)), the decay of
// linear probing's runs at any bucket size; over random homes, with 1 to 16 slots
// a bucket and loads from 0.65 to 0.9, it was 0.0035 times that per key.
__device__ __forceinline__ bool crowded_by_load(float load, float keys) {
  return 0.0035f * keys * expf(-kRunMax * (load - 1.f - logf(load))) > 0.25f;
}

// The long sets' descriptors, the prefix sums of their items, and which are
// crowded by their load or inserted by a warp each for their number (one block).
__global__ void __launch_bounds__(1024)
    long_plan_kernel(const int32_t* __restrict__ off, const int32_t* __restrict__ len,
                     const int64_t* __restrict__ off64, const int32_t* __restrict__ list, int n,
                     int b, float all_keys, int warp_keys, LongSet* __restrict__ sets,
                     LongSet* __restrict__ huge, int32_t* __restrict__ crowded) {
  using Scan = cub::BlockScan<int, 1024>;
  __shared__ typename Scan::TempStorage tmp;
  int keys = 0, buckets = 0, work = 0;  // items before this pass
  for (int base = 0; base < n; base += 1024) {
    const int i = base + threadIdx.x;
    LongSet s{};
    int ki = 0, bi = 0, wi = 0;
    if (i < n) {
      const int u = list[i];
      s.rs = off[u];
      s.d = off[u + 1] - s.rs;
      const int l = len[u];
      s.lg = 31 - __clz(l);
      s.toff = off64[u];
      bi = (l + kBucketItem - 1) / kBucketItem;
      s.crowded = s.d < warp_keys ||
                  crowded_by_load((float)s.d / ((float)l * (float)b),
                                  s.d >= kHugeKeys ? (float)s.d : all_keys);
      crowded[i] = s.crowded;
      if (!s.crowded) {
        ki = (s.d + kKeyItem - 1) / kKeyItem;
        wi = bi;
      }
    }
    int total;
    __syncthreads();
    Scan(tmp).ExclusiveSum(ki, s.key_item, total);
    s.key_item += keys;
    keys += total;
    __syncthreads();
    Scan(tmp).ExclusiveSum(bi, s.bucket_item, total);
    s.bucket_item += buckets;
    buckets += total;
    __syncthreads();
    Scan(tmp).ExclusiveSum(wi, s.work_item, total);
    s.work_item += work;
    work += total;
    if (i < n) sets[i] = s;
  }
  if (threadIdx.x == 0) {
    LongSet end{};
    end.key_item = keys;
    end.bucket_item = buckets;
    end.work_item = work;
    sets[n] = end;
    huge[0] = LongSet{};
  }
}

// The set whose items hold `item` (-1: past the last), found by thread 0.
template <int32_t LongSet::*FIRST>
__device__ __forceinline__ int long_set_of(const LongSet* __restrict__ sets, int n, int item) {
  __shared__ int s_i;
  if (threadIdx.x == 0) {
    // largest i with first item <= item
    int lo = sets[n].*FIRST <= item ? n : 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sets[mid].*FIRST <= item) lo = mid; else hi = mid - 1;
    }
    s_i = lo < n ? lo : -1;
  }
  __syncthreads();
  return s_i;
}

__global__ void __launch_bounds__(kThreads)
    long_clear_kernel(const LongSet* __restrict__ sets, int n, int64_t bucket_num, int b,
                      int32_t* __restrict__ table) {
  const int i = long_set_of<&LongSet::work_item>(sets, n, blockIdx.x);
  if (i < 0) return;
  const LongSet s = sets[i];
  const int h0 = ((int)blockIdx.x - s.work_item) * kBucketItem;
  const int q = min(kBucketItem, (1 << s.lg) - h0) >> 2;
  const int4 neg = make_int4(-1, -1, -1, -1);
  for (int k = 0; k < b; ++k) {
    int4* P = reinterpret_cast<int4*>(table + s.toff + h0 + (int64_t)k * bucket_num);
    for (int j = threadIdx.x; j < q; j += kThreads) P[j] = neg;
  }
}

template <bool HIER>
__global__ void __launch_bounds__(kThreads)
    long_insert_kernel(const int32_t* __restrict__ elems, const LongSet* __restrict__ sets, int n,
                       int64_t bucket_num, int b, int lg_max, int32_t* __restrict__ table,
                       int32_t* __restrict__ crowded) {
  const int i = long_set_of<&LongSet::key_item>(sets, n, blockIdx.x);
  if (i < 0) return;
  const LongSet s = sets[i];
  const int j0 = ((int)blockIdx.x - s.key_item) * kKeyItem;
  int32_t* G = table + s.toff;
  const int lmask = (1 << s.lg) - 1;
  constexpr int kPer = kKeyItem / kThreads;
  int h[kPer];
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int j = j0 + r * kThreads + threadIdx.x;
    h[r] = j < s.d ? home_bucket<HIER>(__ldg(elems + s.rs + j), s.lg, lg_max) : -1;
  }
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    if (h[r] < 0) continue;
    const int j = j0 + r * kThreads + threadIdx.x;
    int hh = h[r], k = 0, walked = 0;
    while (atomicCAS(G + hh + (int64_t)k * bucket_num, -1, j) != -1) {
      if (++k < b) continue;
      k = 0;
      hh = (hh + 1) & lmask;
      if (++walked == kWalkMax || *(volatile int32_t*)(crowded + i)) {
        crowded[i] = 1;  // (the key is left out: the set is built again)
        break;
      }
    }
  }
}

// The runs that start in a bucket item (step 2 above).
template <bool HIER>
__global__ void __launch_bounds__(kThreads)
    long_fix_kernel(const int32_t* __restrict__ elems, const LongSet* __restrict__ sets, int n,
                    int64_t bucket_num, int b, int lg_max, int32_t* __restrict__ table,
                    int32_t* __restrict__ crowded) {
  const int i = long_set_of<&LongSet::work_item>(sets, n, blockIdx.x);
  if (i < 0) return;
  const LongSet s = sets[i];
  if (crowded[i]) return;
  int32_t* G = table + s.toff;
  const int lmask = (1 << s.lg) - 1;
  const int h0 = ((int)blockIdx.x - s.work_item) * kBucketItem;
  const int h1 = min(h0 + kBucketItem, lmask + 1);
  const int64_t last = (int64_t)(b - 1) * bucket_num;  // a bucket's last slot
  for (int h = h0 + threadIdx.x; h < h1; h += kThreads) {
    // an occupied slot holds an index or, once its run is done, a key (>= 0)
    if (__ldcg(G + h) == -1 || __ldcg(G + ((h - 1) & lmask) + last) != -1) continue;
    int idx[kRunMax];
    int t = 0;
    bool fits = true;
    for (int e = h;; e = (e + 1) & lmask) {  // the run's indices, in order
      bool full = true;
      for (int k = 0; k < b; ++k) {
        const int v = __ldcg(G + e + (int64_t)k * bucket_num);
        if (v == -1) {
          full = false;
          break;
        }
        if (t == kRunMax) {
          fits = false;
          break;
        }
        int p = t++;
        for (; p > 0 && idx[p - 1] > v; --p) idx[p] = idx[p - 1];
        idx[p] = v;
      }
      if (!full || !fits) break;
    }
    if (!fits) {
      crowded[i] = 1;
      continue;
    }
    unsigned char fill[kRunMax];  // keys placed per bucket of the run
    for (int j = 0; j < t; ++j) fill[j] = 0;
    for (int j = 0; j < t; ++j) {
      const int x = __ldg(elems + s.rs + idx[j]);
      int p = (home_bucket<HIER>(x, s.lg, lg_max) - h) & lmask;
      while (fill[p] == b) ++p;
      G[((h + p) & lmask) + (int64_t)fill[p] * bucket_num] = x;
      ++fill[p];
    }
  }
}

// Crowded sets, sequentially, a CTA each (those of kHugeKeys keys or more are
// listed for build_huge, huge[0].d of them from huge[1] on).
template <bool HIER>
__global__ void __launch_bounds__(kThreads)
    long_crowded_kernel(const int32_t* __restrict__ elems, const LongSet* __restrict__ sets,
                        const int32_t* __restrict__ crowded, int64_t bucket_num, int b, int lg_max,
                        int32_t* __restrict__ table, LongSet* __restrict__ huge,
                        int32_t* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char fill[];
  if (!crowded[blockIdx.x]) return;
  const LongSet s = sets[blockIdx.x];
  if (s.d >= kHugeKeys) {
    if (threadIdx.x == 0) huge[1 + atomicAdd(&huge->d, 1)] = s;
    return;
  }
  const int l = 1 << s.lg;
  int32_t* G = table + s.toff;
  const int tid = threadIdx.x;
  {
    const int4 neg = make_int4(-1, -1, -1, -1);
    for (int k = 0; k < b; ++k) {
      int4* P = reinterpret_cast<int4*>(G + (int64_t)k * bucket_num);
      for (int i = tid; i < (l >> 2); i += kThreads) P[i] = neg;
    }
    if (l <= kBigFillSmemMax) {
      int32_t* F = reinterpret_cast<int32_t*>(fill);
      for (int i = tid; i < (l >> 2); i += kThreads) F[i] = 0;
    }
  }
  __syncthreads();
  if (tid < 32) {
    if (l <= kBigFillSmemMax)
      insert_set_warp<HIER>(elems + s.rs, s.d, s.lg, lg_max, b,
                            GlobalSlotsSmemFill{G, bucket_num, fill}, status);
    else
      insert_set_warp<HIER>(elems + s.rs, s.d, s.lg, lg_max, b,
                            GlobalSlotsScan{G, bucket_num, b}, status);
  }
}

// The long sets' rows in bucket order: a set's non-empty slots in (bucket,
// slot) order, compacted.  long_count: per bucket item, then a scan over all
// items; long_rows writes.
__global__ void __launch_bounds__(kThreads)
    long_count_kernel(const LongSet* __restrict__ sets, int n, int64_t bucket_num, int b,
                      const int32_t* __restrict__ table, int32_t* __restrict__ blk_cnt) {
  __shared__ int s_c[kWarps];
  const int i = long_set_of<&LongSet::bucket_item>(sets, n, blockIdx.x);
  int c = 0;
  if (i >= 0) {
    const LongSet s = sets[i];
    const int h0 = ((int)blockIdx.x - s.bucket_item) * kBucketItem;
    const int h1 = min(h0 + kBucketItem, 1 << s.lg);
    for (int k = 0; k < b; ++k) {
      const int32_t* P = table + s.toff + (int64_t)k * bucket_num;
      for (int h = h0 + threadIdx.x; h < h1; h += kThreads) c += P[h] != -1;
    }
  }
  c = __reduce_add_sync(kFull, c);
  if ((threadIdx.x & 31) == 0) s_c[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w) c += s_c[w];
    blk_cnt[blockIdx.x] = c;
  }
}

__global__ void __launch_bounds__(kThreads)
    long_rows_kernel(const LongSet* __restrict__ sets, int n, int64_t bucket_num, int b,
                     const int32_t* __restrict__ table, const int32_t* __restrict__ blk_off,
                     int32_t* __restrict__ hash_out) {
  using Scan = cub::BlockScan<int, kThreads>;
  __shared__ typename Scan::TempStorage tmp;
  const int i = long_set_of<&LongSet::bucket_item>(sets, n, blockIdx.x);
  if (i < 0) return;
  const LongSet s = sets[i];
  const int h0 = ((int)blockIdx.x - s.bucket_item) * kBucketItem;
  const int h1 = min(h0 + kBucketItem, 1 << s.lg);
  int32_t* out = hash_out + s.rs + (blk_off[blockIdx.x] - blk_off[s.bucket_item]);
  for (int hb = h0; hb < h1; hb += kThreads) {
    const int h = hb + threadIdx.x;
    const int32_t* P = table + s.toff + h;
    int f = 0;
    if (h < h1)
      while (f < b && P[(int64_t)f * bucket_num] != -1) ++f;
    int at, total;
    __syncthreads();
    Scan(tmp).ExclusiveSum(f, at, total);
    for (int k = 0; k < f; ++k) out[at + k] = P[(int64_t)k * bucket_num];
    out += total;
  }
}

// ----------------------------------------------------------- huge build --
//
// One set of d >= kHugeKeys keys that long_insert_kernel found too crowded,
// built in parallel with exactly the slots of sequential CSR-order insertion:
//  1. home bucket of every key, keys per home bucket (cnt);
//  2. the final fills: in linear probing they do not depend on the
//     insertion order -- the keys carried from bucket h to h+1 are
//     c(h+1) = max(0, c(h) + cnt(h) - b), a max-plus recurrence solved by
//     one scan (c -> max(P, c + Q) composes); the table is circular and
//     holds fewer keys than slots, so the carry into bucket 0 is the P of
//     the whole composition;
//  3. clusters = runs of buckets a carry flows through (a bucket with carry
//     0 starts one); keys never leave their home bucket's cluster;
//  4. keys stably sorted by cluster (so CSR order within each), then one
//     thread per cluster replays the sequential rule on its keys.

struct CarryFn {  // c -> max(p, c + q)
  long long p, q;
};
struct ComposeCarry {  // apply a, then b
  __host__ __device__ CarryFn operator()(const CarryFn& a, const CarryFn& b) const {
    return CarryFn{max(b.p, a.p + b.q), a.q + b.q};
  }
};
struct MaxI32 {
  __host__ __device__ int32_t operator()(int32_t a, int32_t b) const { return a > b ? a : b; }
};

template <bool HIER>
__global__ void huge_home_kernel(const int32_t* __restrict__ keys, int64_t d, int lg,
                                 int lg_max, int32_t* __restrict__ home,
                                 int32_t* __restrict__ cnt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < d;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int h = home_bucket<HIER>(__ldg(keys + i), lg, lg_max);
    home[i] = h;
    atomicAdd(cnt + h, 1);
  }
}

// Carry functions of the buckets; nxt[h] = the next bucket (circular).
__global__ void huge_fn_kernel(const int32_t* __restrict__ cnt, int64_t l, int b,
                               CarryFn* __restrict__ fn, int32_t* __restrict__ nxt) {
  for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < l;
       h += (int64_t)gridDim.x * blockDim.x) {
    fn[h] = CarryFn{0, (long long)cnt[h] - b};
    nxt[h] = (int32_t)((h + 1) & (l - 1));
  }
}

// start[h] = h where the carry into bucket h is 0, else -1 (fn holds the
// inclusive prefix compositions).
__global__ void huge_start_kernel(const CarryFn* __restrict__ fn, int64_t l,
                                  int32_t* __restrict__ start) {
  const long long c0 = fn[l - 1].p;
  for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < l;
       h += (int64_t)gridDim.x * blockDim.x) {
    const long long c = h == 0 ? c0 : max(fn[h - 1].p, c0 + fn[h - 1].q);
    start[h] = c == 0 ? (int32_t)h : -1;
  }
}

// Cluster of every key: the last carry-free bucket at or before its home
// (before bucket 0: the last one of the table, the cluster that wraps).
__global__ void huge_cluster_kernel(const int32_t* __restrict__ home, int64_t d,
                                    const int32_t* __restrict__ cstart, int64_t l,
                                    int32_t* __restrict__ cid, int32_t* __restrict__ idx) {
  const int32_t wrap = cstart[l - 1];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < d;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = cstart[home[i]];
    cid[i] = c >= 0 ? c : wrap;
    idx[i] = (int32_t)i;
  }
}

// One thread per cluster: its keys (sorted_idx[seg .. seg + len), CSR
// order) inserted by the sequential rule; fill[] starts at 0.
__global__ void huge_place_kernel(const int32_t* __restrict__ keys,
                                  const int32_t* __restrict__ home,
                                  const int32_t* __restrict__ sorted_idx,
                                  const int32_t* __restrict__ run_len,
                                  const int32_t* __restrict__ run_off,
                                  const int32_t* __restrict__ n_runs, int64_t l, int b,
                                  int64_t bn, int32_t* __restrict__ fill,
                                  int32_t* __restrict__ nxt, int32_t* __restrict__ G,
                                  int32_t* __restrict__ status) {
  const int64_t nr = *n_runs;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nr;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t s0 = run_off[r], s1 = s0 + run_len[r];
    for (int32_t j = s0; j < s1; ++j) {
      const int32_t i = sorted_idx[j];
      // first bucket with room at or after the home bucket: full buckets
      // point further along (nxt, compressed on the way), so a run of
      // repeated keys does not rescan its cluster for every key
      int64_t h = home[i];
      int64_t guard = 0;
      while (fill[h] >= b && guard < l) {
        h = nxt[h];
        ++guard;
      }
      if (guard >= l) {
        atomicOr(status, kErrTableFull);
        continue;
      }
      for (int64_t x = home[i]; x != h && fill[x] >= b;) {  // compress
        const int64_t y = nxt[x];
        nxt[x] = (int32_t)h;
        x = y;
      }
      const int k = fill[h]++;
      G[h + (int64_t)k * bn] = keys[i];
    }
  }
}

// ------------------------------------------------- standalone extraction --

__global__ void __launch_bounds__(kThreads)
    extract_kernel(const int32_t* __restrict__ off,
                   const int64_t* __restrict__ off64, int32_t n,
                   const int32_t* __restrict__ table, int64_t bucket_num,
                   int b, int32_t* __restrict__ out) {
  const int warps = gridDim.x * kWarps;
  for (int s = blockIdx.x * kWarps + (threadIdx.x >> 5); s < n; s += warps) {
    int rs = off[s], d = off[s + 1] - rs;
    if (d <= 0) continue;
    int64_t toff = off64[s];
    int l = (int)(off64[s + 1] - toff);
    const int32_t* G = table + toff;
    extract_set_warp(l, b, out + rs, [&](int bb, int k) {
      return __ldg(G + bb + (int64_t)k * bucket_num);
    });
  }
}

int grid_for(int64_t items, int threads, int per_sm = 8) {
  int64_t g = (items + threads - 1) / threads;
  int64_t cap = (int64_t)sm_count() * per_sm;
  if (g > cap) g = cap;
  return (int)(g > 0 ? g : 1);
}

}  // namespace

reset_status make_chunk_rows(const int32_t* d_off, int32_t n, int64_t m,
                             int32_t** d_rows_out, cudaStream_t st) {
  int64_t nc = (m + 31) / 32;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(d_rows_out),
                           sizeof(int32_t) * (nc > 0 ? nc : 1), st));
  RST_CUDA(cudaMemsetAsync(*d_rows_out, 0, sizeof(int32_t) * (nc > 0 ? nc : 1), st));
  note_launch(); chunk_rows_kernel<<<grid_for(n, kThreads), kThreads, 0, st>>>(d_off, n, nc,
                                                                             *d_rows_out);
  RST_CUDA(cudaGetLastError());
  return RESET_OK;
}

// Descriptors for offsets other than the build CSR; the table offsets and
// lengths still come from the table.
__global__ void redesc_kernel(const int32_t* __restrict__ off,
                              const int4* __restrict__ src, int32_t n,
                              int4* __restrict__ dst) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n;
       u += (int64_t)gridDim.x * blockDim.x) {
    int4 d = src[u];
    int s = off[u];
    d.x = s;
    d.y = off[u + 1] - s;
    dst[u] = d;
  }
}

reset_status make_desc(const reset_table* t, const int32_t* d_off,
                       int4** d_desc_out, cudaStream_t st) {
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(d_desc_out),
                           sizeof(int4) * (t->n > 0 ? t->n : 1), st));
  note_launch(); redesc_kernel<<<grid_for(t->n, 256), 256, 0, st>>>(d_off, t->d_desc, t->n,
                                                     *d_desc_out);
  RST_CUDA(cudaGetLastError());
  return RESET_OK;
}

// Table memory comes from a library-owned stream-ordered pool per device
// whose release threshold is unlimited: freeing a table keeps its pages
// mapped for the next build, so rebuilding a multi-GB table costs no
// cudaMalloc/cudaFree page mapping (reset_release_cached_memory() returns
// them).
namespace {
constexpr int kPoolDevices = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kPoolDevices] = {};
}  // namespace

reset_status table_pool(cudaMemPool_t* out) {
  int dev = 0;
  RST_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kPoolDevices) return arg_fail("device ordinal too large");
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool;
    RST_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = UINT64_MAX;
    RST_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pool[dev] = pool;
  }
  *out = g_pool[dev];
  return RESET_OK;
}

cudaError_t scratch_malloc(void** p, size_t bytes, cudaStream_t st) {
  cudaMemPool_t pool;
  if (table_pool(&pool) != RESET_OK) return cudaErrorMemoryAllocation;
  return cudaMallocFromPoolAsync(p, bytes, pool, st);
}

void release_pools() {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  for (int d = 0; d < kPoolDevices; ++d)
    if (g_pool[d]) cudaMemPoolTrimTo(g_pool[d], 0);
}

}  // namespace rst

using namespace rst;

namespace {

void destroy(reset_table* t) {
  if (!t) return;
  // stream-ordered frees into the table pool (callers synchronise first)
  if (t->d_table) cudaFreeAsync(t->d_table, 0);
  if (t->d_block) cudaFreeAsync(t->d_block, 0);
  delete t;
}

// The parallel build of one huge set (see huge_home_kernel): row start rs,
// d keys, table length l (a power of two) at offset toff.  Scratch comes
// from the table pool, stream-ordered; no host synchronisation.
template <bool HIER>
reset_status build_huge(const reset_table* t, const int32_t* d_elems, int64_t rs, int64_t d,
                        int64_t l, int64_t toff, cudaStream_t st) {
  const int b = t->bucket;
  const int64_t bn = t->bucket_num;
  const int lg = 63 - __builtin_clzll((unsigned long long)l);
  int32_t* G = t->d_table + toff;
  for (int k = 0; k < b; ++k)
    RST_CUDA(cudaMemsetAsync(G + (int64_t)k * bn, 0xFF, sizeof(int32_t) * (size_t)l, st));
  if (d <= 0) return RESET_OK;
  const int di = (int)d, li = (int)l;
  const int32_t* keys = d_elems + rs;
  // CUB temporary sizes
  size_t tb[5] = {0, 0, 0, 0, 0};
  CarryFn* nf = nullptr;
  int32_t* ni = nullptr;
  RST_CUDA(cub::DeviceScan::InclusiveScan(nullptr, tb[0], nf, nf, ComposeCarry(), li, st));
  RST_CUDA(cub::DeviceScan::InclusiveScan(nullptr, tb[1], ni, ni, MaxI32(), li, st));
  RST_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb[2], ni, ni, ni, ni, di, 0,
                                           std::max(lg, 1), st));
  RST_CUDA(cub::DeviceRunLengthEncode::Encode(nullptr, tb[3], ni, ni, ni, ni, di, st));
  RST_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb[4], ni, ni, di, st));
  size_t tmp = 0;
  for (size_t x : tb) tmp = std::max(tmp, x);
  // one scratch block: 8 arrays of d ints, 5 of l ints, l carry functions
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t sd = al(4 * (size_t)d), sl = al(4 * (size_t)l);
  const size_t bytes = 8 * sd + 5 * sl + al(sizeof(CarryFn) * (size_t)l) + al(16) + al(tmp);
  char* base = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&base), bytes, st));
  char* q = base;
  auto carve = [&q](size_t n) {
    char* r = q;
    q += n;
    return r;
  };
  int32_t* home = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* cid = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* idx = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* cid_s = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* idx_s = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* runs = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* run_len = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* run_off = reinterpret_cast<int32_t*>(carve(sd));
  int32_t* cnt = reinterpret_cast<int32_t*>(carve(sl));
  int32_t* start = reinterpret_cast<int32_t*>(carve(sl));
  int32_t* cstart = reinterpret_cast<int32_t*>(carve(sl));
  int32_t* fill = reinterpret_cast<int32_t*>(carve(sl));
  int32_t* nxt = reinterpret_cast<int32_t*>(carve(sl));
  CarryFn* fn = reinterpret_cast<CarryFn*>(carve(al(sizeof(CarryFn) * (size_t)l)));
  int32_t* n_runs = reinterpret_cast<int32_t*>(carve(al(16)));
  void* ctmp = carve(al(tmp));

  reset_status rs_out = RESET_OK;
  auto run = [&]() -> reset_status {
    RST_CUDA(cudaMemsetAsync(cnt, 0, 4 * (size_t)l, st));
    RST_CUDA(cudaMemsetAsync(fill, 0, 4 * (size_t)l, st));
    note_launch();
    huge_home_kernel<HIER><<<grid_for(d, kThreads), kThreads, 0, st>>>(keys, d, lg, t->lg_max,
                                                                      home, cnt);
    note_launch();
    huge_fn_kernel<<<grid_for(l, kThreads), kThreads, 0, st>>>(cnt, l, b, fn, nxt);
    size_t x = tmp;
    RST_CUDA(cub::DeviceScan::InclusiveScan(ctmp, x, fn, fn, ComposeCarry(), li, st));
    note_launch();
    huge_start_kernel<<<grid_for(l, kThreads), kThreads, 0, st>>>(fn, l, start);
    x = tmp;
    RST_CUDA(cub::DeviceScan::InclusiveScan(ctmp, x, start, cstart, MaxI32(), li, st));
    note_launch();
    huge_cluster_kernel<<<grid_for(d, kThreads), kThreads, 0, st>>>(home, d, cstart, l, cid,
                                                                    idx);
    x = tmp;
    RST_CUDA(cub::DeviceRadixSort::SortPairs(ctmp, x, cid, cid_s, idx, idx_s, di, 0,
                                             std::max(lg, 1), st));
    x = tmp;
    RST_CUDA(cub::DeviceRunLengthEncode::Encode(ctmp, x, cid_s, runs, run_len, n_runs, di, st));
    x = tmp;
    RST_CUDA(cub::DeviceScan::ExclusiveSum(ctmp, x, run_len, run_off, di, st));
    note_launch();
    huge_place_kernel<<<grid_for(d, kThreads), kThreads, 0, st>>>(
        keys, home, idx_s, run_len, run_off, n_runs, l, b, bn, fill, nxt, G, t->d_status);
    RST_CUDA(cudaGetLastError());
    return RESET_OK;
  };
  rs_out = run();
  cudaFreeAsync(base, st);
  return rs_out;
}

template <bool HIER>
reset_status launch_builds(const reset_table* t, const int32_t* d_off, const int32_t* d_elems,
                           const int32_t* d_tile_first, int32_t n_tiles, const Geom& g,
                           const int32_t* d_long, const BuildInfo& info,
                           int32_t* d_hash_out, cudaStream_t st) {
  if (n_tiles > 0) {
    // (the same for every bucket size: other threads may be between here and a
    // launch; g.smem is at most the budget)
    RST_CUDA(cudaFuncSetAttribute(tile_build_kernel<HIER>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kTileSmemBudget));
    note_launch(); tile_build_kernel<HIER><<<n_tiles, kTileThreads, g.smem, st>>>(
        d_off, d_elems, t->d_len, t->d_off64, d_tile_first, t->bucket_num,
        t->bucket, t->lg_max, g.R_max, g.LT, t->d_table, d_hash_out,
        t->d_status);
    RST_CUDA(cudaGetLastError());
  }
  if (info.n_long == 0) return RESET_OK;
  // at most one partly filled item per set
  const int n = info.n_long, b = t->bucket;
  const int64_t bn = t->bucket_num;
  const int64_t key_items = (int64_t)(info.long_keys / kKeyItem) + n;
  const int64_t bucket_items = (int64_t)(info.long_buckets / kBucketItem) + n;
  if (bucket_items > INT32_MAX) return arg_fail("too many buckets in long sets");
  size_t scan_bytes = 0;
  if (d_hash_out)
    RST_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (int32_t*)nullptr,
                                           (int32_t*)nullptr, (int)bucket_items, st));
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t sz_sets = al(sizeof(LongSet) * ((size_t)n + 1)), sz_flag = al(4 * (size_t)n);
  const size_t sz_blk = d_hash_out ? al(4 * (size_t)bucket_items) : 0;
  char* base = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&base),
                          2 * sz_sets + sz_flag + 2 * sz_blk + al(scan_bytes), st));
  LongSet* sets = reinterpret_cast<LongSet*>(base);
  LongSet* huge = reinterpret_cast<LongSet*>(base + sz_sets);
  int32_t* crowded = reinterpret_cast<int32_t*>(base + 2 * sz_sets);
  int32_t* blk = reinterpret_cast<int32_t*>(base + 2 * sz_sets + sz_flag);
  int32_t* blk_off = reinterpret_cast<int32_t*>(base + 2 * sz_sets + sz_flag + sz_blk);
  void* scan_tmp = base + 2 * sz_sets + sz_flag + 2 * sz_blk;
  // Sets short enough beside their number: a warp each fills the chip and takes
  // fewer accesses per key, but no less than the longest one's chain.  Without
  // rows, us, key-parallel / a warp per set: 10,000 sets of 1500 keys, 5 slots
  // 914 / 780, one slot 1624 / 834; 2000 of 3000, one slot 723 / 382; 400 of 5000, 5
  // slots 290 / 690.
  int warp_keys = 0;
  unsigned long long below = 0, by_warps = 0;
  for (int i = 0; i < 16; ++i) {
    below += info.keys_lg[i];
    if (below >= 1000ull << (i + 1)) {
      warp_keys = 2 << i;
      by_warps = below;
    }
  }
  const bool parallel = by_warps < info.long_keys;  // some are left
  auto run = [&]() -> reset_status {
    const int fill_smem = kBigFillSmemMax;
    RST_CUDA(cudaFuncSetAttribute(long_crowded_kernel<HIER>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, fill_smem));
    note_launch(parallel ? 5 : 2);
    long_plan_kernel<<<1, 1024, 0, st>>>(d_off, t->d_len, t->d_off64, d_long, n, b,
                                         (float)info.long_keys, warp_keys, sets, huge, crowded);
    if (parallel) {
      long_clear_kernel<<<(unsigned)bucket_items, kThreads, 0, st>>>(sets, n, bn, b, t->d_table);
      long_insert_kernel<HIER><<<(unsigned)key_items, kThreads, 0, st>>>(
          d_elems, sets, n, bn, b, t->lg_max, t->d_table, crowded);
      long_fix_kernel<HIER><<<(unsigned)bucket_items, kThreads, 0, st>>>(
          d_elems, sets, n, bn, b, t->lg_max, t->d_table, crowded);
    }
    long_crowded_kernel<HIER><<<n, kThreads, fill_smem, st>>>(
        d_elems, sets, crowded, bn, b, t->lg_max, t->d_table, huge, t->d_status);
    RST_CUDA(cudaGetLastError());
    if (info.n_huge > 0) {  // one more sync, only for tables that have such sets
      const size_t count = (size_t)info.n_huge + 1;
      std::unique_ptr<LongSet[]> list(new (std::nothrow) LongSet[count]);
      if (!list) return cuda_fail(cudaErrorMemoryAllocation, "long sets", __FILE__, __LINE__);
      RST_CUDA(cudaMemcpyAsync(list.get(), huge, sizeof(LongSet) * count, cudaMemcpyDeviceToHost,
                               st));
      RST_CUDA(cudaStreamSynchronize(st));
      for (int i = 1; i <= list[0].d; ++i) {
        const LongSet& s = list[i];
        RST_CHECK(build_huge<HIER>(t, d_elems, s.rs, s.d, (int64_t)1 << s.lg, s.toff, st));
      }
    }
    if (d_hash_out) {
      note_launch(2);
      long_count_kernel<<<(unsigned)bucket_items, kThreads, 0, st>>>(sets, n, bn, b, t->d_table,
                                                                     blk);
      size_t x = scan_bytes;
      RST_CUDA(cub::DeviceScan::ExclusiveSum(scan_tmp, x, blk, blk_off, (int)bucket_items, st));
      long_rows_kernel<<<(unsigned)bucket_items, kThreads, 0, st>>>(sets, n, bn, b, t->d_table,
                                                                    blk_off, d_hash_out);
      RST_CUDA(cudaGetLastError());
    }
    return RESET_OK;
  };
  const reset_status rs = run();
  cudaFreeAsync(base, st);
  return rs;
}

}  // namespace

extern "C" {

reset_status reset_table_build(const int32_t* d_off, const int32_t* d_elems,
                               int32_t n, int64_t m, const reset_params* params,
                               int32_t hierarchical, int32_t* d_hash_out,
                               reset_table** out, reset_stream_t stream) {
  if (!out) return arg_fail("out is NULL");
  *out = nullptr;
  reset_params p;
  reset_params_default(&p);
  if (params) p = *params;
  if (n < 0 || m < 0) return arg_fail("negative n or m");
  if (!d_off) return arg_fail("d_off is NULL");
  if (m > 0 && !d_elems) return arg_fail("d_elems is NULL");
  if (!(p.alpha > 0.f && p.alpha <= 1.f))
    return arg_fail("alpha must be in (0, 1]");
  if (p.bucket < 1 || p.bucket > 16) return arg_fail("bucket must be in 1..16");
  if (m > INT32_MAX) return arg_fail("m exceeds the int32 CSR range");
  cudaStream_t st = as_stream(stream);
  const Geom g = tile_geom(p.bucket);

  reset_table* t = new reset_table();
  t->n = n;
  t->m = m;
  t->bucket = p.bucket;
  t->alpha = p.alpha;
  t->hier = hierarchical ? 1 : 0;
  t->build_off = d_off;
  cudaGetDevice(&t->device);

  char* scratch = nullptr;
  auto fail = [&](reset_status s) {
    cudaStreamSynchronize(st);
    if (scratch) cudaFreeAsync(scratch, st);
    cudaStreamSynchronize(st);
    destroy(t);
    return s;
  };
#define BUILD_CUDA(call)                                                   \
  do {                                                                     \
    cudaError_t _e = (call);                                               \
    if (_e != cudaSuccess) return fail(cuda_fail(_e, #call, __FILE__, __LINE__)); \
  } while (0)

  // what the table keeps but its slots, in one allocation
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t n1 = n > 0 ? n : 1;
  t->n_chunks = (m + 31) / 32;
  const size_t sz_len = al(sizeof(int32_t) * n1), sz_off = al(sizeof(int64_t) * ((size_t)n + 1));
  const size_t sz_desc = al(sizeof(int4) * n1);
  const size_t sz_rows = al(sizeof(int32_t) * (t->n_chunks > 0 ? t->n_chunks : 1));
  BUILD_CUDA(scratch_malloc(&t->d_block, 256 + sz_len + sz_off + sz_desc + sz_rows, st));
  char* q = static_cast<char*>(t->d_block);
  t->d_status = reinterpret_cast<int32_t*>(q); q += 256;
  t->d_len = reinterpret_cast<int32_t*>(q); q += sz_len;
  t->d_off64 = reinterpret_cast<int64_t*>(q); q += sz_off;
  t->d_desc = reinterpret_cast<int4*>(q); q += sz_desc;
  t->d_chunk_row = reinterpret_cast<int32_t*>(q);

  // scratch: what the host reads back, the blocks' sums, the long sets (each
  // has LT buckets' keys at the least) and the tiles' first sets (len is at
  // most 8 or twice the buckets its keys need at the load factor)
  const int64_t blocks = n > 0 ? std::min<int64_t>((n + 4 * kThreads - 1) / (4 * kThreads),
                                                   (int64_t)sm_count() * 4) : 0;
  const int64_t per = blocks > 0 ? (n + blocks - 1) / blocks : 0;
  const double long_least = std::max(1.0, (double)p.alpha * p.bucket * g.LT * 0.99);
  int64_t long_cap = std::min<int64_t>(n, (int64_t)((double)m / long_least) + 1);
  const int64_t bn_cap = 8 * (int64_t)n +
                         (int64_t)(2.02 * (double)m / ((double)p.alpha * p.bucket)) + 16;
  int64_t tile_cap = bn_cap / g.T + 3;
  const size_t sz_sum = al(sizeof(int64_t) * (blocks > 0 ? blocks : 1));
  BuildInfo info{};
  BuildInfo* d_info = nullptr;
  int32_t *d_long = nullptr, *d_tile_first = nullptr;
  BUILD_CUDA(cudaMemsetAsync(t->d_status, 0, sizeof(int32_t), st));
  if (n == 0) {
    BUILD_CUDA(cudaMemsetAsync(t->d_off64, 0, sizeof(int64_t), st));
    BUILD_CUDA(cudaStreamSynchronize(st));
  }
  while (n > 0) {
    const size_t sz_long = al(sizeof(int32_t) * (size_t)(long_cap > 0 ? long_cap : 1));
    BUILD_CUDA(scratch_malloc(reinterpret_cast<void**>(&scratch),
                              256 + sz_sum + sz_long + al(sizeof(int32_t) * (size_t)tile_cap), st));
    d_info = reinterpret_cast<BuildInfo*>(scratch);
    int64_t* d_sum = reinterpret_cast<int64_t*>(scratch + 256);
    d_long = reinterpret_cast<int32_t*>(scratch + 256 + sz_sum);
    d_tile_first = reinterpret_cast<int32_t*>(scratch + 256 + sz_sum + sz_long);
    BUILD_CUDA(cudaMemsetAsync(d_info, 0, sizeof(BuildInfo), st));
    note_launch(2);
    meta_kernel<<<(int)blocks, kThreads, 0, st>>>(d_off, n, per, p.alpha, p.bucket, g.LT, t->d_len,
                                                  d_sum, d_long, long_cap, d_info, t->d_status);
    layout_kernel<<<(int)blocks, kThreads, 0, st>>>(d_off, t->d_len, n, per, d_sum, t->d_off64,
                                                    t->d_desc, t->n_chunks, t->d_chunk_row,
                                                    d_tile_first, tile_cap, g.T, d_info);
    BUILD_CUDA(cudaGetLastError());
    BUILD_CUDA(cudaMemcpyAsync(&info, d_info, sizeof(info), cudaMemcpyDeviceToHost, st));
    BUILD_CUDA(cudaStreamSynchronize(st));
    const int64_t tiles = (info.bucket_num + g.T - 1) / g.T + 1;
    if (info.n_long <= long_cap && tiles <= tile_cap) break;
    // offsets that descend (an error that reset_table_check reports) can make
    // more of them than m keys do: once more, with room for all
    long_cap = n;
    tile_cap = tiles;
    cudaFreeAsync(scratch, st);
    scratch = nullptr;
  }
  const int64_t bn = info.bucket_num;
  t->bucket_num = bn;
  t->max_len = n > 0 ? info.max_len : 8;
  t->lg_max = 31 - __builtin_clz((unsigned)t->max_len);
  if (bn >= ((int64_t)1 << 56)) return fail(arg_fail("table too large"));
  const int64_t n_tiles64 = (bn + g.T - 1) / g.T;
  if (n_tiles64 > INT32_MAX) return fail(arg_fail("too many tiles"));
  size_t tbytes = sizeof(int32_t) * (size_t)bn * p.bucket;
  BUILD_CUDA(scratch_malloc(reinterpret_cast<void**>(&t->d_table), tbytes > 0 ? tbytes : 16, st));
  if (n > 0) {
    const reset_status rs =
        t->hier ? launch_builds<true>(t, d_off, d_elems, d_tile_first, (int32_t)n_tiles64, g,
                                      d_long, info, d_hash_out, st)
                : launch_builds<false>(t, d_off, d_elems, d_tile_first, (int32_t)n_tiles64, g,
                                       d_long, info, d_hash_out, st);
    if (rs != RESET_OK) return fail(rs);
  }
  if (scratch) cudaFreeAsync(scratch, st);
#undef BUILD_CUDA
  *out = t;
  return RESET_OK;
}

reset_status reset_table_info(const reset_table* t, reset_table_view* v) {
  if (!t || !v) return arg_fail("NULL table or view");
  v->n = t->n;
  v->bucket = t->bucket;
  v->max_len = t->max_len;
  v->hierarchical = t->hier;
  v->bucket_num = t->bucket_num;
  v->m = t->m;
  v->alpha = t->alpha;
  v->pad = 0;
  v->d_table = t->d_table;
  v->d_len = t->d_len;
  v->d_off = t->d_off64;
  return RESET_OK;
}

reset_status reset_table_free(reset_table* t) {
  if (!t) return RESET_OK;
  cudaError_t e = cudaDeviceSynchronize();
  destroy(t);
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceSynchronize", __FILE__, __LINE__);
  return RESET_OK;
}

reset_status reset_table_free_async(reset_table* t, reset_stream_t stream) {
  if (!t) return RESET_OK;
  cudaStream_t st = as_stream(stream);
  cudaError_t e = cudaSuccess;
  for (void* p : {static_cast<void*>(t->d_table), t->d_block})
    if (p) {
      cudaError_t e2 = cudaFreeAsync(p, st);
      if (e == cudaSuccess) e = e2;
    }
  delete t;
  if (e != cudaSuccess) return cuda_fail(e, "cudaFreeAsync", __FILE__, __LINE__);
  return RESET_OK;
}

reset_status reset_release_cached_memory(void) {
  RST_CUDA(cudaDeviceSynchronize());
  release_pools();
  return RESET_OK;
}

reset_status reset_table_check(reset_table* t, reset_stream_t stream) {
  if (!t) return arg_fail("NULL table");
  cudaStream_t st = as_stream(stream);
  int32_t bits = 0;
  RST_CUDA(cudaMemcpyAsync(&bits, t->d_status, sizeof(bits),
                           cudaMemcpyDeviceToHost, st));
  RST_CUDA(cudaStreamSynchronize(st));
  if (bits) {
    RST_CUDA(cudaMemsetAsync(t->d_status, 0, sizeof(int32_t), st));
    RST_CUDA(cudaStreamSynchronize(st));
  }
  if (bits & kErrTableFull) {
    set_error("a set did not fit its table (or a CSR row had negative length)");
    return RESET_ERR_TABLE_FULL;
  }
  if (bits & kErrProbeLimit) {
    set_error("a probe walked a whole table without finding an empty slot");
    return RESET_ERR_PROBE_LIMIT;
  }
  if (bits & kErrBadId) {
    set_error("invalid argument: a row, pair or query id was outside [0, n)");
    return RESET_ERR_ARG;
  }
  if (bits & kErrStageTimeout) {
    set_error("a bounded wait for a shared-memory bulk copy gave up");
    return RESET_ERR_TIMEOUT;
  }
  return RESET_OK;
}

reset_status reset_csr_hash_order(const reset_table* t, const int32_t* d_off,
                                  int32_t* d_cols_out, reset_stream_t stream) {
  if (!t || !d_off || (!d_cols_out && t->m > 0))
    return arg_fail("NULL table, offsets or output");
  if (t->n == 0) return RESET_OK;
  cudaStream_t st = as_stream(stream);
  note_launch(); extract_kernel<<<grid_for((int64_t)t->n * 32, kThreads), kThreads, 0, st>>>(
      d_off, t->d_off64, t->n, t->d_table, t->bucket_num, t->bucket,
      d_cols_out);
  RST_CUDA(cudaGetLastError());
  return RESET_OK;
}

}  // extern "C"
