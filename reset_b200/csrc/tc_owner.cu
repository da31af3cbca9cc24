// Owner-grouped triangle counting: every probed table is read from HBM once,
// into shared memory, and the keys of all sets that probe it stream through.
//
// Same count as dynamic_triangle_count (triangle-count/TC.cu:128-190): for
// every oriented edge (u, v) the keys of the smaller row are looked up in the
// larger row's table (ties: u's keys in v's table, TC.cu:148-157) with the
// reference's bucket layout, hash and probe rule (search_in_hashtable,
// TC.cu:11-31), so rows with repeated entries give the reference's number.
//
// What changes is the order of the work.  Probing edge by edge costs every
// key a random 4-byte table read in HBM, which moves a whole 32-byte sector,
// from tables far larger than L2.  Here the edges are first grouped by the
// set whose table they probe -- its "owner", the larger row -- so
//   * each owner's table is read from HBM once per group;
//   * the keys of its probers (whole CSR rows) stream past it with 128-bit
//     loads; every lookup then reads shared memory only.
// HBM traffic per probe drops from ~4 B of key + a 32 B sector to ~4 B.
//
// The staged form of a table is not its copy: the set it holds is inserted
// into an open-addressing table of 8192 slots (1024 for a warp) with a
// multiplicative hash, whatever the reference table's load, bucket size and
// hash.  Almost every lookup is then settled by ONE shared memory read (a copy
// of the reference table takes two, and with 5-slot buckets one lookup in four
// goes further), and the count runs at the same speed for every table
// parameter.  Inserting is cheap: it reads the slots
// once, where a group's probers bring hundreds of keys per slot.
//
// Passes (all stream-ordered, no host synchronisation):
//   pad_rows_kernel     the key rows padded to whole 32-byte chunks (long ones
//                       by pad_long_kernel)
//   own_count_kernel    owner of every edge; probers per owner
//   CUB exclusive scan  group offsets
//   own_scatter_kernel  (first chunk, keys) of every edge's prober,
//                       grouped by owner
//   own_classify_kernel one of four bins per owner:
//     CTA    large groups (or sets above a warp's share of shared memory):
//            the whole CTA stages the set, its warps split the probers,
//            groups of more than kSeg probers are cut into several units;
//     warp   a warp stages the set in its own region and walks the probers;
//     large  sets above a CTA's share: one CTA per SM stages them in 32768
//            slots;
//     direct small groups, where staging costs more than it saves, and
//            sets too large for shared memory: probes go to the HBM table,
//            flattened across the lanes (thread granularity).
//   tc_owner_kernel     one persistent launch: CTA units, then direct units,
//                       warp owners and direct owners, each from its own work
//                       counter.
//   tc_owner_large_kernel  only for tables that have larger sets: large units,
//                       then the direct units of still larger ones.
//
// Bound by the shared-memory pipe: a lookup's slot read takes 3.1 wavefronts
// for 32 random banks, 25 of the ~40 wavefronts of a step of 256 keys, at
// 72% of the issue slots.  R-MAT scale 24, count call, ms: probing copies of
// the reference tables, two slot reads and a ballot per lookup, 124 (b = 1) /
// 144 (b = 5); one slot read in a set of its own 94; rows padded, keys
// mixed, rows followed without shuffles 85; rows in class order, one random
// read per edge in the grouping passes 73 (b = 1 and 5).
#include <cub/cub.cuh>

#include <algorithm>

#include "common.cuh"
#include "probe_common.cuh"
#include "staged.cuh"

namespace rst {
namespace {

// ------------------------------------------------------------- passes ----

// Keys in the count kernel's rows and staged sets are mixed: multiplied by an
// odd constant (Knuth's, from the golden ratio) modulo 2^31, a bijection of
// [0, 2^31), so the top bits of a mixed key are its hash and no multiply is
// left per lookup.  Vertex ids are < n <= 2^31 - 2 (checked on the host), so
// the images of the two largest values are free: kNoKey pads rows, kFree
// marks free slots.
__host__ __device__ constexpr int mix_key(int x) {
  return (int)(((unsigned)x * 0x9E3779B1u) & 0x7fffffffu);
}
__host__ __device__ constexpr int unmix_key(int y) {  // (the constant's inverse modulo 2^31)
  return (int)(((unsigned)y * 0xe8b2f51u) & 0x7fffffffu);
}
constexpr int kNoKey = mix_key(0x7fffffff), kFree = mix_key(0x7ffffffe);
static_assert(unmix_key(kNoKey) == 0x7fffffff && unmix_key(kFree) == 0x7ffffffe, "inverse");

// The padded rows for flat_probe: a row starts at a chunk, its keys are mixed.
struct PaddedRows {
  static __device__ __forceinline__ int key(const int32_t* rows, int chunk, int j) {
    return unmix_key(__ldg(rows + (int64_t)(unsigned)chunk * 8 + j));
  }
};

// Rows padded to whole chunks of 8 mixed keys (32 bytes, aligned): the count
// kernel then loads whole chunks without a thought for where a row starts or
// ends, which took a third of its instructions.
//
// Inside a row the keys are put in order of their vertex's class, one of
// kClasses by degree (in + out), cut so that each holds about as many keys.
// An owner's set has a lowest class, and a prober's keys below it cannot be in
// the set: the prober's row is read from the chunk where that class starts.
// With edges oriented low -> high by degree every key of w's row has at least
// w's class, so near half of a row that probes its edges' targets drops out;
// in any other graph, whatever the lowest classes show.
constexpr int kClasses = 24;
constexpr int kClassRow = 2040;  // longest row put in order (chunk places in a byte)
// Longer rows are padded by pad_long_kernel, in parts: 8 lanes take 7.6 ms for a
// row of 900,000 keys.  (Launched where the table may have such sets.)
constexpr int kPadPart = 8192;

// A key row's length and lowest class in one word, so that an edge costs one
// random read (of n words, in L2) for its target; rows of kLongRow keys or
// more keep their length in koff.
constexpr int kLongRow = (1 << 27) - 1;
__device__ __forceinline__ int row_len(unsigned info, const int32_t* __restrict__ koff, int u) {
  const int d = (int)(info & kLongRow);
  return d < kLongRow ? d : __ldg(koff + u + 1) - __ldg(koff + u);
}

// Chunk (of the row) to read from when classes below c are not wanted.
struct __align__(8) ClassPlaces {
  uint8_t at[kClasses];
};

__global__ void __launch_bounds__(kOT)
    key_count_kernel(const int32_t* __restrict__ kcols, int64_t mk, int32_t n,
                     int32_t* __restrict__ indeg) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mk;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int x = __ldg(kcols + i);
    if ((unsigned)x < (unsigned)n) atomicAdd(indeg + x, 1);
  }
}

// Degrees in steps of 1/8 octave.
constexpr int kDegSteps = 256;
__device__ __forceinline__ int deg_step(int deg) {
  return deg < 1 ? 0 : min(kDegSteps - 1, (int)(__float_as_uint((float)deg) >> 20) - (127 << 3));
}

// Keys by the degree step of their vertex.
__global__ void __launch_bounds__(kOT)
    degree_hist_kernel(const int32_t* __restrict__ koff, const int32_t* __restrict__ indeg,
                       int32_t n, unsigned* __restrict__ hist) {
  __shared__ unsigned s_h[kDegSteps];
  for (int i = threadIdx.x; i < kDegSteps; i += kOT) s_h[i] = 0;
  __syncthreads();
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n;
       u += (int64_t)gridDim.x * blockDim.x) {
    const int in = indeg[u];
    if (in > 0) atomicAdd(&s_h[deg_step(in + __ldg(koff + u + 1) - __ldg(koff + u))], (unsigned)in);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kDegSteps; i += kOT)
    if (s_h[i]) atomicAdd(hist + i, s_h[i]);
}

// Class of every vertex: degree steps cut into kClasses of about as many keys.
__global__ void __launch_bounds__(kOT)
    class_kernel(const int32_t* __restrict__ koff, const int32_t* __restrict__ indeg, int32_t n,
                 const unsigned* __restrict__ hist, uint8_t* __restrict__ cls) {
  __shared__ uint8_t s_c[kDegSteps];
  if (threadIdx.x < 32) {  // a lane per 8 steps
    constexpr int kPer = kDegSteps / 32;
    unsigned h[kPer];
    int sum = 0, total;
    for (int i = 0; i < kPer; ++i) sum += (int)(h[i] = hist[threadIdx.x * kPer + i]);
    unsigned before = (unsigned)warp_excl_scan(sum, &total);
    for (int i = 0; i < kPer; ++i) {
      const unsigned mid = before + h[i] / 2;
      s_c[threadIdx.x * kPer + i] =
          (uint8_t)min((unsigned long long)kClasses - 1,
                       (unsigned long long)mid * kClasses / (unsigned)max(total, 1));
      before += h[i];
    }
  }
  __syncthreads();
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n;
       u += (int64_t)gridDim.x * blockDim.x)
    cls[u] = s_c[deg_step(indeg[u] + __ldg(koff + u + 1) - __ldg(koff + u))];
}

// The first chunk of the padded row u of n, whose keys start at s of mk: a
// chunk per 8 keys and one more per row is room enough, or, in fewer chunks
// where rows have hardly a key each, a chunk per key.  So no scan over the
// rows is needed (three launches, 12 of 264 us at scale 16), and the rows take
// no more memory than packed ones and the scan's result.
__host__ __device__ __forceinline__ int64_t padded_chunks(int64_t n, int64_t mk) {
  return mk / 8 + n < mk ? mk / 8 + n : mk;
}
__device__ __forceinline__ unsigned first_chunk(int s, int u, int64_t n, int64_t mk) {
  const unsigned at = (unsigned)min((int64_t)max(s, 0), mk);
  return mk / 8 + n < mk ? (at >> 3) + (unsigned)u : at;
}

// The padded rows, 8 lanes to a row, in class order with their lowest class
// and class places (cls NULL: in the order they come); a chunk without keys at
// `none`.
__global__ void __launch_bounds__(kOT)
    pad_rows_kernel(const int32_t* __restrict__ koff, const int32_t* __restrict__ kcols,
                    int32_t n, int64_t mk, const uint8_t* __restrict__ cls,
                    int32_t* __restrict__ padded, int32_t* __restrict__ none,
                    unsigned* __restrict__ info, ClassPlaces* __restrict__ places,
                    int2* __restrict__ parts, int max_parts, int* __restrict__ n_parts) {
  __shared__ int s_cnt[kOT / 8][kClasses];
  constexpr int kPer = kClasses / 8;  // classes a lane looks after
  constexpr int kHold = 6;
  const int l8 = threadIdx.x & 7;
  const unsigned group = 0xffu << (threadIdx.x & 24);
  int* cnt = s_cnt[threadIdx.x >> 3];
  const int64_t step = ((int64_t)gridDim.x * blockDim.x) >> 3;
  if (blockIdx.x == 0 && threadIdx.x < 8) none[threadIdx.x] = kNoKey;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3; u < n; u += step) {
    const int s = max(__ldg(koff + u), 0);
    const int d = (int)min((int64_t)(__ldg(koff + u + 1) - s), mk - s);
    int32_t* out = padded + (int64_t)first_chunk(s, (int)u, n, mk) * 8;
    int place[kPer];
    int lowest = 0;
    for (int i = 0; i < kPer; ++i) place[i] = 0;
    if (cls && d > 8 && d <= kClassRow) {
      for (int i = 0; i < kPer; ++i) cnt[l8 * kPer + i] = 0;
      __syncwarp(group);
      // a lane's first kHold keys and classes stay in registers
      int x[kHold], c[kHold];
#pragma unroll
      for (int i = 0; i < kHold; ++i) x[i] = l8 + 8 * i < d ? __ldg(kcols + s + l8 + 8 * i) : -1;
#pragma unroll
      for (int i = 0; i < kHold; ++i) c[i] = (unsigned)x[i] < (unsigned)n ? __ldg(cls + x[i]) : 0;
#pragma unroll
      for (int i = 0; i < kHold; ++i)
        if (l8 + 8 * i < d) atomicAdd(cnt + c[i], 1);
#pragma unroll 4
      for (int j = l8 + 8 * kHold; j < d; j += 8) {
        const int z = __ldg(kcols + s + j);
        atomicAdd(cnt + ((unsigned)z < (unsigned)n ? __ldg(cls + z) : 0), 1);
      }
      __syncwarp(group);
      int sum = 0, mine = kClasses;
      for (int i = kPer - 1; i >= 0; --i) {
        place[i] = cnt[l8 * kPer + i];
        sum += place[i];
        if (place[i]) mine = l8 * kPer + i;
      }
      int before = sum;  // keys in lower lanes' classes
      for (int o = 1; o < 8; o <<= 1) {
        const int t = __shfl_up_sync(group, before, o, 8);
        if (l8 >= o) before += t;
      }
      before -= sum;
      for (int o = 1; o < 8; o <<= 1) mine = min(mine, __shfl_xor_sync(group, mine, o, 8));
      lowest = mine;
      for (int i = 0; i < kPer; ++i) {
        const int k = place[i];
        cnt[l8 * kPer + i] = before;
        place[i] = before >> 3;
        before += k;
      }
      __syncwarp(group);
#pragma unroll
      for (int i = 0; i < kHold; ++i)
        if (l8 + 8 * i < d) out[atomicAdd(cnt + c[i], 1)] = mix_key(x[i]);
#pragma unroll 4
      for (int j = l8 + 8 * kHold; j < d; j += 8) {
        const int z = __ldg(kcols + s + j);
        out[atomicAdd(cnt + ((unsigned)z < (unsigned)n ? __ldg(cls + z) : 0), 1)] = mix_key(z);
      }
      __syncwarp(group);
    } else {
      int at = max_parts;
      const int np = (d + kPadPart - 1) / kPadPart;
      if (d > kClassRow && max_parts > 0) {
        if (l8 == 0) at = atomicAdd(n_parts, np);
        at = __shfl_sync(group, at, 0, 8);
      }
      if (at <= max_parts - np) {  // left to pad_long_kernel
        for (int i = l8; i < np; i += 8) parts[at + i] = make_int2((int)u, i * kPadPart);
      } else {
        if (at < max_parts) {  // (places it took without filling them)
          for (int i = at + l8; i < max_parts; i += 8) parts[i] = make_int2(-1, 0);
        }
        for (int j = l8; j < d; j += 8) out[j] = mix_key(__ldg(kcols + s + j));
      }
    }
    const int pad = d + l8;
    if (d > 0 && pad < ((d + 7) & ~7)) out[pad] = kNoKey;
    if (cls)
      for (int i = 0; i < kPer; ++i) places[u].at[l8 * kPer + i] = (uint8_t)place[i];
    if (l8 == 0) info[u] = (unsigned)min(max(d, 0), kLongRow) | (unsigned)lowest << 27;
  }
}

// The long rows, a CTA per kPadPart keys.
__global__ void __launch_bounds__(kOT)
    pad_long_kernel(const int32_t* __restrict__ koff, const int32_t* __restrict__ kcols, int32_t n,
                    int64_t mk, const int2* __restrict__ parts, int max_parts,
                    const int* __restrict__ n_parts, int32_t* __restrict__ padded) {
  const int np = min(*n_parts, max_parts);
  for (int i = blockIdx.x; i < np; i += gridDim.x) {
    const int2 part = __ldg(parts + i);
    if (part.x < 0) continue;
    const int s = max(__ldg(koff + part.x), 0);
    const int d = (int)min((int64_t)(__ldg(koff + part.x + 1) - s), mk - s);
    int32_t* out = padded + (int64_t)first_chunk(s, part.x, n, mk) * 8;
    const int end = min(d, part.y + kPadPart);
#pragma unroll 4
    for (int j = part.y + threadIdx.x; j < end; j += kOT) out[j] = mix_key(__ldg(kcols + s + j));
  }
}

// Owners of 32 * kIlp consecutive edges of the edge CSR, kIlp a lane, from
// edge 32 * c on: v of edge (u, v) unless u's key row is longer
// (TC.cu:148-157); the prober is the other end.  Rows come from the key CSR,
// which for plain triangle counting is the edge CSR itself and for an element
// shard its filtered rows.  owner < 0: past the end, or a bad id.
constexpr int kIlp = 4;
struct EdgeOwners {
  int owner[kIlp], prober[kIlp], len[kIlp], low[kIlp];
};

__device__ __forceinline__ EdgeOwners edge_owners(const int32_t* __restrict__ eoff,
                                                  const int32_t* __restrict__ ecols,
                                                  const int32_t* __restrict__ chunk_row,
                                                  const int32_t* __restrict__ koff,
                                                  const unsigned* __restrict__ info, int n,
                                                  int64_t me, int64_t c, int32_t* status) {
  const int lane = threadIdx.x & 31;
  const int64_t n_chunks = (me + 31) >> 5;
  int u[kIlp], v[kIlp];
  bool valid[kIlp];
#pragma unroll
  for (int i = 0; i < kIlp; ++i) {
    const int64_t e = (c + i) * 32 + lane;
    valid[i] = e < me;
    v[i] = __ldg(ecols + (valid[i] ? e : me - 1));
  }
#pragma unroll
  for (int i = 0; i < kIlp; ++i) {
    int u0 = __ldg(chunk_row + min(c + i, n_chunks - 1));
    if ((unsigned)u0 >= (unsigned)n) u0 = 0;
    u[i] = row_of_edge(eoff, n, u0, (int)min((c + i) * 32 + lane, me - 1));
  }
  EdgeOwners r;
  unsigned iu[kIlp], iv[kIlp];
#pragma unroll
  for (int i = 0; i < kIlp; ++i) {
    if (valid[i] && ((unsigned)u[i] >= (unsigned)n || (unsigned)v[i] >= (unsigned)n)) {
      atomicOr(status, kErrBadId);
      valid[i] = false;
    }
    if (!valid[i]) u[i] = v[i] = 0;
    iu[i] = __ldg(info + u[i]);
    iv[i] = __ldg(info + v[i]);
  }
#pragma unroll
  for (int i = 0; i < kIlp; ++i) {
    const int du = row_len(iu[i], koff, u[i]), dv = row_len(iv[i], koff, v[i]);
    const bool own_u = du > dv;
    r.owner[i] = !valid[i] ? -1 : own_u ? u[i] : v[i];
    r.prober[i] = own_u ? v[i] : u[i];
    r.len[i] = own_u ? dv : du;
    r.low[i] = (int)((own_u ? iu[i] : iv[i]) >> 27);
  }
  return r;
}

__global__ void __launch_bounds__(kOT)
    own_count_kernel(const int32_t* __restrict__ eoff, const int32_t* __restrict__ ecols,
                     const int32_t* __restrict__ chunk_row, const int32_t* __restrict__ koff,
                     const unsigned* __restrict__ info, int32_t n, int64_t m,
                     int32_t* __restrict__ cnt, int32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t me = min(m, (int64_t)__ldg(eoff + n));
  const int64_t n_chunks = (me + 31) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * kIlp; c < n_chunks;
       c += nw * kIlp) {
    const EdgeOwners eo = edge_owners(eoff, ecols, chunk_row, koff, info, n, me, c, status);
#pragma unroll
    for (int i = 0; i < kIlp; ++i) {
      const unsigned grp = __match_any_sync(kFull, eo.owner[i]);
      if (eo.owner[i] >= 0 && lane == __ffs(grp) - 1) atomicAdd(cnt + eo.owner[i], __popc(grp));
    }
  }
}

// ent: a prober's row is read from its owner's lowest class on (places NULL:
// all of it).  left[w] starts at the end of w's group and counts down.
__global__ void __launch_bounds__(kOT)
    own_scatter_kernel(const int32_t* __restrict__ eoff, const int32_t* __restrict__ ecols,
                       const int32_t* __restrict__ chunk_row, const int32_t* __restrict__ koff,
                       const unsigned* __restrict__ info, int32_t n, int64_t m,
                       int64_t mk,
                       const ClassPlaces* __restrict__ places, int32_t* __restrict__ left,
                       int2* __restrict__ ent, int32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t me = min(m, (int64_t)__ldg(eoff + n));
  const int64_t n_chunks = (me + 31) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * kIlp; c < n_chunks;
       c += nw * kIlp) {
    const EdgeOwners eo = edge_owners(eoff, ecols, chunk_row, koff, info, n, me, c, status);
    unsigned grp[kIlp];
    int top[kIlp];
    int2 row[kIlp];
#pragma unroll
    for (int i = 0; i < kIlp; ++i) {
      grp[i] = __match_any_sync(kFull, eo.owner[i]);
      top[i] = 0;
      if (eo.owner[i] >= 0 && lane == __ffs(grp[i]) - 1)
        top[i] = atomicSub(left + eo.owner[i], __popc(grp[i]));
    }
#pragma unroll
    for (int i = 0; i < kIlp; ++i) {
      const bool ok = eo.owner[i] >= 0;
      row[i] = make_int2(
          ok ? (int)first_chunk(__ldg(koff + eo.prober[i]), eo.prober[i], n, mk) : 0, eo.len[i]);
      const int from = ok && eo.low[i] ? __ldg(&places[eo.prober[i]].at[eo.low[i]]) : 0;
      row[i].x += from;
      row[i].y -= 8 * from;
    }
#pragma unroll
    for (int i = 0; i < kIlp; ++i) {
      const int t = __shfl_sync(kFull, top[i], __ffs(grp[i]) - 1);
      if (eo.owner[i] >= 0)
        ent[t - __popc(grp[i]) + __popc(grp[i] & lanemask_lt())] = row[i];
    }
  }
}

// Launch shape and bins of the count kernel.  CTAs of 256 threads with a
// 32 KB table, five to an SM: while one CTA stages or waits for its last
// warp, four others stream.
constexpr int kTT = 256;          // threads per CTA
constexpr int kTW = kTT / 32;     // warps per CTA
constexpr int kTab = 8192;        // slots of a CTA's staged table
constexpr int kWTab = kTab / kTW;  // ... of a warp's
constexpr int kSeg = 512;         // probers per CTA unit
constexpr int kRing = 64;         // rows a warp holds
constexpr int kTake = 16;         // ... and takes at a time from a CTA unit
constexpr int kQueueLane = 8;     // lookups a lane may have to walk on before all do
constexpr int kCtaProbers = 128;  // groups above this, or with this many keys
constexpr int kCtaKeys = 8192;    // to look up, are CTA work
static_assert((kWTab & (kWTab - 1)) == 0 && kTake <= 32 && kRing >= 64, "staged table shapes");

// Sets of more than kTab / 2 keys, by a launch of its own: one CTA of 1024
// threads per SM with a table of 128 KB, up to 5/8 full (the reference's tables
// of up to 20480 slots, at any load).  The direct units of larger sets are in
// this launch too: they read HBM tables through L1, of which tc_owner_kernel's
// five tables leave nothing.  500 rows of 8000 keys among 20,000 vertices, ms a
// count, probing HBM tables in tc_owner_kernel / this way: alpha 0.5, 4 slots
// 53 / 3.3 (staged whole with 20480 slots, 4.7); alpha 0.2, 5 slots 32 / 3.4.
constexpr int kLT = 1024;
constexpr int kLW = kLT / 32;
constexpr int kLTab = 32768;
constexpr int kLargeKeys = 20480;
constexpr int kLSeg = 2048;  // probers per large unit
constexpr int kLDirSeg = 16;  // ... per direct unit: 32 rows of 30,000 keys held one warp 7 ms
constexpr size_t kLargeSmem = sizeof(int) * (kLTab + kLW * 32 * kQueueLane) + 8 * kLW * kRing;

// Lists of the bins, and the counters in ctr: entries, then the cursors.
enum : int {
  kCtrUnits = 0, kCtrWarp = 1, kCtrDirect = 2, kCtrDirectUnits = 6,
  kCtrUnitsNext = 3, kCtrWarpNext = 4, kCtrDirectNext = 5, kCtrDirectUnitsNext = 7,
  kCtrLarge = 8, kCtrLargeDirect = 9, kCtrLargeNext = 10, kCtrLargeDirectNext = 11,
  kCtrPadParts = 12, kCtrs = 13
};

// Bin of every owner with a non-empty group (see the file comment).  The lists
// of the large launch grow from the ends of the other launch's: an owner is in
// one bin, so they do not meet.
__global__ void __launch_bounds__(kOT)
    own_classify_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ goff,
                        const int2* __restrict__ ent, int32_t n, int b, float alpha,
                        int2* __restrict__ units, int32_t* __restrict__ wlist,
                        int32_t* __restrict__ dlist, int2* __restrict__ dunits,
                        int2* __restrict__ units_last, int2* __restrict__ dunits_last,
                        int32_t* __restrict__ ctr) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < n; base += stride) {
    const int64_t w = base + threadIdx.x;
    int bin = -1, nunits = 0;
    if (w < n) {
      const int g0 = __ldg(goff + w), P = __ldg(goff + w + 1) - g0;
      if (P > 0) {
        const int4 d = __ldg(desc + w);
        const int64_t T = (int64_t)b << desc_lg(d);  // table ints
        const float keys = alpha * (float)T;  // the set has at most this many, + 1
        bool big = P > kCtaProbers;
        int64_t work = 0;
        if (!big) {
          for (int i = 0; i < P; ++i) work += __ldg(&ent[g0 + i].y);
          big = work >= kCtaKeys;
        }
        // staging pays when there are at most ~4 slots to insert per lookup;
        // a CTA's staged table is at most half full, and probing rows (no
        // longer than the owner's) of 2^20 keys keep a unit's quads within 32
        // bits
        const bool small = keys <= kTab / 2;
        if ((!small && keys > kLargeKeys) || d.y > (1 << 20) ||
            !(P > kCtaProbers || T <= 4 * work)) {
          bin = P <= 32 ? 2 : small ? 3 : 5;
          const int seg = bin == 5 ? kLDirSeg : kDirSeg;
          if (bin != 2) nunits = (P + seg - 1) / seg;
        } else if (!small) {
          bin = 4;
          nunits = (P + kLSeg - 1) / kLSeg;
        } else if (big || keys > kWTab / 4) {
          bin = 0;
          nunits = (P + kSeg - 1) / kSeg;
        } else {
          bin = 1;
        }
      }
    }
    // warp-aggregated appends
    auto append = [&](int which, int at, int2* list, int step) {
      int tot;
      const int pre = warp_excl_scan(bin == which ? nunits : 0, &tot);
      int b0 = 0;
      if (lane == 0 && tot) b0 = atomicAdd(ctr + at, tot);
      b0 = __shfl_sync(kFull, b0, 0);
      // (a hub's many units by all lanes)
      const int mine = bin == which ? nunits : 0;
      if (mine <= 32)
        for (int s = 0; s < mine; ++s) list[step * (b0 + pre + s)] = make_int2((int)w, s);
      for (unsigned wide = __ballot_sync(kFull, mine > 32); wide; wide &= wide - 1) {
        const int k = __ffs(wide) - 1;
        const int hub = __shfl_sync(kFull, (int)w, k), from = __shfl_sync(kFull, b0 + pre, k);
        const int ns = __shfl_sync(kFull, mine, k);
        for (int s = lane; s < ns; s += 32) list[step * (from + s)] = make_int2(hub, s);
      }
    };
    append(0, kCtrUnits, units, 1);
    append(3, kCtrDirectUnits, dunits, 1);
    if (__any_sync(kFull, bin >= 4)) {
      append(4, kCtrLarge, units_last, -1);
      append(5, kCtrLargeDirect, dunits_last, -1);
    }
#pragma unroll
    for (int which = 1; which <= 2; ++which) {
      const unsigned bm = __ballot_sync(kFull, bin == which);
      int b0 = 0;
      if (lane == 0 && bm) b0 = atomicAdd(ctr + (which == 1 ? kCtrWarp : kCtrDirect), __popc(bm));
      b0 = __shfl_sync(kFull, b0, 0);
      if (bin == which) (which == 1 ? wlist : dlist)[b0 + __popc(bm & lanemask_lt())] = (int)w;
    }
  }
}

// A staged set: 1 << LG slots at shared-memory ints S, linear probing from a
// mixed key's top bits.  A slot is kFree or a mixed key, whose sign bit is set
// once a later key with that HOME slot had to go further.  So a lookup that
// meets another key without the bit has missed: at 1 key per 32 slots, 3% of
// the lookups meet another key but only 1 in 2000 of those that miss, and
// the 1.5% of the keys that went further, have to walk on.
template <int LG>
struct Staged {
  int* S;
  static __device__ __forceinline__ unsigned home(int y) { return (unsigned)y >> (31 - LG); }
  static __device__ __forceinline__ unsigned next(unsigned h) {
    return (h + 1) & ((1u << LG) - 1u);
  }
  static __device__ __forceinline__ int key(int s) { return s & 0x7fffffff; }
  // (ends: the table is at most 5/8 full)
  __device__ __forceinline__ void insert(int y) const {
    unsigned h = home(y);
    int old = atomicCAS(S + h, kFree, y);
    if (old == kFree || key(old) == y) return;
    atomicOr(S + h, 0x80000000);
    do {
      h = next(h);
      old = atomicCAS(S + h, kFree, y);
    } while (old != kFree && key(old) != y);
  }
  // y in the set, given that its home slot holds another key with the bit set
  __device__ __forceinline__ bool walk(int y) const {
    for (unsigned h = next(home(y));; h = next(h)) {
      const int s = key(S[h]);
      if (s == y) return true;
      if (s == kFree) return false;
    }
  }
};

// Clears the staged table and inserts the keys of the set's table (b planes
// of 1 << lg slots, plane k at table + toff + k*bn; 16-byte aligned).  sync
// separates the two steps and publishes the table.
template <int LG, class Sync>
__device__ __forceinline__ void stage_set(const Staged<LG>& st, const int32_t* __restrict__ table,
                                          int64_t toff, int lg, int64_t bn, int b, int t, int nt,
                                          Sync sync) {
  const int4 free4 = make_int4(kFree, kFree, kFree, kFree);
  int4* S4 = reinterpret_cast<int4*>(st.S);
  for (int i = t; i < (1 << LG) / 4; i += nt) S4[i] = free4;
  sync();
  const int q = 1 << (lg - 2);  // 16-byte groups of a plane
  for (int k = 0; k < b; ++k) {
    const int4* P = reinterpret_cast<const int4*>(table + toff + k * bn);
    for (int i = t; i < q; i += nt) {
      const int4 v = __ldg(P + i);
      if (v.x != -1) st.insert(mix_key(v.x));
      if (v.y != -1) st.insert(mix_key(v.y));
      if (v.z != -1) st.insert(mix_key(v.z));
      if (v.w != -1) st.insert(mix_key(v.w));
    }
  }
  sync();
}

// y[j], without an indexed register array.
__device__ __forceinline__ int pick8(const int (&y)[8], int j) {
  const int p0 = j & 1 ? y[1] : y[0], p1 = j & 1 ? y[3] : y[2];
  const int p2 = j & 1 ? y[5] : y[4], p3 = j & 1 ? y[7] : y[6];
  const int q0 = j & 2 ? p1 : p0, q1 = j & 2 ? p3 : p2;
  return j & 4 ? q1 : q0;
}

// A lane's lookups that must walk on: its own column of a shared-memory
// queue of kQueueLane rows.
struct OpenQueue {
  int* q;     // this lane's column
  int n = 0;  // its entries
  __device__ __forceinline__ void push(const int (&y)[8], int j) { q[n++ * 32] = pick8(y, j); }
  template <int LG>
  __device__ __forceinline__ unsigned drain(const Staged<LG>& st) {
    unsigned hits = 0;
    for (; n > 0; --n) hits += st.walk(q[(n - 1) * 32]);
    __syncwarp();
    return hits;
  }
};

// A row of the warp's ring: the rows' chunks are numbered one after the
// other; this row's end there, and what leads from a number to the chunk.
struct RingRow {
  unsigned end, at;
};

// The keys of probing rows ({first chunk, keys} in the padded rows) looked up
// in a staged set.  The rows' chunks of 8 keys are flattened across the
// lanes, without a gap from row to row: lane i of a step finds chunk base + i,
// following the rows in the warp's ring in shared memory with an index of its
// own; two lanes then share a chunk, so that each of the two loads reads 512
// consecutive bytes (of a long row) and not every other 16, and each key reads
// one slot.  Shuffles (a binary search over the rows) and predicated stores
// cost the shared-memory pipe as much as a load each, so there are two
// shuffles and no store in a step: the lookups that must walk on are noted in
// a bit mask, and queued after the step if there are any.
// none: a chunk of kNoKey.  grab(): the next rows of the caller's,
// ent[x .. x + y), y <= 32 (warp-uniform; y = 0: no more).  Returns this
// lane's hits.
template <int LG, class Grab>
__device__ __forceinline__ unsigned stream_rows(const int2* __restrict__ ent, Grab grab,
                                                const int4* __restrict__ quads, unsigned none,
                                                const Staged<LG>& st, OpenQueue& open,
                                                RingRow* ring) {
  const int lane = threadIdx.x & 31;
  unsigned hits = 0;
  unsigned base = 0, run = 0;  // chunks taken, chunks in the ring
  int have = 0;                // rows put into the ring
  bool more = true;
  int k = -1;  // this lane's row
  RingRow row{0, 0};
  for (;;) {
    while (more && run < base + 32 && have - __shfl_sync(kFull, k, 0) <= kRing - 32) {
      const int2 g = grab();
      more = g.y > 0;
      const int2 e = lane < g.y ? __ldg(ent + g.x + lane) : make_int2(0, 0);
      const unsigned nc = (unsigned)(max(e.y, 0) + 7) >> 3;
      const unsigned kept = __ballot_sync(kFull, nc > 0);
      int total;
      const unsigned start = run + (unsigned)warp_excl_scan((int)nc, &total);
      if (nc > 0)
        ring[(have + __popc(kept & lanemask_lt())) & (kRing - 1)] =
            RingRow{start + nc, (unsigned)e.x - start};
      have += __popc(kept);
      run += (unsigned)total;
      __syncwarp();
    }
    if (run == base) break;
    const unsigned end = min(base + 32, run);
    const unsigned f = base + lane;
    // (lanes past the last chunk follow too: lane 0's row stays the earliest
    // that any lane has yet to leave)
    while (f >= row.end && k + 1 < have) row = ring[++k & (kRing - 1)];
    const unsigned c = f < end ? row.at + f : none;
    base = end;
    const unsigned c0 = __shfl_sync(kFull, c, lane >> 1);
    const unsigned c1 = __shfl_sync(kFull, c, 16 + (lane >> 1));
    const int4 a = __ldg(quads + (2 * (size_t)c0 + (lane & 1)));
    const int4 b = __ldg(quads + (2 * (size_t)c1 + (lane & 1)));
    const int y[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    int s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = st.S[st.home(y[j])];
    unsigned todo = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const bool hit = st.key(s[j]) == y[j];
      if (hit) ++hits;
      if (!hit && s[j] < 0) todo |= 1u << j;
    }
    if (todo) {
      open.push(y, __ffs(todo) - 1);
      todo &= todo - 1;
      if (todo) {
        open.push(y, __ffs(todo) - 1);
        // more than two of a lane's eight: rare, walked at once
        while (todo &= todo - 1) hits += st.walk(pick8(y, __ffs(todo) - 1));
      }
    }
    if (__any_sync(kFull, open.n > kQueueLane - 2)) hits += open.drain(st);
  }
  return hits;
}

// This warp's `hits` credited to owner w (OWN; warp-collective).
template <bool OWN>
__device__ __forceinline__ void credit(unsigned long long* owner_hits, int w,
                                       unsigned long long hits) {
  if (OWN) {
    const unsigned long long d = warp_sum_u64(hits);
    if ((threadIdx.x & 31) == 0 && d) atomicAdd(owner_hits + w, d);
  }
}

// CTA units: the whole CTA (NT threads) stages one set, its warps share the
// SEG probers of a unit; unit i at units[STEP * i].  Returns this lane's hits.
template <int LG, int NT, int SEG, int STEP, bool OWN>
__device__ __forceinline__ unsigned long long cta_units(
    const Staged<LG>& st, const int4* __restrict__ desc, const int32_t* __restrict__ goff,
    const int2* __restrict__ ent, const int4* __restrict__ quads, unsigned none,
    const int2* __restrict__ units, int n_units, int32_t* __restrict__ cursor,
    const int32_t* __restrict__ table, int64_t bn, int b, OpenQueue& open, RingRow* ring,
    unsigned long long* __restrict__ owner_hits) {
  __shared__ int s_item, s_next;
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned long long hits = 0;
  for (;;) {
    if (tid == 0) {
      s_item = atomicAdd(cursor, 1);
      s_next = 0;
    }
    __syncthreads();
    const int ui = s_item;
    if (ui >= n_units) break;
    const int2 unit = __ldg(units + STEP * ui);
    const int4 dw = __ldg(desc + unit.x);
    stage_set(st, table, desc_toff(dw), desc_lg(dw), bn, b, tid, NT, [] { __syncthreads(); });
    const int g0 = __ldg(goff + unit.x) + unit.y * SEG;
    const int g1 = min(__ldg(goff + unit.x + 1), g0 + SEG);
    unsigned long long h = stream_rows(
        ent,
        [&] {
          int g = 0;
          if (lane == 0) g = g0 + atomicAdd(&s_next, kTake);
          g = __shfl_sync(kFull, g, 0);
          return make_int2(g, max(0, min(kTake, g1 - g)));
        },
        quads, none, st, open, ring);
    h += open.drain(st);
    credit<OWN>(owner_hits, unit.x, h);
    hits += h;
    __syncthreads();
  }
  return hits;
}

// Direct units: up to SEG probers of one owner whose table stays in HBM, 32
// probers at a time, their probes flattened across the lanes; unit i at
// dunits[STEP * i].
template <bool HIER, int SEG, int STEP, bool OWN>
__device__ __forceinline__ unsigned long long direct_units(
    const int4* __restrict__ desc, const int32_t* __restrict__ goff, const int2* __restrict__ ent,
    const int32_t* __restrict__ rows, const int2* __restrict__ dunits, int n_dunits,
    int32_t* __restrict__ cursor, const int32_t* __restrict__ table, int64_t bn, int b, int lg_max,
    unsigned long long* __restrict__ owner_hits, int32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  unsigned long long hits = 0;
  for (;;) {
    int ui = 0;
    if (lane == 0) ui = atomicAdd(cursor, 1);
    ui = __shfl_sync(kFull, ui, 0);
    if (ui >= n_dunits) break;
    const int2 unit = __ldg(dunits + STEP * ui);
    const int4 dw = __ldg(desc + unit.x);
    const int g0 = __ldg(goff + unit.x) + unit.y * SEG;
    const int g1 = min(__ldg(goff + unit.x + 1), g0 + SEG);
    unsigned long long h = 0;
    for (int g = g0; g < g1; g += 32) {
      const int2 e = g + lane < g1 ? __ldg(ent + g + lane) : make_int2(0, 0);
      h += flat_probe<HIER, PaddedRows>(rows, table, e.y, e.x, desc_toff(dw), desc_lg(dw), lg_max,
                                        bn, b, status, [](int) {});
    }
    credit<OWN>(owner_hits, unit.x, h);
    hits += h;
  }
  return hits;
}

// OWN: every owner's hits are also added to owner_hits[owner] (per-graph
// counts of a batch of disjoint graphs are sums over their vertex ranges).
template <bool HIER, bool OWN = false>
__global__ void __launch_bounds__(kTT, 5)
    tc_owner_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ goff,
                    const int2* __restrict__ ent, const int32_t* __restrict__ rows,
                    unsigned none, const int2* __restrict__ units, const int32_t* __restrict__ wlist,
                    const int32_t* __restrict__ dlist, const int2* __restrict__ dunits,
                    int32_t* __restrict__ ctr,
                    const int32_t* __restrict__ table, int64_t bn, int b, int lg_max,
                    unsigned long long* __restrict__ count,
                    unsigned long long* __restrict__ owner_hits, int32_t* __restrict__ status) {
  extern __shared__ __align__(128) int sm[];  // the CTA's staged table or the warps', queues, rings
  constexpr int kLgTab = 31 - __builtin_clz(kTab), kLgWTab = 31 - __builtin_clz(kWTab);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int4* quads = reinterpret_cast<const int4*>(rows);
  int* queue = sm + kTab + warp * 32 * kQueueLane;
  RingRow* ring = reinterpret_cast<RingRow*>(sm + kTab + kTW * 32 * kQueueLane) + warp * kRing;
  OpenQueue open{queue + lane};
  const int n_warp = ctr[kCtrWarp], n_direct = ctr[kCtrDirect];
  unsigned long long hits =
      cta_units<kLgTab, kTT, kSeg, 1, OWN>(Staged<kLgTab>{sm}, desc, goff, ent, quads, none, units,
                                        ctr[kCtrUnits], ctr + kCtrUnitsNext, table, bn, b, open,
                                        ring, owner_hits);
  hits += direct_units<HIER, kDirSeg, 1, OWN>(desc, goff, ent, rows, dunits, ctr[kCtrDirectUnits],
                                  ctr + kCtrDirectUnitsNext, table, bn, b, lg_max, owner_hits,
                                  status);

  // ---- warp owners: each warp stages a set in its own region
  for (;;) {
    int wi = 0;
    if (lane == 0) wi = atomicAdd(ctr + kCtrWarpNext, 1);
    wi = __shfl_sync(kFull, wi, 0);
    if (wi >= n_warp) break;
    const int w = __ldg(wlist + wi);
    const int4 dw = __ldg(desc + w);
    const int lg = desc_lg(dw);
    const Staged<kLgWTab> st{sm + warp * kWTab};
    stage_set(st, table, desc_toff(dw), lg, bn, b, lane, 32, [] { __syncwarp(); });
    const int g0 = __ldg(goff + w), g1 = __ldg(goff + w + 1);
    int g = g0;
    unsigned long long h = stream_rows(
        ent,
        [&] {
          const int2 r = make_int2(g, min(32, g1 - g));
          g += r.y;
          return r;
        },
        quads, none, st, open, ring);
    h += open.drain(st);
    credit<OWN>(owner_hits, w, h);
    hits += h;
  }

  // ---- direct owners: 32 owners per warp, their (owner, prober) pairs
  // flattened across the lanes, probes into the HBM tables flattened again
  for (;;) {
    int ci = 0;
    if (lane == 0) ci = atomicAdd(ctr + kCtrDirectNext, 1);
    ci = __shfl_sync(kFull, ci, 0);
    const int64_t i = (int64_t)ci * 32 + lane;
    if ((int64_t)ci * 32 >= n_direct) break;
    int g0 = 0, P = 0, lg = 3, w = 0;
    int64_t toff = 0;
    if (i < n_direct) {
      w = __ldg(dlist + i);
      const int4 dw = __ldg(desc + w);
      g0 = __ldg(goff + w);
      P = __ldg(goff + w + 1) - g0;
      lg = desc_lg(dw);
      toff = desc_toff(dw);
    }
    int TP;
    const int Q = warp_excl_scan(P, &TP);
    // OWN: the queue (idle in this phase) holds, per pair lane, its owner
    // lane and, per owner lane, its hits
    int* pair_owner = queue;
    int* own_hits = pair_owner + 32;
    if (OWN) own_hits[lane] = 0;
    for (int base = 0; base < TP; base += 32) {
      const int f = base + lane;
      const int k = owner_lane(Q, f);
      const int kq = __shfl_sync(kFull, Q, k);
      const int kg = __shfl_sync(kFull, g0, k);
      const int klg = __shfl_sync(kFull, lg, k);
      const int64_t kt = __shfl_sync(kFull, toff, k);
      const int2 e = f < TP ? __ldg(ent + kg + (f - kq)) : make_int2(0, 0);
      if (OWN) {
        pair_owner[lane] = k;
        __syncwarp();
      }
      hits += flat_probe<HIER, PaddedRows>(rows, table, e.y, e.x, kt, klg, lg_max, bn, b, status,
                               [&](int kk) {
                                 if (OWN) atomicAdd(own_hits + pair_owner[kk], 1);
                               });
      if (OWN) __syncwarp();
    }
    if (OWN && i < n_direct && own_hits[lane])
      atomicAdd(owner_hits + w, (unsigned long long)own_hits[lane]);
    if (OWN) __syncwarp();
  }
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(count, hits);
}

template <bool HIER, bool OWN = false>
__global__ void __launch_bounds__(kLT, 1)
    tc_owner_large_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ goff,
                          const int2* __restrict__ ent, const int32_t* __restrict__ rows,
                          unsigned none, const int2* __restrict__ units_last,
                          const int2* __restrict__ dunits_last, int32_t* __restrict__ ctr,
                          const int32_t* __restrict__ table, int64_t bn, int b, int lg_max,
                          unsigned long long* __restrict__ count,
                          unsigned long long* __restrict__ owner_hits,
                          int32_t* __restrict__ status) {
  extern __shared__ __align__(128) int sm[];  // the staged table, the warps' queues, rings
  constexpr int kLg = 31 - __builtin_clz(kLTab);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  OpenQueue open{sm + kLTab + warp * 32 * kQueueLane + lane};
  RingRow* ring = reinterpret_cast<RingRow*>(sm + kLTab + kLW * 32 * kQueueLane) + warp * kRing;
  unsigned long long hits = cta_units<kLg, kLT, kLSeg, -1, OWN>(
      Staged<kLg>{sm}, desc, goff, ent, reinterpret_cast<const int4*>(rows), none, units_last,
      ctr[kCtrLarge], ctr + kCtrLargeNext, table, bn, b, open, ring, owner_hits);
  hits += direct_units<HIER, kLDirSeg, -1, OWN>(desc, goff, ent, rows, dunits_last, ctr[kCtrLargeDirect],
                                  ctr + kCtrLargeDirectNext, table, bn, b, lg_max, owner_hits,
                                  status);
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(count, hits);
}

// Key rows are put in class order from this many keys on: the passes cost
// ~25 us and ~20 ps a key, and what they save grows with the row lengths.
// Measured without / with (R-MAT, edge factor 16): scale 18 573 / 620 us,
// scale 20 2631 / 2673 us, scale 22 14.0 / 13.5 ms, scale 24 81 / 73 ms.
constexpr int64_t kClassEdges = 1 << 24;

int grid_stride_blocks(int64_t items_per_block_unit, int cap) {
  if (items_per_block_unit < 1) items_per_block_unit = 1;
  return (int)std::min<int64_t>(items_per_block_unit, cap);
}

}  // namespace

// Owner-grouped sum over the edges (u, v) of the edge CSR (eoff, ecols, me;
// echunk_rows its 32-edge chunk rows) of |K(u) ∩ K(v)|, K = the key CSR
// (koff, kcols, mk; kdesc its descriptors) that table t was built on.  For
// triangle counting both CSRs are the graph.  *count must already be zeroed.
reset_status tc_owner(const reset_table* t, const int4* kdesc, const int32_t* koff,
                      const int32_t* kcols, int64_t mk, const int32_t* eoff,
                      const int32_t* ecols, const int32_t* echunk_rows, int64_t me,
                      unsigned long long* count, cudaStream_t st,
                      unsigned long long* owner_hits) {
  const int64_t n = t->n;
  const int64_t m = me;
  if (n == 0 || me == 0 || mk == 0) return RESET_OK;
  if (mk > INT32_MAX - 16)
    return arg_fail("the owner-grouped count takes at most 2^31 - 17 keys");
  if (n == INT32_MAX) return arg_fail("the owner-grouped count takes at most 2^31 - 2 sets");
  // scratch, one allocation
  size_t cub_bytes = 0;
  RST_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, cub_bytes, (int32_t*)nullptr,
                                         (int32_t*)nullptr, (int)(n + 1), st));
  // the largest set, as own_classify_kernel bounds it
  const bool large = t->alpha * (float)((int64_t)t->bucket << t->lg_max) > kTab / 2;
  const int64_t max_units = n + m / kSeg + 1;
  const int64_t max_dunits = n + m / (large ? kLDirSeg : kDirSeg) + 1;
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t sz_cnt = al(sizeof(int32_t) * (n + 1)), sz_goff = sz_cnt;
  const size_t sz_ent = al(sizeof(int2) * m), sz_units = al(sizeof(int2) * max_units);
  const size_t sz_list = al(sizeof(int32_t) * n), sz_ctr = al(sizeof(int32_t) * kCtrs);
  const size_t sz_dunits = al(sizeof(int2) * max_dunits);
  const int64_t pad_chunks = padded_chunks(n, mk) + 1;  // (and one without keys)
  const size_t sz_pad = al(8 * sizeof(int32_t) * (size_t)(pad_chunks + 1));
  // classes need the rows to be the sets of the tables (the CSR they were
  // built on), and pay on more edges than the passes cost
  const bool classes = koff == t->build_off && mk == t->m && mk >= kClassEdges;
  const size_t sz_deg = classes ? al(sizeof(int32_t) * ((size_t)n + kDegSteps)) : 0;
  const size_t sz_info = al(sizeof(unsigned) * (size_t)n);
  // (rows of more than kClassRow keys: at most mk / kClassRow)
  const bool pad_long = t->alpha * (float)((int64_t)t->bucket << t->lg_max) > kClassRow;
  const int max_parts = pad_long ? (int)(mk / kPadPart + mk / kClassRow + 1) : 0;
  const size_t sz_parts = al(sizeof(int2) * (size_t)max_parts);
  const size_t sz_cls = classes ? al((size_t)n) : 0;
  const size_t sz_places = classes ? al(sizeof(ClassPlaces) * (size_t)n) : 0;
  const size_t total = sz_cnt + sz_goff + sz_ent + sz_units + 2 * sz_list + sz_dunits +
                       sz_ctr + sz_pad + sz_info + sz_deg + sz_cls + sz_places + sz_parts +
                       al(cub_bytes);
  char* base = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&base), total, st));
  char* p = base;
  int32_t* cnt = reinterpret_cast<int32_t*>(p); p += sz_cnt;
  int32_t* ctr = reinterpret_cast<int32_t*>(p); p += sz_ctr;
  int32_t* goff = reinterpret_cast<int32_t*>(p); p += sz_goff;
  int2* ent = reinterpret_cast<int2*>(p); p += sz_ent;
  int2* units = reinterpret_cast<int2*>(p); p += sz_units;
  int32_t* wlist = reinterpret_cast<int32_t*>(p); p += sz_list;
  int32_t* dlist = reinterpret_cast<int32_t*>(p); p += sz_list;
  int2* dunits = reinterpret_cast<int2*>(p); p += sz_dunits;
  int2 *units_last = units + max_units - 1, *dunits_last = dunits + max_dunits - 1;
  int32_t* padded = reinterpret_cast<int32_t*>(p); p += sz_pad;
  int32_t* indeg = reinterpret_cast<int32_t*>(p); p += sz_deg;
  unsigned* hist = reinterpret_cast<unsigned*>(indeg + n);
  uint8_t* cls = classes ? reinterpret_cast<uint8_t*>(p) : nullptr; p += sz_cls;
  unsigned* info = reinterpret_cast<unsigned*>(p); p += sz_info;
  ClassPlaces* places = reinterpret_cast<ClassPlaces*>(p); p += sz_places;
  int2* parts = reinterpret_cast<int2*>(p); p += sz_parts;
  void* cub_tmp = p;

  cudaError_t e = cudaMemsetAsync(cnt, 0, sz_cnt + sz_ctr, st);
  const int sms = sm_count();
  const int64_t chunks = (m + 31) / 32;
  const int g_edges = grid_stride_blocks((chunks + kOW * kIlp - 1) / (kOW * kIlp), sms * 8);
  if (e == cudaSuccess && classes) {
    e = cudaMemsetAsync(indeg, 0, sizeof(int32_t) * ((size_t)n + kDegSteps), st);
    if (e == cudaSuccess) {
      note_launch(3);
      key_count_kernel<<<grid_stride_blocks((mk + kOT - 1) / kOT, sms * 8), kOT, 0, st>>>(
          kcols, mk, t->n, indeg);
      const int g = grid_stride_blocks((n + kOT - 1) / kOT, sms * 4);
      degree_hist_kernel<<<g, kOT, 0, st>>>(koff, indeg, t->n, hist);
      class_kernel<<<g, kOT, 0, st>>>(koff, indeg, t->n, hist, cls);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) {
    note_launch();
    pad_rows_kernel<<<grid_stride_blocks((n * 8 + kOT - 1) / kOT, sms * 16), kOT, 0, st>>>(
        koff, kcols, t->n, mk, cls, padded, padded + pad_chunks * 8, info, places, parts,
        max_parts, ctr + kCtrPadParts);
    if (pad_long) {
      note_launch();
      pad_long_kernel<<<sms * 4, kOT, 0, st>>>(koff, kcols, t->n, mk, parts, max_parts,
                                               ctr + kCtrPadParts, padded);
    }
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    note_launch();
    own_count_kernel<<<g_edges, kOT, 0, st>>>(eoff, ecols, echunk_rows, koff, info, t->n, me, cnt,
                                              t->d_status);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cub::DeviceScan::ExclusiveSum(cub_tmp, cub_bytes, cnt, goff, (int)(n + 1), st);
  if (e == cudaSuccess)  // the groups' ends, counted down by the scatter
    e = cudaMemcpyAsync(cnt, goff + 1, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess) {
    note_launch();
    own_scatter_kernel<<<g_edges, kOT, 0, st>>>(eoff, ecols, echunk_rows, koff, info, t->n, me,
                                                mk, places, cnt, ent, t->d_status);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    note_launch();
    own_classify_kernel<<<grid_stride_blocks((n + kOT - 1) / kOT, sms * 8), kOT, 0, st>>>(
        kdesc, goff, ent, t->n, t->bucket, t->alpha, units, wlist, dlist, dunits, units_last,
        dunits_last, ctr);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    const size_t smem = sizeof(int) * (kTab + kTW * 32 * kQueueLane) + sizeof(RingRow) * kTW * kRing;
    const bool own = owner_hits != nullptr;
#define OWN_K(H, O) tc_owner_kernel<H, O>
    const void* k = t->hier ? (own ? (const void*)OWN_K(true, true) : (const void*)OWN_K(true, false))
                            : (own ? (const void*)OWN_K(false, true)
                                   : (const void*)OWN_K(false, false));
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTT, smem);
    if (e == cudaSuccess) {
      const int grid = sms * (per_sm > 0 ? per_sm : 1);
      note_launch();
#define OWN_LAUNCH(H, O)                                                                   \
  OWN_K(H, O)<<<grid, kTT, smem, st>>>(kdesc, goff, ent, padded, (unsigned)pad_chunks, units, \
                                       wlist, dlist, dunits, ctr, t->d_table, t->bucket_num, t->bucket,  \
                                       t->lg_max, count, owner_hits, t->d_status)
      if (t->hier) {
        if (own) OWN_LAUNCH(true, true); else OWN_LAUNCH(true, false);
      } else {
        if (own) OWN_LAUNCH(false, true); else OWN_LAUNCH(false, false);
      }
#undef OWN_LAUNCH
#undef OWN_K
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && large) {
#define OWN_L(H, O)                                                                             \
  do {                                                                                          \
    e = cudaFuncSetAttribute(tc_owner_large_kernel<H, O>,                                       \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLargeSmem);     \
    if (e != cudaSuccess) break;                                                                \
    note_launch();                                                                              \
    tc_owner_large_kernel<H, O><<<sms, kLT, kLargeSmem, st>>>(                                  \
        kdesc, goff, ent, padded, (unsigned)pad_chunks, units_last, dunits_last, ctr, t->d_table, \
        t->bucket_num, t->bucket, t->lg_max, count, owner_hits, t->d_status);                   \
    e = cudaGetLastError();                                                                     \
  } while (0)
      if (t->hier) {
        if (own) OWN_L(true, true); else OWN_L(true, false);
      } else {
        if (own) OWN_L(false, true); else OWN_L(false, false);
      }
#undef OWN_L
    }
  }
  cudaFreeAsync(base, st);
  if (e != cudaSuccess) return cuda_fail(e, "owner-grouped TC", __FILE__, __LINE__);
  return RESET_OK;
}

}  // namespace rst

using namespace rst;

extern "C" reset_status reset_tc_count_batch(const reset_table* t, const int32_t* d_off,
                                             const int32_t* d_cols, int64_t m,
                                             const int32_t* d_graph_off, int32_t n_graphs,
                                             uint64_t* d_counts, reset_stream_t stream) {
  if (!t || !d_counts || !d_graph_off) return arg_fail("NULL table, graph offsets or counts");
  if (n_graphs < 1) return arg_fail("n_graphs must be >= 1");
  if (m < 0 || m > INT32_MAX - 16) return arg_fail("m out of range");
  if (m > 0 && (!d_cols || !d_off)) return arg_fail("NULL offsets or cols");
  if ((reinterpret_cast<uintptr_t>(d_cols) & 15) != 0)
    return arg_fail("reset_tc_count_batch needs a 16-byte aligned column array");
  if (d_off != t->build_off || m != t->m)
    return arg_fail("d_off/m must be the CSR the table was built on");
  cudaStream_t st = as_stream(stream);
  RST_CUDA(cudaMemsetAsync(d_counts, 0, sizeof(uint64_t) * (size_t)n_graphs, st));
  if (m == 0 || t->n == 0) return RESET_OK;
  size_t cub_bytes = 0;
  RST_CUDA(cub::DeviceSegmentedReduce::Sum(nullptr, cub_bytes, (unsigned long long*)nullptr,
                                           (unsigned long long*)nullptr, n_graphs, d_graph_off,
                                           d_graph_off + 1, st));
  const size_t own_bytes = (sizeof(unsigned long long) * ((size_t)t->n + 1) + 255) & ~(size_t)255;
  char* buf = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&buf), own_bytes + 256 + cub_bytes, st));
  auto* owner_hits = reinterpret_cast<unsigned long long*>(buf);
  auto* total = reinterpret_cast<unsigned long long*>(buf + own_bytes);
  cudaError_t e = cudaMemsetAsync(buf, 0, own_bytes + 256, st);
  reset_status s = RESET_OK;
  if (e == cudaSuccess) {
    const bool sparse = tc_sparse(t);
    if (!sparse)
      s = tc_owner(t, t->d_desc, d_off, d_cols, m, d_off, d_cols, t->d_chunk_row, m, total, st,
                   owner_hits);
    if (s == RESET_ERR_OOM) {  // no memory for the groups
      cudaGetLastError();
      e = cudaMemsetAsync(buf, 0, own_bytes + 256, st);
    }
    if (e == cudaSuccess && (sparse || s == RESET_ERR_OOM))
      s = tc_edges(t, t->d_desc, d_cols, d_off, d_cols, t->d_chunk_row, m, total, st, owner_hits);
  }
  if (e == cudaSuccess && s == RESET_OK)
    e = cub::DeviceSegmentedReduce::Sum(buf + own_bytes + 256, cub_bytes, owner_hits,
                                        reinterpret_cast<unsigned long long*>(d_counts), n_graphs,
                                        d_graph_off, d_graph_off + 1, st);
  cudaFreeAsync(buf, st);
  if (e != cudaSuccess) return cuda_fail(e, "reset_tc_count_batch", __FILE__, __LINE__);
  return s;
}
