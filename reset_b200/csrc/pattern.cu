// Pattern counting (subgraph matching) by multi-way hash-probe
// intersections: SMOG's DFSKernelForGeneral and DFSKernelForClique
// (SMOG/SMOG_hie/subgraph_match_hie.cu:58-406) over this library's tables,
// for any pattern in SMOG's encoding (reset_pattern in reset.h).
//
// One warp per start edge.  The edge fixes m_0 and m_1.  Level l >= 2 builds
// its candidate set C_l in one pass: the base is the reused level's set or
// the shortest row among the listed backward vertices; every base key is
// looked up in the other listed rows (early exit per lane), and the hits are
// compacted into the warp's scratch row of level l (ballot/popc).  A level
// with nothing to look up keeps a view of its base, without a copy.
// The last level is only counted; earlier levels are walked 32 candidates
// at a time, the next m_l being the first lane's key that passes the
// level's check.  Where no later level reuses C_l, keys failing l's check
// are dropped at compaction already.  The reference instead builds C_l by
// one pass per listed row, and walks candidates one by one.
//
// Work distribution: the search below one start edge grows with the square or
// cube of the rows it meets, so on a skewed graph a few hub edges outlast all
// others (R-MAT scale 9, Q6: 8% of the warps active over the run).  Edges
// whose first set may be long are cut into parts, listed ahead of the rest;
// a part builds C_2 again (one pass) and walks its slice of it.
//
// Lookups: a row is its bit row of n bits where the graph's bit matrix fits
// kBitBudget (else the longest rows' bit rows, as many as fit), one load and
// a shift; other rows are probed in their hash table.  Bit rows need all keys
// in [0, n), checked in the pass that finds the longest row.
//
// With strictly ascending rows (checked in the same pass), a restriction
// m_l < m_r cuts the base to its prefix below m_r before any lookup, and a
// last level with nothing to look up is counted without a scan: the prefix
// length, or |C_l| less the earlier vertices in it.  Such a last level is not
// entered at all: the level before it hands one candidate to each lane,
// which counts the last level for it; what does not depend on the candidate
// (which earlier vertices the base holds, and where) is found once per visit.
// A last level that intersects a fixed vertex's row with the row of the
// candidate just picked (N(m_a) ∩ N(x)) is not entered either: such
// intersections of at most kLaneMax keys run one candidate per lane, longer
// ones by the whole warp, as AND + popcount over the two bit rows where that
// is less work than looking up the shorter row's keys; without a bound, on up
// to 16384 vertices, the sizes of all such intersections are computed first
// (codegree_kernel) and a candidate costs a load.  A reusing
// k-clique chain without checks (SMOG's Q0, Q3, Q5, Q7) runs the k-clique
// count (clique.cu).
//
// Bound by instruction issue and, on small graphs, by the longest part.
// Against one edge per warp with every lookup a hash probe (R-MAT, ms):
// Q6 scale 8 / 11: 3.2 / 116 -> 0.16 / 0.81; Q4 scale 8 / 13: 0.57 / 19.8 ->
// 0.15 / 4.8; Q8 scale 13: 20.6 -> 3.7; Q1 scale 8 / 14: 0.16 / 16.3 ->
// 0.12 / 6.5; Q2 scale 14: 11.9 -> 3.1.
//
// Semantics differ from the reference in one case only: where two listed
// vertices of a level map to the same data vertex and that vertex has the
// shortest row, the reference skips both (its count then reads scratch left
// from an earlier edge); here N(x) ∩ N(x) = N(x).  No pattern of the
// reference's table reaches that case: in each, an edge, the distinctness
// check or a restriction separates the two vertices.
#include <algorithm>
#include <cstring>

#include "probe_common.cuh"

namespace rst {
namespace {

constexpr int kPatMax = RESET_PATTERN_MAX;
constexpr int kPtThreads = 256;
constexpr int kPtWarps = kPtThreads / 32;
// Scratch rows of all resident warps together stay below this; a graph
// whose largest row would need more runs fewer warps.
constexpr size_t kPtScratchBudget = size_t(1) << 30;
// Bytes of bit rows at most (2x the L2; n = 46340 vertices get a whole matrix),
// and per unit of the sum of the squared row lengths, which bounds the keys that
// the second level looks up: clearing a matrix that hardly any lookup reads took
// most of a call (40,000 vertices with 200 edges: 260 us, 88 without).
constexpr int64_t kBitBudget = int64_t(1) << 28, kBitPerSquare = 64;
// Rows shorter than this get no bit row of their own on larger graphs: their
// hash table spans no more cache lines than the bit row's hits would.
constexpr int kBitMinRow = 64;
// Start edges whose first set may hold more keys than this are cut into
// parts of about as many; a paired or fused last level right after it takes
// 32 candidates at a time, deeper patterns have far more below a candidate.
constexpr int kPartDeep = 8, kPartFlat = 64;
// ... and are made longer where there would be more parts than this.
constexpr int64_t kMaxParts = int64_t(1) << 20;
// Longest row up to which neither bit rows nor parts are used: a set is then a
// step of a warp, and the launches that prepare them cost more than they save.
// 10,000 vertices with 10 neighbours each, Q6 / Q4: 220 / 197 us with them, 146 / 142
// without; 100 with one each 103 / 90 and 82 / 84.
constexpr int kShortRows = 32;

struct PatternDev {
  int32_t k, flags;
  int32_t restr[kPatMax];          // restriction[l], -1 = none
  int32_t reuse[kPatMax];          // reused level, -1 = none
  int32_t nb[kPatMax];             // listed backward vertices of level l
  int32_t back[kPatMax][kPatMax];  // ... their pattern indices (no -1)
  int32_t filt[kPatMax];           // 1: no later level reuses C_l
  int32_t chain;                   // a reusing clique chain without checks
  int32_t fuse;                    // the last level probes nothing
  int32_t pair;                    // the last level lists {pair_a, k-2} only
  int32_t pair_a;
};

// Intersections of the paired last level up to this length run one per
// lane; longer ones take the whole warp.
constexpr int kLaneMax = 32;

// checkRestriction (SMOG/SMOG_hie/subgraph_match_hie.cu:23-42) with the
// opposite sense: true when key x may be m_l.
__device__ __forceinline__ bool level_ok(const PatternDev& p, int l, int x, const int* map) {
  const int r = p.restr[l];
  if ((p.flags & RESET_PATTERN_DISTINCT) && r < 0)
    for (int i = 0; i < l; ++i)
      if (map[i] == x) return false;
  if ((p.flags & RESET_PATTERN_RESTRICT) && r >= 0 && x >= map[r]) return false;
  return true;
}

// First index of a[0 .. n) whose key is >= x (a ascending); plain loads,
// `a` may be the calling warp's scratch.
__device__ __forceinline__ int lower_bound_key(const int32_t* a, int n, int x) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// The graph's bit rows: row[y] (or y itself, row NULL) is the row of vertex
// y, -1 = none; `words` a row, a multiple of 4.
struct BitRows {
  const uint32_t* bits;
  const int32_t* row;
  int64_t words;
  __device__ __forceinline__ const uint32_t* of(int y) const {
    if (!bits) return nullptr;
    const int r = row ? __ldg(row + y) : y;
    return r < 0 ? nullptr : bits + r * words;
  }
};

__device__ __forceinline__ bool bit_of(const uint32_t* br, int x) {
  return (__ldg(br + (x >> 5)) >> (x & 31)) & 1u;
}

// Rows of at least `shortest` keys get the next bit rows, in any order.
__global__ void bit_assign_kernel(const int4* __restrict__ desc, int32_t n, int shortest,
                                  int32_t* __restrict__ row, int32_t* __restrict__ ctr) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n;
       u += (int64_t)gridDim.x * blockDim.x)
    row[u] = __ldg(desc + u).y >= shortest ? atomicAdd(ctr, 1) : -1;
}

// Sets the bit rows (zeroed, all keys in [0, n)), a warp per row, and counts
// the vertices whose row holds themselves.
__global__ void bit_fill_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ cols,
                                int32_t n, const int32_t* __restrict__ row, int64_t words,
                                uint32_t* __restrict__ bits, int32_t* __restrict__ loops) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < n; u += nw) {
    const int4 du = __ldg(desc + u);
    const int r = row ? __ldg(row + u) : (int)u;
    uint32_t* br = bits + r * words;
    for (int j = lane; j < du.y; j += 32) {
      const int x = __ldg(cols + du.x + j);
      if (r >= 0) atomicOr(br + (x >> 5), 1u << (x & 31));
      if (x == u) atomicAdd(loops, 1);
    }
  }
}

// Keys the first set of start edge (u, v) may hold: the shortest listed row,
// counted no longer than u's so that the parts of all edges are bounded by
// the sum of the squared row lengths.
__device__ __forceinline__ int first_set(const PatternDev& p, int du, int dv) {
  int s = du;
  for (int j = 0; j < p.nb[2]; ++j) s = min(s, p.back[2][j] == 0 ? du : dv);
  return s;
}

// Start edges with a first set above `part` keys, as (u, v, i, parts).  With
// the bit rows of all vertices, also an estimate of the visits of a paired
// last level, from every step-th of these edges: |C_2| (squared where two
// levels walk it), less where rows are short and a visit costs little.
__global__ void pattern_parts_kernel(const int4* __restrict__ desc,
                                     const int32_t* __restrict__ cols, int32_t n, int64_t m,
                                     const PatternDev pat, int part, int4* __restrict__ list,
                                     int32_t* __restrict__ n_list, const BitRows br, int step,
                                     unsigned long long* __restrict__ visits) {
  const int lane = threadIdx.x & 31;
  unsigned long long sum = 0;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < n; u += nw) {
    const int4 du = __ldg(desc + u);
    if (du.y <= part) continue;
    const int d = (int)min((int64_t)du.y, m - du.x);
    for (int j = lane; j - lane < d; j += 32) {
      const int v = j < d ? __ldg(cols + du.x + j) : -1;
      const int map[2] = {(int)u, v};
      int s = 0;
      if ((unsigned)v < (unsigned)n && level_ok(pat, 1, v, map))
        s = first_set(pat, du.y, __ldg(&desc[v].y));
      const int np = s > part ? (s + part - 1) / part : 0;
      int total;
      const int before = warp_excl_scan(np, &total);
      if (total == 0) continue;
      int at = lane == 0 ? atomicAdd(n_list, total) : 0;
      at = __shfl_sync(kFull, at, 0) + before;
      for (int i = 0; i < np; ++i) list[at + i] = make_int4((int)u, v, i, np);
      if (!br.bits) continue;
      for (unsigned todo = __ballot_sync(kFull, np > 0 && (du.x + j) % step == 0); todo;
           todo &= todo - 1) {
        const int g = __ffs(todo) - 1;
        const int vg = __shfl_sync(kFull, v, g), sg = __shfl_sync(kFull, s, g);
        int c = 0;
        for (int w = lane; w < br.words; w += 32) {
          uint32_t x = ~0u;
          for (int i = 0; i < pat.nb[2]; ++i) x &= __ldg(br.of(pat.back[2][i] == 0 ? u : vg) + w);
          c += __popc(x);
        }
        const unsigned long long e = __reduce_add_sync(kFull, c);
        if (lane == 0) sum += (pat.k > 4 ? e * e : e) * min(sg, 64);
      }
    }
  }
  if (lane == 0 && sum) atomicAdd(visits, sum * step / 64);
}

// Co-degrees |N(a) ∩ N(x)| of all pairs of vertices, from the bit rows: where
// the paired last level has no bound, its count for a candidate x is one of
// them, less the earlier vertices, and a visit costs a load where it took the
// AND of two bit rows by the whole warp.  The matrix takes n^3 / 64 word
// steps of three instructions, a visit without it up to 100 warp
// instructions: it is filled (and used) where the visits times kCoVisits reach
// n^3, a quarter of where it pays with long rows.  Decided on the device, where
// the estimate is.  Popcounts bound the matrix (n = 2048: 44 us).  Q6 on R-MAT
// graphs, ms a call, by ANDs / by co-degrees: scale 11 3.41 / 0.81, scale 13
// 62.8 / 6.9 (268 MB of matrix), scale 14 380 / 30 (1 GB); scale 8, whose matrix is
// nothing, 0.26 / 0.16.  A random graph of 8192 vertices and 100 neighbours
// each, with hardly a common one, is walked without.
constexpr unsigned long long kCoVisits = 16384;
constexpr int kCoSmall = 512;  // vertices whose matrix (2 us) costs less than the estimate
constexpr int64_t kCoBudget = int64_t(1) << 30;  // bytes: up to 16384 vertices
constexpr int kCoTile = 64;  // vertices on a side of a block's tile
constexpr int kCoWords = 32;

__device__ __forceinline__ bool co_used(const unsigned long long* visits, int64_t n) {
  return n <= kCoSmall || *visits >= (unsigned long long)(n * n * n) / kCoVisits;
}

__global__ void __launch_bounds__(256)
    codegree_kernel(const uint32_t* __restrict__ bits, int32_t n, int words,
                    const unsigned long long* __restrict__ visits, int32_t* __restrict__ co) {
  if (!co_used(visits, n)) return;
  const int i0 = blockIdx.y * kCoTile, j0 = blockIdx.x * kCoTile;
  if (i0 > j0) return;  // the tile below the diagonal is written with its mirror
  __shared__ uint32_t sa[kCoTile][kCoWords + 1], sb[kCoTile][kCoWords + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  int acc[4][4] = {};
  for (int w0 = 0; w0 < words; w0 += kCoWords) {
    __syncthreads();
    for (int t = threadIdx.x; t < kCoTile * kCoWords; t += 256) {
      const int r = t / kCoWords, w = t % kCoWords;
      const bool in = w0 + w < words;
      sa[r][w] = in && i0 + r < n ? __ldg(bits + (int64_t)(i0 + r) * words + w0 + w) : 0;
      sb[r][w] = in && j0 + r < n ? __ldg(bits + (int64_t)(j0 + r) * words + w0 + w) : 0;
    }
    __syncthreads();
#pragma unroll 4
    for (int w = 0; w < kCoWords; ++w) {
      uint32_t a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = sa[ty + 16 * i][w], b[i] = sb[tx + 16 * i][w];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += __popc(a[i] & b[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t y = i0 + ty + 16 * i, x = j0 + tx + 16 * j;
      if (y >= n || x >= n) continue;
      co[y * n + x] = acc[i][j];
      co[x * n + y] = acc[i][j];
    }
}

template <bool HIER>
__global__ void __launch_bounds__(kPtThreads, 4)
    pattern_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ off,
                   const int32_t* __restrict__ cols, const int32_t* __restrict__ chunk_row,
                   int32_t n, int64_t m, const int32_t* __restrict__ table, int64_t bn, int b,
                   int lg_max, const PatternDev pat, int sorted, const BitRows br,
                   const int32_t* __restrict__ loops, const int32_t* __restrict__ co,
                   const unsigned long long* __restrict__ visits,
                   const int4* __restrict__ parts_list,
                   const int32_t* __restrict__ n_list, int part, int lg_grab,
                   int32_t* __restrict__ scratch, int32_t cap,
                   unsigned long long* __restrict__ count,
                   unsigned long long* __restrict__ cursor, int32_t* __restrict__ status) {
  __shared__ PatternDev sp;
  if (threadIdx.x == 0) sp = pat;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int k = sp.k;
  const int rows = k > 3 ? k - 3 : 1;
  int32_t* Sbase = scratch + gw * (int64_t)cap * rows;
  const int64_t me = min(m, (int64_t)__ldg(off + n));
  const int grab = 1 << lg_grab;  // start edges a warp takes at a time, at most 32
  const int64_t n_grabs = (me + grab - 1) >> lg_grab;
  const int n_parts = part > 0 ? *n_list : 0;
  // no row holds its own vertex (known where bit rows were set)
  const bool loop_free = br.bits && *loops == 0;
  const bool have_co = co && co_used(visits, n);
  unsigned long long hits = 0;
  // level l: m_l, its index in C_l, C_l (cs, sz), the next candidate (it)
  int map[kPatMax], idx[kPatMax], sz[kPatMax], it[kPatMax];
  const int32_t* cs[kPatMax];
  int4 pd[kPatMax];
  const uint32_t* pbits[kPatMax];
  // x in the row of desc dy with bit row by
  auto holds = [&](const uint32_t* by, const int4& dy, int x) {
    return by ? bit_of(by, x)
              : probe_key<HIER>(x, table + desc_toff(dy), desc_lg(dy), lg_max, bn, b, status);
  };
  bool listed = n_parts > 0;
  for (;;) {
    // the next listed part, then the next edges: one start edge per lane
    unsigned long long cc = 0;
    if (lane == 0) cc = atomicAdd(cursor + (listed ? 0 : 1), 1ull);
    const int64_t c = (int64_t)__shfl_sync(kFull, cc, 0);
    int4 item = make_int4(0, 0, 0, 1);
    bool start;
    if (listed) {
      if (c >= n_parts) {
        listed = false;
        continue;
      }
      start = lane == 0;
      if (start) item = __ldg(parts_list + c);
    } else {
      if (c >= n_grabs) break;
      const int64_t e0 = c << lg_grab;
      const int64_t e = min(e0 + min(lane, grab - 1), me - 1);
      int u0 = __ldg(chunk_row + (e0 >> 5));
      if ((unsigned)u0 >= (unsigned)n) u0 = 0;
      item.x = row_of_edge(off, n, u0, (int)e);
      item.y = __ldg(cols + e);
      start = lane < grab && e0 + lane < me && (unsigned)item.x < (unsigned)n;
      if (start && (unsigned)item.y >= (unsigned)n) {
        atomicOr(status, kErrBadId);
        start = false;
      }
      if (start) {
        const int ends[2] = {item.x, item.y};
        start = level_ok(sp, 1, item.y, ends) &&
                !(part > 0 &&
                  first_set(sp, __ldg(&desc[item.x].y), __ldg(&desc[item.y].y)) > part);
      }
    }
    for (unsigned todo = __ballot_sync(kFull, start); todo; todo &= todo - 1) {
      const int f = __ffs(todo) - 1;
      map[0] = __shfl_sync(kFull, item.x, f);
      map[1] = __shfl_sync(kFull, item.y, f);
      const int my_part = __shfl_sync(kFull, item.z, f), parts = __shfl_sync(kFull, item.w, f);
      int end2 = 0;  // candidates of level 2 end here (a part's slice of C_2)
      int lv = 2;    // warp-uniform depth
      bool build = true;
      while (lv >= 2) {
        if (build) {
          build = false;
          // the base of C_lv: the reused set, or the shortest listed row
          const int32_t* src = cols;
          int ns = 0, bv = -1;
          const int r = sp.reuse[lv];
          if (r >= 0) {
            src = cs[r];
            ns = sz[r];
          } else {
            ns = INT_MAX;
            for (int j = 0; j < sp.nb[lv]; ++j) {
              const int y = map[sp.back[lv][j]];
              const int4 dy = __ldg(desc + y);
              if (dy.y < ns) {
                ns = dy.y;
                bv = y;
                src = cols + dy.x;
              }
            }
          }
          // the other listed rows, each once, are looked up
          int np = 0;
          for (int j = 0; j < sp.nb[lv]; ++j) {
            const int y = map[sp.back[lv][j]];
            if (y == bv) continue;
            bool seen = false;
            for (int q = 0; q < j; ++q) seen |= map[sp.back[lv][q]] == y;
            if (seen) continue;
            const int4 dy = __ldg(desc + y);
            if (dy.y == 0) ns = 0;
            pbits[np] = br.of(y);
            pd[np++] = dy;
          }
          const bool last = lv == k - 1;
          const int rr = sp.restr[lv];
          // ascending rows: the keys a restriction m_lv < m_rr admits are a
          // prefix of the base (cut only where no later level reuses C_lv);
          // m_rr's own index where the base is m_rr's set
          if (sorted && (sp.flags & RESET_PATTERN_RESTRICT) && rr >= 0 && (last || sp.filt[lv]))
            ns = rr >= 2 && src == cs[rr] && idx[rr] < ns ? idx[rr]
                                                          : lower_bound_key(src, ns, map[rr]);
          if (last && np == 0 && sorted) {
            // C_lv is the base itself: |C_lv| less the earlier vertices in it
            int c2 = ns;
            if ((sp.flags & RESET_PATTERN_DISTINCT) && rr < 0)
              for (int i = 0; i < lv; ++i) {
                const int y = map[i];
                bool seen = false;
                for (int q = 0; q < i; ++q) seen |= map[q] == y;
                if (seen) continue;
                const int at = lower_bound_key(src, ns, y);
                if (at < ns && src[at] == y) --c2;
              }
            if (lane == 0) hits += c2;
            --lv;
            continue;
          }
          if (np == 0 && !last) {  // a view of the base
            cs[lv] = src;
            sz[lv] = ns;
          } else {
            int32_t* dst = Sbase + (int64_t)(lv - 2) * cap;
            const bool chk = last || sp.filt[lv];
            int nw = 0;
            for (int j0 = 0; j0 < ns; j0 += 32) {
              const int j = j0 + lane;
              bool in = false;
              int x = 0;
              if (j < ns) {
                x = src[j];  // plain load: src may be this warp's scratch
                in = !chk || level_ok(sp, lv, x, map);
                for (int q = 0; in && q < np; ++q) in = holds(pbits[q], pd[q], x);
              }
              if (last) {
                hits += in;
              } else {
                const unsigned msk = __ballot_sync(kFull, in);
                if (in) {
                  const int pos = nw + __popc(msk & lt);
                  if (pos < cap) dst[pos] = x;
                }
                nw += __popc(msk);
              }
            }
            if (!last) {
              if (nw > cap) {  // cannot happen: no set outgrows the longest row
                if (lane == 0) atomicOr(status, kErrProbeLimit);
                nw = cap;
              }
              __syncwarp();
              cs[lv] = dst;
              sz[lv] = nw;
            }
          }
          if (last) {
            --lv;
            continue;
          }
          it[lv] = 0;
          if (lv == 2) {
            it[2] = (int)((int64_t)sz[2] * my_part / parts);
            end2 = (int)((int64_t)sz[2] * (my_part + 1) / parts);
          }
        }
        const int end = lv == 2 ? end2 : sz[lv];
        if (sp.pair && lv == k - 2) {
          // the last level is N(m_a) ∩ N(x) for the candidate x: short
          // intersections run one candidate per lane, long ones afterwards
          // by the warp
          const int L = k - 1, rr = sp.restr[L];
          const bool rcut = sorted && (sp.flags & RESET_PATTERN_RESTRICT) && rr >= 0;
          const bool dist = (sp.flags & RESET_PATTERN_DISTINCT) && rr < 0;
          // keys to be checked one by one: only where rows may be out of
          // order or repeat keys
          const bool chk = !sorted && ((sp.flags & RESET_PATTERN_RESTRICT) || dist);
          const int ma = map[sp.pair_a];
          const int4 da = __ldg(desc + ma);
          const uint32_t* ba = br.of(ma);
          unsigned in_a = 0;  // earlier vertices (each once) that N(m_a) holds
          if (sorted && dist) {
            bool in = false;
            if (lane < lv) {
              in = !(loop_free && map[lane] == ma);
              for (int q = 0; q < lane; ++q) in = in && map[q] != map[lane];
              in = in && da.y > 0 && holds(ba, da, map[lane]);
            }
            in_a = __ballot_sync(kFull, in);
          }
          if (have_co) {  // (ascending rows, no bound, bit rows of all vertices)
            const int32_t* co_a = co + (int64_t)ma * n;
            for (int j = it[lv] + lane; j < end; j += 32) {
              const int x = cs[lv][j];  // (in [0, n): bit rows)
              if (!level_ok(sp, lv, x, map)) continue;
              int c2 = __ldg(co_a + x);
              if (dist && c2 > 0) {
                const uint32_t* bx = br.of(x);
                for (unsigned q = in_a; q; q &= q - 1) c2 -= bit_of(bx, map[__ffs(q) - 1]);
                if (!loop_free && bit_of(bx, x)) {
                  bool seen = false;
                  for (int q = 0; q < lv; ++q) seen |= map[q] == x;
                  if (!seen && bit_of(ba, x)) --c2;
                }
              }
              hits += c2;
            }
            --lv;
            continue;
          }
          for (int j0 = it[lv]; j0 < end; j0 += 32) {
            const int j = j0 + lane;
            int x = j < end ? cs[lv][j] : 0;
            bool act = j < end;
            if (act && (unsigned)x >= (unsigned)n) {
              atomicOr(status, kErrBadId);
              act = false;
            }
            act = act && level_ok(sp, lv, x, map);
            int len = 0, bound = n;
            bool a_base = false;  // the shorter row is m_a's
            const uint32_t* bx = nullptr;
            int4 dx = make_int4(0, 0, 0, 0);
            if (act) {
              dx = __ldg(desc + x);
              a_base = dx.y > da.y;
              len = min(dx.y, da.y);
              bx = br.of(x);
              if (rcut) {
                bound = rr == lv ? x : map[rr];
                len = lower_bound_key(cols + (a_base ? da.x : dx.x), len, bound);
              }
            }
            const int32_t* base = cols + (a_base ? da.x : dx.x);
            const int4 dt = a_base ? dx : da;
            const uint32_t* bt = a_base ? bx : ba;
            const bool big = len > kLaneMax;
            if (!big && len > 0) {
              unsigned long long c2 = 0;
              if (chk) {
                map[lv] = x;
                for (int t = 0; t < len; ++t) {
                  const int z = base[t];
                  c2 += level_ok(sp, L, z, map) && holds(bt, dt, z);
                }
              } else {
#pragma unroll 4
                for (int t = 0; t < len; ++t) c2 += holds(bt, dt, base[t]);
              }
              hits += c2;
            }
            if (sorted && dist && len > 0) {
              // less the earlier vertices in both rows
              for (unsigned q = in_a; q; q &= q - 1) hits -= holds(bx, dx, map[__ffs(q) - 1]);
              if (!loop_free && holds(bx, dx, x)) {
                bool seen = false;
                for (int q = 0; q < lv; ++q) seen |= map[q] == x;
                if (!seen && holds(ba, da, x)) --hits;
              }
            }
            for (unsigned bm = __ballot_sync(kFull, big); bm; bm &= bm - 1) {
              const int g = __ffs(bm) - 1;
              const int xb = __shfl_sync(kFull, x, g);
              const int lb = __shfl_sync(kFull, len, g);
              const int kb = __shfl_sync(kFull, bound, g);
              const uint32_t* bxb = br.of(xb);
              const int full = kb >> 5;  // whole words below the bound
              // a word step is one AND + popcount on 128 words, a key step a
              // lookup of 32 keys: about as many instructions
              if (sorted && ba && bxb && full < 4 * lb) {
                const int4* wa = reinterpret_cast<const int4*>(ba);
                const int4* wx = reinterpret_cast<const int4*>(bxb);
                unsigned t = 0;
                for (int q = lane; 4 * q < full; q += 32) {
                  const int4 p = __ldg(wa + q), r2 = __ldg(wx + q);
                  unsigned w[4] = {(unsigned)(p.x & r2.x), (unsigned)(p.y & r2.y),
                                   (unsigned)(p.z & r2.z), (unsigned)(p.w & r2.w)};
#pragma unroll
                  for (int i = 0; i < 4; ++i) t += 4 * q + i < full ? __popc(w[i]) : 0;
                }
                if (lane == 0 && (kb & 31))
                  t += __popc(__ldg(ba + full) & __ldg(bxb + full) & ((1u << (kb & 31)) - 1));
                hits += t;
                continue;
              }
              const int4 dxb = __ldg(desc + xb);
              const bool ab = dxb.y > da.y;
              const int32_t* bb = cols + (ab ? da.x : dxb.x);
              const int4 dtb = ab ? dxb : da;
              const uint32_t* btb = ab ? bxb : ba;
              if (chk) {
                map[lv] = xb;
                for (int t = lane; t < lb; t += 32) {
                  const int z = bb[t];
                  hits += level_ok(sp, L, z, map) && holds(btb, dtb, z);
                }
              } else {
#pragma unroll 4
                for (int t = lane; t < lb; t += 32) hits += holds(btb, dtb, bb[t]);
              }
            }
          }
          --lv;
          continue;
        }
        if (sorted && sp.fuse && lv == k - 2) {
          // the last level looks up nothing: every key x of C_lv that passes
          // lv's check is m_lv for one lane, which counts the last level's
          // keys for it at once (prefix below the restriction bound, less
          // the earlier vertices found in the base), without building it
          const int L = k - 1, rr = sp.restr[L], ru = sp.reuse[L];
          const bool rcut = (sp.flags & RESET_PATTERN_RESTRICT) && rr >= 0;
          const bool dist = (sp.flags & RESET_PATTERN_DISTINCT) && rr < 0;
          // the base: the same for every x, unless it is x's own row
          const bool fixed = ru >= 0 || sp.back[L][0] != lv;
          const int32_t* base = nullptr;
          int nbase = 0, at_bound = 0, kept = 0;
          if (fixed) {
            if (ru >= 0) {
              base = cs[ru];
              nbase = sz[ru];
            } else {
              const int4 dy = __ldg(desc + map[sp.back[L][0]]);
              base = cols + dy.x;
              nbase = dy.y;
            }
            if (rcut && rr != lv) nbase = lower_bound_key(base, nbase, map[rr]);
            if (dist) {  // (no bound then) the base's keys but the earlier vertices
              bool in = false;
              if (lane < lv) {
                const int y = map[lane];
                bool seen = false;
                for (int q = 0; q < lane; ++q) seen |= map[q] == y;
                const int at = lower_bound_key(base, nbase, y);
                in = !seen && at < nbase && base[at] == y;
              }
              kept = nbase - __popc(__ballot_sync(kFull, in));
            }
          }
          const bool same = fixed && base == cs[lv];  // x's index in the base is j, if below nbase
          for (int j = it[lv] + lane; j < end; j += 32) {
            const int x = cs[lv][j];
            if ((unsigned)x >= (unsigned)n) {
              atomicOr(status, kErrBadId);
              continue;
            }
            if (!level_ok(sp, lv, x, map)) continue;
            int4 dx = make_int4(0, 0, 0, 0);
            if (!fixed) {
              dx = __ldg(desc + x);
              base = cols + dx.x;
              nbase = dx.y;
              if (rcut && rr != lv) nbase = lower_bound_key(base, nbase, map[rr]);
            }
            int c2 = nbase;
            if (rcut && rr == lv)
              c2 = same ? min(j, nbase) : lower_bound_key(base, nbase, x);
            if (dist && fixed) {
              bool seen = false;
              for (int q = 0; q < lv; ++q) seen |= map[q] == x;
              at_bound = same ? j : lower_bound_key(base, nbase, x);
              c2 = kept - (!seen && at_bound < nbase && (same || base[at_bound] == x));
            } else if (dist && nbase > 0) {  // (no bound then) N(x) but the earlier vertices
              const uint32_t* bx = br.of(x);
              for (int i = 0; i <= lv; ++i) {
                if (i == lv && loop_free) break;
                const int y = i == lv ? x : map[i];
                bool seen = false;
                for (int q = 0; q < i; ++q) seen |= map[q] == y;
                if (!seen) c2 -= holds(bx, dx, y);
              }
            }
            hits += c2;
          }
          --lv;
          continue;
        }
        // the next key of C_lv that passes the level's check becomes m_lv
        int x = -1;
        while (it[lv] < end) {
          const int j = it[lv] + lane;
          const int y = j < end ? cs[lv][j] : 0;
          const bool bad = j < end && (unsigned)y >= (unsigned)n;
          if (bad) atomicOr(status, kErrBadId);
          const bool ok = j < end && !bad && level_ok(sp, lv, y, map);
          const unsigned msk = __ballot_sync(kFull, ok);
          if (msk) {
            const int g = __ffs(msk) - 1;
            x = __shfl_sync(kFull, y, g);
            idx[lv] = it[lv] + g;
            it[lv] += g + 1;
            break;
          }
          it[lv] += 32;
        }
        if (x < 0) {
          --lv;
          continue;
        }
        map[lv] = x;
        ++lv;
        build = true;
      }
    }
  }
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(count, hits);
}

// Checks a pattern and lays it out for the kernel.
reset_status compile_pattern(const reset_pattern* p, PatternDev* d) {
  if (!p) return arg_fail("NULL pattern");
  const int k = p->k;
  if (k < 3 || k > kPatMax) return arg_fail("pattern k must be in 3..RESET_PATTERN_MAX");
  if (p->flags & ~(RESET_PATTERN_RESTRICT | RESET_PATTERN_DISTINCT))
    return arg_fail("unknown pattern flags");
  if (!p->offsets || !p->backward) return arg_fail("NULL pattern offsets or backward");
  if (p->offsets[0] != 0 || p->offsets[1] != 1 || p->backward[0] != 0)
    return arg_fail("pattern level 1 must list exactly vertex 0");
  std::memset(d, 0, sizeof(*d));
  d->k = k;
  d->flags = p->flags;
  for (int l = 0; l < k; ++l) {
    d->restr[l] = p->restriction ? p->restriction[l] : -1;
    d->reuse[l] = p->reuse ? p->reuse[l] : -1;
    d->filt[l] = 1;
  }
  if (d->restr[0] != -1) return arg_fail("restriction[0] must be -1");
  for (int l = 1; l < k; ++l)
    if (d->restr[l] < -1 || d->restr[l] >= l)
      return arg_fail("restriction[l] must be -1 or an earlier vertex");
  for (int l = 0; l < k; ++l) {
    const int r = d->reuse[l];
    if (r == -1) continue;
    if (l < 3 || r < 2 || r >= l) return arg_fail("reuse[l] must be -1 or a level in [2, l)");
    d->filt[r] = 0;
  }
  for (int l = 2; l < k; ++l) {
    const int a = p->offsets[l - 1], z = p->offsets[l];
    if (z < a || z - a > kPatMax) return arg_fail("pattern offsets must rise by at most RESET_PATTERN_MAX");
    int minus = 0, nb = 0;
    for (int i = a; i < z; ++i) {
      const int j = p->backward[i];
      if (j == -1) {
        ++minus;
        continue;
      }
      if (j < 0 || j >= l) return arg_fail("backward entries must be -1 or earlier vertices");
      d->back[l][nb++] = j;
    }
    if (minus != (d->reuse[l] >= 0 ? 1 : 0))
      return arg_fail("a reusing level lists exactly one -1, other levels none");
    if (nb == 0 && d->reuse[l] < 0)
      return arg_fail("every level needs a listed vertex or a reused set");
    d->nb[l] = nb;
  }
  // The reusing k-clique chain (SMOG's Q0, Q3, Q5, Q7): level 2 lists
  // {0, 1}, every later level l reuses l-1 and lists l-1; with no active
  // check its count is the k-clique search's.
  bool checks = (d->flags & RESET_PATTERN_DISTINCT) != 0;
  for (int l = 1; l < k; ++l) checks |= (d->flags & RESET_PATTERN_RESTRICT) && d->restr[l] >= 0;
  bool chain = !checks && d->nb[2] == 2 && d->reuse[2] < 0 &&
               ((d->back[2][0] == 0 && d->back[2][1] == 1) || (d->back[2][0] == 1 && d->back[2][1] == 0));
  for (int l = 3; l < k && chain; ++l)
    chain = d->reuse[l] == l - 1 && d->nb[l] == 1 && d->back[l][0] == l - 1;
  d->chain = chain ? 1 : 0;
  d->fuse = k >= 4 && ((d->reuse[k - 1] >= 0 && d->nb[k - 1] == 0) ||
                       (d->reuse[k - 1] < 0 && d->nb[k - 1] == 1));
  d->pair = 0;
  if (k >= 4 && d->reuse[k - 1] < 0 && d->nb[k - 1] == 2) {
    const int a = d->back[k - 1][0], c = d->back[k - 1][1];
    if ((a == k - 2) != (c == k - 2)) {
      d->pair = 1;
      d->pair_a = a == k - 2 ? c : a;
    }
  }
  return RESET_OK;
}

// SMOG's query patterns (SMOG/SMOG_hie/script_hie.py:85-152) and the graph
// each is counted on (SMOG/SMOG_hie/common_hie.cu:72-85).
struct NamedPattern {
  const char* name;
  int32_t k, flags, oriented;
  int32_t offsets[kPatMax], backward[2 * kPatMax], restriction[kPatMax], reuse[kPatMax];
  bool has_restriction, has_reuse;
};

constexpr int32_t kRD = RESET_PATTERN_RESTRICT | RESET_PATTERN_DISTINCT;
const NamedPattern kNamed[] = {
    {"Q0", 3, 0, 1, {0, 1, 3}, {0, 0, 1}, {}, {}, false, false},
    {"Q1", 4, RESET_PATTERN_RESTRICT, 0, {0, 1, 2, 4}, {0, 0, 1, 2}, {-1, 0, 1, 0}, {},
     true, false},
    {"Q2", 4, RESET_PATTERN_RESTRICT, 0, {0, 1, 3, 5}, {0, 0, 1, 1, 2}, {-1, -1, 1, 0}, {},
     true, false},
    {"Q3", 4, 0, 1, {0, 1, 3, 5}, {0, 0, 1, -1, 2}, {}, {-1, -1, -1, 2}, false, true},
    {"Q4", 5, kRD, 0, {0, 1, 3, 5, 6}, {0, 0, 1, -1, 2, -1}, {-1, 0, -1, 2, -1},
     {-1, -1, -1, 2, 2}, true, true},
    {"Q5", 5, 0, 1, {0, 1, 3, 5, 7}, {0, 0, 1, -1, 2, -1, 3}, {}, {-1, -1, -1, 2, 3}, false,
     true},
    {"Q6", 5, kRD, 0, {0, 1, 3, 4, 6}, {0, 0, 1, -1, 2, 3}, {-1, 0, -1, 2, -1},
     {-1, -1, -1, 2, -1}, true, true},
    {"Q7", 6, 0, 1, {0, 1, 3, 5, 7, 9}, {0, 0, 1, -1, 2, -1, 3, -1, 4}, {},
     {-1, -1, -1, 2, 3, 4}, false, true},
    {"Q8", 5, RESET_PATTERN_RESTRICT, 0, {0, 1, 3, 5, 6}, {0, 0, 1, -1, 2, -1},
     {-1, 0, -1, -1, 3}, {-1, -1, -1, 2, 3}, true, true},
};

}  // namespace
}  // namespace rst

using namespace rst;

extern "C" reset_status reset_pattern_named(const char* name, reset_pattern* out,
                                            int32_t* oriented) {
  if (!name || !out) return arg_fail("NULL name or pattern");
  for (const NamedPattern& q : kNamed) {
    if (std::strcmp(q.name, name) != 0) continue;
    out->k = q.k;
    out->flags = q.flags;
    out->offsets = q.offsets;
    out->backward = q.backward;
    out->restriction = q.has_restriction ? q.restriction : nullptr;
    out->reuse = q.has_reuse ? q.reuse : nullptr;
    if (oriented) *oriented = q.oriented;
    return RESET_OK;
  }
  return arg_fail("unknown pattern name (SMOG's table has Q0..Q8)");
}

extern "C" reset_status reset_pattern_count(const reset_table* t, const int32_t* d_off,
                                            const int32_t* d_cols, int64_t m,
                                            const reset_pattern* p, uint64_t* d_count,
                                            reset_stream_t stream) {
  if (!t || !d_count) return arg_fail("NULL table or count");
  PatternDev pat;
  {
    const reset_status s = compile_pattern(p, &pat);
    if (s != RESET_OK) return s;
  }
  if (m < 0 || m > INT32_MAX) return arg_fail("m out of range");
  if (m > 0 && (!d_off || !d_cols)) return arg_fail("NULL offsets or cols");
  if (d_off != t->build_off || m != t->m)
    return arg_fail("d_off/m must be the CSR the table was built on");
  if (pat.chain) return reset_clique_count(t, d_off, d_cols, m, pat.k, d_count, stream);
  cudaStream_t st = as_stream(stream);
  RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), st));
  if (m == 0 || t->n == 0) return RESET_OK;
  RowStats stats;
  RST_CHECK(row_stats(d_off, d_cols, t->n, m, st, &stats));
  const int32_t cap = stats.longest > 0 ? (int32_t)stats.longest : 1;
  const int sorted = stats.ascending() ? 1 : 0;
  const int64_t rows = pat.k > 3 ? pat.k - 3 : 1;
  const int sms = sm_count();
  const void* kf = t->hier ? (const void*)pattern_kernel<true> : (const void*)pattern_kernel<false>;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kf, kPtThreads, 0);
  if (per_sm < 1) per_sm = 1;
  const size_t per_block = sizeof(int32_t) * (size_t)cap * (size_t)rows * kPtWarps;
  const int64_t fit = std::max<int64_t>(1, (int64_t)(kPtScratchBudget / per_block));
  int64_t grid = std::min<int64_t>((int64_t)sms * per_sm, fit);
  // bit rows: all vertices', or those of the longest rows that fit
  BitRows br{nullptr, nullptr, ((int64_t)t->n + 127) / 128 * 4};
  int64_t bit_rows = 0;
  int bit_min = 0;
  const bool short_rows = stats.longest <= kShortRows;
  if (stats.outside == 0 && !short_rows) {
    const int64_t squares = (int64_t)std::min<unsigned long long>(stats.squares, kBitBudget);
    const int64_t budget = std::min(kBitBudget, std::max<int64_t>(1 << 20, kBitPerSquare * squares));
    const int64_t most = budget / (4 * br.words);
    if (t->n <= most) {
      bit_rows = t->n;
    } else {
      for (int i = 30; i >= 0 && (1 << i) >= kBitMinRow; --i) {
        if (bit_rows + (int64_t)stats.lg_rows[i] > most) break;
        bit_rows += (int64_t)stats.lg_rows[i];
        bit_min = 1 << i;
      }
    }
  }
  // parts of long start edges: there are at most 2 * squares / part of them
  int part = 0;
  int64_t max_parts = 0;
  if (pat.k > 3 && !short_rows) {
    const int least = pat.k > 4 ? kPartDeep : kPartFlat;
    const unsigned long long by_count = 2 * stats.squares / (unsigned long long)kMaxParts;
    part = (int)std::min<unsigned long long>(std::max<unsigned long long>(least, by_count), INT_MAX);
    max_parts = (int64_t)(2 * stats.squares / part) + 1;
  }
  // up to 32 start edges at a time, fewer where that leaves warps idle; warps
  // beyond the work items (parts, grabs of edges) have nothing to do
  int lg_grab = 0;
  while (lg_grab < 5 && (m >> (lg_grab + 1)) >= grid * kPtWarps * 8) ++lg_grab;
  grid = std::min<int64_t>(grid, ((m >> lg_grab) + 1 + max_parts + kPtWarps - 1) / kPtWarps);
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  bool some = false;
  size_t sz_scr = 0, sz_bits = 0, sz_row = 0, sz_list = 0;
  char* base = nullptr;
  auto allocate = [&]() {
    some = bit_rows > 0 && bit_rows < t->n;
    sz_scr = al(per_block * (size_t)grid);
    sz_bits = al(sizeof(uint32_t) * (size_t)(bit_rows * br.words));
    sz_row = some ? al(sizeof(int32_t) * (size_t)t->n) : 0;
    sz_list = al(sizeof(int4) * (size_t)max_parts);
    return scratch_malloc(reinterpret_cast<void**>(&base),
                          sz_scr + sz_bits + sz_row + sz_list + 256, st);
  };
  if (allocate() != cudaSuccess) {  // without memory for them: no bit rows, no parts
    cudaGetLastError();
    bit_rows = 0;
    part = 0;
    max_parts = 0;
    RST_CUDA(allocate());
  }
  int32_t* scr = reinterpret_cast<int32_t*>(base);
  uint32_t* bits = reinterpret_cast<uint32_t*>(base + sz_scr);
  int32_t* row = reinterpret_cast<int32_t*>(base + sz_scr + sz_bits);
  int4* list = reinterpret_cast<int4*>(base + sz_scr + sz_bits + sz_row);
  // [0..1] work cursors, the visits (u64), then the listed parts,
  // self-loops, bit rows
  auto* cursor = reinterpret_cast<unsigned long long*>(base + sz_scr + sz_bits + sz_row + sz_list);
  auto* visits = cursor + 2;
  int32_t* ctr = reinterpret_cast<int32_t*>(cursor + 3);
  const int warp_grid = (int)std::min<int64_t>(((int64_t)t->n + 7) / 8, (int64_t)sms * 8);
  cudaError_t e = cudaMemsetAsync(cursor, 0, 256, st);
  if (e == cudaSuccess && bit_rows > 0) {
    br.bits = bits;
    e = cudaMemsetAsync(bits, 0, sizeof(uint32_t) * (size_t)(bit_rows * br.words), st);
    if (e == cudaSuccess && some) {
      br.row = row;
      note_launch();
      bit_assign_kernel<<<warp_grid, 256, 0, st>>>(t->d_desc, t->n, bit_min, row, ctr + 2);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
      note_launch();
      bit_fill_kernel<<<warp_grid, 256, 0, st>>>(t->d_desc, d_cols, t->n, br.row, br.words, bits,
                                                 ctr + 1);
      e = cudaGetLastError();
    }
  }
  // co-degrees, where the paired last level has no bound; without memory for
  // them the walk does as well
  const bool bounded = (pat.flags & RESET_PATTERN_RESTRICT) && pat.restr[pat.k - 1] >= 0;
  const int64_t co_bytes = (int64_t)sizeof(int32_t) * t->n * t->n;
  // (the visits at most: of |C_2| or |C_2|^2 per edge)
  const double most_visits = pat.k > 4 ? stats.cubes : (double)stats.squares;
  const bool co_may = pat.pair && sorted && !bounded && bit_rows == t->n && part > 0 &&
                      co_bytes <= kCoBudget &&
                      (t->n <= kCoSmall ||
                       most_visits >= (double)t->n * t->n * t->n / kCoVisits);
  int32_t* co = nullptr;
  if (e == cudaSuccess && part > 0) {
    const int step = (int)std::max<int64_t>(1, m >> 10);  // about 2^10 edges looked at
    note_launch();
    pattern_parts_kernel<<<warp_grid, 256, 0, st>>>(t->d_desc, d_cols, t->n, m, pat, part, list,
                                                    ctr, co_may && t->n > kCoSmall ? br : BitRows{}, step,
                                                    visits);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && co_may) {
    if (scratch_malloc(reinterpret_cast<void**>(&co), (size_t)co_bytes, st) != cudaSuccess) {
      cudaGetLastError();
      co = nullptr;
    } else {
      const unsigned tiles = (unsigned)((t->n + kCoTile - 1) / kCoTile);
      note_launch();
      codegree_kernel<<<dim3(tiles, tiles), 256, 0, st>>>(bits, t->n, (int)br.words, visits, co);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) {
    note_launch();
#define PT_LAUNCH(H)                                                                           \
  pattern_kernel<H><<<(int)grid, kPtThreads, 0, st>>>(                                         \
      t->d_desc, d_off, d_cols, t->d_chunk_row, t->n, m, t->d_table, t->bucket_num, t->bucket, \
      t->lg_max, pat, sorted, br, ctr + 1, co, visits, list, ctr, part, lg_grab, scr, cap,    \
      reinterpret_cast<unsigned long long*>(d_count), cursor, t->d_status)
    if (t->hier) PT_LAUNCH(true); else PT_LAUNCH(false);
#undef PT_LAUNCH
    e = cudaGetLastError();
  }
  if (co) cudaFreeAsync(co, st);
  cudaFreeAsync(base, st);
  if (e != cudaSuccess) return cuda_fail(e, "pattern_kernel", __FILE__, __LINE__);
  return RESET_OK;
}
