// k-clique counting on an oriented graph: the clique DFS of SMOG
// (SMOG/SMOG_hie/subgraph_match_hie.cu:58-247, DFSKernelForClique) over this
// library's tables.
//
// With edges oriented low -> high (degree, then id), every k-clique is found
// exactly once, from its first two vertices:
//   count = sum over edges (u, v) of chains w_1 .. w_{k-2},
//           w_1 in C_0 = N+(u) ∩ N+(v), w_{j+1} in C_j = C_{j-1} ∩ N+(w_j).
// Two forms:
//  * clique_bits_kernel, rows strictly ascending (sets): the graph on N+(u)
//    as bit rows in shared memory, found by one round of hash probes per
//    vertex; per edge, the sub-graph on C_0 packed into bit rows of |C_0|
//    bits, on which the remaining levels are AND + popcount.
//  * clique_k_kernel, any rows (repeated or unordered keys, whose
//    multiplicity counts), and edges too large for the bit rows: one warp
//    per edge, every candidate set found by hash probes.
#include <algorithm>

#include "probe_common.cuh"

namespace rst {
namespace {

constexpr int kCqThreads = 256;
constexpr int kCqWarps = kCqThreads / 32;

// k-cliques, 4 <= k <= kMaxClique, as a warp-level depth-first search over
// hash-probe intersections.  An edge (u, v) fixes two vertices;
// the candidates of the third are C0 = N+(u) ∩ N+(v); after picking w from
// C_j, the candidates of the next vertex are C_{j+1} = C_j ∩ N+(w) (the
// keys of C_j probed into w's table, hits compacted into the warp's scratch
// row of level j+1).  The last level is only counted: sum over w in C_j of
// |C_j ∩ N+(w)|.  Scratch: k-3 rows of `cap` ints per warp (levels 0..k-4).
// With elist, only the edges elist[0 .. *n_list) are searched.
constexpr int kMaxClique = 16;

template <bool HIER>
__global__ void __launch_bounds__(kCqThreads)
    clique_k_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ off,
                    const int32_t* __restrict__ cols, const int32_t* __restrict__ chunk_row,
                    int32_t n, int64_t m, const int32_t* __restrict__ table, int64_t bn, int b,
                    int lg_max, int k, int32_t* __restrict__ scratch, int32_t cap,
                    const int32_t* __restrict__ elist, const int32_t* __restrict__ n_list,
                    unsigned long long* __restrict__ count,
                    unsigned long long* __restrict__ cursor, int32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int levels = k - 3;
  int32_t* Cbase = scratch + gw * (int64_t)cap * levels;
  const int64_t me = min(m, (int64_t)__ldg(off + n));
  const int64_t n_chunks = (me + 31) >> 5;
  unsigned long long hits = 0;
  int sz[kMaxClique], it[kMaxClique];
  int u = 0;
  for (;;) {
    unsigned long long cc = 0;
    if (lane == 0) cc = atomicAdd(cursor, 1ull);
    int64_t e = (int64_t)__shfl_sync(kFull, cc, 0);
    if (elist) {
      if (e >= *n_list) break;
      e = elist[e];
    }
    if (e >= me) break;
    // row of edge e: largest u with off[u] <= e, searched between the rows
    // of the 32-edge chunks around e (lane 0)
    if (lane == 0) {
      const int64_t c = e >> 5;
      int lo = __ldg(chunk_row + c);
      int hi = c + 1 < n_chunks ? __ldg(chunk_row + c + 1) : n - 1;
      if ((unsigned)lo >= (unsigned)n) lo = 0;
      if (hi < lo || hi >= n) hi = n - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= e) lo = mid; else hi = mid - 1;
      }
      u = lo;
    }
    u = __shfl_sync(kFull, u, 0);
    const int v = __ldg(cols + e);
    if ((unsigned)v >= (unsigned)n) {
      if (lane == 0) atomicOr(status, kErrBadId);
      continue;
    }
    const int4 du = __ldg(desc + u), dv = __ldg(desc + v);
    const bool sw = du.y > dv.y;
    const int4 A = sw ? dv : du, Bd = sw ? du : dv;
    const int32_t* tb = table + desc_toff(Bd);
    const int blg = desc_lg(Bd);
    // level 0: C0 = N+(u) ∩ N+(v)
    int32_t* C0 = Cbase;
    int nw = 0;
    for (int j0 = 0; j0 < A.y; j0 += 32) {
      const int j = j0 + lane;
      bool in = false;
      int x = 0;
      if (j < A.y) {
        x = __ldg(cols + A.x + j);
        in = probe_key<HIER>(x, tb, blg, lg_max, bn, b, status);
      }
      const unsigned msk = __ballot_sync(kFull, in);
      if (in) {
        const int pos = nw + __popc(msk & lt);
        if (pos < cap) C0[pos] = x;
      }
      nw += __popc(msk);
    }
    if (nw > cap) {  // cannot happen when cap >= the largest out-degree
      if (lane == 0) atomicOr(status, kErrProbeLimit);
      continue;
    }
    __syncwarp();
    sz[0] = nw;
    it[0] = 0;
    int lv = 0;  // warp-uniform depth
    while (lv >= 0) {
      int32_t* C = Cbase + (int64_t)lv * cap;
      if (lv == k - 4) {  // last level: count, do not store
        for (int t = 0; t < sz[lv]; ++t) {
          const int4 dw = __ldg(desc + C[t]);
          if (dw.y == 0) continue;
          const int32_t* tw = table + desc_toff(dw);
          const int wlg = desc_lg(dw);
          for (int j = lane; j < sz[lv]; j += 32)
            hits += probe_key<HIER>(C[j], tw, wlg, lg_max, bn, b, status);
        }
        --lv;
        continue;
      }
      if (it[lv] >= sz[lv]) {
        --lv;
        continue;
      }
      const int4 dw = __ldg(desc + C[it[lv]]);
      ++it[lv];
      int32_t* D = C + cap;
      int nd = 0;
      if (dw.y > 0) {
        const int32_t* tw = table + desc_toff(dw);
        const int wlg = desc_lg(dw);
        for (int j0 = 0; j0 < sz[lv]; j0 += 32) {
          const int j = j0 + lane;
          bool in = false;
          int x = 0;
          if (j < sz[lv]) {
            x = C[j];
            in = probe_key<HIER>(x, tw, wlg, lg_max, bn, b, status);
          }
          const unsigned msk = __ballot_sync(kFull, in);
          if (in) D[nd + __popc(msk & lt)] = x;
          nd += __popc(msk);
        }
      }
      __syncwarp();
      if (nd == 0) continue;  // no clique grows from this pick
      ++lv;
      sz[lv] = nd;
      it[lv] = 0;
    }
    __syncwarp();
  }
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(count, hits);
}

// ------------------------------------------------------------ bit rows ----
//
// One CTA per vertex u (or a share of its edges) with row length
// d = |N+(u)| > 32; one warp per shorter row.
//  1. A[i], i < d: the positions j < d with N+(u)[j] in N+(N+(u)[i]), as
//     W = ceil(d/32) words: d^2 probes, 32 to a ballot, in shared memory.
//  2. Per edge (u, N+(u)[i]): C_0 = A[i].  Its c = |C_0| positions are listed
//     and the graph on them packed into c rows of ceil(c/32) words (one bit
//     test per pair), held in the warp's own 2 KB; edges with c > 128 are
//     packed by the whole CTA over all warps' regions.
//  3. The chain w_1 .. w_{k-2} on the packed rows: a lane per w_1, nested
//     loops over the set bits, the last level a popcount.
// Packing matters: |C_0| is ~30-120 where d is 250 (R-MAT scale 16), so a
// step touches 1-4 words, held in registers, instead of a row of N+(u), and
// each costs a few instructions where a hash probe costs ~30 and a dependent
// load.  Bound by instruction issue; measured beside the launch below.
constexpr int kCbThreads = 512;
constexpr int kCbWarps = kCbThreads / 32;
constexpr int kCbPackInts = 512;              // a warp's packed rows: 128 rows of 4 words
constexpr int kCbWarpMax = 128;               // |C_0| a warp packs
constexpr int kCbCtaMax = 512;                // |C_0| a CTA packs (16 words a row)
constexpr int kCbRowMax = 1216;               // longest row held as bits
constexpr int kCbPack = kCbWarps * kCbPackInts;  // ints of packed rows per CTA
static_assert(kCbCtaMax * (kCbCtaMax / 32) <= kCbPack, "packed rows of a CTA edge");
static_assert(kCbRowMax <= kCbPack, "the row's keys overlay the packed rows");

// Words of shared memory for the bit rows of a vertex with d out-edges.  An
// odd row stride spreads equal word indices of different rows over the banks.
__host__ __device__ __forceinline__ int cb_stride(int d) { return ((d + 31) >> 5) | 1; }

// Chains below the set D: T(D, 0) = |D|, T(D, r) = sum over x in D of
// T(D ∩ B[x], r - 1).
template <int WP, int R>
struct Chains {
  static __device__ __forceinline__ unsigned long long count(const uint32_t* B,
                                                             const uint32_t (&D)[WP]) {
    unsigned long long t = 0;
#pragma unroll
    for (int w = 0; w < WP; ++w) {
      uint32_t bits = D[w];
      while (bits) {
        const int x = w * 32 + __ffs(bits) - 1;
        bits &= bits - 1;
        const uint32_t* Bx = B + x * WP;
        uint32_t E[WP];
#pragma unroll
        for (int v = 0; v < WP; ++v) E[v] = D[v] & Bx[v];
        t += Chains<WP, R - 1>::count(B, E);
      }
    }
    return t;
  }
};
template <int WP>
struct Chains<WP, 0> {
  static __device__ __forceinline__ unsigned count(const uint32_t*, const uint32_t (&D)[WP]) {
    unsigned t = 0;
#pragma unroll
    for (int w = 0; w < WP; ++w) t += __popc(D[w]);
    return t;
  }
};

// T(D, r) for any r <= kMaxClique with an explicit stack.
template <int WP>
__device__ __noinline__ unsigned long long chains_deep(const uint32_t* B, const uint32_t* D0,
                                                       int r) {
  uint32_t D[kMaxClique][WP], todo[kMaxClique][WP];
  unsigned long long t = 0;
  for (int w = 0; w < WP; ++w) D[0][w] = todo[0][w] = D0[w];
  int lv = 0;
  while (lv >= 0) {
    int x = -1;
    for (int w = 0; w < WP && x < 0; ++w)
      if (todo[lv][w]) {
        x = w * 32 + __ffs(todo[lv][w]) - 1;
        todo[lv][w] &= todo[lv][w] - 1;
      }
    if (x < 0) {
      --lv;
      continue;
    }
    unsigned n = 0;
    uint32_t* E = D[lv + 1];
    for (int w = 0; w < WP; ++w) {
      E[w] = D[lv][w] & B[x * WP + w];
      n += __popc(E[w]);
    }
    if (n == 0) continue;
    if (lv + 1 == r) {
      t += n;
    } else {
      ++lv;
      for (int w = 0; w < WP; ++w) todo[lv][w] = E[w];
    }
  }
  return t;
}

// Sum over rows a = t, t + nt, .. < rows of T(B[a], levels - 1): this
// thread's share of the chains of length `levels` + 1 of the packed graph
// (levels >= 2).
template <int WP>
__device__ __forceinline__ unsigned long long count_rows(const uint32_t* B, int rows, int levels,
                                                         int t, int nt) {
  unsigned long long hits = 0;
  for (int a = t; a < rows; a += nt) {
    uint32_t D[WP];
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < WP; ++w) any |= D[w] = B[a * WP + w];
    if (!any) continue;
    if (levels == 2)
      hits += Chains<WP, 1>::count(B, D);
    else if (levels == 3)
      hits += Chains<WP, 2>::count(B, D);
    else
      hits += chains_deep<WP>(B, D, levels - 1);
  }
  return hits;
}

// Rows a = t, t + nt, .. < c of the graph on the listed positions, packed:
// bit q of row a is bit list[q] of A[list[a]].
template <int WP>
__device__ __forceinline__ void pack_rows(const uint32_t* A, int stride, const uint16_t* list,
                                          int c, uint32_t* B, int t, int nt) {
  for (int a = t; a < c; a += nt) {
    const uint32_t* Ra = A + list[a] * stride;
#pragma unroll
    for (int w = 0; w < WP; ++w) {
      const int q1 = min(32, c - w * 32);
      uint32_t word = 0;
      for (int q = q1 - 1; q >= 0; --q) {
        const int j = list[w * 32 + q];
        // bit j of the row moved to the top, then shifted in from below
        word = __funnelshift_l(Ra[j >> 5] << (31 - (j & 31)), word, 1);
      }
      B[a * WP + w] = word;
    }
  }
}

// The set positions of a row of W words, ascending, into list (warp).
__device__ __forceinline__ void list_bits(const uint32_t* Ai, int W, uint16_t* list) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int w0 = 0; w0 < W; w0 += 32) {
    const int w = w0 + lane;
    uint32_t bits = w < W ? Ai[w] : 0;
    int total;
    int pos = base + warp_excl_scan(__popc(bits), &total);
    while (bits) {
      list[pos++] = (uint16_t)(w * 32 + __ffs(bits) - 1);
      bits &= bits - 1;
    }
    base += total;
  }
}

// A probe of set dv (all lanes of the warp; inactive lanes pass act false).
template <bool HIER>
__device__ __forceinline__ bool probe_set(int x, bool act, const int4& dv,
                                          const int32_t* __restrict__ table, int64_t bn, int b,
                                          int lg_max, int32_t* status) {
  if (!act) return false;
  const int32_t* tb = table + desc_toff(dv);
  const int lg = desc_lg(dv);
  const int h = home_bucket<HIER>(x, lg, lg_max);
  const int s0 = __ldg(tb + h);
  const int s1 = b > 1 ? __ldg(tb + h + bn) : -1;
  return probe_resolve2<HIER>(x, s0, s1, tb, lg, h, bn, b, status);
}

// Work lists: items (u, first edge, end) of CTA work and the short rows.
// A vertex's work grows about as d^3; one with more than 1/parts of the sum
// is cut into shares of its edges (each share finds the bit rows again, which
// costs d^2 probes, so a share has at least 16 edges).  Edges of rows above
// dcap go to elist.  ctr: [0] items, [1] short rows, [4] listed edges.
__global__ void clique_items_kernel(const int4* __restrict__ desc, int32_t n, int64_t m, int dcap,
                                    double d3_sum, int parts, int4* __restrict__ items,
                                    int32_t* __restrict__ small, int32_t* __restrict__ elist,
                                    int32_t* __restrict__ ctr) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n;
       u += (int64_t)gridDim.x * blockDim.x) {
    const int4 du = __ldg(desc + u);
    const int d = (int)min((int64_t)du.y, m - du.x);
    if (d <= 0) continue;
    if (d <= 32) {
      small[atomicAdd(ctr + 1, 1)] = (int)u;
    } else if (d <= dcap) {
      const double share = (double)d * d * d / d3_sum * parts;
      const int ns = max(1, min((int)share + 1, d / 16));
      const int at = atomicAdd(ctr + 0, ns);
      for (int s = 0; s < ns; ++s)
        items[at + s] = make_int4((int)u, (int)((int64_t)d * s / ns),
                                  (int)((int64_t)d * (s + 1) / ns), 0);
    } else {
      const int at = atomicAdd(ctr + 4, d);
      for (int i = 0; i < d; ++i) elist[at + i] = du.x + i;
    }
  }
}

template <bool HIER>
__global__ void __launch_bounds__(kCbThreads, 2)
    clique_bits_kernel(const int4* __restrict__ desc, const int32_t* __restrict__ cols,
                       int32_t n, int64_t m, const int32_t* __restrict__ table, int64_t bn, int b,
                       int lg_max, int k, const int4* __restrict__ items,
                       const int32_t* __restrict__ small, int32_t* __restrict__ elist,
                       int32_t* __restrict__ ctr, unsigned long long* __restrict__ count,
                       int32_t* __restrict__ status) {
  extern __shared__ __align__(16) uint32_t cb_sm[];
  __shared__ uint16_t s_list[kCbWarps][kCbWarpMax];  // (a CTA edge's list: the first rows)
  __shared__ uint16_t s_big[kCbRowMax];
  __shared__ int s_item, s_next, s_nbig;
  static_assert(kCbCtaMax <= kCbWarps * kCbWarpMax, "list of a CTA edge");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* P = cb_sm;            // packed rows; the row's keys while A is built
  uint32_t* A = cb_sm + kCbPack;  // bit rows of u
  uint32_t* Pw = P + warp * kCbPackInts;
  uint16_t* Lw = s_list[warp];
  const int n_items = ctr[0], n_small = ctr[1];
  unsigned long long hits = 0;

  // ---- rows of more than 32 keys
  for (;;) {
    if (tid == 0) s_item = atomicAdd(ctr + 2, 1);
    __syncthreads();
    const int it = s_item;
    if (it >= n_items) break;
    const int4 item = __ldg(items + it);
    const int4 du = __ldg(desc + item.x);
    const int d = (int)min((int64_t)du.y, m - du.x);
    const int W = (d + 31) >> 5, S = cb_stride(d);
    int32_t* keys = reinterpret_cast<int32_t*>(P);
    for (int j = tid; j < d; j += kCbThreads) keys[j] = __ldg(cols + du.x + j);
    if (tid == 0) {
      s_next = item.y;
      s_nbig = 0;
    }
    __syncthreads();
    for (int i = warp; i < d; i += kCbWarps) {
      const int v = keys[i];
      const bool ok = (unsigned)v < (unsigned)n;
      if (!ok && lane == 0) atomicOr(status, kErrBadId);
      const int4 dv = ok ? __ldg(desc + v) : make_int4(0, 0, 0, 0);
      uint32_t* Ai = A + i * S;
#pragma unroll 4
      for (int w = 0; w < W; ++w) {
        const int j = w * 32 + lane;
        const bool act = j < d && dv.y > 0;
        const unsigned word = __ballot_sync(
            kFull, probe_set<HIER>(act ? keys[j] : 0, act, dv, table, bn, b, lg_max, status));
        if (lane == 0) Ai[w] = word;
      }
    }
    __syncthreads();
    // edges i of this share, one per warp
    for (;;) {
      int i = 0;
      if (lane == 0) i = atomicAdd(&s_next, 1);
      i = __shfl_sync(kFull, i, 0);
      if (i >= item.z) break;
      const uint32_t* Ai = A + i * S;
      int c = 0;
      for (int w = lane; w < W; w += 32) c += __popc(Ai[w]);
      c = __reduce_add_sync(kFull, c);
      if (c == 0) continue;
      if (k == 4) {  // sum over j in C_0 of |C_0 ∩ N+(j)|, on the rows of u
        unsigned t = 0;
        const bool listed = c <= kCbWarpMax;
        if (listed) {
          list_bits(Ai, W, Lw);
          __syncwarp();
        }
        for (int q = lane; q < (listed ? c : d); q += 32) {
          const int j = listed ? Lw[q] : q;
          if (!listed && !((Ai[j >> 5] >> (j & 31)) & 1u)) continue;
          const uint32_t* Aj = A + j * S;
          for (int w = 0; w < W; ++w) t += __popc(Ai[w] & Aj[w]);
        }
        hits += t;
        __syncwarp();
        continue;
      }
      if (c > kCbWarpMax) {  // the whole CTA's, below
        if (lane == 0) s_big[atomicAdd(&s_nbig, 1)] = (uint16_t)i;
        continue;
      }
      list_bits(Ai, W, Lw);
      __syncwarp();
      if (c <= 32) {
        pack_rows<1>(A, S, Lw, c, Pw, lane, 32);
        __syncwarp();
        hits += count_rows<1>(Pw, c, k - 3, lane, 32);
      } else if (c <= 64) {
        pack_rows<2>(A, S, Lw, c, Pw, lane, 32);
        __syncwarp();
        hits += count_rows<2>(Pw, c, k - 3, lane, 32);
      } else {
        pack_rows<4>(A, S, Lw, c, Pw, lane, 32);
        __syncwarp();
        hits += count_rows<4>(Pw, c, k - 3, lane, 32);
      }
      __syncwarp();
    }
    __syncthreads();
    const int nbig = s_nbig;
    for (int g = 0; g < nbig; ++g) {
      const int i = s_big[g];
      const uint32_t* Ai = A + i * S;
      int c = 0;
      for (int w = lane; w < W; w += 32) c += __popc(Ai[w]);
      c = __reduce_add_sync(kFull, c);  // the same in every warp
      if (c > kCbCtaMax) {
        if (tid == 0) elist[atomicAdd(ctr + 4, 1)] = du.x + i;
        continue;
      }
      uint16_t* L = &s_list[0][0];
      if (warp == 0) list_bits(Ai, W, L);
      __syncthreads();
      if (c <= 256)
        pack_rows<8>(A, S, L, c, P, tid, kCbThreads);
      else
        pack_rows<16>(A, S, L, c, P, tid, kCbThreads);
      __syncthreads();
      if (c <= 256)
        hits += count_rows<8>(P, c, k - 3, tid, kCbThreads);
      else
        hits += count_rows<16>(P, c, k - 3, tid, kCbThreads);
      __syncthreads();
    }
  }

  // ---- rows of at most 32 keys: a warp each, the bit rows as packed rows
  __syncthreads();
  for (;;) {
    int q = 0;
    if (lane == 0) q = atomicAdd(ctr + 3, 1);
    q = __shfl_sync(kFull, q, 0);
    if (q >= n_small) break;
    const int4 du = __ldg(desc + __ldg(small + q));
    const int d = (int)min((int64_t)du.y, m - du.x);
    const int x = lane < d ? __ldg(cols + du.x + lane) : -1;
    const bool ok = (unsigned)x < (unsigned)n;
    if (lane < d && !ok) atomicOr(status, kErrBadId);
    const int4 mine = ok ? __ldg(desc + x) : make_int4(0, 0, 0, 0);
    uint32_t row = 0;
    for (int i = 0; i < d; ++i) {
      int4 dv = make_int4(0, __shfl_sync(kFull, mine.y, i), 0, 0);
      if (dv.y == 0) continue;
      dv.z = __shfl_sync(kFull, mine.z, i);
      dv.w = __shfl_sync(kFull, mine.w, i);
      const unsigned word = __ballot_sync(
          kFull, probe_set<HIER>(x, lane < d, dv, table, bn, b, lg_max, status));
      if (lane == i) row = word;
    }
    Pw[lane] = row;
    __syncwarp();
    hits += count_rows<1>(Pw, d, k - 2, lane, 32);
    __syncwarp();
  }
  hits = warp_sum_u64(hits);
  if (lane == 0 && hits) atomicAdd(count, hits);
}

// One pass over a CSR for RowStats.
__global__ void __launch_bounds__(256)
    row_stats_kernel(const int32_t* __restrict__ off, const int32_t* __restrict__ cols,
                     int32_t n, int64_t m, RowStats* __restrict__ out) {
  __shared__ unsigned s_lg[32];
  if (threadIdx.x < 32) s_lg[threadIdx.x] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int mx = 0;
  unsigned long long desc_pairs = 0, edges = 0, outside = 0, d2 = 0;
  double d3 = 0;
  for (int64_t i = t0; i < n; i += stride) {
    const int a = __ldg(off + i), z = __ldg(off + i + 1), d = z - a;
    mx = max(mx, d);
    if (d > 0) {
      d2 += (unsigned long long)d * d;
      d3 += (double)d * d * d;
      atomicAdd(&s_lg[31 - __clz(d)], 1u);
    }
    if (z > a && z < m) edges += __ldg(cols + z - 1) >= __ldg(cols + z);
  }
  for (int64_t e = t0; e < m; e += stride) {
    const int x = __ldg(cols + e);
    outside += (unsigned)x >= (unsigned)n;
    if (e + 1 < m) desc_pairs += x >= __ldg(cols + e + 1);
  }
  for (int o = 16; o; o >>= 1) {
    mx = max(mx, __shfl_xor_sync(kFull, mx, o));
    desc_pairs += __shfl_xor_sync(kFull, desc_pairs, o);
    edges += __shfl_xor_sync(kFull, edges, o);
    outside += __shfl_xor_sync(kFull, outside, o);
    d2 += __shfl_xor_sync(kFull, d2, o);
    d3 += __shfl_xor_sync(kFull, d3, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out->longest, (unsigned long long)mx);
    if (desc_pairs) atomicAdd(&out->descending, desc_pairs);
    if (edges) atomicAdd(&out->straddling, edges);
    if (outside) atomicAdd(&out->outside, outside);
    if (d2) {
      atomicAdd(&out->squares, d2);
      atomicAdd(&out->cubes, d3);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32 && s_lg[threadIdx.x])
    atomicAdd(&out->lg_rows[threadIdx.x], (unsigned long long)s_lg[threadIdx.x]);
}

}  // namespace

reset_status row_stats(const int32_t* d_off, const int32_t* d_cols, int32_t n, int64_t m,
                       cudaStream_t st, RowStats* out) {
  *out = RowStats{};
  RowStats* d_st = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_st), sizeof(RowStats), st));
  cudaError_t e = cudaMemsetAsync(d_st, 0, sizeof(RowStats), st);
  if (e == cudaSuccess) {
    note_launch();
    row_stats_kernel<<<sm_count() * 4, 256, 0, st>>>(d_off, d_cols, n, m, d_st);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_st, sizeof(RowStats), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFreeAsync(d_st, st);
  if (e != cudaSuccess) return cuda_fail(e, "row stats", __FILE__, __LINE__);
  return RESET_OK;
}

namespace {

// The hash-probe search over all edges, or over elist[0 .. *n_list).
// *d_count is added to.
reset_status clique_probe(const reset_table* t, const int32_t* d_off, const int32_t* d_cols,
                          int64_t m, int32_t k, int64_t longest, const int32_t* elist,
                          const int32_t* n_list, unsigned long long* d_count, cudaStream_t st) {
  const int32_t cap = longest > 0 ? (int32_t)longest : 1;
  const void* kf = t->hier ? (const void*)clique_k_kernel<true> : (const void*)clique_k_kernel<false>;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kf, kCqThreads, 0);
  if (per_sm < 1) per_sm = 1;
  const int64_t grid = std::min<int64_t>((int64_t)sm_count() * per_sm, (m + kCqWarps - 1) / kCqWarps);
  const int64_t warps = grid * kCqWarps;
  const int64_t levels = k - 3;
  int32_t* d_scr = nullptr;
  unsigned long long* d_cur = nullptr;
  RST_CUDA(scratch_malloc(reinterpret_cast<void**>(&d_scr),
                          sizeof(int32_t) * (size_t)warps * (size_t)cap * (size_t)levels, st));
  cudaError_t e = scratch_malloc(reinterpret_cast<void**>(&d_cur), sizeof(unsigned long long), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_cur, 0, sizeof(unsigned long long), st);
  if (e == cudaSuccess) {
    note_launch();
#define CQ_LAUNCH(H)                                                                          \
  clique_k_kernel<H><<<(int)grid, kCqThreads, 0, st>>>(                                       \
      t->d_desc, d_off, d_cols, t->d_chunk_row, t->n, m, t->d_table, t->bucket_num, t->bucket, \
      t->lg_max, k, d_scr, cap, elist, n_list, d_count, d_cur, t->d_status)
    if (t->hier) CQ_LAUNCH(true); else CQ_LAUNCH(false);
#undef CQ_LAUNCH
    e = cudaGetLastError();
  }
  cudaFreeAsync(d_scr, st);
  if (d_cur) cudaFreeAsync(d_cur, st);
  if (e != cudaSuccess) return cuda_fail(e, "clique_k_kernel", __FILE__, __LINE__);
  return RESET_OK;
}

// The bit-row search (strictly ascending rows), or the hash-probe search where
// its lists find no memory.  *d_count, 0 before, is the count.
//
// R-MAT scale 16, k = 5 (15.7M triangles): hash probes 62 ms, bit rows 1.77 ms.
reset_status clique_bits(const reset_table* t, const int32_t* d_off, const int32_t* d_cols,
                         int64_t m, int32_t k, const RowStats& rs, unsigned long long* d_count,
                         cudaStream_t st) {
  const int sms = sm_count();
  // Shared memory for the longest row.  Up to 768 keys two CTAs fit an SM;
  // above it one, and rows above kCbRowMax are searched by hash probes.
  const int dcap = (int)std::min<unsigned long long>(rs.longest, kCbRowMax);
  const size_t smem = sizeof(uint32_t) * (kCbPack + (size_t)dcap * cb_stride(dcap));
  const void* kf =
      t->hier ? (const void*)clique_bits_kernel<true> : (const void*)clique_bits_kernel<false>;
  // (the same for every graph: other threads may be between here and a launch)
  RST_CUDA(cudaFuncSetAttribute(
      kf, cudaFuncAttributeMaxDynamicSharedMemorySize,
      (int)sizeof(uint32_t) * (kCbPack + kCbRowMax * cb_stride(kCbRowMax))));
  int per_sm = 0;
  RST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kf, kCbThreads, smem));
  if (per_sm < 1) return arg_fail("clique bit rows do not fit shared memory");
  const int parts = sms * per_sm * 4;
  const bool overflow = rs.longest > kCbCtaMax;  // some edge may need hash probes
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t sz_items = al(sizeof(int4) * ((size_t)t->n + parts + 1));
  const size_t sz_small = al(sizeof(int32_t) * ((size_t)t->n + 1));
  const size_t sz_edges = overflow ? al(sizeof(int32_t) * (size_t)m) : 0;
  char* base = nullptr;
  if (scratch_malloc(reinterpret_cast<void**>(&base),
                     sz_items + sz_small + sz_edges + al(sizeof(int32_t) * 8), st) != cudaSuccess) {
    cudaGetLastError();  // no memory for the work lists
    return clique_probe(t, d_off, d_cols, m, k, (int64_t)rs.longest, nullptr, nullptr, d_count, st);
  }
  int4* items = reinterpret_cast<int4*>(base);
  int32_t* small = reinterpret_cast<int32_t*>(base + sz_items);
  int32_t* elist = reinterpret_cast<int32_t*>(base + sz_items + sz_small);
  int32_t* ctr = reinterpret_cast<int32_t*>(base + sz_items + sz_small + sz_edges);
  cudaError_t e = cudaMemsetAsync(ctr, 0, sizeof(int32_t) * 8, st);
  if (e == cudaSuccess) {
    note_launch();
    clique_items_kernel<<<std::min((t->n + 255) / 256, sms * 8), 256, 0, st>>>(
        t->d_desc, t->n, m, dcap, rs.cubes, parts, items, small, elist, ctr);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    note_launch();
#define CB_LAUNCH(H)                                                                         \
  clique_bits_kernel<H><<<sms * per_sm, kCbThreads, smem, st>>>(                             \
      t->d_desc, d_cols, t->n, m, t->d_table, t->bucket_num, t->bucket, t->lg_max, k, items, \
      small, elist, ctr, d_count, t->d_status)
    if (t->hier) CB_LAUNCH(true); else CB_LAUNCH(false);
#undef CB_LAUNCH
    e = cudaGetLastError();
  }
  reset_status s = RESET_OK;
  if (e == cudaSuccess && overflow)
    s = clique_probe(t, d_off, d_cols, m, k, (int64_t)rs.longest, elist, ctr + 4, d_count, st);
  cudaFreeAsync(base, st);
  if (e != cudaSuccess) return cuda_fail(e, "clique bit rows", __FILE__, __LINE__);
  if (s == RESET_ERR_OOM) {  // the lists left no memory for the probes: all edges anew
    cudaGetLastError();
    RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(*d_count), st));
    s = clique_probe(t, d_off, d_cols, m, k, (int64_t)rs.longest, nullptr, nullptr, d_count, st);
  }
  return s;
}

}  // namespace
}  // namespace rst

using namespace rst;

extern "C" reset_status reset_clique4_count(const reset_table* t, const int32_t* d_off,
                                            const int32_t* d_cols, int64_t m,
                                            uint64_t* d_count, reset_stream_t stream) {
  return reset_clique_count(t, d_off, d_cols, m, 4, d_count, stream);
}

extern "C" reset_status reset_clique_count(const reset_table* t, const int32_t* d_off,
                                           const int32_t* d_cols, int64_t m, int32_t k,
                                           uint64_t* d_count, reset_stream_t stream) {
  if (!t || !d_count) return arg_fail("NULL table or count");
  if (k < 3 || k > kMaxClique) return arg_fail("k must be in 3..16");
  if (m < 0 || m > INT32_MAX) return arg_fail("m out of range");
  if (m > 0 && (!d_off || !d_cols)) return arg_fail("NULL offsets or cols");
  if (d_off != t->build_off || m != t->m)
    return arg_fail("d_off/m must be the CSR the table was built on");
  // triangles: the same sum, over tables staged in shared memory
  if (k == 3) return reset_tc_count(t, d_off, d_cols, m, d_count, stream);
  cudaStream_t st = as_stream(stream);
  RST_CUDA(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), st));
  if (m == 0 || t->n == 0) return RESET_OK;
  RowStats rs;
  RST_CHECK(row_stats(d_off, d_cols, t->n, m, st, &rs));
  unsigned long long* cnt = reinterpret_cast<unsigned long long*>(d_count);
  if (rs.ascending()) return clique_bits(t, d_off, d_cols, m, k, rs, cnt, st);
  return clique_probe(t, d_off, d_cols, m, k, (int64_t)rs.longest, nullptr, nullptr, cnt, st);
}
