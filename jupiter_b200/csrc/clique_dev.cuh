// Device building blocks of the vertex-rooted local-bitmap k-clique count, shared by the
// plain per-query kernels (clique_tiers.cuh) and the batched persistent kernels (batch.cu).
//
// The graph is the rank DAG (RankDag): vertices renumbered by descending (degree, id) rank, so
// id 0 is the highest-ranked vertex, every arc runs from a larger id to a smaller one, and rows
// are sorted.  For a root u with out-degree d, L = N+(u) ascending, the bitmap rows
//     R_i bit j  <=>  L[j] in N+(L[i])        (only j < i can be set)
// are the level-1 sets of the reference's edge-rooted plans (W of arc (u, L[i]));
// K_k(u) = sum_i C_{k-3}(R_i) with C_0(m) = popc(m), C_t(m) = sum_{j in m} C_{t-1}(m & R_j).
//
// Level 1, pair tests.  A row is built by testing its pairs (i, j < i), lane j for list entry j:
// when L[i] is one of the graph's top h vertices, by one load from the adjacency bitmap kept
// for them (RankDag::bits, a lower triangle), else by a binary search in the row of L[i], the
// lanes in lockstep.  The ballot of 32 tests is one word of the row.  Scanning the rows N+(L[i])
// instead, and searching L for each of their elements, looks at four to five times as many
// elements on R-MAT graphs (scale 22, edge factor 4: 2,262 M scanned against 521 M pairs) and
// spends about 50 instructions on each, against about 8 warp instructions for 32 pair tests.
//
// Level 2, in the same pass.  Rows come in order of i and R_i needs only R_j with j < i, so a
// warp keeps R_j in registers of the lane that owns entry j: once the words m of row i are
// known, every lane j with bit j set adds popc(m & R_j) (4-cliques of the root).  5-cliques
// apply the same scheme to the members of each row (row_triangles).
//
// Modes of the root kernels:
//   ETRI   (k = 3) every triangle adds one to each of its three DAG arcs in tri[] (edge
//          triangles);
//   PAIRS  ETRI whose adds return the old value; an add of k to a counter holding o creates
//          k*o + C(k, 2) new pairs of triangles on that edge, so the sum over all adds is
//          sum_e C(t_e, 2) -- the diamond count -- in one pass (tri[] starts at zero).
//   TT     (k = 4, with ETRI and PAIRS) the vertex-induced tailed-triangle count in the same
//          pass: I(TT) = N(TT) - 4 N(diamond) + 12 K4, where N(TT) = sum over triangles of
//          (d_a - 2) + (d_b - 2) + (d_c - 2) with d the symmetric degree.  Each root returns
//          12 K4 - 4 pairs + its triangles' degree terms in wrapping 64-bit arithmetic; the
//          sum over all roots is the exact (non-negative) count.
//   The root kernels return the pair count in PAIRS mode, the TT value in TT mode and the
//   clique count otherwise.

#pragma once
#include "jgpm_internal.h"
#include "setops.cuh"

namespace jgpm {

// Pairs of triangles created on one edge by adding k to a counter that held o.
__device__ __forceinline__ acc_t pair_gain(unsigned o, unsigned k) {
  return (acc_t)k * (acc_t)o + (acc_t)k * (acc_t)(k - 1) / 2;
}

// Largest power of two <= n (0 for n <= 0).
__device__ __forceinline__ int top_pow2(int n) { return n > 0 ? 1 << (31 - __clz(n)) : 0; }

// Elements of the sorted shared-memory array a[0..n) below x, by binary lifting (top = top_pow2(n)).
__device__ __forceinline__ int count_below(const int* a, int n, int top, int x) {
  int p = 0;
  for (int step = top; step > 0; step >>= 1)
    if (p + step <= n && a[p + step - 1] < x) p += step;
  return p;
}

// Symmetric degree minus two (the tailed-triangle degree term of a triangle vertex).
__device__ __forceinline__ acc_t tt_deg(const RankDag& g, vid_t v) {
  return (acc_t)g.sdeg[v] - 2ull;
}

constexpr uint32_t kNoRow = 0xffffffffu;  // bitmap row of a vertex outside the top h

// First bitmap word of vertex x, or kNoRow.
__device__ __forceinline__ uint32_t bit_row(const RankDag& g, vid_t x) {
  return x < g.h ? rank_bits_row(x) : kNoRow;
}

// Slot (index into col) of the arc x -> w whose bit is set in `word`, word `at` of the bitmap;
// s is the start of x's row.
__device__ __forceinline__ eid_t bit_slot(const RankDag& g, eid_t s, uint32_t at, uint32_t word,
                                          vid_t w) {
  return s + g.rk[at] + __popc(word & ((1u << (w & 31)) - 1u));
}

// Position of the r-th set bit (r counted from 0) of the W-word row.
__device__ __forceinline__ int select_bit(const uint32_t* row, int W, int r) {
  for (int q = 0; q < W; ++q) {
    const uint32_t w = row[q];
    const int c = __popc(w);
    if (r < c) return q * 32 + (int)__fns(w, 0, r + 1);
    r -= c;
  }
  return 0;  // not reached: r < popc(row)
}

// Word w of a register array, by an unrolled select (the array stays in registers).
template <int WMAX>
__device__ __forceinline__ uint32_t pick_word(const uint32_t (&m)[WMAX], int w) {
  uint32_t r = 0u;
#pragma unroll
  for (int q = 0; q < WMAX; ++q) r = (q == w) ? m[q] : r;
  return r;
}

// ---------------------------------------------------------------- single-word rows
template <int D, bool STATS>
struct SmallCount {
  // m: candidate set (bits over L), R: rows, deg: out-degrees of L (stats only)
  __device__ __forceinline__ static acc_t run(uint32_t m, const uint32_t* R, const int* deg,
                                              acc_t& elems) {
    acc_t s = 0;
    const int pm = __popc(m);
    uint32_t it = m;
    while (it) {
      const int j = __ffs(it) - 1;
      it &= it - 1;
      if (STATS) elems += (acc_t)pm + (acc_t)deg[j];
      s += SmallCount<D - 1, STATS>::run(m & R[j], R, deg, elems);
    }
    return s;
  }
};

template <bool STATS>
struct SmallCount<0, STATS> {
  __device__ __forceinline__ static acc_t run(uint32_t m, const uint32_t*, const int*, acc_t&) {
    return (acc_t)__popc(m);
  }
};

// Rows of more than this many elements are cut to the range of the root's list before a scan.
constexpr int kRangeCut = 32;

// Scans rows for a root's list, one root per group of G lanes: lane j of a group holds list entry
// Lj (ascending, INT32_MAX past the end) and, if row j is to be scanned, its start s and length
// len (else 0).  The rows' elements are flattened over the group's lanes, read in order, and
// looked up in the list by shuffles, kScanAhead elements of a lane at a time so that their loads
// overlap.  hits(in, i, p, e) is called by the whole warp for each such step: in[t] <=> this lane's
// t-th element, slot e[t] of row i[t], is list entry p[t].
constexpr int kScanAhead = 4;
template <int G, typename Hits>
__device__ __forceinline__ void scan_rows(const RankDag& g, vid_t Lj, int d, eid_t s, int len,
                                          Hits&& hits) {
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const vid_t lo_key = __shfl_sync(kFull, Lj, 0, G);
  const vid_t hi_key = __shfl_sync(kFull, Lj, d > 0 ? d - 1 : 0, G);
  if (len > kRangeCut) {
    const int lb = lower_bound_g(g.col + s, len, lo_key);
    const int ub = upper_bound_g(g.col + s, len, hi_key);
    s += lb;
    len = ub > lb ? ub - lb : 0;
  }
  int off = len;  // inclusive scan of the row lengths within the group
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
    const int t = __shfl_up_sync(kFull, off, o, G);
    if (gl >= o) off += t;
  }
  const int T = __shfl_sync(kFull, off, G - 1, G);
  const int Tmax = G == 32 ? T : (int)__reduce_max_sync(kFull, (unsigned)T);
  s -= off - len;  // element t of the flattened rows is col[s + t] while it is in this row
  for (int t0 = 0; t0 < Tmax; t0 += kScanAhead * G) {
    int i[kScanAhead], p[kScanAhead];
    eid_t e[kScanAhead];
    vid_t x[kScanAhead];
    bool in[kScanAhead];
#pragma unroll
    for (int q = 0; q < kScanAhead; ++q) {
      const int t = t0 + q * G + gl;
      i[q] = 0;  // rows of the group that end at or before t
#pragma unroll
      for (int step = G / 2; step > 0; step >>= 1) {
        const int ov = __shfl_sync(kFull, off, i[q] + step - 1, G);
        if (ov <= t) i[q] += step;
      }
      e[q] = __shfl_sync(kFull, s, i[q], G) + t;
      in[q] = t < T;
      x[q] = in[q] ? __ldg(g.col + e[q]) : INT32_MIN;
    }
#pragma unroll
    for (int q = 0; q < kScanAhead; ++q) {
      p[q] = 0;
#pragma unroll
      for (int step = G / 2; step > 0; step >>= 1) {
        const vid_t lv = __shfl_sync(kFull, Lj, p[q] + step - 1, G);
        if (lv < x[q]) p[q] += step;
      }
      const vid_t lp = __shfl_sync(kFull, Lj, p[q], G);
      in[q] = in[q] && lp == x[q];
    }
    hits(in, i, p, e);
  }
}

// One root per group of G lanes (G in {4, 8, 16, 32}); every lane of the warp calls this
// with its group's root u (or u < 0 for an idle group).  Lane j of a group holds list entry j and
// its row.  R and DG point at the group's G shared words (used where rows are scanned, for k >= 5
// and for the accounting).  Returns this lane's partial count.  tri (edge-triangle mode) receives
// one count per triangle arc.
//
// Rows of the graph's top h vertices are tested pair by pair in the bitmap, four rows at a time so
// that their loads overlap (eight in a triangle count, which keeps nothing of them).  The other rows, which are short, are scanned (scan_rows): their
// elements are read once, in order, where a binary search per pair is a chain of scattered loads
// (R-MAT, 1,048,576 vertices, edge factor 16, a = 0.45, 84 % of the pairs outside the bitmap: a
// triangle count of 1.79 ms with searches, 0.80 ms with scans; kScanAhead = 1: 0.85 ms).
template <int G, int K, bool STATS, bool ETRI, bool PAIRS = false, bool TT = false>
__device__ __forceinline__ acc_t group_root(const RankDag& g, vid_t u, uint32_t* R, int* DG,
                                            uint32_t* tri, acc_t& elems) {
  constexpr bool STORE = K >= 5 || STATS;
  constexpr int U = K == 3 && !ETRI && !STATS && G >= 8 ? 8 : 4;
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1);
  const int gsh = lane & ~(G - 1);
  eid_t base = 0;
  int d = 0;
  if (u >= 0) {
    base = g.rp[u];
    d = (int)(g.rp[u + 1] - base);
  }
  const vid_t Lj = gl < d ? __ldg(g.col + base + gl) : INT32_MAX;
  const uint32_t rb = gl < d ? bit_row(g, Lj) : 0u;
  const bool out = gl < d && rb == kNoRow;
  const bool scan = __any_sync(kFull, out);
  // start and length of the rows that are scanned (all rows where the slots are needed)
  eid_t s = 0;
  int len = 0;
  if (gl < d && (ETRI || STATS || out)) {
    s = g.rp[Lj];
    len = (int)(g.rp[Lj + 1] - s);
  }
  if (STORE || scan) {
    __syncwarp();
    R[gl] = 0u;
    if (STATS) DG[gl] = len;
    else if (ETRI) DG[gl] = 0;  // hits per list entry in the scanned rows
  }
  // the list ascends, so the rows in the bitmap are the first hc
  const int hc = G == 32 ? d - __popc(__ballot_sync(kFull, out))
                         : d - __popc((__ballot_sync(kFull, out) >> gsh) & ((1u << (G & 31)) - 1u));
  const int hmax = G == 32 ? hc : (int)__reduce_max_sync(kFull, (unsigned)hc);
  const uint32_t wi = (uint32_t)Lj >> 5, bi = (uint32_t)Lj & 31u;
  acc_t cnt = 0, pairs = 0, tt = 0;
  uint32_t row = 0;             // R_gl
  unsigned rowc = 0, colc = 0;  // ETRI: popc(R_gl), rows with bit gl
  for (int i0 = 1; i0 < hmax; i0 += U) {
    uint32_t xb[U], word[U];
    bool hit[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int i = i0 + t;
      xb[t] = __shfl_sync(kFull, rb, i & (G - 1), G);
      word[t] = 0u;
      if (i < hc && gl < i) word[t] = __ldg(g.bits + xb[t] + wi);
    }
#pragma unroll
    for (int t = 0; t < U; ++t) hit[t] = ((word[t] >> bi) & 1u) != 0u;
    if (ETRI) {  // triangles (u, L[i], L[gl]): the arcs L[i] -> L[gl] get their counts now
      eid_t e[U];
      unsigned old[U];
#pragma unroll
      for (int t = 0; t < U; ++t) {
        e[t] = __shfl_sync(kFull, s, (i0 + t) & (G - 1), G);
        if (hit[t]) e[t] = bit_slot(g, e[t], xb[t] + wi, word[t], Lj);
      }
#pragma unroll
      for (int t = 0; t < U; ++t) {
        old[t] = 0u;
        if (hit[t]) {
          old[t] = atomicAdd(tri + e[t], 1u);
          ++colc;
        }
      }
      if (PAIRS) {
#pragma unroll
        for (int t = 0; t < U; ++t) pairs += (acc_t)old[t];
      }
    }
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int i = i0 + t;
      if (K == 3 && !ETRI && !STATS) {
        cnt += hit[t] ? 1u : 0u;
        continue;
      }
      const unsigned all = __ballot_sync(kFull, hit[t]);
      const uint32_t m = G == 32 ? all : (all >> gsh) & ((1u << (G & 31)) - 1u);
      if (ETRI && gl == i) rowc = (unsigned)__popc(m);
      if (K == 3 && !PAIRS) cnt += hit[t] ? 1u : 0u;
      if (K >= 4) {
        if (K == 4 && !STATS && hit[t]) cnt += (acc_t)__popc(m & row);
        if (gl == i) row = m;
      }
      if ((STORE || (K >= 4 && scan)) && gl == i && i < hc) R[gl] = m;
    }
  }
  if (scan) {
    __syncwarp();
    constexpr int A = kScanAhead;
    scan_rows<G>(g, Lj, d, s, out ? len : 0,
                 [&](const bool (&in)[A], const int (&i)[A], const int (&p)[A], const eid_t (&e)[A]) {
      unsigned old[A];
#pragma unroll
      for (int q = 0; q < A; ++q) {
        old[q] = 0u;
        if (!in[q]) continue;
        if (ETRI) {
          old[q] = atomicAdd(tri + e[q], 1u);
          atomicAdd(&DG[p[q]], 1);
        }
        if (K == 3 && !ETRI && !STATS) ++cnt;
        else atomicOr(&R[i[q]], 1u << p[q]);
      }
      if (PAIRS) {
#pragma unroll
        for (int q = 0; q < A; ++q) pairs += (acc_t)old[q];
      }
    });
    __syncwarp();
    if (ETRI && out) rowc = (unsigned)__popc(R[gl]);
    if (ETRI && gl < d) colc += (unsigned)DG[gl];
    if (K == 3 && ETRI && !PAIRS) cnt += out ? rowc : 0u;
    if (K == 4 && !STATS && out) cnt += SmallCount<1, false>::run(R[gl], R, DG, elems);
  }
  if (STORE) {
    __syncwarp();
    if (gl < d) cnt = SmallCount<K - 3, STATS>::run(R[gl], R, DG, elems);
  }
  if (STORE || scan) __syncwarp();
  if (ETRI && gl < d) {
    // the root's own arc (u, L[gl]) lies on popc(R_gl) + (rows with bit gl) triangles
    const unsigned tu = rowc + colc;
    if (tu) {
      const unsigned o = atomicAdd(tri + base + gl, tu);
      if (PAIRS) pairs += pair_gain(o, tu);
      // L[gl] is the middle vertex of popc(R_gl) of the root's triangles and the top of colc
      if (TT) {
        const acc_t dg = tt_deg(g, Lj);
        tt = (acc_t)rowc * (tt_deg(g, u) + dg) + (acc_t)colc * dg;
      }
    }
  }
  if (TT) return 12ull * cnt - 4ull * pairs + tt;
  return PAIRS ? pairs : cnt;
}

// ---------------------------------------------------------------- multi-word rows
// Row loads: rows in global memory (GR) are built with L2 atomics, so they are read at L2
// (ld.global.cg), never from a possibly stale L1 line; shared-memory rows are read directly.
template <bool GR>
__device__ __forceinline__ uint32_t ld_row(const uint32_t* p) {
  if (GR) return __ldcg(p);
  return *p;
}

// Mask distributed over the warp, WPL words per lane: lane l holds words l + 32 q (q < WPL,
// word index < W).  Rows are W words long.
template <int D, int WPL, bool STATS, bool GR = false>
struct DistCount {
  __device__ __forceinline__ static acc_t run(const uint32_t (&mw)[WPL], const uint32_t* R,
                                              int W, const int* deg, acc_t& elems, int S) {
    const int lane = threadIdx.x & 31;
    acc_t s = 0;
    int pm = 0;
    if (STATS) {
      int c = 0;
#pragma unroll
      for (int q = 0; q < WPL; ++q) c += __popc(mw[q]);
      pm = __reduce_add_sync(kFull, (unsigned)c);
    }
    // one recursive call site per level (a rolled loop over the lane's words, picked from
    // registers), so the code does not grow as WPL^depth
#pragma unroll 1
    for (int q = 0; q < WPL; ++q) {
      const uint32_t mq = pick_word<WPL>(mw, q);
      unsigned nz = __ballot_sync(kFull, mq != 0u);
      while (nz) {
        const int lw = __ffs(nz) - 1;
        nz &= nz - 1;
        uint32_t word = __shfl_sync(kFull, mq, lw);
        while (word) {
          const int b = __ffs(word) - 1;
          word &= word - 1;
          const int j = (q * 32 + lw) * 32 + b;
          if (STATS && lane == 0) elems += (acc_t)pm + (acc_t)deg[j];
          const uint32_t* Rj = R + (size_t)j * S;
          uint32_t nxt[WPL];
#pragma unroll
          for (int r = 0; r < WPL; ++r) {
            const int w = r * 32 + lane;
            nxt[r] = w < W ? (mw[r] & ld_row<GR>(Rj + w)) : 0u;
          }
          s += DistCount<D - 1, WPL, STATS, GR>::run(nxt, R, W, deg, elems, S);
        }
      }
    }
    return s;
  }
};

template <int WPL, bool STATS, bool GR>
struct DistCount<0, WPL, STATS, GR> {
  __device__ __forceinline__ static acc_t run(const uint32_t (&mw)[WPL], const uint32_t*, int,
                                              const int*, acc_t&, int) {
    acc_t s = 0;  // per-lane partial; summed at the end
#pragma unroll
    for (int q = 0; q < WPL; ++q) s += (acc_t)__popc(mw[q]);
    return s;
  }
};

// Row-parallel counting with the candidate mask in registers (WMAX words, W <= WMAX used):
// one thread owns one first-level row and walks the deeper levels itself.  Each level has a
// single recursive call site (code size stays linear in the depth); words are picked out of
// the register array with an unrolled select so the masks never go to local memory.

template <int D, int WMAX, bool STATS>
struct RowCount {
  __device__ static acc_t run(const uint32_t (&m)[WMAX], const uint32_t* R, int W,
                              const int* deg, acc_t& elems, int S) {
    acc_t s = 0;
    int pm = 0;
    if (STATS) {
#pragma unroll
      for (int w = 0; w < WMAX; ++w) pm += __popc(m[w]);
    }
    int w = 0;
    uint32_t bits = m[0];
    for (;;) {
      while (bits == 0u) {
        if (++w >= W) return s;
        bits = pick_word<WMAX>(m, w);
      }
      const int j = w * 32 + __ffs(bits) - 1;
      bits &= bits - 1;
      if (STATS) elems += (acc_t)pm + (acc_t)deg[j];
      uint32_t nxt[WMAX];
      const uint32_t* Rj = R + (size_t)j * S;
#pragma unroll
      for (int q = 0; q < WMAX; ++q) nxt[q] = q < W ? (m[q] & Rj[q]) : 0u;
      s += RowCount<D - 1, WMAX, STATS>::run(nxt, R, W, deg, elems, S);
    }
  }
};

template <int WMAX, bool STATS>
struct RowCount<0, WMAX, STATS> {
  __device__ __forceinline__ static acc_t run(const uint32_t (&m)[WMAX], const uint32_t*, int,
                                              const int*, acc_t&, int) {
    acc_t s = 0;
#pragma unroll
    for (int w = 0; w < WMAX; ++w) s += (acc_t)__popc(m[w]);
    return s;
  }
};

// One 32 x 32 tile of a root's pair tests, by one warp: rows 32 B + r, r < nrow, against this
// lane's list entry w of column block b; `first` is the first row the entry is tested in (0 in a
// block left of the diagonal; on it, lane + 1).  A row costs its bitmap base, one load and one
// ballot; four rows at a time, so that their loads overlap.  The first nbm rows are in the bitmap
// (base(r) is the row's first word), the others (vertex id(r)) are searched in lockstep.
// Returns, in lane r, word b of row 32 B + r (0 past the last row).  add(r, e) is called for each
// hit of this lane in the edge-triangle mode, e the slot of the arc from the row's vertex to w;
// got collects what it returns (the old values of counter adds), after the four rows' adds are
// all on their way: waiting for each kept the warps idle for most of a diamond count.
template <bool ETRI, typename Base, typename Id, typename Add>
__device__ __forceinline__ uint32_t test_tile(const RankDag& g, vid_t w, int first, int nrow,
                                              int nbm, Base&& base, Id&& id, acc_t& got,
                                              Add&& add) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const uint32_t* col = g.bits + ((uint32_t)w >> 5);
  const uint32_t bit = 1u << (w & 31);
  uint32_t keep = 0u;
  for (int r0 = 0; r0 < nbm; r0 += U) {
    uint32_t word[U], xb[U];
    eid_t s[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int r = r0 + t;
      word[t] = 0u;
      xb[t] = base(r);
      if (r < nbm && r >= first) word[t] = __ldg(col + xb[t]);
      if (ETRI) s[t] = r < nbm ? g.rp[id(r)] : 0;
    }
    unsigned before[U], old[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int r = r0 + t;
      const bool h = (word[t] & bit) != 0u;
      const uint32_t m = __ballot_sync(kFull, h);
      if (lane == r) keep = m;
      if (ETRI) before[t] = h ? g.rk[xb[t] + ((uint32_t)w >> 5)] : 0u;
    }
    if (ETRI) {
#pragma unroll
      for (int t = 0; t < U; ++t) {
        old[t] = 0u;
        if (word[t] & bit)
          old[t] = add(r0 + t, s[t] + before[t] + __popc(word[t] & (bit - 1u)));
      }
#pragma unroll
      for (int t = 0; t < U; ++t) got += (acc_t)old[t];
    }
  }
  for (int r0 = nbm; r0 < nrow; r0 += U) {
    const vid_t* rowp[U];
    int len[U], pos[U], lmax = 0;
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int r = r0 + t;
      const vid_t x = id(r);
      rowp[t] = g.col;
      len[t] = pos[t] = 0;
      if (r < nrow) {
        const eid_t s = g.rp[x];
        rowp[t] = g.col + s;
        len[t] = (int)(g.rp[x + 1] - s);
      }
      lmax = max(lmax, len[t]);
    }
    for (int step = top_pow2(lmax); step > 0; step >>= 1) {
#pragma unroll
      for (int t = 0; t < U; ++t)
        if (pos[t] + step <= len[t] && __ldg(rowp[t] + pos[t] + step - 1) < w) pos[t] += step;
    }
    bool h[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int r = r0 + t;
      h[t] = r < nrow && r >= first && pos[t] < len[t] && __ldg(rowp[t] + pos[t]) == w;
      const uint32_t m = __ballot_sync(kFull, h[t]);
      if (lane == r) keep = m;
    }
    if (ETRI) {
      unsigned old[U];
#pragma unroll
      for (int t = 0; t < U; ++t) {
        old[t] = 0u;
        if (h[t]) old[t] = add(r0 + t, (rowp[t] - g.col) + pos[t]);
      }
#pragma unroll
      for (int t = 0; t < U; ++t) got += (acc_t)old[t];
    }
  }
  return keep;
}

// Triangles among the members of one row, in the sub-DAG that the rows induce on them: the
// 5-cliques through that row.  Pw[0..c) holds the members' list positions, ascending; c <= 32 P.
// Lane y keeps the induced row A_y of its members y, y + 32, ... in registers; row x's words
// m come from one ballot per 32 members, and every lane y < x in A_x adds popc(m & A_y).  About
// a dozen instructions for each x and 32 members; a first form that read x's position from
// shared memory and compared y with x took half as many again (5-clique band of out-degree
// 129..256 on the scale 22 graph: 1.73 G warp instructions, now 1.37 G).
template <int P>
__device__ __forceinline__ int row_triangles(const uint32_t* R, int S, const uint16_t* Pw,
                                             int c) {
  const int lane = threadIdx.x & 31;
  int row[P], pw[P];  // first word of the member's row, word and bit of its position
  uint32_t bit[P];    // (0 past the last member: never hit)
#pragma unroll
  for (int b = 0; b < P; ++b) {
    const int y = 32 * b + lane;
    const int p = y < c ? (int)Pw[y] : 0;
    row[b] = p * S;
    pw[b] = p >> 5;
    bit[b] = y < c ? 1u << (p & 31) : 0u;
  }
  uint32_t A[P][P];
#pragma unroll
  for (int b = 0; b < P; ++b)
#pragma unroll
    for (int q = 0; q < P; ++q) A[b][q] = 0u;
  int s = 0;
#pragma unroll
  for (int B = 0; B < P; ++B) {
    const int lim = min(32, c - 32 * B);
    if (lim <= 0) break;
#pragma unroll 4
    for (int ii = 0; ii < lim; ++ii) {
      const uint32_t* Rx = R + __shfl_sync(kFull, row[B], ii);
      uint32_t m[P];
      bool hit[P];
#pragma unroll
      for (int b = 0; b <= B; ++b) {  // rows are triangular: no bit at or after x itself
        hit[b] = (Rx[pw[b]] & bit[b]) != 0u;
        m[b] = __ballot_sync(kFull, hit[b]);
      }
#pragma unroll
      for (int b = 0; b <= B; ++b) {
        int t = 0;
#pragma unroll
        for (int q = 0; q <= b; ++q) t += __popc(m[q] & A[b][q]);
        if (hit[b]) s += t;
      }
#pragma unroll
      for (int q = 0; q <= B; ++q)
        if (lane == ii) A[B][q] = m[q];
    }
  }
  return s;
}

// The same for rows of at most G members, 32 / G rows at a time, one per group of G lanes; Pw
// and c are the group's row (c = 0: none).
template <int G, typename T>
__device__ __forceinline__ int group_triangles(const uint32_t* R, int S, const T* Pw, int c) {
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gsh = lane & ~(G - 1);
  const int p = gl < c ? (int)Pw[gl] : 0;
  const int row = p * S, pw = p >> 5;
  const uint32_t bit = gl < c ? 1u << (p & 31) : 0u;
  const int cmax = (int)__reduce_max_sync(kFull, (unsigned)c);
  uint32_t A = 0u;
  int s = 0;
  for (int x = 1; x < cmax; ++x) {
    const bool hit = (R[__shfl_sync(kFull, row, x, G) + pw] & bit) != 0u;
    const uint32_t m = (__ballot_sync(kFull, hit) >> gsh) & ((1u << G) - 1u);
    const int t = __popc(m & A);
    if (hit) s += t;
    if (gl == x) A = m;
  }
  return s;
}

// Writes the list positions of the members of row Ri (w_d words) to Pw, ascending, and returns
// their number (warp-uniform); Pw must hold them all.
__device__ __forceinline__ int row_members(const uint32_t* Ri, int w_d, uint16_t* Pw) {
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  int c = 0;
  for (int q = 0; q < w_d; ++q) {
    const uint32_t m = Ri[q];
    if ((m >> lane) & 1u) Pw[c + __popc(m & below)] = (uint16_t)(q * 32 + lane);
    c += __popc(m);
  }
  return c;
}

// One root of out-degree d <= kLightOutDegree of a graph without a rank DAG, on a CTA of 256
// threads: the warps scan the rows, four at a time, and look their elements up in the list in shared
// memory.  Such roots are few, so what counts is how long one takes.
struct ScanSmem {
  eid_t s[kLightOutDegree];
  int len[kLightOutDegree];
  int L[kLightOutDegree];
  int hits[kLightOutDegree];  // per list entry (ETRI)
  uint32_t R[kLightOutDegree * 2];
};
template <int K, bool STATS, bool ETRI, bool PAIRS = false, bool TT = false>
__device__ __forceinline__ acc_t scan_root(const RankDag& g, vid_t u, ScanSmem& sm, uint32_t* tri,
                                           acc_t& elems) {
  static_assert(kLightOutDegree == 64, "two row elements a lane, four threads a row");
  constexpr int U = 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const eid_t base = g.rp[u];
  const int d = (int)(g.rp[u + 1] - base);
  __syncthreads();  // the last root's readers are done
  if (tid < kLightOutDegree) {
    const vid_t x = tid < d ? __ldg(g.col + base + tid) : INT32_MAX;
    const eid_t s = tid < d ? g.rp[x] : 0;
    sm.L[tid] = x;
    sm.s[tid] = s;
    sm.len[tid] = tid < d ? (int)(g.rp[x + 1] - s) : 0;
    sm.hits[tid] = 0;
    sm.R[2 * tid] = sm.R[2 * tid + 1] = 0u;
  }
  __syncthreads();
  acc_t cnt = 0, pairs = 0, tt = 0;
  for (int i0 = warp; i0 < d; i0 += 8 * U) {
    eid_t e[U][2];
    vid_t x[U][2];
    unsigned old[U][2];
#pragma unroll
    for (int t = 0; t < U; ++t) {
      const int i = min(i0 + 8 * t, kLightOutDegree - 1), ln = i0 + 8 * t < d ? sm.len[i] : 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        e[t][h] = sm.s[i] + 32 * h + lane;
        x[t][h] = 32 * h + lane < ln ? __ldg(g.col + e[t][h]) : -1;
      }
    }
#pragma unroll
    for (int t = 0; t < U; ++t) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        old[t][h] = 0u;
        int p = 0;
#pragma unroll
        for (int step = 32; step > 0; step >>= 1)
          if (sm.L[p + step - 1] < x[t][h]) p += step;
        if (x[t][h] < 0 || sm.L[p] != x[t][h]) continue;
        if (ETRI) {
          old[t][h] = atomicAdd(tri + e[t][h], 1u);
          atomicAdd(&sm.hits[p], 1);
        }
        if (K == 3) ++cnt;
        atomicOr(&sm.R[2 * (i0 + 8 * t) + (p >> 5)], 1u << (p & 31));
      }
    }
    if (PAIRS) {
#pragma unroll
      for (int t = 0; t < U; ++t) pairs += (acc_t)old[t][0] + (acc_t)old[t][1];
    }
  }
  __syncthreads();
  const int i = tid >> 2;
  if (K > 3 && i < d) {  // four threads take the members of row i in turn
    const uint32_t m[2] = {sm.R[2 * i], sm.R[2 * i + 1]};
    const int pm = __popc(m[0]) + __popc(m[1]);
    int at = tid & 3;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      for (uint32_t w = m[q]; w != 0u; w &= w - 1u, ++at) {
        if ((at & 3) != 0) continue;
        const int j = 32 * q + __ffs(w) - 1;
        if (STATS) elems += (acc_t)pm + (acc_t)sm.len[j];
        const uint32_t nxt[2] = {m[0] & sm.R[2 * j], m[1] & sm.R[2 * j + 1]};
        cnt += RowCount<(K > 3 ? K - 4 : 0), 2, STATS>::run(nxt, sm.R, 2, sm.len, elems, 2);
      }
    }
  }
  if (ETRI && tid < d) {  // the root's own arcs, as in group_root
    const unsigned rowc = (unsigned)(__popc(sm.R[2 * tid]) + __popc(sm.R[2 * tid + 1]));
    const unsigned colc = (unsigned)sm.hits[tid], tu = rowc + colc;
    if (tu) {
      const unsigned o = atomicAdd(tri + base + tid, tu);
      if (PAIRS) pairs += pair_gain(o, tu);
      if (TT) {
        const acc_t di = tt_deg(g, sm.L[tid]);
        tt += (acc_t)rowc * (tt_deg(g, u) + di) + (acc_t)colc * di;
      }
    }
  }
  if (TT) return 12ull * cnt - 4ull * pairs + tt;
  return PAIRS ? pairs : cnt;
}

// ---------------------------------------------------------------- warp per root
// One root of out-degree 32 < d <= kWarpMaxDeg per warp, with the warp's own slice of shared
// memory (no CTA barriers).
constexpr int kWarpMaxDeg = 128;
constexpr int kWarpW = kWarpMaxDeg / 32;

// Rows of at most this many members count their triangles several to a warp.
constexpr int kRowFew = 16;

// Shared memory of a warp root: nothing for the plain counts of k <= 4, whose rows stay in
// registers; the rows and a row's members for k = 5; the pair offsets for k >= 6 and the
// accounting.
struct WarpSmem {
  uint32_t R[kWarpMaxDeg * kWarpW];
  union {
    struct {
      uint16_t mem[kWarpMaxDeg];            // members of one row
      uint8_t few[kWarpMaxDeg][kRowFew];    // members of the rows with at most kRowFew
      uint8_t list[kWarpMaxDeg];            // rows: few by slot, then the others from the end
      uint8_t cnt[kWarpMaxDeg];             // their sizes (few)
    };
    struct {
      int off[kWarpMaxDeg + 1];
      int deg[kWarpMaxDeg];
    };
  };
};
template <int K, bool STATS>
constexpr size_t warp_smem_bytes() {
  return K <= 4 && !STATS ? 0 : 8 * sizeof(WarpSmem);
}

template <int K, bool STATS, bool ETRI, bool PAIRS = false, bool TT = false>
__device__ __forceinline__ acc_t warp_root(const RankDag& g, vid_t u, WarpSmem* wsp,
                                           uint32_t* tri, acc_t& elems) {
  constexpr int NB = kWarpW;
  constexpr bool STORE = K >= 5 || STATS;
  constexpr bool FUSE4 = K == 4 && !STATS;
  const int lane = threadIdx.x & 31;
  const eid_t base = g.rp[u];
  const int d = (int)(g.rp[u + 1] - base);
  const int w_d = (d + 31) >> 5;
  vid_t L[NB];
  uint32_t rb[NB];
  int hc = 0;  // rows below hc are tested in the bitmap (L ascends)
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = 32 * b + lane;
    L[b] = j < d ? __ldg(g.col + base + j) : INT32_MAX;
    rb[b] = bit_row(g, L[b]);
    hc += __popc(__ballot_sync(kFull, rb[b] != kNoRow));
  }
  if (STORE) __syncwarp();  // the last root's readers are done
  if (STATS) {
    for (int j = lane; j < d; j += 32) {
      const vid_t x = __ldg(g.col + base + j);
      wsp->deg[j] = (int)(g.rp[x + 1] - g.rp[x]);
    }
  }
  // Lane r holds the words of rows r, 32 + r, ...: Rr[B][b], b <= B
  uint32_t Rr[NB][NB];
  unsigned colc[NB];  // ETRI: rows with bit j, per list entry of this lane
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    colc[b] = 0u;
#pragma unroll
    for (int q = 0; q < NB; ++q) Rr[b][q] = 0u;
  }
  unsigned c32 = 0;
  acc_t pairs = 0;
#pragma unroll
  for (int B = 0; B < NB; ++B) {
    const int nrow = min(32, d - 32 * B);
    if (nrow <= 0) break;
    const int nbm = max(0, min(nrow, hc - 32 * B));
#pragma unroll
    for (int b = 0; b <= B; ++b)
      Rr[B][b] = test_tile<ETRI>(
          g, L[b], b < B ? 0 : lane + 1, nrow, nbm,
          [&](int r) { return __shfl_sync(kFull, rb[B], r & 31); },
          [&](int r) { return __shfl_sync(kFull, L[B], r & 31); },
          pairs, [&](int, eid_t e) {
            const unsigned o = atomicAdd(tri + e, 1u);
            ++colc[b];
            return PAIRS ? o : 0u;
          });
    unsigned c = 0;
#pragma unroll
    for (int b = 0; b <= B; ++b) c += (unsigned)__popc(Rr[B][b]);
    if (K == 3 && !PAIRS) c32 += c;
    if (FUSE4) {
      // rows of two bits or more: every lane j in the row adds popc(R_i & R_j)
      for (unsigned live = __ballot_sync(kFull, c >= 2u); live != 0u; live &= live - 1u) {
        const int ii = __ffs(live) - 1;
        uint32_t m[NB];
#pragma unroll
        for (int q = 0; q <= B; ++q) m[q] = __shfl_sync(kFull, Rr[B][q], ii);
#pragma unroll
        for (int b = 0; b <= B; ++b) {
          unsigned v = 0;
#pragma unroll
          for (int q = 0; q <= b; ++q) v += (unsigned)__popc(m[q] & Rr[b][q]);
          if ((m[b] >> lane) & 1u) c32 += v;
        }
      }
    }
    if (STORE && 32 * B + lane < d) {
#pragma unroll
      for (int q = 0; q < NB; ++q)
        if (q < w_d) wsp->R[(32 * B + lane) * w_d + q] = q <= B ? Rr[B][q] : 0u;
    }
  }
  acc_t cnt = (acc_t)c32;
  if (STORE) {
    __syncwarp();
    const uint32_t* R = wsp->R;
    if (K == 5 && !STATS) {
      // rows by their number of members c: those of c <= 8 and c <= 16 get their members listed
      // one row per lane and are counted four and two to a warp; on the scale 22 graph 83 % of
      // the rows with c >= 3 are of these (a warp for each: 1.56 ms for the warp tier;
      // so: 1.01 ms)
      int n8 = 0, n16 = 0, nbig = 0;
      auto list_few = [&](int lo, int hi, int at) {
        int n = 0;
        for (int i0 = 0; i0 < d; i0 += 32) {
          const int i = i0 + lane;
          uint32_t w[NB];
          int c = 0;
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            w[q] = i < d && q < w_d ? R[i * w_d + q] : 0u;
            c += __popc(w[q]);
          }
          const bool mine = c >= lo && c <= hi;
          const unsigned all = __ballot_sync(kFull, mine);
          if (mine) {
            const int slot = at + n + __popc(all & ((1u << lane) - 1u));
            wsp->cnt[slot] = (uint8_t)c;
            if (hi <= kRowFew) {
              uint8_t* out = wsp->few[slot];
#pragma unroll
              for (int q = 0; q < NB; ++q)
                for (uint32_t m = w[q]; m != 0u; m &= m - 1u)
                  *out++ = (uint8_t)(32 * q + __ffs(m) - 1);
            } else {
              wsp->list[slot] = (uint8_t)i;
            }
          }
          n += __popc(all);
        }
        return n;
      };
      n8 = list_few(3, 8, 0);
      n16 = list_few(9, kRowFew, n8);
      nbig = list_few(kRowFew + 1, kWarpMaxDeg, n8 + n16);
      __syncwarp();
      for (int r = 0; r < n8; r += 4) {
        const int q = r + (lane >> 3);
        const int at = q < n8 ? q : 0;
        cnt += (acc_t)group_triangles<8>(R, w_d, wsp->few[at], q < n8 ? wsp->cnt[at] : 0);
      }
      for (int r = 0; r < n16; r += 2) {
        const int q = r + (lane >> 4);
        const int at = n8 + (q < n16 ? q : 0);
        cnt += (acc_t)group_triangles<16>(R, w_d, wsp->few[at], q < n16 ? wsp->cnt[at] : 0);
      }
      for (int r = 0; r < nbig; ++r) {
        const int i = wsp->list[n8 + n16 + r];
        const int c = row_members(R + i * w_d, w_d, wsp->mem);
        __syncwarp();
        cnt += (acc_t)row_triangles<NB>(R, w_d, wsp->mem, c);
        __syncwarp();
      }
    } else if (K >= 5) {
      // k >= 6 (and the accounting of k = 5): the first two levels flattened over the lanes as
      // (row i, bit j of R_i) pairs, so one dense row does not hold up the warp.  off[i] =
      // pairs before row i.
      int* off = wsp->off;
      const int b0 = min(d, lane * NB), b1 = min(d, b0 + NB);
      int local = 0;
      for (int i = b0; i < b1; ++i) {
        int c = 0;
        for (int q = 0; q < w_d; ++q) c += __popc(R[i * w_d + q]);
        off[i] = c;
        local += c;
      }
      int incl = local;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
      }
      int run = incl - local;
      for (int i = b0; i < b1; ++i) {
        const int c = off[i];
        off[i] = run;
        run += c;
      }
      if (lane == 31) off[d] = incl;
      __syncwarp();
      const int P = off[d], topO = top_pow2(d - 1);
      for (int p = lane; p < P; p += 32) {
        const int i = count_below(off + 1, d - 1, topO, p + 1);
        const uint32_t* Ri = R + i * w_d;
        const int j = select_bit(Ri, w_d, p - off[i]);
        const uint32_t* Rj = R + j * w_d;
        uint32_t m2[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q) m2[q] = q < w_d ? (Ri[q] & Rj[q]) : 0u;
        if (STATS) elems += (acc_t)(off[i + 1] - off[i]) + (acc_t)wsp->deg[j];
        cnt += RowCount<(K >= 5 ? K - 4 : 1), NB, STATS>::run(m2, R, w_d, wsp->deg, elems, w_d);
      }
    } else {  // accounting of k <= 4
      for (int i = lane; i < d; i += 32) {
        uint32_t m[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q) m[q] = q < w_d ? R[i * w_d + q] : 0u;
        const acc_t c = RowCount<K - 3, NB, STATS>::run(m, R, w_d, wsp->deg, elems, w_d);
        if (K != 3) cnt += c;
      }
    }
    __syncwarp();
  }
  acc_t tt = 0;
  if (ETRI) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int i = 32 * b + lane;
      unsigned rowc = 0;
#pragma unroll
      for (int q = 0; q <= b; ++q) rowc += (unsigned)__popc(Rr[b][q]);
      const unsigned tu = rowc + colc[b];
      if (i < d && tu) {
        const unsigned o = atomicAdd(tri + base + i, tu);
        if (PAIRS) pairs += pair_gain(o, tu);
        if (TT) {
          const acc_t di = tt_deg(g, L[b]);
          tt += (acc_t)rowc * (tt_deg(g, u) + di) + (acc_t)colc[b] * di;
        }
      }
    }
  }
  if (TT) return 12ull * cnt - 4ull * pairs + tt;
  return PAIRS ? pairs : cnt;
}

// Row stride in words of a root with w_d-word rows in shared memory: odd, so that the rows that
// the threads of a warp read at the same word index fall into different banks; for k = 4, which
// reads four words at a time, an odd multiple of four.  Rows in global memory (GR) are packed.
template <int K>
__host__ __device__ __forceinline__ int row_stride(int w_d, bool global_rows) {
  if (global_rows) return w_d;
  return K == 4 ? (((w_d + 3) >> 2) | 1) << 2 : (w_d | 1);
}
// Words that a layout allots per row of up to W words: none for the triangle counts, which keep no
// rows (K = 3 without accounting), else the most that any k takes.  (The 5-clique bands are the
// slower with only their own: one CTA more per SM takes L1 from the pair tests; 65,536 vertices,
// edge factor 16: 0.96 ms, 1.36 ms so.)
template <int K, bool STATS = false>
__host__ __device__ constexpr int row_words(int W) {
  const int odd = W | 1, four = (((W + 3) >> 2) | 1) << 2;
  return K == 3 && !STATS ? 0 : odd > four ? odd : four;
}

// Balanced 5-clique count of the widest band (BAL, rows of up to 32 words): per warp, the
// R_i & R_j masks of 32 (i, j) pairs (RW words each, word q of lane l at q * 32 + l) and a list
// of kBalCap packed items (k | lane << 10).
constexpr int kBalCap = 512;
__host__ __device__ __forceinline__ size_t bal_bytes(int rw) {
  return (size_t)8 * ((size_t)rw * 32 * 4 + (size_t)kBalCap * 2);
}

// 5-cliques of a CTA root: the members of one row per warp (rows of up to 16 words).
constexpr int kRowMembers = 512;
constexpr int kCtaWarps = 8;
// Rows of up to 32 kTriWords members are counted by row_triangles, denser ones pair by pair.
// Four words keep the kernel at 64 registers; on the R-MAT scale 22 graph 2,072 of 1.86 M rows of
// the <= 256 band have more than 128 members.
constexpr int kTriWords = 4;
// Buffers of the 5-clique count for masks of rw words: counters, then (rw <= 16) the members of
// one row per warp, the members of the rows with at most kRowFew, and the rows by size, or (rw =
// 32) the item buffers, over the same memory.
__host__ __device__ __forceinline__ size_t k5_bytes(int rw, int dmax) {
  if (rw <= 0) return 0;
  const size_t b = rw <= 16 ? (size_t)kCtaWarps * kRowMembers * 2 +
                                  (size_t)dmax * kRowFew * 2 + (size_t)dmax * 4
                            : bal_bytes(rw);
  return 16 + b + 16;  // counters, buffers, alignment slack
}

// Shared layout for one mid-tier root (dynamic shared memory):
//   L[dmax] ids | rb[dmax] bitmap rows | off[dmax+1] pair offsets, or row counts | deg[dmax]
//   out-degrees, or column counts | R[dmax * row_w] rows | 8 warp sums | 5-clique buffers (bal_rw)
struct MidLayout {
  int dmax;
  int row_w;       // words allotted per row (row_words)
  int bal_rw = 0;  // mask words of the 5-clique buffers (0: none)
  __host__ __device__ size_t bytes() const {
    return bytes_no_rows() + (size_t)dmax * row_w * 4;
  }
  __host__ __device__ size_t bytes_no_rows() const {
    return (size_t)dmax * 16 + 4 + 16 + 64 + 64 + k5_bytes(bal_rw, dmax);
  }
};

struct MidSmem {
  vid_t* L;
  uint32_t* rb;
  int* off;
  int* deg;
  uint32_t* R;
  int* wsum;
  int* k5_next;        // 5-clique count: next task, rows of <= 8, <= 16 and more members
  uint16_t* mem;       // members: 8 warps x kRowMembers
  uint16_t* few;       // members of the rows of <= kRowFew, kRowFew each
  uint16_t* list;      // those rows' sizes from the front (<= 8) and the back (<= 16)
  uint16_t* big;       // rows with more members
  uint32_t* bal_m;     // item form: 8 warps x RW x 32 mask words
  uint16_t* bal_list;  // item form: 8 warps x kBalCap items
  // rows = nullptr: the rows follow in shared memory (MidLayout); otherwise they live at
  // rows (dmax * W words of global scratch for this CTA) and shared memory holds the rest
  // (MidLayout::bytes_no_rows).
  __device__ __forceinline__ static MidSmem carve(unsigned char* smem, int dmax, int row_w,
                                                  uint32_t* rows = nullptr, int bal_rw = 0) {
    MidSmem m;
    m.L = reinterpret_cast<vid_t*>(smem);
    m.rb = reinterpret_cast<uint32_t*>(m.L + dmax);
    m.deg = reinterpret_cast<int*>(m.rb + dmax);
    m.off = m.deg + dmax;
    // rows start on 16 bytes
    uint32_t* after = reinterpret_cast<uint32_t*>(
        (reinterpret_cast<uintptr_t>(m.off + dmax + 1) + 15) & ~uintptr_t(15));
    if (rows) {
      m.R = rows;
      m.wsum = reinterpret_cast<int*>(after);
    } else {
      m.R = after;
      m.wsum = reinterpret_cast<int*>(m.R + (size_t)dmax * row_w);
    }
    m.k5_next = reinterpret_cast<int*>(
        (reinterpret_cast<uintptr_t>(m.wsum + 8) + 15) & ~uintptr_t(15));
    m.bal_m = reinterpret_cast<uint32_t*>(m.k5_next + 4);
    m.bal_list = reinterpret_cast<uint16_t*>(m.bal_m + (size_t)8 * bal_rw * 32);
    m.mem = reinterpret_cast<uint16_t*>(m.bal_m);
    m.few = m.mem + kCtaWarps * kRowMembers;
    m.list = m.few + (size_t)dmax * kRowFew;
    m.big = m.list + dmax;
    return m;
  }
};

// Rows up to this many words (out-degree <= 512) are counted row-parallel from registers.
constexpr int kCtaRowWords = 16;

// Exclusive scan of off[0..d) in place over the CTA (blocked per thread, then across
// warps); off[d] receives the total.
__device__ __forceinline__ void cta_exclusive_scan(int* off, int d, int* wsum) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthreads = blockDim.x;
  const int per = (d + nthreads - 1) / nthreads;
  const int b0 = min(d, tid * per), b1 = min(d, b0 + per);
  int local = 0;
  for (int i = b0; i < b1; ++i) local += off[i];
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int wbase = 0;
  for (int w = 0; w < warp; ++w) wbase += wsum[w];
  int run = wbase + incl - local;
  __syncthreads();
  for (int i = b0; i < b1; ++i) {
    const int l = off[i];
    off[i] = run;
    run += l;
  }
  if (tid == nthreads - 1) off[d] = run;
  __syncthreads();
}

// Items t = lane, lane + 32, ... < nit of a balanced round: popc(M_owner & R_k) over the
// first W words (W a compile-time multiple of 4 >= w_d; the mask words past w_d are zero).
template <int W>
__device__ __forceinline__ acc_t bal_items_w(const uint16_t* Lw, int nit, const uint32_t* Mw,
                                             const uint32_t* R, int S) {
  acc_t cnt = 0;
  for (int t2 = threadIdx.x & 31; t2 < nit; t2 += 32) {
    const uint32_t v = Lw[t2];
    const uint32_t* Rk = R + (size_t)(v & 1023u) * S;
    const uint32_t* Mo = Mw + (v >> 10);
    int s = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) s += __popc(Mo[q * 32] & Rk[q]);
    cnt += (acc_t)s;
  }
  return cnt;
}

// Rows of 17 to 32 words (the band of out-degree 513 to 1,024).
__device__ __forceinline__ acc_t bal_items(const uint16_t* Lw, int nit, const uint32_t* Mw,
                                           const uint32_t* R, int S, int w_d) {
  switch ((w_d + 3) >> 2) {
    case 5: return bal_items_w<20>(Lw, nit, Mw, R, S);
    case 6: return bal_items_w<24>(Lw, nit, Mw, R, S);
    case 7: return bal_items_w<28>(Lw, nit, Mw, R, S);
    default: return bal_items_w<32>(Lw, nit, Mw, R, S);
  }
}

// 5-cliques of one root from its bitmap rows, with the work spread evenly over the lanes.
// off[0..d] holds the exclusive prefix of the row popcounts (P = off[d] pairs (i, j), j a
// bit of R_i).  A warp takes 32 pairs at a time: each lane forms m = R_i & R_j, then the
// bits k of all 32 masks are expanded into an item list (at most kBalCap per round) that
// the lanes take round-robin; an item adds popc(m & R_k).  The work per item is the same
// for every lane, whatever the masks' sizes.
template <int RW>
__device__ __forceinline__ acc_t bal_count5(const int* off, int d, int topO,
                                            const uint32_t* R, int w_d, int S,
                                            uint32_t* Mw, uint16_t* Lw) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int P = off[d];
  acc_t cnt = 0;
  for (int base = warp * 32; base < P; base += nwarps * 32) {
    const int p = base + lane;
    uint32_t m2[RW];
    int c = 0;
    if (p < P) {
      const int i = count_below(off + 1, d - 1, topO, p + 1);
      const uint32_t* Ri = R + (size_t)i * S;
      const int j = select_bit(Ri, w_d, p - off[i]);
      const uint32_t* Rj = R + (size_t)j * S;
#pragma unroll
      for (int q = 0; q < RW; ++q) {
        m2[q] = q < w_d ? (Ri[q] & Rj[q]) : 0u;
        c += __popc(m2[q]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < RW; ++q) m2[q] = 0u;
    }
#pragma unroll
    for (int q = 0; q < RW; ++q)
      if (q < ((w_d + 3) & ~3)) Mw[q * 32 + lane] = m2[q];  // m2[q] = 0 for q >= w_d
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    const int first = incl - c;
    const int C = __shfl_sync(kFull, incl, 31);
    for (int r0 = 0; r0 < C; r0 += kBalCap) {
      // this lane's items with index in [r0, r0 + kBalCap)
      const int tend = min(first + c, r0 + kBalCap);
      int t = first;
      if (t < tend) {
#pragma unroll
        for (int q = 0; q < RW; ++q) {
          uint32_t w = m2[q];
          const int pc = __popc(w);
          if (t + pc <= r0) {  // the whole word lies before this round
            t += pc;
            continue;
          }
          while (w != 0u && t < tend) {
            const int b = __ffs(w) - 1;
            w &= w - 1;
            if (t >= r0) Lw[t - r0] = (uint16_t)((q * 32 + b) | (lane << 10));
            ++t;
          }
        }
      }
      __syncwarp();
      const int nit = min(C - r0, kBalCap);
      cnt += bal_items(Lw, nit, Mw, R, S, w_d);
      __syncwarp();
    }
  }
  return cnt;
}

// Row block and column block of tile t of the lower triangle (t = B (B + 1) / 2 + b).
__device__ __forceinline__ void tile_at(int t, int& B, int& b) {
  B = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (B * (B + 1) / 2 > t) --B;
  while ((B + 1) * (B + 2) / 2 <= t) ++B;
  b = t - B * (B + 1) / 2;
}

// 4-cliques of a root's tile (B, b), by one warp: sum of popc(R_i & R_j) over the rows i of block
// B and the bits j of R_i in block b.  Lane j holds four words of R_j at a time; R_i is read
// for the whole warp.  Words past b are zero in R_j.  (Out-degree 129..256 of the scale 22 graph's
// 4-clique count, tests and pairs: 727 us row by row, 469 us by tiles.)
__device__ __forceinline__ unsigned tile_pairs(const uint32_t* R, int S, int B, int b, int d) {
  const int lane = threadIdx.x & 31;
  const int nrow = min(32, d - 32 * B);
  const uint32_t* Ri = R + (size_t)(32 * B) * S;
  const uint32_t mine = lane < nrow ? Ri[(size_t)lane * S + b] : 0u;
  unsigned live = __ballot_sync(kFull, mine != 0u);  // rows with a bit in block b
  if (live == 0u) return 0u;
  const int j = 32 * b + lane;
  unsigned c = 0;
  for (int q0 = 0; q0 <= b; q0 += 4) {
    uint4 rj = make_uint4(0u, 0u, 0u, 0u);
    if (j < d) rj = *reinterpret_cast<const uint4*>(R + (size_t)j * S + q0);
#pragma unroll 4
    for (int r = 0; r < nrow; ++r) {
      const uint32_t m = __shfl_sync(kFull, mine, r);
      const uint4 ri = *reinterpret_cast<const uint4*>(Ri + (size_t)r * S + q0);
      const unsigned t = __popc(ri.x & rj.x) + __popc(ri.y & rj.y) + __popc(ri.z & rj.z) +
                         __popc(ri.w & rj.w);
      if ((m >> lane) & 1u) c += t;
    }
  }
  return c;
}

// One root of out-degree 32 < d <= dmax processed by the whole CTA (blockDim = 256).
// Every thread calls it; returns this thread's partial count.  Pairs are tested in tiles, one
// per warp (test_tile).  k = 4 counts from rows in shared memory by the same tiles (tile_pairs),
// k = 5 row by row (row_triangles, group_triangles); larger k with rows of up to ROWW words flatten the first two levels over the
// threads, with masks in registers; wider ones (or all, with ROWW = 0) are counted
// warp-cooperatively with WPL mask words per lane (rows of up to 32 WPL words).  BAL (k = 5,
// rows of up to ROWW words in shared memory, no accounting): the layout carries the 5-clique
// buffers (MidLayout::bal_rw = ROWW).
template <int K, bool STATS, bool ETRI, bool PAIRS = false, int ROWW = kCtaRowWords,
          int WPL = 1, bool GR = false, bool TT = false, bool BAL = false>
__device__ __forceinline__ acc_t cta_root(const RankDag& g, vid_t u, const MidSmem& sm,
                                          uint32_t* tri, acc_t& elems) {
  static_assert(!BAL || (K == 5 && !STATS && !ETRI && !GR && ROWW > 0),
                "the balanced count is for plain 5-clique counts with rows in shared memory");
  static_assert(!GR || ROWW == 0, "rows in global memory are counted warp-cooperatively");
  constexpr bool STORE = K >= 4 || STATS;  // k = 3 counts its hits as they are found
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nthreads = blockDim.x;
  const int nwarps = nthreads >> 5;
  vid_t* L = sm.L;
  int* off = sm.off;
  int* deg = sm.deg;
  uint32_t* R = sm.R;
  const eid_t base = g.rp[u];
  const int d = (int)(g.rp[u + 1] - base);
  const int w_d = (d + 31) >> 5;
  const int S = row_stride<K>(w_d, GR);
  int low = 0;
  for (int j = tid; j < d; j += nthreads) {
    const vid_t x = __ldg(g.col + base + j);
    L[j] = x;
    const uint32_t xb = bit_row(g, x);
    sm.rb[j] = xb;
    low += xb != kNoRow ? 1 : 0;
    // edge-triangle mode: deg[] holds the column counts, off[] the row counts
    if (ETRI || STATS) deg[j] = ETRI ? 0 : (int)(g.rp[x + 1] - g.rp[x]);
    if (ETRI) off[j] = 0;
  }
  if (BAL && tid < 4) sm.k5_next[tid] = 0;
  low = __reduce_add_sync(kFull, (unsigned)low);
  if (lane == 0) sm.wsum[warp] = low;
  __syncthreads();
  int hc = 0;  // rows below hc are tested in the bitmap (L ascends)
  for (int q = 0; q < nwarps; ++q) hc += sm.wsum[q];
  acc_t cnt = 0, pairs = 0, tt = 0;
  unsigned c32 = 0;
  const int tiles = w_d * (w_d + 1) / 2;
  const int wz = !GR && K == 4 ? (w_d + 3) & ~3 : w_d;  // words of a row that are read
  for (int t = warp; t < tiles; t += nwarps) {
    int B, b;
    tile_at(t, B, b);
    unsigned colc = 0;
    const int j = 32 * b + lane, nrow = min(32, d - 32 * B);
    const vid_t w = j < d ? L[j] : INT32_MAX;
    const uint32_t* rb = sm.rb + 32 * B;
    const vid_t* Lx = L + 32 * B;
    const uint32_t word = test_tile<ETRI>(
        g, w, b < B ? 0 : lane + 1, nrow, max(0, min(nrow, hc - 32 * B)),
        [&](int r) { return rb[min(r, nrow - 1)]; }, [&](int r) { return Lx[min(r, nrow - 1)]; },
        pairs, [&](int, eid_t e) {
          const unsigned o = atomicAdd(tri + e, 1u);
          ++colc;
          return PAIRS ? o : 0u;
        });
    const int i = 32 * B + lane;
    if (K == 3 && !PAIRS) c32 += (unsigned)__popc(word);
    if (ETRI) {
      if (word) atomicAdd(&off[i], (int)__popc(word));
      if (colc) atomicAdd(&deg[32 * b + lane], (int)colc);
    }
    if (STORE && i < d) {
      uint32_t* Ri = R + (size_t)i * S;
      if (GR) __stcg(Ri + b, word);
      else Ri[b] = word;
      if (b == B) {  // zeros up to the row's end
        for (int q = B + 1; q < wz; ++q) {
          if (GR) __stcg(Ri + q, 0u);
          else Ri[q] = 0u;
        }
      }
    }
  }
  __syncthreads();
  if (ETRI) {  // the root's own arcs: popc(R_i) + (rows with bit i) triangles each
    for (int i = tid; i < d; i += nthreads) {
      const unsigned pc = (unsigned)off[i];
      const unsigned tu = pc + (unsigned)deg[i];
      if (tu) {
        const unsigned o = atomicAdd(tri + base + i, tu);
        if (PAIRS) pairs += pair_gain(o, tu);
        if (TT) {
          const acc_t di = tt_deg(g, L[i]);
          tt += (acc_t)pc * (tt_deg(g, u) + di) + (acc_t)deg[i] * di;
        }
      }
    }
  }
  if (PAIRS && !TT) {
    __syncthreads();
    return pairs;
  }
  constexpr int RW = ROWW > 0 ? ROWW : 1;
  if (K == 3 && !STATS) {
    cnt = c32;
  } else if (K == 4 && !STATS && !GR) {
    // tiles by weight, heaviest (largest b) first within each warp's share
    for (int t = tiles - 1 - warp; t >= 0; t -= nwarps) {
      int B, b;
      tile_at(t, B, b);
      cnt += (acc_t)tile_pairs(R, S, B, b, d);
    }
  } else if (BAL && RW <= 16 && w_d <= ROWW) {
    // rows by their number of members c: those of c <= 8 and c <= 16 get their members listed
    // one row per thread and are counted four and two to a warp, the others one to a warp
    for (int i = tid; i < d; i += nthreads) {
      const uint32_t* Ri = R + (size_t)i * S;
      int c = 0;
      for (int q = 0; q < w_d; ++q) c += __popc(Ri[q]);
      if (c < 3) continue;
      if (c > kRowFew) {
        sm.big[atomicAdd(&sm.k5_next[3], 1)] = (uint16_t)i;
        continue;
      }
      const int slot = c <= 8 ? atomicAdd(&sm.k5_next[1], 1) : d - 1 - atomicAdd(&sm.k5_next[2], 1);
      sm.list[slot] = (uint16_t)c;
      uint16_t* out = sm.few + (size_t)slot * kRowFew;
      for (int q = 0; q < w_d; ++q)
        for (uint32_t m = Ri[q]; m != 0u; m &= m - 1u) *out++ = (uint16_t)(32 * q + __ffs(m) - 1);
    }
    __syncthreads();
    const int n8 = sm.k5_next[1], n16 = sm.k5_next[2], nbig = sm.k5_next[3];
    const int t16 = (n16 + 1) >> 1, t8 = (n8 + 3) >> 2;
    uint16_t* Pw = sm.mem + (size_t)warp * kRowMembers;
    for (;;) {  // tasks from a shared counter
      int t = 0;
      if (lane == 0) t = atomicAdd(sm.k5_next, 1);
      t = __shfl_sync(kFull, t, 0);
      if (t >= nbig + t16 + t8) break;
      if (t >= nbig + t16) {
        const int q = 4 * (t - nbig - t16) + (lane >> 3);
        const int at = q < n8 ? q : 0;
        cnt += (acc_t)group_triangles<8>(R, S, sm.few + (size_t)at * kRowFew,
                                         q < n8 ? (int)sm.list[at] : 0);
        continue;
      }
      if (t >= nbig) {
        const int q = 2 * (t - nbig) + (lane >> 4);
        const int at = d - 1 - (q < n16 ? q : 0);
        cnt += (acc_t)group_triangles<16>(R, S, sm.few + (size_t)at * kRowFew,
                                          q < n16 ? (int)sm.list[at] : 0);
        continue;
      }
      const uint32_t* Ri = R + (size_t)sm.big[t] * S;
      const int c = row_members(Ri, w_d, Pw);
      __syncwarp();
      if (c <= 32 * kTriWords) {
        cnt += (acc_t)row_triangles<kTriWords>(R, S, Pw, c);
      } else {  // a dense row: pair by pair
        for (int jj = lane; jj < c; jj += 32) {
          const uint32_t* Rj = R + (size_t)Pw[jj] * S;
          uint32_t m2[RW];
#pragma unroll
          for (int q = 0; q < RW; ++q) m2[q] = q < w_d ? (Ri[q] & Rj[q]) : 0u;
          cnt += RowCount<1, RW, false>::run(m2, R, w_d, deg, elems, S);
        }
      }
      __syncwarp();
    }
  } else if (ROWW > 0 && w_d <= ROWW && K >= 5 && !ETRI) {
    // k >= 5: the first two levels flattened over the threads as (row i, bit j of R_i)
    // pairs, so one dense row does not hold up the CTA.  off[i] = pairs before row i.
    for (int i = tid; i < d; i += nthreads) {
      int c = 0;
      for (int q = 0; q < w_d; ++q) c += __popc(R[(size_t)i * S + q]);
      off[i] = c;
    }
    __syncthreads();
    cta_exclusive_scan(off, d, sm.wsum);
    const int topO = top_pow2(d - 1);
    if (BAL) {
      cnt += bal_count5<RW>(off, d, topO, R, w_d, S, sm.bal_m + (size_t)warp * RW * 32,
                            sm.bal_list + (size_t)warp * kBalCap);
    } else {
      const int P = off[d];
      for (int p = tid; p < P; p += nthreads) {
        const int i = count_below(off + 1, d - 1, topO, p + 1);
        const uint32_t* Ri = R + (size_t)i * S;
        const int j = select_bit(Ri, w_d, p - off[i]);
        const uint32_t* Rj = R + (size_t)j * S;
        uint32_t m2[RW];
#pragma unroll
        for (int q = 0; q < RW; ++q) m2[q] = q < w_d ? (Ri[q] & Rj[q]) : 0u;
        if (STATS) elems += (acc_t)(off[i + 1] - off[i]) + (acc_t)deg[j];
        cnt += RowCount<(K >= 5 ? K - 4 : 1), RW, STATS>::run(m2, R, w_d, deg, elems, S);
      }
    }
  } else if (ROWW > 0 && w_d <= ROWW) {
    // accounting: each thread owns rows, masks in registers
    for (int i = tid; i < d; i += nthreads) {
      uint32_t m[RW];
#pragma unroll
      for (int q = 0; q < RW; ++q) m[q] = q < w_d ? R[(size_t)i * S + q] : 0u;
      cnt += RowCount<K - 3, RW, STATS>::run(m, R, w_d, deg, elems, S);
    }
  } else {
    // wide rows: the mask is distributed over the lanes, WPL words each
    for (int i = warp; i < d; i += nwarps) {
      uint32_t mw[WPL];
#pragma unroll
      for (int q = 0; q < WPL; ++q) {
        const int w = q * 32 + lane;
        mw[q] = w < w_d ? ld_row<GR>(R + (size_t)i * S + w) : 0u;
      }
      cnt += DistCount<K - 3, WPL, STATS, GR>::run(mw, R, w_d, deg, elems, S);
    }
  }
  __syncthreads();
  if (TT) return 12ull * cnt - 4ull * pairs + tt;
  return cnt;
}

}  // namespace jgpm
