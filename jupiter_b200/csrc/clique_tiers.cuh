// The per-tier k-clique kernels and their launch templates, shared by the translation units
// that instantiate them (clique_k*.cu, one or two clique sizes each, so the build compiles
// them in parallel).  See clique.cu for the design.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "clique_dev.cuh"
#include "jgpm_internal.h"
#include "setops.cuh"

namespace jgpm {

struct CliqueArgs {
  RankDag dag;
  const vid_t* roots;
  int64_t begin, end;   // root range of this launch: roots[begin + (i - begin) * step],
  int64_t step;         // begin <= i < end (step > 1: one shard's roots of a tier)
  DevControl* ctl;
  int32_t* scratch;     // large tier: per-warp lists
  int64_t scratch_per_warp;
  uint32_t* rows;       // CTA tiers with rows in global memory: dmax * W words per CTA
  int large_chunks;     // list tier: tasks per root (chunks of 32 arcs of the widest root)
  int cursor;           // which ctl->counter this launch steals from
  uint32_t* tri;        // edge-triangle modes: triangles per DAG arc
};

// Kernel variants: PAIRS (with ETRI, K == 3) returns sum_e C(t_e, 2) as the count; TT (with
// ETRI and PAIRS, K == 4) the vertex-induced tailed-triangle count (clique_dev.cuh).

constexpr int kMaxLevels = 6;  // list tier: candidate lists per warp

// Tier indices b, b + step, ..., (e - b) of them.
struct TierRange {
  int64_t b = 0, e = 0;
  int64_t step = 1;
  bool empty() const { return e <= b; }
};

// Root of launch index i (a.begin <= i < a.end).
__device__ __forceinline__ vid_t root_at(const CliqueArgs& a, int64_t i) {
  return a.roots[a.begin + (i - a.begin) * a.step];
}

// Launch plan of one count: the root ranges of each tier.  wide holds the CTA roots of
// out-degree (1024, 4096] (rows in global scratch); mid[0..2] are the CTA-root bands of
// out-degree (512, 1024], (256, 512] and (split, 256].
struct TierPlan {
  TierRange large, wide, mid[3], warp, g32, g16, g8, g4;
  TierRange scan;  // all roots above 32, of a graph without a rank DAG
};

// CTAs and global row words of a wide/global-row band of out-degree <= dmax: at most
// kRowsBudget bytes of rows so that they stay in L2.
constexpr size_t kRowsBudget = (size_t)96 << 20;
inline int rows_band_grid(int dmax, int sms, int64_t roots) {
  const size_t per = (size_t)dmax * ((dmax + 31) / 32) * 4;
  const int64_t by_budget = (int64_t)std::max<size_t>(1, kRowsBudget / per);
  return (int)std::max<int64_t>(
      1, std::min<int64_t>(std::min<int64_t>((int64_t)sms * 4, by_budget), roots));
}

// Launches the tiers of one count for clique size k (3..8).  mode: 0 count, 1 count with the
// set-op accounting, 2 edge triangles (k = 3), 3 diamond pairs (k = 3), 4 vertex-induced
// tailed triangles (k = 4).  Returns the number of kernels launched.
int launch_tiers_k3(int mode, const CliqueArgs& a, const TierPlan& p, int sms, cudaStream_t s,
                    int max_out);
int launch_tiers_k4(int mode, const CliqueArgs& a, const TierPlan& p, int sms, cudaStream_t s,
                    int max_out);
int launch_tiers_k5(int mode, const CliqueArgs& a, const TierPlan& p, int sms, cudaStream_t s,
                    int max_out);
int launch_tiers_k6(int mode, const CliqueArgs& a, const TierPlan& p, int sms, cudaStream_t s,
                    int max_out);
int launch_tiers_k78(int k, int mode, const CliqueArgs& a, const TierPlan& p, int sms,
                     cudaStream_t s, int max_out);

namespace {

// The tier kernels of one count share nothing but their atomic result adds (each has its own
// cursor and its own scratch), so every tier after the first is launched with programmatic
// stream serialization and overlaps the previous tier's last CTAs (pdl_open / pdl_close).

// Adds a warp's count (and accounting elements) to the control block: one atomic per CTA.
// Every thread of the CTA calls it, at its end.
template <bool STATS>
__device__ __forceinline__ void add_result(DevControl* ctl, acc_t cnt, acc_t elems) {
  __shared__ acc_t s_sum[2];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(kFull, cnt, o);
    if (STATS) elems += __shfl_xor_sync(kFull, elems, o);
  }
  __syncthreads();
  if (lane == 0 && cnt) atomicAdd(&s_sum[0], cnt);
  if (STATS && lane == 0 && elems) atomicAdd(&s_sum[1], elems);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_sum[0]) atomicAdd(&ctl->count[0], s_sum[0]);
    if (STATS && s_sum[1]) atomicAdd(&ctl->elements[0], s_sum[1]);
  }
}

// ------------------------------------------------------------------ small tiers (d <= 32)
// The four lane-group tiers in one launch: tasks of 32 / G roots, the wide groups first.  The
// roots are short and bound by the latency of their loads (root, row, list, tests), so each warp
// fetches its next task while it works, and the tiers share one tail.  (Triangles of 1,000
// vertices: 54 us in three launches, 35 us in one.)
struct SmallRanges {
  TierRange g[4];  // groups of 32, 16, 8, 4 lanes
};

template <int G, int K, bool STATS, bool ETRI, bool PAIRS, bool TT>
__device__ __forceinline__ acc_t small_task(const CliqueArgs& a, const TierRange& r, int64_t task,
                                            uint32_t* rows, int* degs, acc_t& elems) {
  const int gi = (threadIdx.x & 31) / G;
  const int64_t i = r.b + task * (32 / G) + gi;
  const vid_t u = i < r.e ? a.roots[r.b + (i - r.b) * r.step] : -1;
  return group_root<G, K, STATS, ETRI, PAIRS, TT>(a.dag, u, rows + gi * G, degs + gi * G, a.tri,
                                                  elems);
}

template <int K, bool STATS, bool ETRI = false, bool PAIRS = false, bool TT = false>
__global__ void __launch_bounds__(256) k_clique_small(CliqueArgs a, SmallRanges r) {
  __shared__ uint32_t rows_s[256];
  __shared__ int degs_s[256];
  const int lane = threadIdx.x & 31;
  uint32_t* rows = rows_s + (threadIdx.x & ~31);
  int* degs = degs_s + (threadIdx.x & ~31);
  pdl_open();
  int64_t end[4], n = 0;  // end of each tier's tasks
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int per = 1 << q;
    n += (r.g[q].e - r.g[q].b + per - 1) >> q;
    end[q] = n;
  }
  acc_t cnt = 0, elems = 0;
  auto fetch = [&]() {
    unsigned long long c = 0;
    if (lane == 0) c = atomicAdd(&a.ctl->counter[a.cursor], 1ull);
    return (int64_t)c;
  };
  int64_t next = fetch();
  for (;;) {
    const int64_t t = __shfl_sync(kFull, next, 0);
    if (t >= n) break;
    next = fetch();
    if (t < end[0])
      cnt += small_task<32, K, STATS, ETRI, PAIRS, TT>(a, r.g[0], t, rows, degs, elems);
    else if (t < end[1])
      cnt += small_task<16, K, STATS, ETRI, PAIRS, TT>(a, r.g[1], t - end[0], rows, degs, elems);
    else if (t < end[2])
      cnt += small_task<8, K, STATS, ETRI, PAIRS, TT>(a, r.g[2], t - end[1], rows, degs, elems);
    else
      cnt += small_task<4, K, STATS, ETRI, PAIRS, TT>(a, r.g[3], t - end[2], rows, degs, elems);
  }
  add_result<STATS>(a.ctl, cnt, elems);
  pdl_close();
}

// ------------------------------------------------------------------ warp tier (d <= 128)
// Four CTAs per SM: 64 registers hold the rows of a root of up to 128 entries.
template <int K, bool STATS, bool ETRI = false, bool PAIRS = false, bool TT = false>
__global__ void __launch_bounds__(256, 4) k_clique_warp(CliqueArgs a) {
  extern __shared__ __align__(16) unsigned char wsmem[];
  WarpSmem* ws = reinterpret_cast<WarpSmem*>(wsmem) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  pdl_open();
  acc_t cnt = 0, elems = 0;
  auto fetch = [&]() {
    unsigned long long c = 0;
    if (lane == 0) c = atomicAdd(&a.ctl->counter[a.cursor], 1ull);
    return (int64_t)c;
  };
  int64_t next = fetch();
  for (;;) {
    const int64_t idx = a.begin + __shfl_sync(kFull, next, 0);
    if (idx >= a.end) break;
    next = fetch();
    cnt += warp_root<K, STATS, ETRI, PAIRS, TT>(a.dag, root_at(a, idx), ws, a.tri, elems);
  }
  add_result<STATS>(a.ctl, cnt, elems);
  pdl_close();
}

// ------------------------------------------- roots above 32 of a graph without a rank DAG
template <int K, bool STATS, bool ETRI = false, bool PAIRS = false, bool TT = false>
__global__ void __launch_bounds__(256) k_clique_scan(CliqueArgs a) {
  __shared__ ScanSmem sm;
  pdl_open();
  acc_t cnt = 0, elems = 0;
  for (int64_t i = a.begin + blockIdx.x; i < a.end; i += gridDim.x)
    cnt += scan_root<K, STATS, ETRI, PAIRS, TT>(a.dag, root_at(a, i), sm, a.tri, elems);
  add_result<STATS>(a.ctl, cnt, elems);
  pdl_close();
}

// --------------------------------------------------- CTA tiers (32 < d <= kWideMaxDeg)
// GR: the bitmap rows live in global scratch (a.rows, dmax * W words per CTA, L2-resident)
// and the shared memory holds only the root's list and row offsets.
// Four CTAs per SM (64 registers) for the counts of k <= 5; the item form of the widest 5-clique
// band and the larger k need more.
template <int K, bool STATS, bool BAL, int ROWW>
constexpr int kMidMinBlocks() {
  return !STATS && (K <= 4 || (BAL && ROWW <= 16)) ? 4 : 1;
}

template <int K, bool STATS, bool ETRI = false, bool PAIRS = false, int ROWW = kCtaRowWords,
          int WPL = 1, bool GR = false, bool TT = false, bool BAL = false>
__global__ void __launch_bounds__(256, kMidMinBlocks<K, STATS, BAL, ROWW>())
    k_clique_mid(CliqueArgs a, int dmax, int W) {
  extern __shared__ __align__(16) unsigned char smem[];
  const MidSmem sm = MidSmem::carve(smem, dmax, row_words<K, STATS>(W),
                                    GR ? a.rows + (size_t)blockIdx.x * dmax * W : nullptr,
                                    BAL ? ROWW : 0);
  __shared__ unsigned long long s_idx[2];
  const int tid = threadIdx.x;
  pdl_open();
  acc_t cnt = 0, elems = 0;
  // the next root is fetched while this one runs: cta_root's barriers lie between the store of a
  // slot and its read, and between its read and its next store
  if (tid == 0) s_idx[0] = atomicAdd(&a.ctl->counter[a.cursor], 1ull);
  __syncthreads();
  for (int it = 0;; ++it) {
    const int64_t idx = (int64_t)s_idx[it & 1] + a.begin;
    if (idx >= a.end) break;
    if (tid == 0) s_idx[(it + 1) & 1] = atomicAdd(&a.ctl->counter[a.cursor], 1ull);
    cnt += cta_root<K, STATS, ETRI, PAIRS, ROWW, WPL, GR, TT, BAL>(a.dag, root_at(a, idx), sm,
                                                                   a.tri, elems);
  }
  __syncthreads();
  add_result<STATS>(a.ctl, cnt, elems);
  pdl_close();
}

// ------------------------------------------------------------------ large tier (d > 1024)
// Edge-rooted, list based: one warp per arc (u, v_i) of a large root.  Candidate lists of
// each level live in the warp's global scratch (kMaxLevels lists of max_out entries).
// REM = levels still to choose (compile-time, so no device-side recursion at run time).
template <int REM, bool STATS>
struct ListClique {
  __device__ static acc_t run(const CliqueArgs& a, const vid_t* cand, int nc, int32_t* buf,
                              int64_t cap, acc_t& elems) {
    const int lane = threadIdx.x & 31;
    acc_t s = 0;
    for (int i = 0; i < nc; ++i) {
      const vid_t v = cand[i];
      const eid_t b = a.dag.rp[v];
      const int dv = (int)(a.dag.rp[v + 1] - b);
      if (STATS && lane == 0) elems += (acc_t)nc + (acc_t)dv;
      if (REM == 1) {
        int c = 0;  // |cand & N+(v)|, lookups of cand (written by this warp) in N+(v)
        for (int q = lane; q < nc; q += 32)
          if (contains_g(a.dag.col + b, dv, cand[q])) ++c;
        s += (acc_t)warp_sum_int(c);
      } else {
        const int t = warp_intersect_w(cand, nc, a.dag.col + b, dv, INT32_MAX, buf);
        if (t > 0)
          s += ListClique<(REM > 1 ? REM - 1 : 1), STATS>::run(a, buf, t, buf + cap, cap, elems);
      }
    }
    return s;
  }
};

template <int K, bool STATS, bool ETRI = false, bool PAIRS = false, bool TT = false>
__global__ void __launch_bounds__(256) k_clique_large(CliqueArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t gwarp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int32_t* buf = a.scratch + gwarp * a.scratch_per_warp;
  const int64_t cap = a.scratch_per_warp / kMaxLevels;
  pdl_open();
  acc_t cnt = 0, elems = 0;
  for (;;) {
    // task t = chunk (t mod large_chunks) of 32 arcs of root begin + t / large_chunks
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(&a.ctl->counter[a.cursor], 1ull);
    t = __shfl_sync(kFull, t, 0);
    const int64_t r = a.begin + (int64_t)(t / (unsigned long long)a.large_chunks);
    if (r >= a.end) break;
    const vid_t u = root_at(a, r);
    const eid_t bu = a.dag.rp[u];
    const int du = (int)(a.dag.rp[u + 1] - bu);
    const int i0 = (int)(t % (unsigned long long)a.large_chunks) * 32;
    for (int i = i0; i < min(du, i0 + 32); ++i) {
      const vid_t v = __ldg(a.dag.col + bu + i);
      const eid_t bv = a.dag.rp[v];
      const int dv = (int)(a.dag.rp[v + 1] - bv);
      int32_t* W = buf;
      const int tw = warp_intersect(a.dag.col + bu, du, a.dag.col + bv, dv, INT32_MAX, W);
      // tw and the ListClique sums are the same in every lane: lane 0 keeps them.  Pair
      // gains enter the TT value with weight -4, 4-cliques with weight 12.
      const acc_t pw = TT ? (acc_t)0 - 4ull : 1ull;
      if (ETRI && tw > 0) {
        if (lane == 0) {
          const unsigned o = atomicAdd(a.tri + bu + i, (unsigned)tw);
          if (PAIRS) cnt += pw * pair_gain(o, (unsigned)tw);
        }
        const acc_t tuv = TT ? tt_deg(a.dag, u) + tt_deg(a.dag, v) : 0ull;
        for (int q = lane; q < tw; q += 32) {
          const vid_t w = W[q];
          const unsigned o1 = atomicAdd(a.tri + bu + lower_bound_g(a.dag.col + bu, du, w), 1u);
          const unsigned o2 = atomicAdd(a.tri + bv + lower_bound_g(a.dag.col + bv, dv, w), 1u);
          if (PAIRS) cnt += pw * ((acc_t)o1 + (acc_t)o2);
          if (TT) cnt += tuv + tt_deg(a.dag, w);
        }
        __syncwarp();
      }
      if (K == 3) {
        if (!PAIRS && lane == 0) cnt += (acc_t)tw;
      } else if (tw > 0 && (!PAIRS || TT)) {
        const acc_t c =
            ListClique<(K > 3 ? K - 3 : 1), STATS>::run(a, W, tw, buf + cap, cap, elems);
        if (lane == 0) cnt += TT ? 12ull * c : c;
      }
      __syncwarp();  // W is rewritten by the next arc
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(kFull, cnt, o);
    if (STATS) elems += __shfl_xor_sync(kFull, elems, o);
  }
  if (lane == 0) {
    if (cnt) atomicAdd(&a.ctl->count[0], cnt);
    if (STATS && elems) atomicAdd(&a.ctl->elements[0], elems);
  }
  pdl_close();
}

// True (with the error recorded) if the kernel just launched failed to launch (rc: the
// launch call's own status), so that a count never silently misses a tier.
inline bool launch_failed(cudaError_t* err, cudaError_t rc = cudaSuccess) {
  const cudaError_t last = cudaGetLastError();
  const cudaError_t e = rc != cudaSuccess ? rc : last;
  if (e == cudaSuccess) return false;
  *err = e;
  jgpm_set_error_(std::string("clique tier launch: ") + cudaGetErrorString(e));
  return true;
}

// Launches one tier kernel of 256 threads; after the first tier of a count (pdl) with
// programmatic stream serialization.
template <typename... Args>
cudaError_t tier_launch(bool pdl, void (*kern)(Args...), int grid, size_t smem, cudaStream_t s,
                        Args... args) {
  return launch_pdl(pdl, kern, grid, 256, smem, s, args...);
}

// Mask words that a CTA band counts from registers.  None (0) where nothing is: the plain counts of
// k <= 4, which work on tiles (one kernel for all bands), and k >= 7, counted warp-cooperatively,
// which keeps the deep register-mask recursion, and its compile time, out of the large sizes.
template <int K, bool STATS>
constexpr int kBandRowWords(int w) { return K >= 7 || (K <= 4 && !STATS) ? 0 : w; }

// The same for the band of out-degree <= 1024 (rows of up to 32 words): k = 5 over (row, bit) pairs
// and the accounting of k = 4 row-parallel, one 32-word mask per thread.
template <int K, bool STATS>
constexpr int kWideBandRowWords() { return (K == 4 && STATS) || K == 5 ? 32 : 0; }

// One CTA-root band: bitmap layout for out-degree <= dmax, masks of up to ROWW words counted
// from registers, wider ones with WPL words per lane; GR puts the rows in global scratch.
// A plain 5-clique count with rows in shared memory counts with the balanced form.
template <int K, bool STATS, bool ETRI, int ROWW, bool GR>
constexpr bool kBandBalanced() { return K == 5 && !STATS && !ETRI && ROWW > 0 && !GR; }

template <int K, bool STATS, bool ETRI, bool PAIRS, int ROWW, int WPL = 1, bool GR = false,
          bool TT = false>
cudaError_t launch_mid_band(CliqueArgs a, const TierRange& r, int cursor, int dmax, int sms,
                            cudaStream_t s, bool pdl) {
  a.begin = r.b;
  a.end = r.e;
  a.step = r.step;
  a.cursor = cursor;
  const int W = (dmax + 31) / 32;
  constexpr bool BAL = kBandBalanced<K, STATS, ETRI, ROWW, GR>();
  const MidLayout lay{dmax, row_words<K, STATS>(W), BAL ? ROWW : 0};
  const size_t sm = GR ? lay.bytes_no_rows() : lay.bytes();
  auto kern = k_clique_mid<K, STATS, ETRI, PAIRS, ROWW, WPL, GR, TT, BAL>;
  raise_smem_limit((const void*)kern, sm);  // a failure shows up as the launch error
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, sm);
  if (per_sm < 1) per_sm = 1;
  const int64_t roots = r.e - r.b;
  int grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)sms * per_sm, roots));
  if (GR) grid = std::min(grid, rows_band_grid(dmax, sms, roots));
  return tier_launch(pdl, kern, grid, sm, s, a, dmax, W);
}

template <int K, bool STATS, bool ETRI, bool PAIRS = false, bool TT = false>
int launch_plan_k(const CliqueArgs& base, const TierPlan& p, int sms, cudaStream_t s,
                  int max_out) {
  CliqueArgs a = base;
  int n = 0;
  cudaError_t err = cudaSuccess;
  // the first tier of a count is an ordinary launch (after the control block's reset in the
  // stream); the later ones overlap their predecessor's last CTAs
  auto pdl = [&]() { return n > 0; };
  if (!p.large.empty()) {
    a.begin = p.large.b;
    a.end = p.large.e;
    a.step = p.large.step;
    a.cursor = 2;
    const cudaError_t rc =
        tier_launch(pdl(), k_clique_large<K, STATS, ETRI, PAIRS, TT>, sms * 2, 0, s, a);
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  if (!p.wide.empty()) {
    const cudaError_t rc = launch_mid_band<K, STATS, ETRI, PAIRS, 0, 4, true, TT>(
        a, p.wide, 9, std::min(max_out, kWideMaxDeg), sms, s, pdl());
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  if (!p.mid[0].empty()) {
    const cudaError_t rc =
        launch_mid_band<K, STATS, ETRI, PAIRS, kWideBandRowWords<K, STATS>(), 1, false, TT>(
            a, p.mid[0], 1, std::min(max_out, kMidMaxDeg), sms, s, pdl());
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  if (!p.mid[1].empty()) {
    const cudaError_t rc =
        launch_mid_band<K, STATS, ETRI, PAIRS, kBandRowWords<K, STATS>(16), 1, false, TT>(
            a, p.mid[1], 0, std::min(max_out, 512), sms, s, pdl());
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  if (!p.mid[2].empty()) {
    const cudaError_t rc =
        launch_mid_band<K, STATS, ETRI, PAIRS, kBandRowWords<K, STATS>(8), 1, false, TT>(
            a, p.mid[2], 8, std::min(max_out, 256), sms, s, pdl());
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  if (!p.warp.empty()) {
    a.begin = p.warp.b;
    a.end = p.warp.e;
    a.step = p.warp.step;
    a.cursor = 7;
    const size_t sm = warp_smem_bytes<K, STATS>();
    raise_smem_limit((const void*)k_clique_warp<K, STATS, ETRI, PAIRS, TT>, sm);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clique_warp<K, STATS, ETRI, PAIRS, TT>,
                                                  256, sm);
    if (per_sm < 1) per_sm = 1;
    const int64_t grid = std::min<int64_t>((int64_t)sms * per_sm, (a.end - a.begin + 7) / 8);
    const cudaError_t rc =
        tier_launch(pdl(), k_clique_warp<K, STATS, ETRI, PAIRS, TT>, (int)grid, sm, s, a);
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  if (!p.scan.empty()) {
    a.begin = p.scan.b;
    a.end = p.scan.e;
    a.step = p.scan.step;
    const int64_t grid = std::min<int64_t>((int64_t)sms * 4, a.end - a.begin);
    const cudaError_t rc =
        tier_launch(pdl(), k_clique_scan<K, STATS, ETRI, PAIRS, TT>, (int)grid, 0, s, a);
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  SmallRanges sr{{p.g32, p.g16, p.g8, p.g4}};
  int64_t tasks = 0;
  for (int q = 0; q < 4; ++q) {
    sr.g[q].e = std::max(sr.g[q].e, sr.g[q].b);
    tasks += (sr.g[q].e - sr.g[q].b + (1 << q) - 1) >> q;
  }
  if (tasks > 0) {
    a.cursor = 3;
    auto kern = k_clique_small<K, STATS, ETRI, PAIRS, TT>;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0);
    // a short launch behind other tiers, whose last CTAs it overlaps, leaves them room: five CTAs
    // per SM (triangles of 65,536 vertices, edge factor 16: 85 us, 88 with as many as fit; a long
    // one, of 4,194,304 vertices, edge factor 4, a = 0.45, b = 0.2391: 0.81 and 0.71 ms)
    if (n > 0 && tasks < (int64_t)sms * 1024) per_sm = std::min(per_sm, 5);
    per_sm = std::max(1, per_sm);
    const int64_t grid = std::min<int64_t>((int64_t)sms * per_sm, (tasks + 7) / 8);
    const cudaError_t rc = tier_launch(pdl(), kern, (int)grid, 0, s, a, sr);
    ++n;
    if (launch_failed(&err, rc)) return -1;
  }
  return n;
}

}  // namespace
}  // namespace jgpm
