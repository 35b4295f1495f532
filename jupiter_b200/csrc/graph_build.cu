// Device-side graph construction: seeded R-MAT generation, CSR build (sort, dedup,
// symmetrise), validation of caller CSRs, degree orientation into a DAG, and the
// out-degree root tiers the clique kernels schedule from.
//
// Orientation keeps u->v iff deg(v) > deg(u) or (deg(v) == deg(u) and v > u), the rule of
// Graph::orientation (common/graph.cc:229-230, :383-384).  Because arcs are visited in
// CSR order, every DAG row stays sorted, as the reference's does.
#include <cub/cub.cuh>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <sstream>

#include "jgpm_internal.h"
#include "rmat.h"

namespace jgpm {

namespace {

__global__ void k_rmat_keys(RmatParams p, int shift, uint64_t* keys, uint64_t invalid) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.num_edges;
       i += stride) {
    int32_t u, v;
    bool ok = rmat_edge(p, (uint64_t)i, &u, &v);
    if (!ok || u == v) {
      keys[2 * i] = invalid;
      keys[2 * i + 1] = invalid;
    } else {
      keys[2 * i] = ((uint64_t)u << shift) | (uint64_t)v;
      keys[2 * i + 1] = ((uint64_t)v << shift) | (uint64_t)u;
    }
  }
}

__global__ void k_edge_keys(const int32_t* src, const int32_t* dst, int64_t ne, int32_t n,
                            int shift, uint64_t* keys, uint64_t invalid, int* bad) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += stride) {
    int32_t u = src[i], v = dst[i];
    if (u < 0 || v < 0 || u >= n || v >= n) {
      atomicExch(bad, 1);
      keys[2 * i] = invalid;
      keys[2 * i + 1] = invalid;
      continue;
    }
    if (u == v) {
      keys[2 * i] = invalid;
      keys[2 * i + 1] = invalid;
    } else {
      keys[2 * i] = ((uint64_t)u << shift) | (uint64_t)v;
      keys[2 * i + 1] = ((uint64_t)v << shift) | (uint64_t)u;
    }
  }
}

__global__ void k_unique_flags(const uint64_t* keys, int64_t nk, uint64_t invalid, int* flags) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nk; i += stride) {
    uint64_t k = keys[i];
    flags[i] = (k != invalid && (i == 0 || keys[i - 1] != k)) ? 1 : 0;
  }
}

__global__ void k_compact_keys(const uint64_t* keys, const int* flags, const int64_t* pos,
                               int64_t nk, uint64_t mask, uint64_t* ukeys, int32_t* col) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nk; i += stride) {
    if (flags[i]) {
      uint64_t k = keys[i];
      ukeys[pos[i]] = k;
      col[pos[i]] = (int32_t)(k & mask);
    }
  }
}

// rowptr[v] = first unique key with source >= v.
__global__ void k_rowptr_from_keys(const uint64_t* ukeys, int64_t m, int32_t n, int shift,
                                   int64_t* rowptr) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += stride) {
    uint64_t target = (uint64_t)v << shift;
    int64_t lo = 0, hi = m;
    while (lo < hi) {
      int64_t mid = (lo + hi) >> 1;
      if (ukeys[mid] < target) lo = mid + 1;
      else hi = mid;
    }
    rowptr[v] = lo;
  }
}

// Expands rowptr into the source of every arc (one warp per vertex).
__global__ void k_arc_src(const int64_t* rowptr, int32_t n, int32_t* src) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
    int64_t b = rowptr[v], e = rowptr[v + 1];
    for (int64_t k = b + lane; k < e; k += 32) src[k] = (int32_t)v;
  }
}

constexpr unsigned kAll = 0xffffffffu;

// Last v with rowptr[v] <= k (0 <= k < rowptr[n]), by one warp: 32 probes a round.
__device__ __forceinline__ int32_t warp_owner(const int64_t* rowptr, int32_t n, int64_t k) {
  const int lane = threadIdx.x & 31;
  int64_t lo = 0, hi = n;  // rowptr[lo] <= k < rowptr[hi]
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t at = lo + (int64_t)(lane + 1) * step;
    const bool le = at < hi && rowptr[at] <= k;
    const int c = __popc(__ballot_sync(kAll, le));
    const int64_t nlo = lo + (int64_t)c * step;
    hi = min(hi, nlo + step);
    lo = nlo;
  }
  return (int32_t)lo;
}

// The owners of the arcs, 32 to a word.  On larger graphs: a bit at the first arc of every row,
// the rows before each word, and the non-empty rows in order, so that an arc's owner is a popcount
// and a load away and independent of the other arcs'.  (Walking the row ends from word to word
// instead took three times as long on 33 M arcs: a chain of loads for every 32 arcs.)  On smaller
// graphs (start == null), where its three launches cost more than they save, a search per word
// (upload, checks, DAG and two counts of R-MAT graphs of edge factor 8, a = 0.45, by searches | bits:
// 30,000 vertices, 0.4 M arcs: 470 | 492 us; 1,000,000, 16 M arcs: 2.66 | 2.57 ms; alike between).
struct ArcOwners {
  const uint32_t* start = nullptr;
  const int32_t* before = nullptr;
  const int32_t* row = nullptr;
};
constexpr int64_t kOwnerArcs = (int64_t)1 << 20;

// Owner of arc 32 w + lane (of the last arc before it for lanes past the end).
__device__ __forceinline__ int32_t arc_owner(const ArcOwners& o, const int64_t* rowptr, int32_t n,
                                             int64_t w) {
  const int lane = threadIdx.x & 31;
  if (o.start) {
    const uint32_t b = o.start[w] & (kAll >> (31 - lane));
    return o.row[o.before[w] + __popc(b) - 1];
  }
  const int64_t k0 = w << 5;
  int64_t base = warp_owner(rowptr, n, k0);
  int32_t own = 0;
  bool found = false;
  for (;; base += 32) {  // row ends after the word's first owner, 32 at a time
    const int64_t r = base + 1 + lane;
    const int64_t rel = r <= n ? rowptr[r] - k0 : 64;
    const int end = rel < 64 ? (int)rel : 64;
    int c = 0;  // ends at or before this lane's arc
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const int e = __shfl_sync(kAll, end, c + step - 1);
      if (e <= lane) c += step;
    }
    const int last = __shfl_sync(kAll, end, 31);
    if (c == 31 && last <= lane) c = 32;
    if (!found) {
      own = (int32_t)(base + c);
      found = c < 32;
    }
    if (last > 31) return own;
  }
}

__global__ void k_row_starts(const int64_t* rowptr, int32_t n, uint32_t* start) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const int64_t b = rowptr[v];
    if (rowptr[v + 1] > b) atomicOr(&start[b >> 5], 1u << (b & 31));
  }
}

__global__ void k_row_index(const int64_t* rowptr, int32_t n, const uint32_t* start,
                            const int32_t* before, int32_t* row) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const int64_t b = rowptr[v];
    if (rowptr[v + 1] > b)
      row[before[b >> 5] + __popc(start[b >> 5] & ((1u << (b & 31)) - 1u))] = (int32_t)v;
  }
}

struct BitsOfWord {
  __host__ __device__ __forceinline__ int32_t operator()(uint32_t w) const {
#ifdef __CUDA_ARCH__
    return __popc(w);
#else
    return __builtin_popcount(w);
#endif
  }
};

constexpr int kWordStep = 4;  // words that a warp takes at a time, so that their loads overlap

// Checks a CSR whose row pointers are in order: ids in range, no self-loops, rows strictly
// increasing, both directions present.  Every arc to the lower-ranked end is looked up in that
// end's (shorter) row; with as many such arcs as others -- `down` counts them -- the lookups pair
// every arc with its reverse.  keep (may be null) receives what k_orient_masks would write: the
// arcs that are not looked up are the DAG's.
__global__ void k_validate(const int64_t* rowptr, const int32_t* col, int32_t n, int64_t m,
                           ArcOwners own, int* bad, unsigned long long* down, uint32_t* keep,
                           int32_t* count) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t words = (m + 31) >> 5;
  unsigned long long nd = 0;
  bool all_ok = true;
  for (int64_t w = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kWordStep; w < words;
       w += warps * kWordStep) {
    {
      int32_t u[kWordStep], v[kWordStep], prev[kWordStep];
      int64_t lo[kWordStep], dv[kWordStep];
      bool ok[kWordStep], dn[kWordStep];
#pragma unroll
      for (int t = 0; t < kWordStep; ++t) {
        const int64_t k = ((w + t) << 5) + lane;
        const bool in = k < m;
        v[t] = in ? col[k] : 0;
        prev[t] = in && k > 0 ? col[k - 1] : -1;
      }
#pragma unroll
      for (int t = 0; t < kWordStep; ++t) {
        ok[t] = v[t] >= 0 && v[t] < n;
        lo[t] = ok[t] ? rowptr[v[t]] : 0;
        dv[t] = ok[t] ? rowptr[v[t] + 1] - lo[t] : 0;
      }
#pragma unroll
      for (int t = 0; t < kWordStep; ++t) {
        dn[t] = false;
        u[t] = w + t < words ? arc_owner(own, rowptr, n, w + t) : 0;
        const int64_t k = ((w + t) << 5) + lane;
        if (k < m) {
          const int64_t bu = rowptr[u[t]], du = rowptr[u[t] + 1] - bu;
          ok[t] = ok[t] && v[t] != u[t] && (k == bu || prev[t] < v[t]);
          dn[t] = ok[t] && (dv[t] < du || (dv[t] == du && v[t] < u[t]));
        } else {
          ok[t] = true;
        }
        const unsigned down_mask = __ballot_sync(kAll, dn[t]);
        nd += (unsigned)__popc(down_mask);
        all_ok = all_ok && ok[t];
        if (keep && lane == 0 && w + t < words) {
          const int64_t left = m - ((w + t) << 5);
          const uint32_t up = ~down_mask & (left >= 32 ? kAll : (1u << left) - 1u);
          keep[w + t] = up;
          count[w + t] = __popc(up);
        }
      }
      // u must be in N(v): the four rows are searched in lockstep
      int len[kWordStep], pos[kWordStep], lmax = 0;
#pragma unroll
      for (int t = 0; t < kWordStep; ++t) {
        len[t] = dn[t] ? (int)dv[t] : 0;
        pos[t] = 0;
        lmax = max(lmax, len[t]);
      }
      for (int step = lmax > 0 ? 1 << (31 - __clz(lmax)) : 0; step > 0; step >>= 1) {
#pragma unroll
        for (int t = 0; t < kWordStep; ++t)
          if (pos[t] + step <= len[t] && col[lo[t] + pos[t] + step - 1] < u[t]) pos[t] += step;
      }
#pragma unroll
      for (int t = 0; t < kWordStep; ++t)
        if (dn[t]) all_ok = all_ok && pos[t] < len[t] && col[lo[t] + pos[t]] == u[t];
    }
  }
  if (!all_ok) atomicExch(bad, 1);
  if (lane == 0 && nd) atomicAdd(down, nd);
}

struct DegreeStats {
  int most;
  unsigned long long squares;  // sum of the squared degrees
};

// Every thread of a full warp calls it.
__device__ __forceinline__ void add_degree_stats(int most, unsigned long long squares,
                                                 DegreeStats* out) {
  for (int o = 16; o > 0; o >>= 1) {
    most = max(most, __shfl_xor_sync(kAll, most, o));
    squares += __shfl_xor_sync(kAll, squares, o);
  }
  if ((threadIdx.x & 31) == 0 && most) {
    atomicMax(&out->most, most);
    atomicAdd(&out->squares, squares);
  }
}

__global__ void k_rowptr_check(const int64_t* rowptr, int32_t n, int64_t m, int* bad,
                               DegreeStats* stats) {
  int most = 0;
  unsigned long long squares = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const int64_t d = rowptr[v + 1] - rowptr[v];
    if (d < 0 || d > INT32_MAX) {
      atomicExch(bad, 1);
    } else {
      most = max(most, (int)d);
      squares += (unsigned long long)d * (unsigned long long)d;
    }
  }
  add_degree_stats(most, squares, stats);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (rowptr[0] != 0 || rowptr[n] != m) atomicExch(bad, 1);
  }
}

// Bit k of keep: arc k of the CSR is a DAG arc (its head has the higher (degree, id)); count[w] =
// bits of word w.
__global__ void k_orient_masks(const int64_t* rowptr, const int32_t* col, int32_t n, int64_t m,
                               ArcOwners own, uint32_t* keep, int32_t* count) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t words = (m + 31) >> 5;
  for (int64_t w = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kWordStep; w < words;
       w += warps * kWordStep) {
    int32_t u[kWordStep], v[kWordStep];
    int64_t du[kWordStep], dv[kWordStep];
#pragma unroll
    for (int t = 0; t < kWordStep; ++t) {
      const int64_t k = ((w + t) << 5) + lane;
      v[t] = k < m ? col[k] : 0;
      u[t] = w + t < words ? arc_owner(own, rowptr, n, w + t) : 0;
      if (k >= m) u[t] = 0;
    }
#pragma unroll
    for (int t = 0; t < kWordStep; ++t) {
      dv[t] = rowptr[v[t] + 1] - rowptr[v[t]];
      du[t] = rowptr[u[t] + 1] - rowptr[u[t]];
    }
#pragma unroll
    for (int t = 0; t < kWordStep; ++t) {
      const int64_t k = ((w + t) << 5) + lane;
      const bool up = k < m && (dv[t] > du[t] || (dv[t] == du[t] && v[t] > u[t]));
      const uint32_t mask = __ballot_sync(kAll, up);
      if (lane == 0 && w + t < words) {
        keep[w + t] = mask;
        count[w + t] = __popc(mask);
      }
    }
  }
}

__global__ void k_orient_scatter(const int32_t* col, const uint32_t* keep, const int64_t* pos,
                                 int64_t m, int32_t* dag_col) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t words = (m + 31) >> 5;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += warps) {
    const uint32_t mask = keep[w];
    if ((mask >> lane) & 1u)
      dag_col[pos[w] + __popc(mask & ((1u << lane) - 1u))] = col[(w << 5) + lane];
  }
}

// Row pointers of the DAG; out[0] = its largest out-degree, out[1] = its vertices of out-degree above
// 32 (both zero before).  words = words of keep; total = DAG arcs.
__global__ void k_dag_rowptr(const int64_t* rowptr, const uint32_t* keep, const int64_t* pos,
                             int32_t n, int64_t m, int64_t total, int64_t* dag_rowptr,
                             int* out) {
  auto at = [&](int64_t k) {
    return k < m ? pos[k >> 5] + __popc(keep[k >> 5] & ((1u << (k & 31)) - 1u)) : total;
  };
  int most = 0, over = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += stride) {
    const int64_t b = rowptr[v], p = at(b);
    dag_rowptr[v] = p;
    if (v < n) {
      const int64_t e = rowptr[v + 1];
      const int d = e > b ? (int)(at(e) - p) : 0;
      most = max(most, d);
      over += d > 32 ? 1 : 0;
    }
  }
  most = (int)__reduce_max_sync(kAll, (unsigned)most);
  over = (int)__reduce_add_sync(kAll, (unsigned)over);
  if ((threadIdx.x & 31) == 0 && most) {
    atomicMax(out, most);
    if (over) atomicAdd(out + 1, over);
  }
}

__global__ void k_degree_stats(const int64_t* rowptr, int32_t n, DegreeStats* out) {
  int most = 0;
  unsigned long long squares = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const int d = (int)(rowptr[v + 1] - rowptr[v]);
    most = max(most, d);
    squares += (unsigned long long)d * (unsigned)d;
  }
  add_degree_stats(most, squares, out);
}

std::mutex g_pool_mu;
cudaMemPool_t g_pools[64] = {};

// The library's pool on `dev`: it keeps every byte freed into it (no release threshold), so
// repeated graph life cycles reuse the same memory.  Callers that need the memory elsewhere
// get it back by the trim on an allocation failure.
cudaMemPool_t device_pool(int dev) {
  if (dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pools[dev]) {
    cudaMemPoolProps props;
    memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    uint64_t keep = UINT64_MAX;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    g_pools[dev] = pool;
  }
  return g_pools[dev];
}

// Pinned host mirrors of the graphs' control blocks: slots of pinned slabs, reused.
std::mutex g_ctl_mu;
std::vector<DevControl*> g_ctl_free;

DevControl* ctl_slot() {
  std::lock_guard<std::mutex> lk(g_ctl_mu);
  if (g_ctl_free.empty()) {
    constexpr int kSlots = 256;
    DevControl* slab = nullptr;
    if (cudaMallocHost((void**)&slab, kSlots * sizeof(DevControl)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    for (int i = kSlots - 1; i >= 0; --i) g_ctl_free.push_back(slab + i);
  }
  DevControl* p = g_ctl_free.back();
  g_ctl_free.pop_back();
  return p;
}

void ctl_release(DevControl* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_ctl_mu);
  g_ctl_free.push_back(p);
}

int grid_for(int64_t work, int threads = 256) {
  int64_t b = (work + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 148 * 32) b = 148 * 32;
  return (int)b;
}

}  // namespace

namespace {
std::atomic<int64_t> g_fail_alloc{-1};  // jgpm_fail_alloc_
}

int gmalloc(void** p, size_t bytes, cudaStream_t s) {
  if (g_fail_alloc.load(std::memory_order_relaxed) >= 0 && g_fail_alloc.fetch_sub(1) == 0) {
    *p = nullptr;
    jgpm_set_error_("device allocation refused (jgpm_fail_alloc_)");
    return JGPM_ENOMEM;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  cudaMemPool_t pool = device_pool(dev);
  cudaError_t e = pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaErrorMemoryAllocation;
  if (e == cudaErrorMemoryAllocation && pool) {  // return the cached memory, then retry once
    cudaGetLastError();
    cudaDeviceSynchronize();
    cudaMemPoolTrimTo(pool, 0);
    e = cudaMallocFromPoolAsync(p, bytes, pool, s);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    jgpm_set_error_(std::string("device allocation of ") + std::to_string(bytes) +
                    " bytes: " + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? JGPM_ENOMEM : JGPM_ECUDA;
  }
  return JGPM_OK;
}

void gfree(void* p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

namespace {

template <typename T>
int dalloc(T** p, size_t count, cudaStream_t s) {
  return gmalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T), s);
}

// A temporary device buffer, returned to the pool in the order of stream s.
struct DevBuf {
  cudaStream_t s;
  void* p = nullptr;
  explicit DevBuf(cudaStream_t stream) : s(stream) {}
  ~DevBuf() {
    if (p) gfree(p, s);
  }
  // Hands the buffer over to a graph.
  template <typename T>
  void publish(T** to) {
    *to = (T*)p;
    p = nullptr;
  }
};

// The arc owners of a CSR, in buf.
int build_owners(const int64_t* rowptr, int32_t n, int64_t m, DevBuf& buf, ArcOwners* o) {
  if (m < kOwnerArcs) return JGPM_OK;
  cudaStream_t s = buf.s;
  const int64_t words = (m + 31) >> 5;
  auto room = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
  const size_t wb = room((size_t)words * 4), rb = room((size_t)n * 4);
  size_t tb = 0;
  using Bits = cub::TransformInputIterator<int32_t, BitsOfWord, const uint32_t*>;
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, Bits(nullptr, BitsOfWord()),
                                              (int32_t*)nullptr, words, s));
  int rc;
  if ((rc = dalloc((char**)&buf.p, 2 * wb + rb + tb, s))) return rc;
  uint32_t* start = (uint32_t*)buf.p;
  int32_t* before = (int32_t*)((char*)buf.p + wb);
  int32_t* row = (int32_t*)((char*)buf.p + 2 * wb);
  JGPM_CUDA_TRY(cudaMemsetAsync(start, 0, (size_t)words * 4, s));
  k_row_starts<<<grid_for(n), 256, 0, s>>>(rowptr, n, start);
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveSum((char*)buf.p + 2 * wb + rb, tb,
                                              Bits(start, BitsOfWord()), before, words, s));
  k_row_index<<<grid_for(n), 256, 0, s>>>(rowptr, n, start, before, row);
  JGPM_CUDA_TRY(cudaGetLastError());
  o->start = start;
  o->before = before;
  o->row = row;
  return JGPM_OK;
}

// Sorts 2*ne keys, removes duplicates and the invalid key, and fills g's symmetric CSR.
int keys_to_csr(jgpm_graph* g, int32_t n, uint64_t* d_keys, int64_t nk, int shift,
                uint64_t invalid, int end_bit) {
  cudaStream_t s = g->stream;
  DevBuf alt(g->stream), tmp(g->stream), flags(g->stream), pos(g->stream);
  int rc;
  if ((rc = dalloc((uint64_t**)&alt.p, nk, g->stream))) return rc;
  size_t tbytes = 0, tb2 = 0;
  cub::DoubleBuffer<uint64_t> db(d_keys, (uint64_t*)alt.p);
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, tbytes, db, nk, 0, end_bit, s));
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb2, (int*)nullptr, (int64_t*)nullptr,
                                              nk, s));
  tbytes = std::max(tbytes, tb2);
  if ((rc = dalloc((char**)&tmp.p, tbytes, g->stream))) return rc;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp.p, tbytes, db, nk, 0, end_bit, s));
  uint64_t* sorted = db.Current();
  uint64_t* spare = db.Alternate();
  if ((rc = dalloc((int**)&flags.p, nk, g->stream))) return rc;
  if ((rc = dalloc((int64_t**)&pos.p, nk + 1, g->stream))) return rc;
  k_unique_flags<<<grid_for(nk), 256, 0, s>>>(sorted, nk, invalid, (int*)flags.p);
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(tmp.p, tbytes, (int*)flags.p, (int64_t*)pos.p,
                                              nk, s));
  int64_t last_pos = 0;
  int last_flag = 0;
  if (nk > 0) {
    JGPM_CUDA_TRY(cudaMemcpyAsync(&last_pos, (int64_t*)pos.p + nk - 1, sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, s));
    JGPM_CUDA_TRY(cudaMemcpyAsync(&last_flag, (int*)flags.p + nk - 1, sizeof(int),
                                  cudaMemcpyDeviceToHost, s));
    JGPM_CUDA_TRY(cudaStreamSynchronize(s));
  }
  const int64_t m = last_pos + last_flag;
  if ((rc = dalloc(&g->d_col, m, g->stream))) return rc;
  if ((rc = dalloc(&g->d_rowptr, (size_t)n + 1, g->stream))) return rc;
  uint64_t* ukeys = spare;  // nk >= m entries, free after the sort
  k_compact_keys<<<grid_for(nk), 256, 0, s>>>(sorted, (int*)flags.p, (int64_t*)pos.p, nk,
                                              (1ull << shift) - 1, ukeys, g->d_col);
  k_rowptr_from_keys<<<grid_for((int64_t)n + 1), 256, 0, s>>>(ukeys, m, n, shift,
                                                              g->d_rowptr);
  JGPM_CUDA_TRY(cudaGetLastError());
  g->n = n;
  g->m = m;
  return JGPM_OK;
}

int finish_sym(jgpm_graph* g) {
  DevBuf md(g->stream);
  int rc;
  if ((rc = dalloc((DegreeStats**)&md.p, 1, g->stream))) return rc;
  JGPM_CUDA_TRY(cudaMemsetAsync(md.p, 0, sizeof(DegreeStats), g->stream));
  k_degree_stats<<<grid_for(g->n), 256, 0, g->stream>>>(g->d_rowptr, g->n, (DegreeStats*)md.p);
  DegreeStats h = {0, 0};
  JGPM_CUDA_TRY(cudaMemcpyAsync(&h, md.p, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
  JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));
  g->max_degree = h.most;
  g->degree_squares = h.squares;
  return JGPM_OK;
}

int shift_for(int32_t n) {
  int s = 1;
  while ((int64_t(1) << s) <= (int64_t)n) ++s;  // ids and the invalid source n fit
  return s;
}

}  // namespace

int raise_smem_limit(const void* func, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> limits;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& cur = limits[std::make_pair(dev, func)];
  if (bytes <= cur) return JGPM_OK;
  const cudaError_t e =
      cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) {
    jgpm_set_error_(std::string("raise_smem_limit: ") + cudaGetErrorString(e));
    return JGPM_ECUDA;
  }
  cur = bytes;
  return JGPM_OK;
}

int device_sm_count(int device) {
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return 148;
  return sms;
}

int rmat_build(jgpm_graph* g, int64_t n, int64_t num_edges, double a, double b, double c,
               uint64_t seed) {
  if (n < 2 || n > INT32_MAX - 1 || num_edges < 0 || a < 0 || b < 0 || c < 0 ||
      a + b + c > 1.0 + 1e-12) {
    jgpm_set_error_("jgpm_graph_rmat: bad parameters");
    return JGPM_EINVAL;
  }
  RmatParams p = rmat_params(n, num_edges, a, b, c, seed);
  const int shift = shift_for((int32_t)n);
  const uint64_t invalid = (uint64_t)n << shift;
  const int end_bit = 2 * shift;
  const int64_t nk = 2 * num_edges;
  DevBuf keys(g->stream);
  int rc;
  if ((rc = dalloc((uint64_t**)&keys.p, nk, g->stream))) return rc;
  k_rmat_keys<<<grid_for(num_edges), 256, 0, g->stream>>>(p, shift, (uint64_t*)keys.p, invalid);
  JGPM_CUDA_TRY(cudaGetLastError());
  if ((rc = keys_to_csr(g, (int32_t)n, (uint64_t*)keys.p, nk, shift, invalid, end_bit)))
    return rc;
  return finish_sym(g);
}

int edges_build(jgpm_graph* g, const int32_t* src, const int32_t* dst, int64_t ne, int32_t n) {
  if (n < 1 || ne < 0) {
    jgpm_set_error_("jgpm_graph_from_edges: bad sizes");
    return JGPM_EINVAL;
  }
  const int shift = shift_for(n);
  const uint64_t invalid = (uint64_t)n << shift;
  DevBuf ds(g->stream), dd(g->stream), keys(g->stream), bad(g->stream);
  int rc;
  if ((rc = dalloc((int32_t**)&ds.p, ne, g->stream))) return rc;
  if ((rc = dalloc((int32_t**)&dd.p, ne, g->stream))) return rc;
  if ((rc = dalloc((uint64_t**)&keys.p, 2 * ne, g->stream))) return rc;
  if ((rc = dalloc((int**)&bad.p, 1, g->stream))) return rc;
  JGPM_CUDA_TRY(cudaMemcpyAsync(ds.p, src, ne * sizeof(int32_t), cudaMemcpyDefault, g->stream));
  JGPM_CUDA_TRY(cudaMemcpyAsync(dd.p, dst, ne * sizeof(int32_t), cudaMemcpyDefault, g->stream));
  JGPM_CUDA_TRY(cudaMemsetAsync(bad.p, 0, sizeof(int), g->stream));
  k_edge_keys<<<grid_for(ne), 256, 0, g->stream>>>((int32_t*)ds.p, (int32_t*)dd.p, ne, n, shift,
                                                   (uint64_t*)keys.p, invalid, (int*)bad.p);
  int hbad = 0;
  JGPM_CUDA_TRY(cudaMemcpyAsync(&hbad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, g->stream));
  JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));
  if (hbad) {
    jgpm_set_error_("jgpm_graph_from_edges: vertex id out of range");
    return JGPM_EINVAL;
  }
  if ((rc = keys_to_csr(g, n, (uint64_t*)keys.p, 2 * ne, shift, invalid, 2 * shift))) return rc;
  return finish_sym(g);
}

int upload_csr(jgpm_graph* g, const int64_t* rowptr, const int32_t* col, int32_t n, int64_t m,
               int validate, int orient) {
  if (n < 1 || m < 0 || !rowptr || (m > 0 && !col)) {
    jgpm_set_error_("jgpm_graph_from_csr: bad arguments");
    return JGPM_EINVAL;
  }
  int rc;
  if ((rc = dalloc(&g->d_rowptr, (size_t)n + 1, g->stream))) return rc;
  if ((rc = dalloc(&g->d_col, m, g->stream))) return rc;
  JGPM_CUDA_TRY(cudaMemcpyAsync(g->d_rowptr, rowptr, ((size_t)n + 1) * sizeof(int64_t),
                                cudaMemcpyDefault, g->stream));
  if (m > 0)
    JGPM_CUDA_TRY(cudaMemcpyAsync(g->d_col, col, (size_t)m * sizeof(int32_t), cudaMemcpyDefault,
                                  g->stream));
  g->n = n;
  g->m = m;
  if (validate) {
    struct Check {
      int bad;
      DegreeStats degrees;
      unsigned long long down;
    } h;
    DevBuf st(g->stream);
    if ((rc = dalloc((Check**)&st.p, 1, g->stream))) return rc;
    Check* d = (Check*)st.p;
    JGPM_CUDA_TRY(cudaMemsetAsync(d, 0, sizeof(Check), g->stream));
    k_rowptr_check<<<grid_for(n), 256, 0, g->stream>>>(g->d_rowptr, n, m, &d->bad,
                                                       &d->degrees);
    JGPM_CUDA_TRY(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
    JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));
    if (!h.bad && m > 0) {
      g->max_degree = h.degrees.most;
      g->degree_squares = h.degrees.squares;
      DevBuf ob(g->stream);
      ArcOwners own;
      if ((rc = build_owners(g->d_rowptr, n, m, ob, &own))) return rc;
      // the orientation is decided on the way: its masks stay until ensure_dag takes them
      const int64_t words = (m + 31) >> 5;
      if (orient && (rc = dalloc(&g->d_keep, 2 * words + 1, g->stream))) return rc;
      k_validate<<<grid_for((m + kWordStep - 1) / kWordStep), 256, 0, g->stream>>>(
          g->d_rowptr, g->d_col, n, m, own, &d->bad, &d->down, g->d_keep,
          g->d_keep ? (int32_t*)g->d_keep + words : nullptr);
      JGPM_CUDA_TRY(cudaGetLastError());
      JGPM_CUDA_TRY(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
      JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));
      if (2 * h.down != (unsigned long long)m) h.bad = 1;
    }
    const int hbad = h.bad;
    if (hbad) {
      jgpm_set_error_(
          "jgpm_graph_from_csr: CSR must have rowptr[0]=0, rowptr[n]=m, nondecreasing row "
          "pointers, strictly increasing rows, ids in [0,n), no self-loops and both "
          "directions of every edge");
      return JGPM_EINVAL;
    }
    return JGPM_OK;
  }
  return finish_sym(g);
}

int ensure_dag(jgpm_graph* g) {
  if (g->d_dag_rowptr) return JGPM_OK;
  cudaStream_t s = g->stream;
  const int64_t m = g->m;
  const int32_t n = g->n;
  int rc;
  // the graph gets the arrays when they are complete: a call that failed half-way is as if it
  // had not been made
  DevBuf rowptr(s), col(s);
  if ((rc = dalloc((int64_t**)&rowptr.p, (size_t)n + 1, s))) return rc;
  // one bit per arc, and one prefix per 32 arcs: nothing of the arcs' size but the arcs is
  // written (33 M arcs: 0.80 ms with a source, a flag and a position for each arc)
  const int64_t words = (m + 31) >> 5;
  DevBuf masks(s), pos(s), tmp(s), st(s), ob(s);
  const bool have = g->d_keep != nullptr;  // from the validation of the caller's CSR
  if (have) {
    masks.p = g->d_keep;
    g->d_keep = nullptr;
  } else if ((rc = dalloc((uint32_t**)&masks.p, 2 * words + 1, s))) {
    return rc;
  }
  uint32_t* keep = (uint32_t*)masks.p;
  int32_t* count = (int32_t*)keep + words;
  if ((rc = dalloc((int64_t**)&pos.p, words + 1, s))) return rc;
  if ((rc = dalloc((int**)&st.p, 2, s))) return rc;
  JGPM_CUDA_TRY(cudaMemsetAsync(st.p, 0, 2 * sizeof(int), s));
  JGPM_CUDA_TRY(cudaMemsetAsync(count + words, 0, 4, s));
  if (words > 0 && !have) {
    ArcOwners own;
    if ((rc = build_owners(g->d_rowptr, n, m, ob, &own))) return rc;
    k_orient_masks<<<grid_for((m + kWordStep - 1) / kWordStep), 256, 0, s>>>(
        g->d_rowptr, g->d_col, n, m, own, keep, count);
  }
  size_t tb = 0;
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveScan(nullptr, tb, count, (int64_t*)pos.p,
                                               cub::Sum(), (int64_t)0, words + 1, s));
  if ((rc = dalloc((char**)&tmp.p, tb, s))) return rc;
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveScan(tmp.p, tb, count, (int64_t*)pos.p,
                                               cub::Sum(), (int64_t)0, words + 1, s));
  // every edge is one DAG arc
  const int64_t total = m / 2;
  if ((rc = dalloc((int32_t**)&col.p, total, s))) return rc;
  if (words > 0)
    k_orient_scatter<<<grid_for(m), 256, 0, s>>>(g->d_col, keep, (int64_t*)pos.p, m,
                                                 (int32_t*)col.p);
  k_dag_rowptr<<<grid_for((int64_t)n + 1), 256, 0, s>>>(g->d_rowptr, keep,
                                                        (int64_t*)pos.p, n, m, total,
                                                        (int64_t*)rowptr.p, (int*)st.p);
  JGPM_CUDA_TRY(cudaGetLastError());
  int h[2] = {0, 0};
  JGPM_CUDA_TRY(cudaMemcpyAsync(h, st.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  JGPM_CUDA_TRY(cudaStreamSynchronize(s));
  g->m_dag = total;
  g->max_out_degree = h[0];
  g->over32 = h[1];
  rowptr.publish(&g->d_dag_rowptr);
  col.publish(&g->d_dag_col);
  return JGPM_OK;
}

// Out-degree classes of the tier boundaries: class t holds the out-degrees up to tier_threshold(t)
// that no lower class holds; the last class the rest.
constexpr int kTierClasses = 34 + 8;
constexpr size_t kTierBytes = 256;  // their counters
__host__ __device__ __forceinline__ int tier_class(int64_t d) {
  if (d <= 33) return (int)d;
  int t = 34;
  for (int64_t top = 64; t < kTierClasses - 1 && d > top; top *= 2) ++t;
  return t;
}
static_assert(kTierClasses * 4 <= kTierBytes && kMidMaxDeg == 1024 && kWideMaxDeg == 4096,
              "classes 34.. end at 64, 128, 256, 512, 1024, 2048 and 4096");

// Adds up the classes of a CTA's vertices (every thread calls it, once, with its own count array
// in shared memory zeroed).
__device__ __forceinline__ void add_classes(const int* mine, int32_t* classes) {
  __syncthreads();
  for (int t = threadIdx.x; t < kTierClasses; t += blockDim.x)
    if (mine[t]) atomicAdd(classes + t, mine[t]);
}

// Roots of a class above t: the first index of the descending root list that is at or below it.
// By one warp.
__device__ __forceinline__ int64_t tier_begin(const int32_t* classes, int t) {
  const int lane = threadIdx.x & 31;
  const unsigned a = lane > t ? (unsigned)classes[lane] : 0u;
  const unsigned b =
      lane + 32 > t && lane + 32 < kTierClasses ? (unsigned)classes[lane + 32] : 0u;
  return (int64_t)__reduce_add_sync(kAll, a + b);
}

// ------------------------------------------------------------------- rank DAG
// The rank DAG (RankDag) is the id DAG with vertices renumbered and every row sorted by the new
// ids.  Rows are gathered, relabelled and sorted on chip, by lane groups, warps or CTAs by
// out-degree: each arc is read once and written once (the id DAG's rows give the arcs, so no
// global sort of arc keys is needed), and the rows of the top h vertices set their bits in the
// bitmap on the way.
namespace {

// Sort input of the root list on the id DAG: out-degrees and ids; with them the symmetric degrees
// and the out-degree classes.
__global__ void k_root_keys(const int64_t* dag_rowptr, const int64_t* rowptr, int32_t n,
                            uint32_t* keys, int32_t* vals, int32_t* sdeg, int32_t* classes) {
  __shared__ int mine[kTierClasses];
  for (int t = threadIdx.x; t < kTierClasses; t += blockDim.x) mine[t] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const int64_t d = dag_rowptr[v + 1] - dag_rowptr[v];
    keys[v] = (uint32_t)d;
    vals[v] = (int32_t)v;
    sdeg[v] = (int32_t)(rowptr[v + 1] - rowptr[v]);
    atomicAdd(&mine[tier_class(d)], 1);
  }
  add_classes(mine, classes);
}

// Sort input of the rank DAG: every vertex by its degree.  both: n entries more, with the bit above
// the others set, for every vertex by descending (out-degree, degree, id), so that one ascending
// sort gives both orders; deg_bits and out_bits hold the largest degree and out-degree.
__global__ void k_order_keys(const int64_t* rowptr, const int64_t* dag_rowptr, int32_t n,
                             int deg_bits, int out_bits, bool both, uint32_t* keys, int32_t* vals,
                             int32_t* classes) {
  __shared__ int mine[kTierClasses];
  for (int t = threadIdx.x; t < kTierClasses; t += blockDim.x) mine[t] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const uint32_t d = (uint32_t)(dag_rowptr[v + 1] - dag_rowptr[v]);
    const uint32_t deg = (uint32_t)(rowptr[v + 1] - rowptr[v]);
    keys[v] = deg;
    vals[v] = (int32_t)v;
    if (both) {
      const uint32_t top = (2u << out_bits) - 1u;  // the bit, and all ones for an out-degree of 0
      const int64_t at = 2 * (int64_t)n - 1 - v;
      keys[at] = ((top - d) << deg_bits) | (((1u << deg_bits) - 1u) - deg);
      vals[at] = (int32_t)v;
    }
    atomicAdd(&mine[tier_class(d)], 1);
  }
  add_classes(mine, classes);
}

// order[p] = the vertex at position p of the ascending (degree, id) order; its new id is
// n - 1 - p.  outdeg gets a zero at index n (the end of the row-pointer scan).  keys and vals (may
// be null): the sort input for the vertices by out-degree, in the order of the new ids.
__global__ void k_rank_label(const int32_t* order, const int64_t* dag_rowptr,
                             const int64_t* rowptr, int32_t n, int32_t* newid, int64_t* outdeg,
                             int32_t* sdeg, uint32_t* keys, int32_t* vals) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const int32_t v = order[p];
    const int64_t x = n - 1 - p;
    newid[v] = (int32_t)x;
    const int64_t d = dag_rowptr[v + 1] - dag_rowptr[v];
    outdeg[x] = d;
    sdeg[x] = (int32_t)(rowptr[v + 1] - rowptr[v]);
    if (keys) {
      keys[x] = (uint32_t)d;
      vals[x] = v;
    }
    if (p == 0) outdeg[n] = 0;
  }
}

// k_rank_label and the row-pointer scan in one launch, for graphs of at most kRankOneCta vertices,
// whose first count is bound by the number of launches.
constexpr int32_t kRankOneCta = 8192;
__global__ void __launch_bounds__(1024)
    k_rank_label_scan(const int32_t* order, const int64_t* dag_rowptr, const int64_t* rowptr,
                      int32_t n, int32_t* newid, int64_t* rp, int32_t* sdeg, uint32_t* keys,
                      int32_t* vals) {
  __shared__ int64_t sums[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + 1023) / 1024;
  const int x0 = min(n, tid * per), x1 = min(n, x0 + per);
  int64_t sum = 0;
  for (int x = x0; x < x1; ++x) {
    const int32_t v = order[n - 1 - x];
    const int64_t d = dag_rowptr[v + 1] - dag_rowptr[v];
    newid[v] = x;
    rp[x] = d;
    sdeg[x] = (int32_t)(rowptr[v + 1] - rowptr[v]);
    if (keys) {
      keys[x] = (uint32_t)d;
      vals[x] = v;
    }
    sum += d;
  }
  int64_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t t = __shfl_up_sync(kAll, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  int64_t run = incl - sum;
  for (int w = 0; w < warp; ++w) run += sums[w];
  for (int x = x0; x < x1; ++x) {
    const int64_t d = rp[x];
    rp[x] = run;
    run += d;
  }
  if (tid == 1023) rp[n] = run;
}

// Sorts a[0..n) ascending: bitonic merges whose comparators all point the same way, so the
// missing elements past n count as infinity and are never touched.
template <typename Sync>
__device__ __forceinline__ void bitonic_sort(int32_t* a, int n, int tid, int nthreads,
                                             Sync&& sync) {
  int N = 1;
  while (N < n) N <<= 1;
  auto exchange = [&](int i, int j) {
    if (j < n) {
      const int32_t x = a[i], y = a[j];
      if (x > y) {
        a[i] = y;
        a[j] = x;
      }
    }
  };
  for (int k = 2; k <= N; k <<= 1) {
    for (int t = tid; t < N / 2; t += nthreads) {
      const int i = ((t & ~(k / 2 - 1)) << 1) | (t & (k / 2 - 1));
      exchange(i, i ^ (k - 1));
    }
    sync();
    for (int h = k >> 2; h > 0; h >>= 1) {
      for (int t = tid; t < N / 2; t += nthreads) {
        const int i = ((t & ~(h - 1)) << 1) | (t & (h - 1));
        exchange(i, i + h);
      }
      sync();
    }
  }
}

struct RowArgs {
  const int32_t* verts;  // id-DAG vertices by descending out-degree
  const int64_t* dag_rowptr;
  const int32_t* dag_col;
  const int32_t* newid;
  const int64_t* rp;
  int32_t* col;
  uint32_t* bits;
  int32_t* roots;          // receives the new ids of verts
  const int32_t* classes;  // out-degree classes: where the kernels' ranges of verts begin
  int32_t h;
};

__device__ __forceinline__ void set_bit(const RowArgs& a, int32_t x, int32_t w) {
  if (x < a.h) atomicOr(a.bits + rank_bits_row((uint32_t)x) + ((uint32_t)w >> 5), 1u << (w & 31));
}

// Rows of out-degree 1..G, one per group of G lanes, sorted in registers; kRowsAhead at a time, so
// that their chains of gathers (vertex, row, arcs, new ids) overlap: one task at a time took 380 us
// on 16.7 M arcs of 4,194,304 vertices.
constexpr int kRowsAhead = 4;
template <int G>
__device__ __forceinline__ void rank_rows_group(const RowArgs& a, int64_t b, int64_t e,
                                                int64_t task) {
  constexpr int U = kRowsAhead;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  int32_t v[U], x[U], key[U];
  int64_t s[U], o[U];
  int d[U];
#pragma unroll
  for (int q = 0; q < U; ++q) {
    const int64_t idx = b + (task * U + q) * (32 / G) + lane / G;
    v[q] = idx < e ? a.verts[idx] : -1;
  }
#pragma unroll
  for (int q = 0; q < U; ++q) {
    const bool in = v[q] >= 0;
    x[q] = in ? a.newid[v[q]] : -1;
    s[q] = in ? a.dag_rowptr[v[q]] : 0;
    d[q] = in ? (int)(a.dag_rowptr[v[q] + 1] - s[q]) : 0;
  }
#pragma unroll
  for (int q = 0; q < U; ++q) {
    const int64_t idx = b + (task * U + q) * (32 / G) + lane / G;
    o[q] = x[q] >= 0 ? a.rp[x[q]] : 0;
    if (x[q] >= 0 && gl == 0) a.roots[idx] = x[q];
    key[q] = gl < d[q] ? a.dag_col[s[q] + gl] : -1;
  }
#pragma unroll
  for (int q = 0; q < U; ++q) key[q] = key[q] >= 0 ? a.newid[key[q]] : INT32_MAX;
#pragma unroll
  for (int q = 0; q < U; ++q) {
#pragma unroll
    for (int k = 2; k <= G; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const int32_t other = __shfl_xor_sync(0xffffffffu, key[q], j);
        const bool up = (gl & k) == 0, low = (gl & j) == 0;
        key[q] = (up == low) ? min(key[q], other) : max(key[q], other);
      }
    }
    if (gl < d[q]) {
      a.col[o[q] + gl] = key[q];
      set_bit(a, x[q], key[q]);
    }
  }
}

// Vertices of out-degree 17..32 | 9..16 | 5..8 | 1..4.
__global__ void k_rank_rows_small(RowArgs a) {
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t b[5] = {tier_begin(a.classes, 32), tier_begin(a.classes, 16),
                        tier_begin(a.classes, 8), tier_begin(a.classes, 4),
                        tier_begin(a.classes, 0)};
  int64_t end[4], n = 0;  // end of each range's tasks
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int per = kRowsAhead << q;
    n += (b[q + 1] - b[q] + per - 1) / per;
    end[q] = n;
  }
  for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += warps) {
    if (t < end[0]) rank_rows_group<32>(a, b[0], b[1], t);
    else if (t < end[1]) rank_rows_group<16>(a, b[1], b[2], t - end[0]);
    else if (t < end[2]) rank_rows_group<8>(a, b[2], b[3], t - end[1]);
    else rank_rows_group<4>(a, b[3], b[4], t - end[2]);
  }
}

constexpr int kClassMid = 38;  // the class that ends at kMidMaxDeg

// Rows of out-degree 33..kMidMaxDeg, one per warp, sorted in the warp's slice of shared memory.
__global__ void __launch_bounds__(256) k_rank_rows_warp(RowArgs a) {
  __shared__ int32_t buf[8][kMidMaxDeg];
  int32_t* k = buf[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t b = tier_begin(a.classes, kClassMid), e = tier_begin(a.classes, 32);
  for (int64_t q = b + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); q < e; q += warps) {
    const int32_t v = a.verts[q], x = a.newid[v];
    const int64_t s = a.dag_rowptr[v], o = a.rp[x];
    const int d = (int)(a.dag_rowptr[v + 1] - s);
    if (lane == 0) a.roots[q] = x;
    for (int t = lane; t < d; t += 32) k[t] = a.newid[a.dag_col[s + t]];
    __syncwarp();
    bitonic_sort(k, d, lane, 32, [] { __syncwarp(); });
    for (int t = lane; t < d; t += 32) {
      a.col[o + t] = k[t];
      set_bit(a, x, k[t]);
    }
    __syncwarp();
  }
}

// Longer rows, one per CTA: in shared memory up to kRankCtaRow entries, else in place.
constexpr int kRankCtaRow = 4096;
__global__ void __launch_bounds__(1024) k_rank_rows_cta(RowArgs a) {
  __shared__ int32_t buf[kRankCtaRow];
  const int64_t e = tier_begin(a.classes, kClassMid);
  for (int64_t q = blockIdx.x; q < e; q += gridDim.x) {
    const int32_t v = a.verts[q], x = a.newid[v];
    const int64_t s = a.dag_rowptr[v], o = a.rp[x];
    const int d = (int)(a.dag_rowptr[v + 1] - s);
    int32_t* k = d <= kRankCtaRow ? buf : a.col + o;
    if (threadIdx.x == 0) a.roots[q] = x;
    for (int t = threadIdx.x; t < d; t += blockDim.x) k[t] = a.newid[a.dag_col[s + t]];
    __syncthreads();
    bitonic_sort(k, d, threadIdx.x, blockDim.x, [] { __syncthreads(); });
    for (int t = threadIdx.x; t < d; t += blockDim.x) {
      const int32_t w = k[t];
      if (k == buf) a.col[o + t] = w;
      set_bit(a, x, w);
    }
    __syncthreads();
  }
}

// rk of every bitmap word: the bits before it in its row.  One warp per row.
__global__ void k_rank_prefix(const uint32_t* bits, int32_t h, uint16_t* rk) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < h; x += warps) {
    const uint32_t base = rank_bits_row((uint32_t)x);
    const int nw = (int)(x >> 5) + 1;
    int run = 0;
    for (int q0 = 0; q0 < nw; q0 += 32) {
      const int c = q0 + lane < nw ? __popc(bits[base + q0 + lane]) : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (q0 + lane < nw) rk[base + q0 + lane] = (uint16_t)(run + incl - c);
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}

// Vertices kept as bitmap rows (a multiple of 32; at most 65,536, so that a row's prefix counts
// fit 16 bits).  The bitmap takes h^2 / 16 bytes: twice the arcs' bytes, at least 256 KB and at
// most 64 MB, so that it stays in L2 (126 MB) beside the arcs.
constexpr int32_t kRankMaxTop = 32768;
int32_t rank_top(int32_t n, int64_t m_dag) {
  int64_t h = 2048;
  while (h < kRankMaxTop && h * h < 128 * m_dag) h += 512;
  return (int32_t)std::min<int64_t>(h, ((int64_t)n + 31) & ~(int64_t)31);
}

size_t rank_bits_words(int32_t h) { return (size_t)rank_bits_row((uint32_t)h); }

// The tier boundaries from the out-degree classes, brought back to the host (waits for the stream,
// so the structures queued before it are complete: batches and server slots read them on streams
// of their own).
int read_tiers(jgpm_graph* g, const int32_t* classes) {
  int32_t c[kTierClasses];
  JGPM_CUDA_TRY(cudaMemcpyAsync(c, classes, sizeof(c), cudaMemcpyDeviceToHost, g->stream));
  JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));
  int64_t first[kTierClasses];  // roots above each class
  int64_t above = 0;
  for (int t = kTierClasses - 1; t >= 0; --t) {
    first[t] = above;
    above += c[t];
  }
  RootTiers& t = g->tiers;
  for (int x = 0; x < 34; ++x) t.deg_begin[x] = first[x];
  t.small_end = first[0];
  t.mid_end = first[32];
  t.large_end = first[38];   // d <= kMidMaxDeg
  t.wide_begin = first[40];  // d <= kWideMaxDeg
  const int le[6] = {32, 34, 35, 36, 37, 39};  // 32, 64, 128, 256, 512, 2048
  for (int x = 0; x < 6; ++x) t.le_begin[x] = first[le[x]];
  return JGPM_OK;
}

int bits_for(int32_t most) { return std::max(1, 32 - __builtin_clz((unsigned)std::max(1, most))); }

// The tiers of a graph whose out-degrees are all small, on the id DAG.
int build_light_tiers(jgpm_graph* g) {
  cudaStream_t s = g->stream;
  const int32_t n = g->n;
  int rc;
  const int out_bits = bits_for(g->max_out_degree);
  size_t tb = 0;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(
      nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr, (int32_t*)nullptr,
      n, 0, out_bits, s));
  const size_t vec = ((size_t)n * 4 + 255) & ~(size_t)255;
  DevBuf buf(s);  // classes, two key arrays, values, cub's space
  if ((rc = dalloc((char**)&buf.p, kTierBytes + 3 * vec + tb, s))) return rc;
  char* at = (char*)buf.p + kTierBytes;
  int32_t* classes = (int32_t*)buf.p;
  uint32_t *k0 = (uint32_t*)at, *k1 = (uint32_t*)(at + vec);
  int32_t* v0 = (int32_t*)(at + 2 * vec);
  if ((rc = dalloc((char**)&g->d_rd_mem, 2 * vec, s))) return rc;
  g->d_rd_sdeg = (int32_t*)g->d_rd_mem;
  g->tiers.d_roots = (int32_t*)((char*)g->d_rd_mem + vec);
  JGPM_CUDA_TRY(cudaMemsetAsync(classes, 0, kTierBytes, s));
  k_root_keys<<<grid_for(n), 256, 0, s>>>(g->d_dag_rowptr, g->d_rowptr, n, k0, v0, g->d_rd_sdeg,
                                          classes);
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(
      at + 3 * vec, tb, k0, k1, v0, g->tiers.d_roots, n, 0, out_bits, s));
  JGPM_CUDA_TRY(cudaGetLastError());
  g->tiers.light = true;
  return read_tiers(g, classes);
}

// Largest graph whose two vertex orders come from one sort of 2n entries: three launches and two
// memsets less, for up to two passes over the entries more.
constexpr int32_t kOneSort = 1 << 18;
// Up to this size a sort is one launch anyway.
constexpr int32_t kTwoSorts = 4096;

// Renumbers the vertices and sorts the roots: g->d_rd_rowptr, d_rd_sdeg, tiers; then the rows
// and the bitmap.  Every range of the kernels follows from the out-degree classes on the device:
// the host waits once, at the end.
int build_rank_dag(jgpm_graph* g) {
  cudaStream_t s = g->stream;
  const int32_t n = g->n;
  int rc;
  const int deg_bits = bits_for(g->max_degree), out_bits = bits_for(g->max_out_degree);
  const bool both = n > kTwoSorts && n <= kOneSort && deg_bits + out_bits < 32;
  const int64_t entries = both ? 2 * (int64_t)n : n;
  const int bits = both ? deg_bits + out_bits + 1 : deg_bits;
  size_t tb = 0, tb2 = 0, tb3 = 0;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint32_t*)nullptr,
                                                (uint32_t*)nullptr, (int32_t*)nullptr,
                                                (int32_t*)nullptr, entries, 0, bits, s));
  if (!both)
    JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(
        nullptr, tb2, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr, (int32_t*)nullptr,
        (int64_t)n, 0, out_bits, s));
  JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb3, (int64_t*)nullptr, (int64_t*)nullptr,
                                              n + 1, s));
  tb = std::max(tb, std::max(tb2, tb3));
  auto room = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
  const size_t vec = room((size_t)n * 4), sorted = room((size_t)entries * 4);
  // one temporary allocation: keys and values, in and out, new ids, vertices by out-degree, cub's
  // space
  DevBuf buf(s);
  if ((rc = dalloc((char**)&buf.p, 4 * sorted + 2 * vec + tb, s))) return rc;
  char* at = (char*)buf.p;
  uint32_t *k0 = (uint32_t*)at, *k1 = (uint32_t*)(at + sorted);
  int32_t *v0 = (int32_t*)(at + 2 * sorted), *order = (int32_t*)(at + 3 * sorted),
          *newid = (int32_t*)(at + 4 * sorted), *verts = (int32_t*)(at + 4 * sorted + vec);
  if (both) verts = order + n;
  void* tmp = at + 4 * sorted + 2 * vec;
  // one allocation: row pointers, degrees, roots, arcs, bitmap, out-degree classes
  g->rd_h = rank_top(n, g->m_dag);
  const size_t bit_bytes = room(rank_bits_words(g->rd_h) * 4);
  const size_t rp_bytes = room(((size_t)n + 1) * 8), arc_bytes = room((size_t)g->m_dag * 4);
  if ((rc = dalloc((char**)&g->d_rd_mem, rp_bytes + 2 * vec + arc_bytes + bit_bytes + kTierBytes,
                   s)))
    return rc;
  g->d_rd_rowptr = (int64_t*)g->d_rd_mem;
  char* own = (char*)g->d_rd_mem + rp_bytes;
  g->d_rd_sdeg = (int32_t*)own;
  g->tiers.d_roots = (int32_t*)(own + vec);
  g->d_rd_col = (int32_t*)(own + 2 * vec);
  g->d_rd_bits = (uint32_t*)(own + 2 * vec + arc_bytes);
  int32_t* classes = (int32_t*)(own + 2 * vec + arc_bytes + bit_bytes);
  JGPM_CUDA_TRY(cudaMemsetAsync(g->d_rd_bits, 0, bit_bytes + kTierBytes, s));
  k_order_keys<<<grid_for(n), 256, 0, s>>>(g->d_rowptr, g->d_dag_rowptr, n, deg_bits, out_bits,
                                           both, k0, v0, classes);
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, k0, k1, v0, order, entries, 0, bits, s));
  uint32_t* k2 = both ? nullptr : k0;  // the second sort's input
  int32_t* v2 = both ? nullptr : v0;
  if (n <= kRankOneCta) {
    k_rank_label_scan<<<1, 1024, 0, s>>>(order, g->d_dag_rowptr, g->d_rowptr, n, newid,
                                         g->d_rd_rowptr, g->d_rd_sdeg, k2, v2);
  } else {
    k_rank_label<<<grid_for(n), 256, 0, s>>>(order, g->d_dag_rowptr, g->d_rowptr, n, newid,
                                             g->d_rd_rowptr, g->d_rd_sdeg, k2, v2);
    JGPM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(tmp, tb, g->d_rd_rowptr, g->d_rd_rowptr, n + 1,
                                                s));
  }
  if (!both)
    JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(tmp, tb, k0, k1, v0, verts, (int64_t)n,
                                                            0, out_bits, s));
  const RowArgs a{verts, g->d_dag_rowptr, g->d_dag_col, newid, g->d_rd_rowptr, g->d_rd_col,
                  g->d_rd_bits, g->tiers.d_roots, classes, g->rd_h};
  k_rank_rows_small<<<grid_for((int64_t)n * 2), 256, 0, s>>>(a);
  if (g->max_out_degree > 32)
    k_rank_rows_warp<<<(int)std::min<int64_t>(148 * 6, ((int64_t)n + 7) / 8), 256, 0, s>>>(a);
  if (g->max_out_degree > kMidMaxDeg) k_rank_rows_cta<<<148 * 2, 1024, 0, s>>>(a);
  JGPM_CUDA_TRY(cudaGetLastError());
  return read_tiers(g, classes);
}

void free_rank_dag(jgpm_graph* g) {
  gfree(g->d_rd_mem, g->stream);
  gfree(g->d_rd_rk, g->stream);
  g->d_rd_mem = nullptr;
  g->d_rd_rowptr = nullptr;
  g->d_rd_col = nullptr;
  g->d_rd_sdeg = nullptr;
  g->d_rd_bits = nullptr;
  g->d_rd_rk = nullptr;
  g->rd_h = 0;
  g->tiers = RootTiers();
}

}  // namespace

int ensure_tiers(jgpm_graph* g) {
  int rc;
  if ((rc = ensure_dag(g))) return rc;
  if (g->tiers.d_roots) return JGPM_OK;
  if ((rc = light_dag(g) ? build_light_tiers(g) : build_rank_dag(g))) free_rank_dag(g);
  return rc;
}

int ensure_rank_dag(jgpm_graph* g) {
  int rc;
  if ((rc = ensure_dag(g))) return rc;
  if (g->d_rd_rowptr) return JGPM_OK;
  free_rank_dag(g);  // tiers on the id DAG
  if ((rc = build_rank_dag(g))) free_rank_dag(g);
  return rc;
}

// Graphs that are counted on the id DAG, every row by scans: renumbering them costs more than it
// saves, where rows are short and few lie in the bitmap.  R-MAT, first call | later calls in us, rank
// DAG and id DAG: 4-cliques of 40,000 vertices, edge factor 8, a = 0.51: 165 and 122 | 54 and 53; of
// 4,194,304 vertices, edge factor 4, a = 0.51 (out-degrees up to 44): 1,186 and 767 | 574 and 620.
// A graph that lies in the bitmap whole, with some 12 arcs a vertex or more, is better off there
// (2,500 vertices, edge factor 32, a = 0.45: 116 and 88 | 40 and 49), and so are graphs with many
// roots above 32 entries, whose pairs grow with the square, or of less than 4 M arcs with a few of
// them, which cost a launch more (8,273 vertices, edge factor 16, a = 0.451: 160 and 127 | 44 and
// 59).
bool light_dag(const jgpm_graph* g) {
  if (g->max_out_degree > kLightOutDegree) return false;
  if (g->over32 > 0) return g->m_dag >= (int64_t)1 << 22 && g->over32 <= g->m_dag / 2048;
  return g->m_dag < 12 * (int64_t)g->n || rank_top(g->n, g->m_dag) < g->n;
}

int ensure_rank_prefix(jgpm_graph* g) {
  if (g->d_rd_rk) return JGPM_OK;
  int rc;
  if ((rc = ensure_tiers(g))) return rc;
  if (!g->d_rd_rowptr) return JGPM_OK;  // no bitmap
  if ((rc = dalloc(&g->d_rd_rk, rank_bits_words(g->rd_h), g->stream))) return rc;
  k_rank_prefix<<<grid_for((int64_t)g->rd_h * 32), 256, 0, g->stream>>>(g->d_rd_bits, g->rd_h,
                                                                        g->d_rd_rk);
  JGPM_CUDA_TRY(cudaGetLastError());
  JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));  // read on other streams by batches
  return JGPM_OK;
}

RankDag rank_dag(const jgpm_graph* g) {
  RankDag r;
  r.rp = g->d_rd_rowptr ? g->d_rd_rowptr : g->d_dag_rowptr;
  r.col = g->d_rd_rowptr ? g->d_rd_col : g->d_dag_col;
  r.bits = g->d_rd_bits;
  r.rk = g->d_rd_rk;
  r.sdeg = g->d_rd_sdeg;
  r.h = g->rd_h;
  return r;
}

uint64_t rank_dag_bytes(const jgpm_graph* g) {
  if (!g->d_rd_rowptr) return g->d_rd_mem ? (uint64_t)g->n * 4 : 0;  // degrees
  const uint64_t words = rank_bits_words(g->rd_h);
  return (uint64_t)(g->n + 1) * 8 + (uint64_t)g->m_dag * 4 + (uint64_t)g->n * 4 + words * 4 +
         (g->d_rd_rk ? words * 2 : 0);
}

int ensure_control(jgpm_graph* g) {
  if (g->d_ctl) return JGPM_OK;
  int rc;
  if (!g->ev0) JGPM_CUDA_TRY(cudaEventCreate(&g->ev0));
  if (!g->ev1) JGPM_CUDA_TRY(cudaEventCreate(&g->ev1));
  if (!g->h_ctl && !(g->h_ctl = ctl_slot())) {
    jgpm_set_error_("pinned host allocation of a control block failed");
    return JGPM_ENOMEM;
  }
  memset(g->h_ctl, 0, sizeof(DevControl));
  if ((rc = dalloc(&g->d_ctl, 1, g->stream))) return rc;
  return JGPM_OK;
}

int ensure_scratch(jgpm_graph* g, size_t bytes) {
  if (g->scratch_bytes >= bytes) return JGPM_OK;
  if (g->d_scratch) gfree(g->d_scratch, g->stream);
  g->d_scratch = nullptr;
  g->scratch_bytes = 0;
  int rc;
  if ((rc = dalloc((char**)&g->d_scratch, bytes, g->stream))) return rc;
  g->scratch_bytes = bytes;
  return JGPM_OK;
}

int ensure_aux(jgpm_graph* g, size_t bytes) {
  if (g->aux_bytes >= bytes) return JGPM_OK;
  if (g->d_aux) gfree(g->d_aux, g->stream);
  g->d_aux = nullptr;
  g->aux_bytes = 0;
  int rc;
  if ((rc = dalloc((char**)&g->d_aux, bytes, g->stream))) return rc;
  g->aux_bytes = bytes;
  return JGPM_OK;
}

namespace {
// Gives back every array of a graph but its control block; the graph is as before its upload.
void drop_arrays(jgpm_graph* g) {
  auto drop = [&](auto*& p) {
    gfree(p, g->stream);
    p = nullptr;
  };
  drop(g->d_rowptr);
  drop(g->d_col);
  drop(g->d_dag_rowptr);
  drop(g->d_dag_col);
  drop(g->d_keep);
  drop(g->d_rank_rowptr);
  drop(g->d_rank_col);
  drop(g->d_c4_small);
  drop(g->d_c4_mid);
  drop(g->d_c4_large);
  drop(g->d_scratch);
  drop(g->d_aux);
  free_rank_dag(g);
  g->aux_bytes = g->scratch_bytes = 0;
  g->c4_nsmall = -1;
  g->c4_nmid = g->c4_nlarge = g->c4_ndense = 0;
  g->c4_large_keys.clear();
}
}  // namespace

void free_graph_device(jgpm_graph* g) {
  drop_arrays(g);
  gfree(g->d_ctl, g->stream);
  ctl_release(g->h_ctl);
  if (g->ev0) cudaEventDestroy(g->ev0);
  if (g->ev1) cudaEventDestroy(g->ev1);
  if (g->stream) cudaStreamDestroy(g->stream);
}

}  // namespace jgpm

// ------------------------------------------------------------------- rank relabelling
namespace jgpm {
namespace {

__global__ void k_rank_keys(const int64_t* rowptr, int32_t n, uint64_t* keys, int32_t* vals) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    keys[v] = ((uint64_t)(rowptr[v + 1] - rowptr[v]) << 32) | (uint64_t)v;
    vals[v] = (int32_t)v;
  }
}

__global__ void k_invert(const int32_t* order, int32_t n, int32_t* rank) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
    rank[order[p]] = (int32_t)p;
}

__global__ void k_rank_arc_keys(const int32_t* src, const int32_t* col, const int32_t* rank,
                                int64_t m, int shift, uint64_t* keys) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += stride)
    keys[k] = ((uint64_t)rank[src[k]] << shift) | (uint64_t)rank[col[k]];
}

__global__ void k_low_bits(const uint64_t* keys, int64_t m, uint64_t mask, int32_t* col) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += stride)
    col[k] = (int32_t)(keys[k] & mask);
}

}  // namespace

// Relabels the symmetric CSR by rank -- position in (degree, id) order, the order the DAG
// orientation uses -- and sorts every row by rank, so "neighbours ranked below v" is a prefix
// of each row.  Built once per graph.
int ensure_rank_csr(jgpm_graph* g) {
  if (g->d_rank_rowptr) return JGPM_OK;
  cudaStream_t s = g->stream;
  const int32_t n = g->n;
  const int64_t m = g->m;
  const int shift = shift_for(n);
  int rc;
  DevBuf k0(g->stream), k1(g->stream), v0(g->stream), v1(g->stream), rank(g->stream), src(g->stream), tmp(g->stream);
  if ((rc = dalloc((uint64_t**)&k0.p, n, g->stream))) return rc;
  if ((rc = dalloc((uint64_t**)&k1.p, n, g->stream))) return rc;
  if ((rc = dalloc((int32_t**)&v0.p, n, g->stream))) return rc;
  if ((rc = dalloc((int32_t**)&v1.p, n, g->stream))) return rc;
  if ((rc = dalloc((int32_t**)&rank.p, n, g->stream))) return rc;
  k_rank_keys<<<grid_for(n), 256, 0, s>>>(g->d_rowptr, n, (uint64_t*)k0.p, (int32_t*)v0.p);
  size_t tb = 0;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint64_t*)k0.p, (uint64_t*)k1.p,
                                                (int32_t*)v0.p, (int32_t*)v1.p, n, 0, 64, s));
  if ((rc = dalloc((char**)&tmp.p, tb, g->stream))) return rc;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, tb, (uint64_t*)k0.p, (uint64_t*)k1.p,
                                                (int32_t*)v0.p, (int32_t*)v1.p, n, 0, 64, s));
  k_invert<<<grid_for(n), 256, 0, s>>>((int32_t*)v1.p, n, (int32_t*)rank.p);
  // arcs as (rank(u), rank(v)) keys, sorted
  DevBuf ak(g->stream), ak2(g->stream), tmp2(g->stream);
  if ((rc = dalloc((int32_t**)&src.p, m, g->stream))) return rc;
  if ((rc = dalloc((uint64_t**)&ak.p, m, g->stream))) return rc;
  if ((rc = dalloc((uint64_t**)&ak2.p, m, g->stream))) return rc;
  k_arc_src<<<grid_for((int64_t)n * 32), 256, 0, s>>>(g->d_rowptr, n, (int32_t*)src.p);
  k_rank_arc_keys<<<grid_for(m), 256, 0, s>>>((int32_t*)src.p, g->d_col, (int32_t*)rank.p, m,
                                              shift, (uint64_t*)ak.p);
  cub::DoubleBuffer<uint64_t> db((uint64_t*)ak.p, (uint64_t*)ak2.p);
  size_t tb2 = 0;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, tb2, db, m, 0, 2 * shift, s));
  if ((rc = dalloc((char**)&tmp2.p, tb2, g->stream))) return rc;
  JGPM_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp2.p, tb2, db, m, 0, 2 * shift, s));
  if ((rc = dalloc(&g->d_rank_rowptr, (size_t)n + 1, g->stream))) return rc;
  if ((rc = dalloc(&g->d_rank_col, m, g->stream))) {
    gfree(g->d_rank_rowptr, g->stream);
    g->d_rank_rowptr = nullptr;
    return rc;
  }
  k_low_bits<<<grid_for(m), 256, 0, s>>>(db.Current(), m, (1ull << shift) - 1, g->d_rank_col);
  k_rowptr_from_keys<<<grid_for((int64_t)n + 1), 256, 0, s>>>(db.Current(), m, n, shift,
                                                              g->d_rank_rowptr);
  JGPM_CUDA_TRY(cudaGetLastError());
  JGPM_CUDA_TRY(cudaStreamSynchronize(s));
  return JGPM_OK;
}

}  // namespace jgpm

// ------------------------------------------------------------------- file I/O (host)
namespace jgpm {

// Reads the reference's on-disk CSR (common/graph.cc:26-46): prefix.meta.txt holds
// "n m vid_size eid_size vlabel_size elabel_size max_degree feat_len nvclasses neclasses".
int read_reference_files(const std::string& prefix, std::vector<int64_t>& rowptr,
                         std::vector<int32_t>& col, int32_t* n_out) {
  std::ifstream meta(prefix + ".meta.txt");
  if (!meta) {
    jgpm_set_error_("cannot open " + prefix + ".meta.txt");
    return JGPM_EIO;
  }
  int64_t n = 0, m = 0;
  int vid_size = 0, eid_size = 0;
  meta >> n >> m >> vid_size >> eid_size;
  if (!meta || n < 1 || m < 0 || vid_size != 4 || eid_size != 8 || n > INT32_MAX) {
    jgpm_set_error_(prefix + ".meta.txt: expected n, m, vid size 4, eid size 8");
    return JGPM_EIO;
  }
  rowptr.resize((size_t)n + 1);
  col.resize((size_t)m);
  std::ifstream fv(prefix + ".vertex.bin", std::ios::binary);
  std::ifstream fe(prefix + ".edge.bin", std::ios::binary);
  if (!fv || !fe) {
    jgpm_set_error_("cannot open " + prefix + ".vertex.bin / .edge.bin");
    return JGPM_EIO;
  }
  fv.read(reinterpret_cast<char*>(rowptr.data()), (std::streamsize)((n + 1) * 8));
  fe.read(reinterpret_cast<char*>(col.data()), (std::streamsize)(m * 4));
  if (!fv || (m > 0 && !fe)) {
    jgpm_set_error_(prefix + ": truncated .vertex.bin or .edge.bin");
    return JGPM_EIO;
  }
  *n_out = (int32_t)n;
  return JGPM_OK;
}

// Writes the reference's on-disk CSR as Graph::dump_binary does (common/graph.cc:727-753).
int write_reference_files(const std::string& prefix, const std::vector<int64_t>& rowptr,
                          const std::vector<int32_t>& col, int32_t n, int32_t max_degree) {
  std::ofstream fv(prefix + ".vertex.bin", std::ios::binary);
  std::ofstream fe(prefix + ".edge.bin", std::ios::binary);
  std::ofstream meta(prefix + ".meta.txt");
  if (!fv || !fe || !meta) {
    jgpm_set_error_("cannot write " + prefix + ".*");
    return JGPM_EIO;
  }
  fv.write(reinterpret_cast<const char*>(rowptr.data()), (std::streamsize)(rowptr.size() * 8));
  fe.write(reinterpret_cast<const char*>(col.data()), (std::streamsize)(col.size() * 4));
  meta << n << "\n" << col.size() << "\n4 8 1 2\n" << max_degree << "\n0\n0\n0\n";
  if (!fv || !fe || !meta) {
    jgpm_set_error_("short write to " + prefix + ".*");
    return JGPM_EIO;
  }
  return JGPM_OK;
}

}  // namespace jgpm

namespace jgpm {

// Frees the device arrays of a graph (CSR, DAG, tiers, scratch) and keeps a host copy of the
// symmetric CSR so the graph can be made resident again (served graph pool eviction).
int evict_graph(jgpm_graph* g, std::vector<int64_t>& h_rowptr, std::vector<int32_t>& h_col) {
  if (!g->d_rowptr) return JGPM_OK;
  if (h_rowptr.empty()) {
    h_rowptr.resize((size_t)g->n + 1);
    h_col.resize((size_t)g->m);
    JGPM_CUDA_TRY(cudaMemcpyAsync(h_rowptr.data(), g->d_rowptr, ((size_t)g->n + 1) * 8,
                                  cudaMemcpyDeviceToHost, g->stream));
    if (g->m)
      JGPM_CUDA_TRY(cudaMemcpyAsync(h_col.data(), g->d_col, (size_t)g->m * 4,
                                    cudaMemcpyDeviceToHost, g->stream));
  }
  JGPM_CUDA_TRY(cudaStreamSynchronize(g->stream));
  drop_arrays(g);
  return JGPM_OK;
}

// Uploads an evicted graph again and rebuilds its DAG and root tiers.  On an error the graph stays
// evicted.
int restore_graph(jgpm_graph* g, const std::vector<int64_t>& h_rowptr,
                  const std::vector<int32_t>& h_col) {
  if (g->d_rowptr) return JGPM_OK;
  int rc = upload_csr(g, h_rowptr.data(), h_col.data(), g->n, (int64_t)h_col.size(), 0, 0);
  if (!rc) rc = ensure_dag(g);
  if (!rc) rc = ensure_tiers(g);
  if (rc) drop_arrays(g);
  return rc;
}

// Device bytes held by a resident graph's arrays.
uint64_t graph_device_bytes(const jgpm_graph* g) {
  if (!g->d_rowptr) return 0;
  uint64_t b = (uint64_t)(g->n + 1) * 8 + (uint64_t)g->m * 4;
  if (g->d_dag_rowptr) b += (uint64_t)(g->n + 1) * 8 + (uint64_t)g->m_dag * 4;
  if (g->tiers.d_roots) b += (uint64_t)g->n * 4 + rank_dag_bytes(g);
  if (g->d_rank_rowptr) b += (uint64_t)(g->n + 1) * 8 + (uint64_t)g->m * 4;
  if (g->d_c4_small) b += (uint64_t)(g->c4_nsmall + g->c4_nmid + g->c4_nlarge) * 4 + 48;
  return b + g->scratch_bytes + g->aux_bytes;
}

}  // namespace jgpm

// Test hook: the `after`-th allocation from the pools from now on (0 = the next), by any thread,
// fails with JGPM_ENOMEM; a negative number calls it off.
extern "C" void jgpm_fail_alloc_(int64_t after) { jgpm::g_fail_alloc.store(after); }
