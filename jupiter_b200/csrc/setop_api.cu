// jgpm_setop / jgpm_setop_batch: the sorted-set operations as library calls.
//
// One warp per operand pair (warp-cooperative primitives of setops.cuh).  Host arrays are
// staged to the device and results copied back; device arrays are used in place.
//
// A call on device arrays is one check kernel (offsets and capacities), one set-op kernel that
// does nothing if the check failed, and one read-back.  Measured on 100,000 pairs of lists of 4 to
// 4,096 ids: 1.63 ms a call when the offsets were copied to the host, checked there, and the call
// made its own stream; 0.39 ms with the check on the device (the set-op kernel 0.36 ms of it, each
// list searched where it lies); 0.25 ms with the pairs handed out and the longer list in tiles.
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "jgpm_internal.h"
#include "setops.cuh"

namespace jgpm {
namespace {

// State of one call, all ones at its start: where the offsets first break a rule (pair index;
// kNone: nowhere), and the pairs handed out.
struct OffsetCheck {
  unsigned long long bad;       // negative or over-long list
  unsigned long long capacity;  // output room too small
  unsigned long long taken;     // the next pair is taken + 1
};
constexpr unsigned long long kNone = ~0ull;

// The next pair of a warp.  Pairs differ by orders of magnitude: handed out one by one, not dealt
// out in advance (which left the SMs half empty).
__device__ __forceinline__ int64_t next_pair(OffsetCheck* st) {
  unsigned long long q = 0;
  if ((threadIdx.x & 31) == 0) q = atomicAdd(&st->taken, 1ull) + 1ull;
  return (int64_t)__shfl_sync(kFull, q, 0);
}

// warp_lookup with B in tiles of kTile ids in the warp's shared memory: every id of both lists is
// read once, in coalesced loads, and the searches, ten dependent steps each, run on chip.  For B
// up to kTileRatio times A's length; above that fewer ids are touched by searching B where it
// lies.  100,000 intersections of lists of 4 to 4,096 ids: see the head of this file; ratios of 4,
// 16 and 64 measure alike there (262, 265 and 266 us in one run).
constexpr int kTile = 512;
constexpr int kTileRatio = 16;
template <typename Visit>
__device__ __forceinline__ void tile_lookup(const int32_t* a, int na, const int32_t* b, int nb,
                                            int32_t* tile, Visit&& visit) {
  if (nb > kTileRatio * (int64_t)na) {
    warp_lookup(a, na, b, nb, visit);
    return;
  }
  const int lane = threadIdx.x & 31;
  int b0 = 0, tl = 0, top = 0;
  auto load = [&]() {
    tl = min(kTile, nb - b0);
    top = tl > 0 ? 1 << (31 - __clz(tl)) : 0;
    int32_t v[kTile / 32];
#pragma unroll
    for (int q = 0; q < kTile / 32; ++q)
      v[q] = q * 32 + lane < tl ? __ldg(b + b0 + q * 32 + lane) : 0;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kTile / 32; ++q) tile[q * 32 + lane] = v[q];
    __syncwarp();
  };
  load();
  int32_t ahead = lane < na ? __ldg(a + lane) : INT32_MAX;
  for (int base = 0; base < na; base += 32) {
    const int32_t key = ahead;
    const bool valid = base + lane < na;
    ahead = base + 32 + lane < na ? __ldg(a + base + 32 + lane) : INT32_MAX;
    bool hit = false, open = valid;
    for (;;) {
      int p = 0;
      for (int step = top; step > 0; step >>= 1)
        if (p + step <= tl && tile[p + step - 1] < key) p += step;
      if (open && p < tl) {
        hit = tile[p] == key;
        open = false;
      }
      if (b0 + tl >= nb || !__any_sync(kFull, open)) break;
      b0 += tl;  // some keys lie past the tile
      load();
    }
    visit(key, valid, hit);
  }
  __syncwarp();
}

// {x in A & B : x < upper}: its size, and the ids in order where out is given.  use_ex leaves ex
// and -1 (the value that stands for no exclusion) out.
__device__ __forceinline__ int pair_intersect(const int32_t* a, int na, const int32_t* b, int nb,
                                              int32_t upper, int32_t ex, bool use_ex,
                                              int32_t* out, int32_t* tile) {
  const int lane = threadIdx.x & 31;
  na = warp_prefix_below(a, na, upper);
  nb = warp_prefix_below(b, nb, upper);
  if (na > nb) {
    const int32_t* t = a; a = b; b = t;
    const int tn = na; na = nb; nb = tn;
  }
  int written = 0;
  tile_lookup(a, na, b, nb, tile, [&](int32_t key, bool valid, bool in_b) {
    const bool f = valid && in_b && !(use_ex && (key == ex || key == -1));
    const unsigned mask = __ballot_sync(kFull, f);
    if (out && f) out[written + __popc(mask & ((1u << lane) - 1u))] = key;
    written += __popc(mask);
  });
  return written;
}

// {x in A : x < upper, x not in B, x != ex}: its size, and the ids in order where out is given.
__device__ __forceinline__ int pair_difference(const int32_t* a, int na, const int32_t* b, int nb,
                                               int32_t upper, int32_t ex, int32_t* out,
                                               int32_t* tile) {
  const int lane = threadIdx.x & 31;
  na = warp_prefix_below(a, na, upper);
  nb = warp_prefix_below(b, nb, upper);
  int written = 0;
  tile_lookup(a, na, b, nb, tile, [&](int32_t key, bool valid, bool in_b) {
    const bool f = valid && key != ex && !in_b;
    const unsigned mask = __ballot_sync(kFull, f);
    if (out && f) out[written + __popc(mask & ((1u << lane) - 1u))] = key;
    written += __popc(mask);
  });
  return written;
}

__global__ void k_check_offsets(const int64_t* a_off, const int64_t* b_off, const int64_t* out_off,
                                int op, int64_t nops, OffsetCheck* st) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nops; i += stride) {
    const int64_t na = a_off[i + 1] - a_off[i], nb = b_off[i + 1] - b_off[i];
    if (na < 0 || nb < 0 || na > INT32_MAX || nb > INT32_MAX ||
        (i == 0 && (a_off[0] < 0 || b_off[0] < 0)))
      atomicMin(&st->bad, (unsigned long long)i);
    else if (out_off && out_off[i + 1] - out_off[i] < (op == JGPM_OP_INTERSECT ? min(na, nb) : na))
      atomicMin(&st->capacity, (unsigned long long)i);
  }
}

__global__ void k_setop_batch(int op, const int32_t* a, const int64_t* a_off, const int32_t* b,
                              const int64_t* b_off, int64_t nops, const int32_t* upper,
                              const int32_t* exclude, int32_t* counts, int32_t* out,
                              const int64_t* out_off, OffsetCheck* st) {
  __shared__ int32_t tiles[8][kTile];
  int32_t* tile = tiles[threadIdx.x >> 5];
  if (st->bad != kNone || st->capacity != kNone) return;
  for (int64_t i = next_pair(st); i < nops; i = next_pair(st)) {
    const int32_t* A = a + a_off[i];
    const int na = (int)(a_off[i + 1] - a_off[i]);
    const int32_t* B = b + b_off[i];
    const int nb = (int)(b_off[i + 1] - b_off[i]);
    const int32_t up = upper ? upper[i] : INT32_MAX;
    const int32_t ex = exclude ? exclude[i] : -1;
    int c = 0;
    switch (op) {
      case JGPM_OP_INTERSECT:
        c = pair_intersect(A, na, B, nb, up, 0, false, out + out_off[i], tile);
        break;
      case JGPM_OP_INTERSECT_COUNT:
        c = pair_intersect(A, na, B, nb, up, ex, true, nullptr, tile);
        break;
      case JGPM_OP_DIFFERENCE:
        c = pair_difference(A, na, B, nb, up, ex, out + out_off[i], tile);
        break;
      case JGPM_OP_DIFFERENCE_COUNT:
        c = pair_difference(A, na, B, nb, up, ex, nullptr, tile);
        break;
    }
    if ((threadIdx.x & 31) == 0) counts[i] = c;
  }
}

// Fused splits, one warp per pair; pair i's outputs sit at the offsets of its operands
// (c and d at a_off[i], e at b_off[i]).
__global__ void k_split_batch(int kind, const int32_t* a, const int64_t* a_off, const int32_t* b,
                              const int64_t* b_off, int64_t nops, const int32_t* upper,
                              int32_t* counts, int32_t* c, int32_t* d, int32_t* e,
                              OffsetCheck* st) {
  if (st->bad != kNone) return;
  for (int64_t i = next_pair(st); i < nops; i = next_pair(st)) {
    const int64_t a0 = a_off[i], b0 = b_off[i];
    const int32_t* A = a + a0;
    const int na = (int)(a_off[i + 1] - a0);
    const int32_t* B = b + b0;
    const int nb = (int)(b_off[i + 1] - b0);
    int r;
    if (kind == JGPM_SPLIT_FUSE) {
      r = na - warp_split_by(A, na, B, nb, INT32_MAX, c + a0, d + a0);  // |A & B|
      warp_split_by(B, nb, A, na, INT32_MAX, e + b0, nullptr);
    } else {
      r = warp_split_by(A, na, B, nb, upper ? upper[i] : INT32_MAX, c + a0, d + a0);
    }
    if ((threadIdx.x & 31) == 0) counts[i] = r;
  }
}

bool is_device_ptr(const void* p) {
  if (!p) return false;
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

// Device copy of a caller array (host or device) of `count` elements.
template <typename T>
struct Staged {
  T* d = nullptr;
  bool owned = false;
  cudaStream_t stream = nullptr;
  cudaError_t init(const T* src, size_t count, cudaStream_t s) {
    if (!src) return cudaSuccess;
    if (is_device_ptr(src)) {
      d = const_cast<T*>(src);
      return cudaSuccess;
    }
    stream = s;
    owned = true;
    if (gmalloc((void**)&d, std::max<size_t>(count, 1) * sizeof(T), s)) {
      d = nullptr;
      return cudaErrorMemoryAllocation;
    }
    if (count) return cudaMemcpyAsync(d, src, count * sizeof(T), cudaMemcpyHostToDevice, s);
    return cudaSuccess;
  }
  ~Staged() {
    if (owned && d) gfree(d, stream);
  }
};

// Streams of the calls: taken for one call, given back idle at its end and kept for the next (at
// most kStreamsKept per device), so that a call does not pay for making one.
constexpr size_t kStreamsKept = 8;
std::mutex g_stream_mu;
std::vector<cudaStream_t> g_streams[64];

struct CallStream {
  cudaStream_t s = nullptr;
  int dev = 0;
  // The stream waits for what the caller has queued on the legacy default stream (inputs written
  // there need no synchronisation first).
  cudaError_t init() {
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64) {
      std::lock_guard<std::mutex> lk(g_stream_mu);
      if (!g_streams[dev].empty()) {
        s = g_streams[dev].back();
        g_streams[dev].pop_back();
      }
    }
    if (!s && (e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)) != cudaSuccess) return e;
    cudaEvent_t ev = nullptr;
    if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) return e;
    e = cudaEventRecord(ev, cudaStreamLegacy);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, ev, 0);
    cudaEventDestroy(ev);
    return e;
  }
  ~CallStream() {
    if (!s) return;
    if (dev < 64) {
      std::lock_guard<std::mutex> lk(g_stream_mu);
      if (g_streams[dev].size() < kStreamsKept) {
        g_streams[dev].push_back(s);
        return;
      }
    }
    cudaStreamDestroy(s);
  }
};

// The offsets of a call: on the device, and checked there or (host arrays) on the host.
struct Offsets {
  Staged<int64_t> a, b, out;
  int64_t a_end = 0, b_end = 0, out_end = 0;  // totals, where staging needs them
  OffsetCheck* check = nullptr;
  cudaStream_t stream = nullptr;
  bool checked = false;  // on the host, or the device check's result is read
  bool a_null = false, b_null = false;  // operand or output arrays that only empty lists allow
  // Returns JGPM_OK or the error.  need_totals: host arrays have to be sized.
  int init(const char* who, const int64_t* a_off, const int64_t* b_off, const int64_t* out_off,
           int op, int64_t nops, bool need_totals, cudaStream_t s) {
    stream = s;
    const bool host = !is_device_ptr(a_off) && !is_device_ptr(b_off) &&
                      (!out_off || !is_device_ptr(out_off));
    if (host) {
      a_end = a_off[nops];
      b_end = b_off[nops];
      out_end = out_off ? out_off[nops] : 0;
      if (a_off[0] < 0 || b_off[0] < 0 || missing()) return bad(who);
      for (int64_t i = 0; i < nops; ++i) {
        const int64_t na = a_off[i + 1] - a_off[i], nb = b_off[i + 1] - b_off[i];
        if (na < 0 || nb < 0 || na > INT32_MAX || nb > INT32_MAX) return bad(who);
        if (out_off && out_off[i + 1] - out_off[i] <
                           (op == JGPM_OP_INTERSECT ? std::min(na, nb) : na))
          return small(who);
      }
    }
    JGPM_CUDA_TRY(a.init(a_off, (size_t)nops + 1, s));
    JGPM_CUDA_TRY(b.init(b_off, (size_t)nops + 1, s));
    JGPM_CUDA_TRY(out.init(out_off, (size_t)nops + 1, s));
    if (gmalloc((void**)&check, sizeof(OffsetCheck), s)) return JGPM_ENOMEM;
    JGPM_CUDA_TRY(cudaMemsetAsync(check, 0xff, sizeof(OffsetCheck), s));
    checked = host;
    if (host) return JGPM_OK;
    k_check_offsets<<<(int)std::min<int64_t>((nops + 255) / 256, 148 * 8), 256, 0, s>>>(
        a.d, b.d, out.d, op, nops, check);
    JGPM_CUDA_TRY(cudaGetLastError());
    if (!need_totals) return JGPM_OK;
    JGPM_CUDA_TRY(cudaMemcpyAsync(&a_end, a.d + nops, 8, cudaMemcpyDeviceToHost, s));
    JGPM_CUDA_TRY(cudaMemcpyAsync(&b_end, b.d + nops, 8, cudaMemcpyDeviceToHost, s));
    if (out_off)
      JGPM_CUDA_TRY(cudaMemcpyAsync(&out_end, out.d + nops, 8, cudaMemcpyDeviceToHost, s));
    JGPM_CUDA_TRY(cudaStreamSynchronize(s));
    if (missing()) return bad(who);
    return verdict(who);
  }
  bool missing() const { return (a_end > 0 && a_null) || (b_end > 0 && b_null); }
  // The device check's result, if it is not read yet (the stream is idle then).
  int verdict(const char* who) {
    if (checked) return JGPM_OK;
    checked = true;
    OffsetCheck h;
    JGPM_CUDA_TRY(cudaMemcpyAsync(&h, check, sizeof(h), cudaMemcpyDeviceToHost, stream));
    JGPM_CUDA_TRY(cudaStreamSynchronize(stream));
    if (h.bad != kNone && h.bad <= h.capacity) return bad(who);
    if (h.capacity != kNone) return small(who);
    return JGPM_OK;
  }
  static int bad(const char* who) {
    jgpm_set_error_(std::string(who) + ": bad offsets or missing array");
    return JGPM_EINVAL;
  }
  static int small(const char* who) {
    jgpm_set_error_(std::string(who) + ": output capacity too small");
    return JGPM_ECAPACITY;
  }
  ~Offsets() {
    if (check) gfree(check, stream);
  }
};

// A caller's output array on the device: used in place when it is device memory, else a
// device copy of its current contents (so entries the kernel does not write keep their
// values either way) that back() returns to the caller.
struct OutArray {
  int32_t* user = nullptr;
  int32_t* d = nullptr;
  size_t n = 0;
  bool staged = false;
  cudaStream_t stream = nullptr;
  cudaError_t init(int32_t* p, size_t count, cudaStream_t s) {
    stream = s;
    user = p;
    n = count;
    if (!p) return cudaSuccess;
    if (is_device_ptr(p)) {
      d = p;
      return cudaSuccess;
    }
    staged = true;
    if (gmalloc((void**)&d, std::max<size_t>(count, 1) * sizeof(int32_t), s)) {
      d = nullptr;
      return cudaErrorMemoryAllocation;
    }
    if (count) return cudaMemcpyAsync(d, p, count * sizeof(int32_t), cudaMemcpyHostToDevice, s);
    return cudaSuccess;
  }
  cudaError_t back(cudaStream_t s) {
    if (!staged || !n) return cudaSuccess;
    return cudaMemcpyAsync(user, d, n * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  }
  ~OutArray() {
    if (staged && d) gfree(d, stream);
  }
};

}  // namespace
}  // namespace jgpm

using namespace jgpm;

extern "C" {

int jgpm_setop_batch(int op, const int32_t* a, const int64_t* a_off, const int32_t* b,
                     const int64_t* b_off, int64_t nops, const int32_t* upper,
                     const int32_t* exclude, int32_t* counts, int32_t* out,
                     const int64_t* out_off) {
  if (op < JGPM_OP_INTERSECT || op > JGPM_OP_DIFFERENCE_COUNT || nops < 0 || !a_off || !b_off ||
      !counts) {
    jgpm_set_error_("jgpm_setop_batch: bad arguments");
    return JGPM_EINVAL;
  }
  const bool mat = (op == JGPM_OP_INTERSECT || op == JGPM_OP_DIFFERENCE);
  if (mat && (!out || !out_off)) {
    jgpm_set_error_("jgpm_setop_batch: materialising ops need out and out_off");
    return JGPM_EINVAL;
  }
  if (nops == 0) return JGPM_OK;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    jgpm_set_error_("no CUDA device");
    return JGPM_ENODEV;
  }
  CallStream cs;
  JGPM_CUDA_TRY(cs.init());
  cudaStream_t s = cs.s;
  // device buffers, freed into the stream on every return path
  Offsets off;
  Staged<int32_t> da, db, dup, dex;
  const bool counts_host = !is_device_ptr(counts);
  const bool out_host = mat && !is_device_ptr(out);
  off.a_null = !a;
  off.b_null = !b;
  int rc = off.init("jgpm_setop_batch", a_off, b_off, mat ? out_off : nullptr, op, nops,
                    out_host || !is_device_ptr(a) || !is_device_ptr(b), s);
  if (rc) return rc;
  JGPM_CUDA_TRY(da.init(a, (size_t)off.a_end, s));
  JGPM_CUDA_TRY(db.init(b, (size_t)off.b_end, s));
  JGPM_CUDA_TRY(dup.init(upper, (size_t)nops, s));
  JGPM_CUDA_TRY(dex.init(exclude, (size_t)nops, s));
  struct DeviceBuf {
    int32_t* p = nullptr;
    cudaStream_t s;
    ~DeviceBuf() { gfree(p, s); }
  } tmp_counts{nullptr, s}, tmp_out{nullptr, s};
  int32_t* dcounts = counts;
  int32_t* dout = out;
  if (counts_host) {
    if ((rc = gmalloc((void**)&tmp_counts.p, nops * sizeof(int32_t), s))) return rc;
    dcounts = tmp_counts.p;
  }
  if (out_host) {
    if ((rc = gmalloc((void**)&tmp_out.p, std::max<int64_t>(1, off.out_end) * 4, s))) return rc;
    dout = tmp_out.p;
  }
  const int64_t blocks = std::min<int64_t>((nops + 7) / 8, 148 * 8);
  k_setop_batch<<<(int)std::max<int64_t>(1, blocks), 256, 0, s>>>(
      op, da.d, off.a.d, db.d, off.b.d, nops, dup.d, dex.d, dcounts, mat ? dout : nullptr,
      mat ? off.out.d : nullptr, off.check);
  cudaError_t e = cudaGetLastError();
  // a refused call writes nothing: the staged results are copied back once the verdict is read
  const bool waits = !off.checked;  // for the kernel, to read the verdict
  if (e == cudaSuccess && (rc = off.verdict("jgpm_setop_batch"))) return rc;
  if (e == cudaSuccess && counts_host)
    e = cudaMemcpyAsync(counts, dcounts, nops * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && out_host && off.out_end > 0)
    e = cudaMemcpyAsync(out, dout, off.out_end * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && (!waits || counts_host || out_host)) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    jgpm_set_error_(std::string("jgpm_setop_batch: ") + cudaGetErrorString(e));
    return JGPM_ECUDA;
  }
  return JGPM_OK;
}

int jgpm_setop_split_batch(int kind, const int32_t* a, const int64_t* a_off, const int32_t* b,
                           const int64_t* b_off, int64_t nops, const int32_t* upper,
                           int32_t* counts, int32_t* c, int32_t* d, int32_t* e) {
  const bool fuse = kind == JGPM_SPLIT_FUSE;
  if ((!fuse && kind != JGPM_SPLIT_DIF_INT) || nops < 0 || !a_off || !b_off || !counts) {
    jgpm_set_error_("jgpm_setop_split_batch: bad arguments");
    return JGPM_EINVAL;
  }
  if (nops == 0) return JGPM_OK;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    jgpm_set_error_("no CUDA device");
    return JGPM_ENODEV;
  }
  CallStream cs;
  JGPM_CUDA_TRY(cs.init());
  cudaStream_t s = cs.s;
  Offsets off;
  bool host_arrays = false;  // arrays that are staged have to be sized
  for (const void* p : {(const void*)a, (const void*)b, (const void*)c, (const void*)d,
                        fuse ? (const void*)e : (const void*)c})
    host_arrays = host_arrays || !is_device_ptr(p);
  off.a_null = !a || !c || !d;
  off.b_null = !b || (fuse && !e);
  int rc = off.init("jgpm_setop_split_batch", a_off, b_off, nullptr, 0, nops, host_arrays, s);
  if (rc) return rc;
  Staged<int32_t> da, db, dup;
  JGPM_CUDA_TRY(da.init(a, (size_t)off.a_end, s));
  JGPM_CUDA_TRY(db.init(b, (size_t)off.b_end, s));
  if (!fuse) JGPM_CUDA_TRY(dup.init(upper, (size_t)nops, s));
  OutArray oc, od, oe, on;
  JGPM_CUDA_TRY(oc.init(c, (size_t)off.a_end, s));
  JGPM_CUDA_TRY(od.init(d, (size_t)off.a_end, s));
  if (fuse) JGPM_CUDA_TRY(oe.init(e, (size_t)off.b_end, s));
  JGPM_CUDA_TRY(on.init(counts, (size_t)nops, s));
  const int64_t blocks = std::min<int64_t>((nops + 7) / 8, 148 * 8);
  k_split_batch<<<(int)std::max<int64_t>(1, blocks), 256, 0, s>>>(
      kind, da.d, off.a.d, db.d, off.b.d, nops, dup.d, on.d, oc.d, od.d, oe.d, off.check);
  cudaError_t err = cudaGetLastError();
  if (err == cudaSuccess) err = on.back(s);
  if (err == cudaSuccess) err = oc.back(s);
  if (err == cudaSuccess) err = od.back(s);
  if (err == cudaSuccess) err = oe.back(s);
  if (err == cudaSuccess && off.checked) err = cudaStreamSynchronize(s);
  if (err != cudaSuccess) {
    jgpm_set_error_(std::string("jgpm_setop_split_batch: ") + cudaGetErrorString(err));
    return JGPM_ECUDA;
  }
  return off.verdict("jgpm_setop_split_batch");
}

int jgpm_setop_split(int kind, const int32_t* a, int32_t na, const int32_t* b, int32_t nb,
                     int32_t upper, int32_t* c, int32_t* d, int32_t* e, int32_t* count) {
  if (na < 0 || nb < 0 || !count || (na > 0 && !a) || (nb > 0 && !b)) {
    jgpm_set_error_("jgpm_setop_split: bad arguments");
    return JGPM_EINVAL;
  }
  const int64_t aoff[2] = {0, na}, boff[2] = {0, nb};
  const int32_t up[1] = {upper};
  int32_t cnt = 0;
  const int rc = jgpm_setop_split_batch(kind, a, aoff, b, boff, 1, up, &cnt, c, d, e);
  if (rc) return rc;
  *count = cnt;
  return JGPM_OK;
}

int jgpm_setop(int op, const int32_t* a, int32_t na, const int32_t* b, int32_t nb,
               int32_t upper, int32_t exclude, int32_t* out, int32_t* out_n) {
  if (na < 0 || nb < 0 || !out_n || (na > 0 && !a) || (nb > 0 && !b)) {
    jgpm_set_error_("jgpm_setop: bad arguments");
    return JGPM_EINVAL;
  }
  const int64_t aoff[2] = {0, na}, boff[2] = {0, nb};
  const bool mat = (op == JGPM_OP_INTERSECT || op == JGPM_OP_DIFFERENCE);
  const int64_t cap = op == JGPM_OP_INTERSECT ? std::min(na, nb) : na;
  const int64_t ooff[2] = {0, cap};
  int32_t cnt = 0;
  const int32_t up[1] = {upper};
  const int32_t ex[1] = {exclude};
  int rc = jgpm_setop_batch(op, a, aoff, b, boff, 1, up, ex, &cnt, mat ? out : nullptr,
                            mat ? ooff : nullptr);
  if (rc) return rc;
  *out_n = cnt;
  return JGPM_OK;
}

}  // extern "C"
