// k_scan.cu -- single-pass exclusive uint32 scan with decoupled look-back,
// the compaction primitive between the stages (the reference's PrefixSum:
// PrefixSum.h:58-248 recursive Blelloch scan, PrefixSum.cpp:73-140).
//
// One CTA scans one tile of SCAN_THREADS * SCAN_ITEMS elements.  Tiles are
// numbered by an atomic ticket in launch order, publish their aggregate, and
// look back over predecessors (a warp reads 32 status words at a time) until
// one with an inclusive prefix is found.  Every wait is bounded: after
// TRAX_SPIN_LIMIT polls the tile records TRAX_EBIT_TIMEOUT, treats the
// missing predecessor as zero and finishes, so a lost tile can never hang
// the GPU.  A launch of one tile needs no ticket, status or cleared scratch,
// nor does one CTA that takes the tiles of a small scan in turn.
//
// A compaction scans count + 1 elements; the tile holding the last one also
// publishes the total (ScanTotal), clamped to the capacity of what follows.
// With the scratch of a whole chain cleared by its first kernel, a
// compaction is one launch instead of three nodes (clear, scan, publish),
// each of them 2 to 3 us in a serial graph.
#include "trax_kernels.h"
#include "trax_lookback.cuh"

namespace trax {

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr uint32_t SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
// Scans of up to this many elements (by capacity) are left to one CTA, which
// takes tile after tile: no tickets, no cleared scratch (a node or a call of its
// own in the host-synced stages), no look-back.  One event by stages 330.6 ->
// 326.0 us, 100 events of 200 tracks 159.0 -> 157.8 us, 37 ttbar-like events
// 436.7 -> 436.5 us, 10 events of 10 muons 117.1 -> 117.8 us; 1024 threads took
// 2 to 4 us more of those last.
constexpr int SCAN_ONE_THREADS = 512;
constexpr uint32_t SCAN_ONE_MAX = 16384;

// One tile of a scan, or all of them by one CTA (ONE).
template <int THREADS, bool ONE>
__device__ __forceinline__ void scan_tile(const ScanJob& job, uint64_t n, uint32_t* err, uint32_t overflowBit,
                                          WaitCtl ctl) {
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[THREADS / 32];
  __shared__ unsigned long long s_wide[THREADS / 32];
  __shared__ uint32_t s_prefix;
  const uint32_t* __restrict__ in = job.in;
  uint32_t* out = job.out;
  uint32_t* ticket = static_cast<uint32_t*>(job.scratch);
  unsigned long long* status = reinterpret_cast<unsigned long long*>(static_cast<char*>(job.scratch) + 256);
  const ScanTotal total = job.total;
  if (threadIdx.x == 0) s_tile = !ONE && gridDim.x > 1 ? atomicAdd(ticket, 1u) : 0u;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned long long carry = 0;  // ONE: the sum of the tiles before
  // (a tile past the end has no successors either)
  for (uint64_t base = (uint64_t)tile * (THREADS * SCAN_ITEMS); base < n; base += THREADS * SCAN_ITEMS) {
    uint32_t v[SCAN_ITEMS];
    const uint64_t i0 = base + (uint64_t)threadIdx.x * SCAN_ITEMS;
    if (i0 + SCAN_ITEMS <= n && ((reinterpret_cast<uintptr_t>(in) & 15u) == 0)) {
      const uint4* p = reinterpret_cast<const uint4*>(in + i0);
#pragma unroll
      for (int q = 0; q < SCAN_ITEMS / 4; ++q) {
        const uint4 a = p[q];
        v[4 * q] = a.x;
        v[4 * q + 1] = a.y;
        v[4 * q + 2] = a.z;
        v[4 * q + 3] = a.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < SCAN_ITEMS; ++k) v[k] = (i0 + k < n) ? in[i0 + k] : 0u;
    }
    uint32_t sum = 0;
    unsigned long long wide = 0;  // exact thread sum, for the tile aggregate
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      uint32_t t = v[k];
      v[k] = sum;
      sum += t;
      wide += t;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) wide += __shfl_down_sync(0xffffffffu, wide, d);
    // block-wide exclusive scan of the per-thread sums
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= (uint32_t)d) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    if (lane == 0) s_wide[warp] = wide;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = (lane < THREADS / 32) ? s_warp[lane] : 0u;
      uint32_t wi = w;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, wi, d);
        if (lane >= (uint32_t)d) wi += t;
      }
      if (lane < THREADS / 32) s_warp[lane] = wi - w;  // exclusive warp offsets
      unsigned long long agg = (lane < THREADS / 32) ? s_wide[lane] : 0ull;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) agg += __shfl_down_sync(0xffffffffu, agg, d);
      agg = __shfl_sync(0xffffffffu, agg, 0);
      // publish and look back (bounded waits); the 32-bit outputs wrap like the
      // reference's uint scan, the exact total flags a count past 2^32
      const unsigned long long excl =
          ONE ? carry : gridDim.x > 1 ? lb_exclusive_prefix(status, tile, agg, err, ctl) : 0ull;
      carry += agg;
      if (lane == 0) {
        s_prefix = (uint32_t)excl;
        if (overflowBit && excl + agg > 0xffffffffull) raise_error(err, overflowBit);
      }
    }
    __syncthreads();
    const uint32_t off = s_prefix + s_warp[warp] + (incl - sum);
    if (i0 + SCAN_ITEMS <= n && ((reinterpret_cast<uintptr_t>(out) & 15u) == 0)) {
      uint4* p = reinterpret_cast<uint4*>(out + i0);
#pragma unroll
      for (int q = 0; q < SCAN_ITEMS / 4; ++q)
        p[q] = make_uint4(off + v[4 * q], off + v[4 * q + 1], off + v[4 * q + 2], off + v[4 * q + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < SCAN_ITEMS; ++k)
        if (i0 + k < n) out[i0 + k] = off + v[k];
    }
    if (total.dst && i0 < n && i0 + SCAN_ITEMS >= n) {  // holds element n - 1
      uint32_t t = 0;
#pragma unroll
      for (int k = 0; k < SCAN_ITEMS; ++k)
        if (i0 + k + 1 == n) t = off + v[k];
      publish_total(total, t, err);
    }
    if (!ONE) break;
    __syncthreads();
  }
}

template <int THREADS, bool ONE>
__global__ void __launch_bounds__(THREADS)
    scan_kernel(Stamp stamp, ScanJob job, uint64_t nHost, const uint32_t* nDev, uint32_t nAdd, uint32_t* err,
                uint32_t overflowBit, WaitCtl ctl) {
  stamp_begin(stamp);
  scan_tile<THREADS, ONE>(job, nDev ? (uint64_t)(*nDev) + nAdd : nHost, err, overflowBit, ctl);
}

// two arrays of one length in one launch (blockIdx.y), each with its own tickets
template <int THREADS, bool ONE>
__global__ void __launch_bounds__(THREADS)
    scan_pair_kernel(Stamp stamp, ScanJob job0, ScanJob job1, uint64_t nHost, const uint32_t* nDev, uint32_t nAdd,
                     uint32_t* err, uint32_t overflowBit, WaitCtl ctl) {
  stamp_begin(stamp);
  scan_tile<THREADS, ONE>(blockIdx.y ? job1 : job0, nDev ? (uint64_t)(*nDev) + nAdd : nHost, err, overflowBit, ctl);
}

// the context's slots and time marks to page-locked host memory
__global__ void slots_to_host_kernel(Stamp stamp, const uint32_t* slots, uint32_t* host, uint32_t n) {
  stamp_begin(stamp);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) host[i] = slots[i];
}

}  // namespace

cudaError_t slots_to_host(const uint32_t* slots, uint32_t* host, uint32_t words, Queue& q) {
  launch(q, slots_to_host_kernel, 1, 128, 0, slots, host, words);
  return cudaGetLastError();
}

size_t scan_scratch_bytes(uint64_t maxN) {
  uint64_t tiles = (maxN + SCAN_TILE - 1) / SCAN_TILE + 1;
  return (256 + tiles * sizeof(unsigned long long) + 255) / 256 * 256;
}

cudaError_t scan_exclusive(const ScanJob* jobs, int nJobs, uint64_t n, const uint32_t* nDev, uint32_t nAdd,
                           uint64_t maxN, bool cleared, uint32_t* err, Queue& q, bool flagOverflow, WaitCtl ctl) {
  uint64_t cap = nDev ? maxN : n;
  if (cap == 0) return cudaSuccess;
  // (a test fault of the look-back needs the look-back)
  const bool one = cap <= SCAN_ONE_MAX && ctl.skipTile == WaitCtl{}.skipTile;
  const uint64_t tiles = one ? 1 : (cap + SCAN_TILE - 1) / SCAN_TILE;
  if (tiles > 1 && !cleared) {
    for (int j = 0; j < nJobs; ++j) {
      cudaError_t e = cudaMemsetAsync(jobs[j].scratch, 0, 256 + tiles * sizeof(unsigned long long), q.st);
      if (e != cudaSuccess) return e;
    }
  }
  const uint32_t overflowBit = flagOverflow ? TRAX_EBIT_OVERFLOW : 0u;
  const bool byOne = one && cap > SCAN_TILE;
  const unsigned threads = byOne ? SCAN_ONE_THREADS : SCAN_THREADS;
  if (nJobs == 1)
    launch(q, byOne ? scan_kernel<SCAN_ONE_THREADS, true> : scan_kernel<SCAN_THREADS, false>, (unsigned)tiles, threads,
           0, jobs[0], n, nDev, nAdd, err, overflowBit, ctl);
  else
    launch(q, byOne ? scan_pair_kernel<SCAN_ONE_THREADS, true> : scan_pair_kernel<SCAN_THREADS, false>,
           dim3((unsigned)tiles, 2), threads, 0, jobs[0], jobs[1], n, nDev, nAdd, err, overflowBit, ctl);
  return cudaGetLastError();
}

cudaError_t scan_exclusive(const uint32_t* in, uint32_t* out, uint64_t n, void* scratch, uint32_t* err, Queue& q,
                           bool flagOverflow, WaitCtl ctl) {
  const ScanJob job{in, out, scratch, ScanTotal{}};
  return scan_exclusive(&job, 1, n, nullptr, 0, n, false, err, q, flagOverflow, ctl);
}

}  // namespace trax

// ------------------------------------------------------------------------
// Allocation-free prefix sum for callers that cannot allocate device memory
// (see trax_prefix_sum_noalloc in include/trax/trax.h).
//
// The single-pass scan needs scratch besides its input and output: a tile
// ticket, an error word and one look-back status word per tile.  Here that
// scratch is a fixed file-scope device array, so the call itself never
// allocates.  It is sized for TRAX_NOALLOC_SCAN_MAX elements and, like any
// __device__ variable, lives on every GPU that loads this library until the
// process exits.  All calls share it: each call clears the part it uses
// before its kernel runs, and two calls whose work overlaps on the GPU (on
// different streams, or from different host threads) race on it.
#include <atomic>
#include <cstdio>

#include "trax/trax.h"

namespace {

constexpr uint64_t NOALLOC_TILES = (TRAX_NOALLOC_SCAN_MAX + trax::SCAN_TILE - 1) / trax::SCAN_TILE;
constexpr size_t NOALLOC_HEADER = 256;  // ticket at byte 0, error word at byte 4 (ScanJob::scratch)
constexpr size_t NOALLOC_BYTES = NOALLOC_HEADER + NOALLOC_TILES * sizeof(unsigned long long);

static __device__ __align__(256) unsigned char g_noalloc_scan_scratch[NOALLOC_BYTES];

// The no-alloc scan's wait settings (trax_noalloc_set_wait), process-wide.
std::atomic<uint32_t> g_noalloc_spin{0}, g_noalloc_skip{0xffffffffu};

trax::WaitCtl noalloc_wait() {
  trax::WaitCtl w;
  w.spinLimit = g_noalloc_spin.load();
  w.skipTile = g_noalloc_skip.load();
  return w;
}

void noalloc_msg(char* buf, size_t len, const char* msg) {
  if (buf && len) {
    snprintf(buf, len, "%s", msg);
  }
}

}  // namespace

extern "C" int trax_prefix_sum_noalloc(const uint32_t* d_in, uint32_t* d_out, uint64_t n, void* stream,
                                       char* err_msg, size_t err_len) {
  noalloc_msg(err_msg, err_len, "");
  if (n == 0) return TRAX_OK;
  if (!d_in || !d_out) {
    noalloc_msg(err_msg, err_len, "trax_prefix_sum_noalloc: null device pointer");
    return TRAX_ERR_ARG;
  }
  if (n > TRAX_NOALLOC_SCAN_MAX) {
    char b[160];
    snprintf(b, sizeof b, "trax_prefix_sum_noalloc: %llu elements exceed the fixed scratch limit of %llu",
             (unsigned long long)n, (unsigned long long)TRAX_NOALLOC_SCAN_MAX);
    noalloc_msg(err_msg, err_len, b);
    return TRAX_ERR_ARG;
  }
  // The array's device address, looked up on every call: an address belongs
  // to a CUDA context, not to a device, so a cached one would be wrong after
  // the caller resets the device or makes another context current.  Host code
  // may not use the symbol itself as a device pointer.  The lookup is cheap
  // next to the stream synchronisation below; the first one in a context also
  // loads this library's device code there.
  void* base = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&base, g_noalloc_scan_scratch);
  if (e != cudaSuccess || !base) {
    char b[200];
    snprintf(b, sizeof b, "trax_prefix_sum_noalloc: cudaGetSymbolAddress failed (%s)",
             e != cudaSuccess ? cudaGetErrorString(e) : "null address");
    noalloc_msg(err_msg, err_len, b);
    return TRAX_ERR_CUDA;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uint64_t tiles = (n + trax::SCAN_TILE - 1) / trax::SCAN_TILE;
  uint32_t* err = static_cast<uint32_t*>(base) + 1;  // behind the ticket
  // the ticket, the error word and the status words of this call start at zero
  e = cudaMemsetAsync(base, 0, NOALLOC_HEADER + tiles * sizeof(unsigned long long), st);
  if (e == cudaSuccess) {
    const trax::ScanJob job{d_in, d_out, base, trax::ScanTotal{}};
    trax::scan_kernel<trax::SCAN_THREADS, false><<<(unsigned)tiles, trax::SCAN_THREADS, 0, st>>>(
        trax::Stamp{}, job, n, nullptr, 0, err, 0u, noalloc_wait());
    e = cudaGetLastError();
  }
  uint32_t hostErr = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hostErr, err, sizeof(hostErr), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    noalloc_msg(err_msg, err_len, cudaGetErrorString(e));
    return TRAX_ERR_CUDA;
  }
  if (hostErr & TRAX_EBIT_TIMEOUT) {
    noalloc_msg(err_msg, err_len, "trax_prefix_sum_noalloc: a bounded look-back wait ran out");
    return TRAX_ERR_TIMEOUT;
  }
  return TRAX_OK;
}

extern "C" int trax_noalloc_set_wait(uint32_t polls, uint32_t skip_tile) {
  g_noalloc_spin.store(polls);
  g_noalloc_skip.store(skip_tile);
  return TRAX_OK;
}
