// Allocation-free BSR3 SpMV with a fused dot product: y = A x and
// dot = (y, w), on device arrays the caller already owns.
//
// Who needs this: code that runs where it must not allocate device memory --
// a solver step inside a host framework that hands out a fixed device arena
// (Flow's linear-solver backends are called between Newton steps and manage
// their own buffers), or a real-time or callback context where cudaMalloc's
// implicit synchronisation is not allowed. The handle API allocates its
// scratch at gbilu_analyze time; this entry point uses no handle and calls
// no cudaMalloc, cudaFree or allocating library routine.
//
// y is written while x and w are read, with no aliasing between them
// assumed by the compiler: y must not alias x or w. (w may alias x.)
//
// Its only scratch is the file-scope device array below: one partial sum per
// CTA plus an arrival counter for the grid-wide reduction. Every GPU that
// loads the library holds this array (about 32 KiB) until the process exits.
// A call writes one partial per CTA (4096 fit). It takes at most 1,048,576
// block rows, the documented limit of the entry point (an earlier kernel needed
// a partial per 256 rows); larger systems are rejected with GBILU_BAD_INPUT.
// Calls share the array: two calls that overlap on the GPU (different streams, or
// different host threads on one device) race on it and give wrong sums, so
// serialise them on one stream.
//
// The device address of the array is looked up once per device, on the
// first call made with that device current (cudaGetSymbolAddress); make that
// first call before any stream capture, since the lookup is not a stream
// operation. Later calls only enqueue work on the given stream. The address
// belongs to the context that was current at the lookup, the device's
// primary context when the caller uses the runtime API: calls made with
// another context current, or after a cudaDeviceReset (which destroys the
// primary context), would use a stale address, so neither is supported.
#include "gbilu.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <mutex>

namespace {

constexpr int kTileRows = 32;             // block rows per tile, one thread per unknown
constexpr int kNoAllocThreads = 3 * kTileRows;
constexpr int kTileBlocks = 256;          // blocks of a tile that fit its buffer
constexpr int kCtasPerSm = 10;            // resident tiles of 19.7 KB each
constexpr int kNoAllocMaxCtas = 4096;     // scratch holds this many partials
constexpr int kNoAllocMaxRows = 1048576;
constexpr int kMaxDevices = 64;

struct NoAllocScratch {
  double partial[kNoAllocMaxCtas];
  // high half: the newest call that used it; low half: its CTAs that arrived
  unsigned long long arrived;
};

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

struct Device {
  NoAllocScratch *scratch;
  int sm_count;
};
std::mutex g_lookup_mutex;
Device g_device[kMaxDevices] = {};
std::atomic<unsigned int> g_calls{0};

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned int)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (unsigned int)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// Component c of a block row: sum over its blocks kb .. ke-1 of the row c of
// each block times x at its column, the gathers of four blocks in flight.
__device__ __forceinline__ double row_component(const double *v, const int *ci, int kb, int ke,
                                                int c, const double *__restrict__ x) {
  double a = 0.0;
  for (int k = kb; k < ke; k += 4) {
    double xv[4][3];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < ke) {
        const double *xs = x + 3 * ci[k + u];
#pragma unroll
        for (int e = 0; e < 3; ++e) xv[u][e] = xs[e];
      }
    const double *b = v + (size_t)k * 9 + 3 * c;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < ke) {
        a = fma(b[9 * u], xv[u][0], a);
        a = fma(b[9 * u + 1], xv[u][1], a);
        a = fma(b[9 * u + 2], xv[u][2], a);
      }
  }
  return a;
}

// Sum of one double per thread, in a fixed order; valid in thread 0.
__device__ __forceinline__ double cta_sum(double d) {
  __shared__ double red[kNoAllocThreads];
  red[threadIdx.x] = d;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
    s = (red[threadIdx.x] + red[threadIdx.x + 32]) + red[threadIdx.x + 64];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  }
  __syncthreads();
  return s;
}

// y_i = sum_k A_ik x_k over the plain BSR rows; (y, w) reduced in a fixed order
// (per thread over the CTA's tiles, per CTA, then the CTAs' partials by the
// last CTA to arrive).
//
// Bound by the FP64 unit: 9 multiply-adds a block, 54 us for the 3.16 M
// blocks of the 500k-cell system against 39 us of HBM time. A tile's blocks
// are one contiguous range of vals, copied to shared memory with coalesced
// asynchronous copies (one thread per row reading its blocks directly
// touched 32 cache lines a load); one thread per unknown then adds its three
// products a block in block order, so y has the bits of a thread per row.
// Ten tiles a SM hide each other's copies, and the dot is summed over all
// tiles of a CTA before its one reduction. A tile too large for the buffer
// is read in place. 500k cells: 194 -> 87 us (a thread per row, and the
// partials added by one thread at 65 cycles each); 4,000 cells: 12.7 -> 9.2 us
// a call, without the launch that cleared the counter.
__global__ void __launch_bounds__(kNoAllocThreads, kCtasPerSm)
k_bsr_spmv_dot_noalloc(int nb, const int *__restrict__ rowptr, const int *__restrict__ colind,
                       const double *__restrict__ vals, const double *__restrict__ x,
                       double *__restrict__ y, const double *__restrict__ w, double *dot,
                       NoAllocScratch *scr, unsigned int call) {
  __shared__ double vbuf[kTileBlocks * 9];
  __shared__ int cbuf[kTileBlocks];
  __shared__ bool last;
  // counts left behind by an earlier call whose CTAs did not all arrive are
  // dropped: the first CTA of a newer call raises the word past them
  if (threadIdx.x == 0) atomicMax(&scr->arrived, (unsigned long long)call << 32);
  const int t = threadIdx.x, c = t % 3;
  double d = 0.0;
  const int tiles = (nb + kTileRows - 1) / kTileRows;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int r0 = tile * kTileRows, r1 = min(r0 + kTileRows, nb);
    const int k0 = rowptr[r0], n = rowptr[r1] - k0;
    const int row = r0 + t / 3;
    const bool act = row < r1;
    const int kb = act ? rowptr[row] : 0, ke = act ? rowptr[row + 1] : 0;
    const bool staged = n <= kTileBlocks;
    const size_t i = 3 * (size_t)r0 + t;
    double wi = 0.0;
    if (staged) {
      const double *vs = vals + (size_t)k0 * 9;
      for (int q = t; q < 9 * n; q += kNoAllocThreads) cp_async8(vbuf + q, vs + q);
      for (int q = t; q < n; q += kNoAllocThreads) cp_async4(cbuf + q, colind + k0 + q);
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    if (act) wi = w[i];
    __syncthreads();
    if (act) {
      const double a = staged ? row_component(vbuf, cbuf, kb - k0, ke - k0, c, x)
                              : row_component(vals, colind, kb, ke, c, x);
      y[i] = a;
      d = fma(a, wi, d);
    }
    __syncthreads();
  }
  d = cta_sum(d);
  if (t == 0) {
    scr->partial[blockIdx.x] = d;
    __threadfence();
    last = (unsigned int)atomicAdd(&scr->arrived, 1ull) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s = 0.0;
  for (unsigned int b = t; b < gridDim.x; b += kNoAllocThreads) s += __ldcg(&scr->partial[b]);
  s = cta_sum(s);
  if (t == 0) {
    *dot = s;
    // leave the count at zero for the next call
    atomicAnd(&scr->arrived, ~0xffffffffull);
  }
}

// Device address of the scratch array for the current device (looked up on
// the first call per device, with that device current).
cudaError_t for_current_device(Device *out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_lookup_mutex);
  if (!g_device[dev].scratch) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&g_device[dev].sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    g_device[dev].scratch = static_cast<NoAllocScratch *>(p);
  }
  *out = g_device[dev];
  return cudaSuccess;
}

}  // namespace

extern "C" int gbilu_bsr_spmv_dot_noalloc(int nb, const int *d_rowptr, const int *d_colind,
                                          const double *d_vals, const double *d_x, double *d_y,
                                          const double *d_w, double *d_dot, void *stream) {
  if (nb <= 0 || !d_rowptr || !d_colind || !d_vals || !d_x || !d_y || !d_w || !d_dot) {
    fprintf(stderr, "ERROR: gbilu_bsr_spmv_dot_noalloc: null pointer or nb <= 0\n");
    return GBILU_BAD_INPUT;
  }
  if (nb > kNoAllocMaxRows) {
    fprintf(stderr,
            "ERROR: gbilu_bsr_spmv_dot_noalloc: nb = %d exceeds the maximum of %d block rows\n",
            nb, kNoAllocMaxRows);
    return GBILU_BAD_INPUT;
  }
  Device dev = {};
  cudaError_t e = for_current_device(&dev);
  if (e != cudaSuccess) {
    fprintf(stderr, "ERROR: gbilu_bsr_spmv_dot_noalloc: cudaGetSymbolAddress: %s\n",
            cudaGetErrorString(e));
    return GBILU_CUDA_ERROR;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int tiles = (nb + kTileRows - 1) / kTileRows;
  const int grid = std::min({tiles, dev.sm_count * kCtasPerSm, kNoAllocMaxCtas});
  k_bsr_spmv_dot_noalloc<<<grid, kNoAllocThreads, 0, s>>>(
      nb, d_rowptr, d_colind, d_vals, d_x, d_y, d_w, d_dot, dev.scratch,
      g_calls.fetch_add(1, std::memory_order_relaxed) + 1);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    fprintf(stderr, "ERROR: gbilu_bsr_spmv_dot_noalloc: %s\n", cudaGetErrorString(e));
    return GBILU_CUDA_ERROR;
  }
  return GBILU_OK;
}
