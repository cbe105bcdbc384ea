// v2c_sort_static.cu -- cell assignment + stable counting sort by cell that
// allocates nothing (v2c_sort_cells_static in include/v2c.h).
//
// Same results as the context path (k_assign + the counting sort of
// v2c_sort.cu): the cell of every marker from the FP64 bisection of
// nxsearch/nysearch (interpolation.c:1536-1573), and the markers of each
// cell in ascending array index.  The difference is where the scratch lives.
// The context path keeps per-cell counters and per-marker slot/rank buffers
// in memory it allocates at v2c_create; this variant keeps its only scratch,
// the per-cell counters and the scan's block sums, in the file-scope array
// g_scratch below, and orders each cell's segment of the caller's perm in
// place, so it needs no per-marker scratch at all.
//
// g_scratch is one array per device (module-scope __device__ storage).
// Calls that overlap on one device -- two streams, two host threads, or a
// call on one stream while another is still running on another -- race on
// it and produce wrong counts; calls must be ordered (one stream, or events).
#include <climits>
#include <cstdio>
#include <mutex>

#include "v2c_internal.cuh"

namespace v2c {

namespace {

constexpr int SB = 1024, SE = 4;  // scan: 1024 threads x 4 counters per block
constexpr long MAX_CELLS = V2C_STATIC_SORT_MAX_CELLS;
constexpr long MAX_BLOCKS = (MAX_CELLS + SB * SE - 1) / (SB * SE);
constexpr long SCRATCH_WORDS = MAX_CELLS + MAX_BLOCKS;  // counters, then block sums

// 4 Mi counters + 1 Ki block sums = 16 MiB + 4 KiB per device.  The counters
// must be zero before the counting pass; every call zeroes them itself on its
// stream, so nothing has to be zero on entry.
static __device__ __align__(256) int32_t g_scratch[SCRATCH_WORDS];

constexpr int MAX_DEVICES = 64;
std::mutex g_setup_mu;
int32_t *g_scratch_ptr[MAX_DEVICES] = {};

// Line search among the upper words of the lines in shared memory, for an x
// without a sign bit: the largest line whose upper word does not exceed x's.
__device__ __forceinline__ int search_upper(const int32_t *upper, const double *g, int n,
                                            double x) {
  const long long xb = __double_as_longlong(x);
  const int32_t xh = (int32_t)(xb >> 32);
  int lo = 0;
  for (int len = n - 1; len > 1;) {  // the line sought is one of lo .. lo + len - 1
    const int half = len >> 1;
    if (upper[lo + half] <= xh) lo += half;
    len -= half;
  }
  if (upper[lo] != xh || __ldg(reinterpret_cast<const long long *>(g) + lo) <= xb) return lo;
  // that line shares x's upper word and lies above it: the one before, unless
  // it shares the word too (lines closer than 2^-20 of the coordinate)
  if (lo == 0 || upper[lo - 1] != xh) return lo > 0 ? lo - 1 : 0;
  return nsearch_bits(g, n, x);
}

// Cells and the markers' slots in them (whatever the atomics give).  The slot
// rides in the upper ten bits of the cell (fewer than 2^22 cells) to k_fill,
// which then needs no atomics; SLOT_LATE stands for that and all above.
// AM markers per thread; LINES: the grid's upper words fit in shared memory.
// 9 M markers on 1501 x 401 lines: 341 us with FP64 comparisons, 97 with
// 64-bit integer ones, 79 so, slots included, and k_fill, which
// waited for its atomics, 57 -> 36.
static_assert(MAX_CELLS <= 1l << 22, "cells and slots share a word");
constexpr int SLOT_SHIFT = 22, SLOT_LATE = 1023;
constexpr int AM = 4;
constexpr int MAX_LINES = 6144;
template <bool LINES>
__global__ void __launch_bounds__(256) k_assign_count(const double *gx, int xn, const double *gy,
                                                      int yn, const double *x, const double *y,
                                                      long n, int32_t *cell, int32_t *count) {
  after_previous();
  extern __shared__ int32_t upper[];
  if (LINES) {
    for (int k = threadIdx.x; k < xn + yn; k += 256)
      upper[k] = __double2hiint(k < xn ? gx[k] : gy[k - xn]);
    __syncthreads();
  }
  const long i0 = blockIdx.x * (256l * AM) + threadIdx.x;
  double xi[AM], yi[AM];
#pragma unroll
  for (int k = 0; k < AM; k++) {
    const bool in = i0 + 256 * k < n;
    xi[k] = in ? x[i0 + 256 * k] : 0.0;
    yi[k] = in ? y[i0 + 256 * k] : 0.0;
  }
  int c[AM];
#pragma unroll
  for (int k = 0; k < AM; k++) {
    int ix, iy;
    if (LINES && (__double2hiint(xi[k]) | __double2hiint(yi[k])) >= 0) {
      ix = search_upper(upper, gx, xn, xi[k]);
      iy = search_upper(upper + xn, gy, yn, yi[k]);
    } else {
      ix = nsearch_bits(gx, xn, xi[k]);
      iy = nsearch_bits(gy, yn, yi[k]);
    }
    c[k] = ix * (yn - 1) + iy;
  }
#pragma unroll
  for (int k = 0; k < AM; k++)
    if (i0 + 256 * k < n) {
      const int slot = atomicAdd(count + c[k], 1);
      cell[i0 + 256 * k] =
          (int32_t)((uint32_t)c[k] | (uint32_t)min(slot, SLOT_LATE) << SLOT_SHIFT);
    }
}

__global__ void k_scan_block_s(const int32_t *in, long m, int32_t *out, int32_t *bsum) {
  after_previous();
  __shared__ int32_t sh[SB];
  const long base = (long)blockIdx.x * SB * SE + (long)threadIdx.x * SE;
  int32_t v[SE], s = 0;
#pragma unroll
  for (int k = 0; k < SE; k++) {
    v[k] = (base + k < m) ? in[base + k] : 0;
    s += v[k];
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int off = 1; off < SB; off <<= 1) {
    const int32_t t = (threadIdx.x >= off) ? sh[threadIdx.x - off] : 0;
    __syncthreads();
    sh[threadIdx.x] += t;
    __syncthreads();
  }
  int32_t run = sh[threadIdx.x] - s;
#pragma unroll
  for (int k = 0; k < SE; k++) {
    if (base + k < m) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == SB - 1) bsum[blockIdx.x] = sh[SB - 1];
}

// exclusive scan of at most SB block sums in one block; the total goes to
// *total (start[ncell])
__global__ void k_scan_sums_s(int32_t *bsum, int nb, int32_t *total) {
  after_previous();
  __shared__ int32_t sh[SB];
  const int32_t v = (threadIdx.x < nb) ? bsum[threadIdx.x] : 0;
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int off = 1; off < SB; off <<= 1) {
    const int32_t t = (threadIdx.x >= off) ? sh[threadIdx.x - off] : 0;
    __syncthreads();
    sh[threadIdx.x] += t;
    __syncthreads();
  }
  if (threadIdx.x < nb) bsum[threadIdx.x] = sh[threadIdx.x] - v;
  if (threadIdx.x == SB - 1) *total = sh[SB - 1];
}

__global__ void k_scan_add_s(int32_t *out, long m, const int32_t *bsum) {
  after_previous();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < m) out[i] += bsum[i / (SB * SE)];
}

// Every marker goes to its slot of its cell's segment (k_order_cells makes
// slot order index order), the late ones to what they count the counter down
// to, and the cells are left without the slots.
constexpr int FM = 4;
__global__ void __launch_bounds__(256) k_fill(int32_t *cell, long n, const int32_t *start,
                                              int32_t *count, int32_t *perm) {
  after_previous();
  const long i0 = blockIdx.x * (256l * FM) + threadIdx.x;
  uint32_t w[FM];
  int at[FM];
#pragma unroll
  for (int k = 0; k < FM; k++) w[k] = i0 + 256 * k < n ? (uint32_t)cell[i0 + 256 * k] : 0u;
#pragma unroll
  for (int k = 0; k < FM; k++) {
    const int c = (int)(w[k] & ((1u << SLOT_SHIFT) - 1)), slot = (int)(w[k] >> SLOT_SHIFT);
    at[k] = __ldg(start + c) + slot;
    if (i0 + 256 * k < n) {
      if (slot == SLOT_LATE) at[k] += atomicSub(count + c, 1) - 1 - SLOT_LATE;
      cell[i0 + 256 * k] = c;
    }
  }
#pragma unroll
  for (int k = 0; k < FM; k++)
    if (i0 + 256 * k < n) perm[at[k]] = (int32_t)(i0 + 256 * k);
}

// ascending over the warp's lanes (W = 32) or each of its halves (W = 16)
template <int W>
__device__ __forceinline__ int32_t bitonic(int32_t key, int lane) {
#pragma unroll
  for (int k = 2; k <= W; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const int32_t other = __shfl_xor_sync(V2C_FULL, key, j);
      const bool keep_min = ((lane & j) == 0) == ((lane & k & (W - 1)) == 0);
      key = keep_min ? min(key, other) : max(key, other);
    }
  return key;
}

// A segment of L > 32 entries: a bitonic network in the form whose every
// compare puts the smaller value at the lower position (first stage of each
// merge compares a with its mirror in the block), so positions past the
// segment act as +infinity and are never touched.  Every position is in one
// pair per stage; __syncwarp() orders the stages' global-memory accesses
// among the warp's lanes.
__device__ __noinline__ void order_large(int32_t *p, int L, int lane) {
  int P = 64;
  while (P < L) P <<= 1;
  for (int k = 2; k <= P; k <<= 1) {
    const int h = k >> 1;
    for (int i = lane; i < P / 2; i += 32) {
      const int blk = i / h, off = i - blk * h;
      const int a = blk * k + off, b = blk * k + k - 1 - off;
      if (b < L) {
        const int32_t va = p[a], vb = p[b];
        if (va > vb) { p[a] = vb; p[b] = va; }
      }
    }
    __syncwarp();
    for (int j = k >> 2; j >= 1; j >>= 1) {
      for (int i = lane; i < P / 2; i += 32) {
        const int blk = i / j, off = i - blk * j;
        const int a = blk * 2 * j + off, b = a + j;
        if (b < L) {
          const int32_t va = p[a], vb = p[b];
          if (va > vb) { p[a] = vb; p[b] = va; }
        }
      }
      __syncwarp();
    }
  }
}

// One warp per OG consecutive cells sorts each cell's segment of perm
// ascending, in place.  The cells' starts come in one read and all their
// entries, one run of perm, in the next (two rounds of memory latency per
// warp, full lines); the entries wait in shared memory, so that the sorting
// code is one loop, which takes two cells at a time, half a warp each, where
// both have at most 16 markers, and go back the way they came.  600 000 cells
// of 15 markers: 144 us with a warp per cell, 79 with a read and a write per
// cell, 72 so.
constexpr int OG = 8;
__global__ void __launch_bounds__(256) k_order_cells(const int32_t *start, long ncell,
                                                     int32_t *perm) {
  after_previous();
  __shared__ int32_t keys[8][OG * 32];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long c0 = (blockIdx.x * 8l + wl) * OG;
  if (c0 >= ncell) return;  // uniform across the warp
  const int ng = (int)min((long)OG, ncell - c0);
  // (lanes past the last cell repeat its end: empty cells)
  const int sv = start[c0 + min(lane, ng)];
  const int s0 = __shfl_sync(V2C_FULL, sv, 0), total = __shfl_sync(V2C_FULL, sv, OG) - s0;
  const int len = __shfl_down_sync(V2C_FULL, sv, 1) - sv;
  if (__any_sync(V2C_FULL, lane < OG && len > 32)) {
#pragma unroll 1
    for (int g = 0; g < ng; g++) {
      const int s = __shfl_sync(V2C_FULL, sv, g), L = __shfl_sync(V2C_FULL, sv, g + 1) - s;
      if (L > 32) {
        order_large(perm + s, L, lane);
      } else if (L > 1) {
        const int32_t key = bitonic<32>(lane < L ? perm[s + lane] : INT_MAX, lane);
        if (lane < L) perm[s + lane] = key;
      }
    }
    return;
  }
  int32_t *buf = keys[wl];
  int32_t val[OG];
#pragma unroll
  for (int k = 0; k < OG; k++) val[k] = k * 32 + lane < total ? perm[s0 + k * 32 + lane] : 0;
#pragma unroll
  for (int k = 0; k < OG; k++) buf[k * 32 + lane] = val[k];
  __syncwarp();
#pragma unroll 1
  for (int g = 0; g < ng; g += 2) {
    const int o0 = __shfl_sync(V2C_FULL, sv, g) - s0, o1 = __shfl_sync(V2C_FULL, sv, g + 1) - s0;
    const int L0 = o1 - o0, L1 = __shfl_sync(V2C_FULL, sv, g + 2) - s0 - o1;
    if (L0 <= 16 && L1 <= 16) {
      const int half = lane >> 4, l = lane & 15, at = (half ? o1 : o0) + l;
      const bool in = l < (half ? L1 : L0);
      const int32_t key = bitonic<16>(in ? buf[at] : INT_MAX, lane);
      if (in) buf[at] = key;
      continue;
    }
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      const int at = (h ? o1 : o0) + lane;
      const bool in = lane < (h ? L1 : L0);
      const int32_t key = bitonic<32>(in ? buf[at] : INT_MAX, lane);
      if (in) buf[at] = key;
    }
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < OG; k++)
    if (k * 32 + lane < total) perm[s0 + k * 32 + lane] = buf[k * 32 + lane];
}

inline unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

// Set-up, once per device, with that device current: the device address of
// g_scratch.  This may load the module on the device, so a caller that
// captures streams makes its first call on each device before capturing.
int scratch_for_current_device(int32_t **out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return V2C_ERR_CUDA;
  if (dev < 0 || dev >= MAX_DEVICES) return V2C_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_setup_mu);
  if (!g_scratch_ptr[dev]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);
    if (e != cudaSuccess || !p) {
      fprintf(stderr, "v2c_sort_cells_static: cudaGetSymbolAddress failed on device %d: %s\n",
              dev, cudaGetErrorString(e));
      return V2C_ERR_CUDA;
    }
    g_scratch_ptr[dev] = static_cast<int32_t *>(p);
  }
  *out = g_scratch_ptr[dev];
  return V2C_OK;
}

}  // namespace

}  // namespace v2c

using namespace v2c;

extern "C" int v2c_sort_cells_static(const double *gx_dev, long xnumx, const double *gy_dev,
                                     long ynumy, const double *x_dev, const double *y_dev,
                                     long n, int32_t *cell_dev, int32_t *perm_dev,
                                     int32_t *start_dev, void *cuda_stream) {
  // sizes first: nothing below the limits reaches the device.  Each factor
  // is bounded before the product is formed, so no size overflows `long` or
  // the int the kernels take.
  if (xnumx < 2 || ynumy < 2 || n < 0 || n > INT_MAX) return V2C_ERR_ARG;
  if (xnumx - 1 > MAX_CELLS || ynumy - 1 > MAX_CELLS / (xnumx - 1)) {
    fprintf(stderr,
            "v2c_sort_cells_static: %ld x %ld grid lines give more than the %ld cells "
            "(V2C_STATIC_SORT_MAX_CELLS) its fixed scratch holds; use the context path\n",
            xnumx, ynumy, MAX_CELLS);
    return V2C_ERR_CAPACITY;
  }
  const long ncell = (xnumx - 1) * (ynumy - 1);
  if (!gx_dev || !gy_dev || !start_dev || (n > 0 && (!x_dev || !y_dev || !cell_dev || !perm_dev)))
    return V2C_ERR_ARG;
  // An error another caller left pending would be reported as this call's
  // own by the checks after each launch below: refuse to start instead, and
  // leave that error in place for its owner.
  if (cudaPeekAtLastError() != cudaSuccess) {
    fprintf(stderr, "v2c_sort_cells_static: an earlier CUDA error is pending (%s); not started\n",
            cudaGetErrorString(cudaPeekAtLastError()));
    return V2C_ERR_CUDA;
  }
  int32_t *scratch = nullptr;
  if (int rc = scratch_for_current_device(&scratch)) return rc;
  int32_t *count = scratch, *bsum = scratch + MAX_CELLS;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  // status of the launch just queued (nothing was pending on entry)
  auto launched = []() { return cudaGetLastError() == cudaSuccess; };

  if (cudaMemsetAsync(count, 0, sizeof(int32_t) * ncell, st) != cudaSuccess) return V2C_ERR_CUDA;
  if (n > 0) {
    const bool lines = xnumx + ynumy <= MAX_LINES;
    launch_after(lines ? k_assign_count<true> : k_assign_count<false>, nblk(n, 256 * AM), 256,
                 lines ? sizeof(int32_t) * (xnumx + ynumy) : 0, st, gx_dev, (int)xnumx, gy_dev,
                 (int)ynumy, x_dev, y_dev, n, cell_dev, count);
    if (!launched()) return V2C_ERR_CUDA;
  }
  const long nb = (ncell + SB * SE - 1) / (SB * SE);
  launch_after(k_scan_block_s, (unsigned)nb, SB, 0, st, count, ncell, start_dev, bsum);
  if (!launched()) return V2C_ERR_CUDA;
  launch_after(k_scan_sums_s, 1, SB, 0, st, bsum, (int)nb, start_dev + ncell);
  if (!launched()) return V2C_ERR_CUDA;
  launch_after(k_scan_add_s, nblk(ncell, 256), 256, 0, st, start_dev, ncell, bsum);
  if (!launched()) return V2C_ERR_CUDA;
  if (n > 0) {
    launch_after(k_fill, nblk(n, 256 * FM), 256, 0, st, cell_dev, n, start_dev, count, perm_dev);
    if (!launched()) return V2C_ERR_CUDA;
    launch_after(k_order_cells, nblk(ncell, 8 * OG), 256, 0, st, start_dev, ncell, perm_dev);
    if (!launched()) return V2C_ERR_CUDA;
  }
  return V2C_OK;
}
