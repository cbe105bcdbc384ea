// v2c_sort.cu -- cell assignment and the counting sort by cell.
//
// Cell assignment (upload) bisects the FP64 grid lines exactly like
// nxsearch/nysearch (interpolation.c:1536-1573), so the integer cell of
// every marker is bit-identical to the reference's.  The counting sort
// orders by cell, within a cell by quarter class q = 2 (v > 1/2) + (u > 1/2)
// and within a class by array index: counts by integer atomics
// (order-independent), exclusive scan, scatter of (q, index) keys into
// per-cell slots, then each cell's keys are ranked, which fixes the order
// whatever order the atomics handed the slots out in.  The sweeps that
// scatter to nodes read each quarter class as one contiguous run.
#include <climits>

#include "v2c_kernels.h"

namespace v2c {

namespace {

__global__ void k_assign(Grid g, const double *x, const double *y, long n, Markers m) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double xi = x[i], yi = y[i];
  int ix = nsearch_bits(g.gx, g.xn, xi), iy = nsearch_bits(g.gy, g.yn, yi);
  double u = (xi - g.gx[ix]) / (g.gx[ix + 1] - g.gx[ix]);
  double v = (yi - g.gy[iy]) / (g.gy[iy + 1] - g.gy[iy]);
  m.cell_in[i] = ix * g.ncy + iy;
  m.u_in[i] = offset32(u);
  m.v_in[i] = offset32(v);
  m.id[i] = (int32_t)i;
}

// Markers of one cell are mostly adjacent in memory, so the lanes of a warp
// share few cells: one atomic per distinct cell in the warp (the leader adds
// the group's size), each lane's slot is the group's base plus its rank
// among the group's lanes.
// Each warp takes MK groups of 32 markers, so that MK cell reads and then MK
// atomics are in flight together (the kernel is their latency; C4: 334 ->
// 152 us).
constexpr int MK = 4;
__global__ void __launch_bounds__(256) k_count(const int32_t *cell, long n, int32_t *counts,
                                               int32_t *slot) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const long i0 = (blockIdx.x * 8l + (threadIdx.x >> 5)) * (32 * MK) + lane;
  int c[MK], base[MK];
  unsigned grp[MK];
#pragma unroll
  for (int k = 0; k < MK; k++) c[k] = i0 + 32 * k < n ? cell[i0 + 32 * k] : -1;
#pragma unroll
  for (int k = 0; k < MK; k++) {
    grp[k] = __match_any_sync(V2C_FULL, c[k]);
    base[k] = 0;
    if (c[k] >= 0 && lane == __ffs(grp[k]) - 1) base[k] = atomicAdd(counts + c[k], __popc(grp[k]));
  }
#pragma unroll
  for (int k = 0; k < MK; k++) {
    const int b = __shfl_sync(V2C_FULL, base[k], __ffs(grp[k]) - 1);
    if (c[k] >= 0) slot[i0 + 32 * k] = b + __popc(grp[k] & ((1u << lane) - 1));
  }
}

// Exclusive scan in two launches.  First each block scans its SB * SE
// elements (4 per thread) and leaves their sum; CLEAR also zeroes the input,
// so that the sort's counters are zero again for its next call.
constexpr int SB = 1024, SE = 4;

// inclusive scan of one value per thread over the block
__device__ __forceinline__ int32_t block_scan(int32_t v, int32_t *warp_sum) {
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t t = __shfl_up_sync(V2C_FULL, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) warp_sum[wl] = v;
  __syncthreads();
  if (wl == 0) {
    int32_t w = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(V2C_FULL, w, o);
      if (lane >= o) w += t;
    }
    warp_sum[lane] = w;
  }
  __syncthreads();
  return v + (wl > 0 ? warp_sum[wl - 1] : 0);
}

template <bool CLEAR>
__global__ void __launch_bounds__(SB) k_scan_block(int32_t *in, long m, int32_t *out,
                                                   int32_t *bsum) {
  after_previous();
  __shared__ int32_t ws[32];
  const long base = (long)blockIdx.x * SB * SE + (long)threadIdx.x * SE;
  int32_t v[SE], s = 0;
#pragma unroll
  for (int k = 0; k < SE; k++) {
    v[k] = (base + k < m) ? in[base + k] : 0;
    s += v[k];
  }
  const int32_t incl = block_scan(s, ws);
  int32_t run = incl - s;
#pragma unroll
  for (int k = 0; k < SE; k++) {
    if (base + k < m) {
      out[base + k] = run;
      if (CLEAR) in[base + k] = 0;
    }
    run += v[k];
  }
  if (threadIdx.x == SB - 1) bsum[blockIdx.x] = incl;
}

// Then each block adds the sum of the blocks before its own (each sums them
// for itself: at most a thousand or so), and the last leaves the total.
__global__ void __launch_bounds__(SB) k_scan_add(int32_t *out, long m, const int32_t *bsum,
                                                 int nb) {
  after_previous();
  __shared__ int32_t ws[32];
  int32_t s = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += SB) s += bsum[i];
  block_scan(s, ws);
  const int32_t before = ws[31];
  const long base = (long)blockIdx.x * SB * SE;
  if (before)
    for (long i = base + threadIdx.x; i < min(base + SB * SE, m); i += SB) out[i] += before;
  if (blockIdx.x == nb - 1 && threadIdx.x == 0) out[m] = before + bsum[nb - 1];
}

// key of marker i: quarter class in bits 30-31, array index below
__global__ void __launch_bounds__(256) k_slots(const int32_t *cell, const float *u, const float *v,
                                               long n, const int32_t *start, const int32_t *slot,
                                               uint32_t *tmp) {
  after_previous();
  const long i0 = blockIdx.x * (256l * MK) + threadIdx.x;
  int c[MK], at[MK];
  uint32_t q[MK];
#pragma unroll
  for (int k = 0; k < MK; k++) {
    const long i = i0 + 256 * k;
    c[k] = i < n ? cell[i] : -1;
    if (c[k] >= 0) {
      at[k] = slot[i];
      q[k] = (v[i] > 0.5f ? 2u : 0u) + (u[i] > 0.5f ? 1u : 0u);
    }
  }
#pragma unroll
  for (int k = 0; k < MK; k++)
    if (c[k] >= 0) tmp[__ldg(start + c[k]) + at[k]] = (q[k] << 30) | (uint32_t)(i0 + 256 * k);
}

constexpr uint32_t KEY_INDEX = (1u << 30) - 1;

// One warp orders the L <= 32 distinct keys of a cell's slots, held one per
// lane in val (lanes >= L hold 0xffffffff, which sorts last: array indices
// stay below 2^30 - 1, so no key equals it), writes their indices in
// ascending key order and returns the counts of quarter classes 0, 1, 2
// (same value in every lane).  The bitonic network is skipped when the
// keys are in order already: a cell whose markers one warp of the count
// pass met keeps their slots in array order, and array order is class
// order for markers that have kept their cell and class since the markers
// were last stored in sorted order.
__device__ __forceinline__ int4 rank_small(uint32_t val, int32_t *perm, int L, int lane) {
  uint32_t key = val;
  const uint32_t next = __shfl_down_sync(V2C_FULL, val, 1);
  if (!__all_sync(V2C_FULL, lane >= L - 1 || val < next)) {
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const uint32_t other = __shfl_xor_sync(V2C_FULL, key, j);
        const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
        key = keep_min ? min(key, other) : max(key, other);
      }
  }
  const bool in = lane < L;
  const uint32_t q = key >> 30;
  int4 cnt;
  cnt.x = __popc(__ballot_sync(V2C_FULL, in && q == 0));
  cnt.y = __popc(__ballot_sync(V2C_FULL, in && q == 1));
  cnt.z = __popc(__ballot_sync(V2C_FULL, in && q == 2));
  cnt.w = 0;
  if (in) perm[lane] = (int32_t)(key & KEY_INDEX);
  return cnt;
}

// The same for a cell of L > 32 keys (read from tmp): each key's rank is
// the number of the cell's keys below it.
__device__ __noinline__ int4 rank_large(const uint32_t *tmp, int32_t *perm, int L, int lane) {
  int4 cnt = make_int4(0, 0, 0, 0);
  for (int b = 0; b < L; b += 32) {
    const int jj = b + lane;
    const uint32_t val = (jj < L) ? tmp[jj] : 0xffffffffu;
    int rank = 0;
    for (int b2 = 0; b2 < L; b2 += 32) {
      const uint32_t other = (b2 + lane < L) ? tmp[b2 + lane] : 0xffffffffu;
#pragma unroll 8
      for (int k = 0; k < 32; k++) rank += (__shfl_sync(V2C_FULL, other, k) < val);
    }
    const bool in = jj < L;
    const uint32_t q = val >> 30;
    cnt.x += __popc(__ballot_sync(V2C_FULL, in && q == 0));
    cnt.y += __popc(__ballot_sync(V2C_FULL, in && q == 1));
    cnt.z += __popc(__ballot_sync(V2C_FULL, in && q == 2));
    if (in) perm[rank] = (int32_t)(val & KEY_INDEX);
  }
  return cnt;
}

// One warp per RG consecutive cells: their starts in one read, then all
// their keys (two rounds of memory latency per warp; the keys wait in shared
// memory, so that the ranking code stays one loop), their quarter class
// starts written together; the largest cell count goes to the status counter
// once per block.  C4: 604 -> 337 us against one cell's keys read ahead.
constexpr int RG = 8;
__global__ void __launch_bounds__(256) k_rank(const int32_t *start, long ncell,
                                              const uint32_t *tmp, int32_t *perm, int4 *qstart,
                                              unsigned long long *stat) {
  after_previous();
  __shared__ int bmax;
  __shared__ uint32_t keys[8][RG][32];
  if (threadIdx.x == 0) bmax = 0;
  __syncthreads();
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long c0 = (blockIdx.x * 8l + wl) * RG;
  if (c0 < ncell) {
    const int ng = (int)min((long)RG, ncell - c0);
    // starts of the group's cells, and the last one's end
    const int sv = start[c0 + min(lane, ng)];
    uint32_t val[RG];
#pragma unroll
    for (int g = 0; g < RG; g++) {
      const int s = __shfl_sync(V2C_FULL, sv, g), L = __shfl_sync(V2C_FULL, sv, g + 1) - s;
      val[g] = (g < ng && lane < L && L <= 32) ? tmp[s + lane] : 0xffffffffu;
    }
#pragma unroll
    for (int g = 0; g < RG; g++) keys[wl][g][lane] = val[g];
    int4 myq = make_int4(0, 0, 0, 0);
    int lmax = 0;
#pragma unroll 1
    for (int g = 0; g < ng; g++) {
      const int s = __shfl_sync(V2C_FULL, sv, g), L = __shfl_sync(V2C_FULL, sv, g + 1) - s;
      lmax = max(lmax, L);
      int4 cnt = make_int4(0, 0, 0, 0);
      if (L > 32) cnt = rank_large(tmp + s, perm + s, L, lane);
      else if (L > 0) cnt = rank_small(keys[wl][g][lane], perm + s, L, lane);
      if (lane == g)
        myq = make_int4(s, s + cnt.x, s + cnt.x + cnt.y, s + cnt.x + cnt.y + cnt.z);
    }
    if (lane < ng) qstart[c0 + lane] = myq;
    if (lane == 0) {
      if (lmax > 0) atomicMax(&bmax, lmax);
      if (c0 + ng == ncell) {
        const int e = start[ncell];
        qstart[ncell] = make_int4(e, e, e, e);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && bmax > 0) atomicMax(stat + ST_MAX_CELL, (unsigned long long)bmax);
}

__global__ void k_f64_to_f32(const double *src, float *dst, long n) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (float)src[i];
}
// FP64 -> float pair hi + lo (hi the nearest float, lo the nearest float to
// the remainder)
__global__ void k_f64_to_pair(const double *src, float *hi, float *lo, long n) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) {
    const double d = src[i];
    const float h = (float)d;
    hi[i] = h;
    lo[i] = (float)(d - (double)h);
  }
}
__global__ void k_unperm_pair(const float *hi, const float *lo, const int32_t *id, double *out,
                              long n) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[id[i]] = (double)hi[i] + (double)lo[i];
}
template <class T>
__global__ void k_gather(const T *src, const int32_t *perm, T *dst, long n) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[perm[i]];
}
__global__ void k_unperm_f32(const float *src, const int32_t *id, double *out, long n) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[id[i]] = (double)src[i];
}
template <class T>
__global__ void k_unperm(const T *src, const int32_t *id, T *out, long n) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[id[i]] = src[i];
}
__global__ void k_positions(Grid g, Markers m, long n, double *x, double *y) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c = m.cell_in[i];
  int ix = c / g.ncy, iy = c - ix * g.ncy;
  int k = m.id[i];
  x[k] = g.gx[ix] + (double)m.u_in[i] * (g.gx[ix + 1] - g.gx[ix]);
  y[k] = g.gy[iy] + (double)m.v_in[i] * (g.gy[iy + 1] - g.gy[iy]);
}

// where each marker of the host's numbering lies (-1: nowhere)
__global__ void k_marker_inverse(const int32_t *id, long n, int32_t *inv) {
  after_previous();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) inv[id[i]] = (int32_t)i;
}
// One row of blocks per field, in the host's order: the device's reads are
// gathered (from L2), the host's arrays written in full lines over the link.
__global__ void __launch_bounds__(256) k_markers_to_host(Grid g, Markers m, long n,
                                                         const __grid_constant__ MarkerFields F,
                                                         const int32_t *inv) {
  after_previous();
  const int f = blockIdx.y, kind = F.kind[f];
  const float *src = F.src[f], *lo = F.lo[f];
  double *dst = F.dst[f];
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
    const int i = inv[k];
    if (i < 0) continue;
    if (kind == MARKER_F32) {
      dst[k] = (double)src[i];
    } else if (kind == MARKER_PAIR) {
      dst[k] = (double)src[i] + (double)lo[i];
    } else {
      int ix, iy;
      g.cell_at(m.cell_in[i], ix, iy);
      dst[k] = kind == MARKER_X ? g.gx[ix] + (double)m.u_in[i] * (g.gx[ix + 1] - g.gx[ix])
                                : g.gy[iy] + (double)m.v_in[i] * (g.gy[iy + 1] - g.gy[iy]);
    }
  }
}

inline unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void launch_assign(const Grid &g, const double *x, const double *y, long n, Markers m,
                   unsigned long long *stat, cudaStream_t st) {
  (void)stat;
  if (n > 0) k_assign<<<nblk(n, 256), 256, 0, st>>>(g, x, y, n, m);
}

long scan_blocks(long m) { return (m + SB * SE - 1) / (SB * SE); }

namespace {
// exclusive scan of in[0, m), m > 0
template <bool CLEAR>
void scan(int32_t *in, long m, int32_t *out, int32_t *blocksum, cudaStream_t st) {
  const int nb = (int)scan_blocks(m);
  launch_after(k_scan_block<CLEAR>, nb, SB, 0, st, in, m, out, blocksum);
  launch_after(k_scan_add, nb, SB, 0, st, out, m, blocksum, nb);
}
}  // namespace

void launch_scan(const int32_t *in, long m, int32_t *out, int32_t *blocksum, cudaStream_t st) {
  if (m > 0) scan<false>(const_cast<int32_t *>(in), m, out, blocksum, st);
  else cudaMemsetAsync(out, 0, sizeof(int32_t), st);
}

void launch_sort(const int32_t *cell, const float *u, const float *v, long n, long ncell,
                 SortBufs &b, unsigned long long *stat, cudaStream_t st) {
  if (n > 0) launch_after(k_count, nblk(n, 256 * MK), 256, 0, st, cell, n, b.counts, b.slot);
  scan<true>(b.counts, ncell, b.start, b.blocksum, st);
  uint32_t *keys = reinterpret_cast<uint32_t *>(b.tmp);
  if (n > 0) launch_after(k_slots, nblk(n, 256 * MK), 256, 0, st, cell, u, v, n, b.start, b.slot,
                          keys);
  launch_after(k_rank, nblk((ncell + RG - 1) / RG * 32, 256), 256, 0, st, b.start, ncell, keys,
               b.perm, b.qstart, stat);
}

void launch_f64_to_f32(const double *src, float *dst, long n, cudaStream_t st) {
  if (n > 0) k_f64_to_f32<<<nblk(n, 256), 256, 0, st>>>(src, dst, n);
}
void launch_f64_to_pair(const double *src, float *hi, float *lo, long n, cudaStream_t st) {
  if (n > 0) k_f64_to_pair<<<nblk(n, 256), 256, 0, st>>>(src, hi, lo, n);
}
void launch_unpermute_pair(const float *hi, const float *lo, const int32_t *id, double *out,
                           long n, cudaStream_t st) {
  if (n > 0) k_unperm_pair<<<nblk(n, 256), 256, 0, st>>>(hi, lo, id, out, n);
}
void launch_gather_f32(const float *src, const int32_t *perm, float *dst, long n, cudaStream_t st) {
  if (n > 0) k_gather<float><<<nblk(n, 256), 256, 0, st>>>(src, perm, dst, n);
}
void launch_gather_i32(const int32_t *src, const int32_t *perm, int32_t *dst, long n, cudaStream_t st) {
  if (n > 0) k_gather<int32_t><<<nblk(n, 256), 256, 0, st>>>(src, perm, dst, n);
}
void launch_gather_i8(const int8_t *src, const int32_t *perm, int8_t *dst, long n, cudaStream_t st) {
  if (n > 0) k_gather<int8_t><<<nblk(n, 256), 256, 0, st>>>(src, perm, dst, n);
}
void launch_gather_u8(const uint8_t *src, const int32_t *perm, uint8_t *dst, long n, cudaStream_t st) {
  if (n > 0) k_gather<uint8_t><<<nblk(n, 256), 256, 0, st>>>(src, perm, dst, n);
}
void launch_unpermute_f32(const float *src, const int32_t *id, double *out, long n, cudaStream_t st) {
  if (n > 0) k_unperm_f32<<<nblk(n, 256), 256, 0, st>>>(src, id, out, n);
}
void launch_unpermute_f64(const double *src, const int32_t *id, double *out, long n, cudaStream_t st) {
  if (n > 0) k_unperm<double><<<nblk(n, 256), 256, 0, st>>>(src, id, out, n);
}
void launch_unpermute_i32(const int32_t *src, const int32_t *id, int32_t *out, long n, cudaStream_t st) {
  if (n > 0) k_unperm<int32_t><<<nblk(n, 256), 256, 0, st>>>(src, id, out, n);
}
void launch_unpermute_u8(const uint8_t *src, const int32_t *id, uint8_t *out, long n, cudaStream_t st) {
  if (n > 0) k_unperm<uint8_t><<<nblk(n, 256), 256, 0, st>>>(src, id, out, n);
}
void launch_unpermute_i8(const int8_t *src, const int32_t *id, int8_t *out, long n, cudaStream_t st) {
  if (n > 0) k_unperm<int8_t><<<nblk(n, 256), 256, 0, st>>>(src, id, out, n);
}
void launch_positions(const Grid &g, const Markers &m, long n, double *x, double *y,
                      cudaStream_t st) {
  if (n > 0) k_positions<<<nblk(n, 256), 256, 0, st>>>(g, m, n, x, y);
}

void launch_markers_to_host(const Grid &g, const Markers &m, long n, const MarkerFields &f,
                            int32_t *inv, cudaStream_t st) {
  if (n <= 0 || f.n <= 0) return;
  cudaMemsetAsync(inv, 0xff, sizeof(int32_t) * n, st);
  launch_after(k_marker_inverse, nblk(n, 256), 256, 0, st, m.id, n, inv);
  // enough blocks to keep the host link busy, no more
  const unsigned want = nblk(n, 256), most = 1216 / (unsigned)f.n + 1;
  launch_after(k_markers_to_host, dim3(want < most ? want : most, (unsigned)f.n), 256, 0, st, g, m,
               n, f, inv);
}

}  // namespace v2c
