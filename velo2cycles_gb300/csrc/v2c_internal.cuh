// v2c_internal.cuh -- device data layout and shared helpers of the GB300
// marker-in-cell step.
//
// HBM layout (one context):
//  * markers, structure of arrays, physically sorted by cell at upload and
//    updated in place afterwards; a per-step permutation `perm` lists them in
//    (cell, array index) order.  Position = int32 cell (ix*(ynumy-1)+iy) +
//    FP32 in-cell offsets (u, v); u, v in [0,1) inside the grid, outside
//    [0,1] only for markers beyond the domain edge.  cell/u/v are double
//    buffered so a kernel can move markers while neighbouring tiles still
//    read the old positions.
//  * node fields, FP32, [V2C_NF_N][nodenum], y fastest (m3 = m1*ynumy+m2),
//    the reference's own layout; they are converted to and from FP64 only
//    when they cross the C ABI.  (GB300 runs FP64 -- conversions included --
//    at 1/64 of the FP32 rate, so FP64 inside the per-marker and per-node
//    loops would dominate the step.)
//  * grid: FP64 lines plus FP32 cell widths for cell-local arithmetic.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/v2c.h"
#include "v2c_f32x2.cuh"

#define V2C_FULL 0xffffffffu

namespace v2c {

// ------------------------------------------------------------ rock table
// FP32 copies and derived constants of the per-type coefficients.
// The _LO entries are the low words of float pairs (hi + lo, ~48 bits) for
// the constants of the Arrhenius exponent, whose rounding to FP32 alone would
// change the viscosity by several parts in 1e6 (see ductile_visc32).
enum {
  RK_GG = 0, RK_INV_GG, RK_NU, RK_LNNU, RK_DH, RK_DV, RK_LNSS, RK_MM,
  RK_RO, RK_BB, RK_AA, RK_CP, RK_KT, RK_HT, RK_KF, RK_KP, RK_LN_N0, RK_LN_N1,
  RK_N0, RK_N1, RK_KIND, RK_IM,
  RK_DH_LO, RK_DV_LO,      // activation energy and volume, low words
  RK_LNK, RK_LNK_LO,       // ln(0.5 nu / ss^(mm-1)), the diffusion-creep prefactor
  RK_LNG, RK_LNG_LO,       // ln G
  RK_SS, RK_SS_LO,         // ss
  RK_EM, RK_EM_LO,         // (mm-1)/mm
  RK_MM1, RK_MM1_LO,       // mm-1
  RK_LNSS_LO,              // low word of ln ss
  RK_N
};
enum { VISC_NEWTON = 0, VISC_POWER = 1, VISC_STICKY = 2, VISC_UNDEF = 3 };

struct Rock {
  const float *f;  // [RK_N][V2C_MAXTMR]
  __device__ __forceinline__ float operator()(int k, int t) const {
    return __ldg(f + k * V2C_MAXTMR + t);
  }
};

// --------------------------------------------------------------- markers
struct Markers {
  int32_t *cell_in, *cell_out;
  float *u_in, *u_out, *v_in, *v_out;
  int32_t *id;
  int8_t *type;
  uint8_t *flags;  // bit0: out-of-grid reset (markd = markw = -1)
  // tk + tk_lo is the temperature as a float pair: the power-law viscosity
  // depends on exp(E/RT) with E/RT up to ~50, so a temperature rounded to
  // FP32 (6e-8) alone would move it by ~3e-6
  float *tk, *e, *p, *sxx, *sxy, *exx, *exy, *vx, *vy, *phi, *coh, *slipv;
  float *tk_lo;
  // markv as a float pair: the y anchor of an immobile marker (type >= 100,
  // whose markk holds the x anchor), moveandrotatemarkers.c:127-133
  float *mv, *mv_lo;
  float *mnu, *mkt, *mro;  // per-step results of the marker physics kernel
};
// RESET: out-of-grid reset, markd = markw = -1; DNEG: markd = -1 only (a
// marker appended or refilled by the immobile-marker rule)
enum { MFLAG_RESET = 1, MFLAG_DNEG = 2 };

// ------------------------------------------------------------------ grid
// Dependent launches.  A step is some twenty-five kernels on one stream, many
// of a few microseconds; in the usual order a kernel's launch begins only
// when everything of the one before has ended and been flushed.  With
// launch_after the two overlap: the kernel's blocks are set up as the last
// blocks of the one before leave, and wait in after_previous(), the first
// statement of every kernel launched that way, until the whole of it, and
// with it everything before, has ended and its writes are visible.  Pass
// times in us, plain launches and these in turn on one build otherwise alike:
//   51 x 21 lines 239 / 200, 301 x 101 417 / 373, 13-node 433 x 187 679 / 631,
//   refined 1001 x 401 2542 / 2507, 4001 x 1001 19847 / 19656 (runs of one
//   side differ by 0.3, 0.2, 0.1, 0.0 and 0.9 %).
// (Letting the next kernel be set up from the start of this one, by
// launch_dependents, was worse at every size: 210 against 199, 379 against
// 372, 2650 against 2620 and 20600 against 20260 us on the first two and last
// two models; the waiting blocks take the room of working ones.)
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem,
                         cudaStream_t st, const A &...args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, P(args)...);
}

struct Grid {
  const double *gx, *gy;  // lines
  const float *wx, *wy;   // cell widths (ncx, ncy)
  int xn, yn, ncx, ncy;
  long nn;
  double xsize, ysize;
  float xsf, ysf;  // (float)xsize, (float)ysize
  unsigned div_m;  // c / ncy = c div_m >> 31 + div_s for 0 <= c < 2^31
  int div_s;
  // cell column and row of cell c = ix ncy + iy, without the division
  __device__ __forceinline__ void cell_at(int c, int &ix, int &iy) const {
    ix = (int)(((unsigned long long)(unsigned)c * div_m) >> (31 + div_s));
    iy = c - ix * ncy;
  }
};

// div_s = ceil(log2 d), div_m = floor(2^(31 + div_s) / d) + 1: with
// e = div_m d - 2^(31 + div_s) in (0, d], the quotient's error
// c e / (d 2^(31 + div_s)) stays below 1 / d for every c < 2^31.
inline void set_divider(Grid &g) {
  g.div_s = 0;
  while ((1l << g.div_s) < g.ncy) g.div_s++;
  g.div_m = (unsigned)((1ull << (31 + g.div_s)) / (unsigned)g.ncy + 1);
}

struct Nodes {
  float *base;
  long nn;
  __host__ __device__ __forceinline__ float *f(int k) const { return base + (long)k * nn; }
};

// scalar parameters the kernels read, converted once per call on the host
struct Scal {
  v2c_params p;
  int antid;        // timesum > 0 && antidiffinter == 1
  int phi_reset0;   // timesum == timestep (calc_RSF.c:287)
  int sticky_cap;   // stickymod == 1 && timesum > 4e7
  float dt;
  float sticky_nu;  // markgg[2]*timestep/100
  float ln_nubeg, ln_nuend;
  // FP32 copies of the double parameters that per-marker and per-node code
  // reads, rounded once here: in a kernel every double->float conversion or
  // double compare issues on the FP64 pipe, 1/64 of the FP32 rate on this GPU
  float fault_y_f, fault_slope_f;
  float fault_hw1_f;  // (float)fault_hw + 1: far-field test margin
  float a_hr_f, b_hr_f, L_hr_f, V0_hr_f;
  float tdeep_f, zdeep_f;
  float zdeep_lo_f;   // (float)zdeep - 1 - 1e-6 |zdeep|: coarse depth test
  float eps2_f, nstress_f, nubeg_f, nuend_f, faultwidth_f;
  float dt_hi, dt_lo, W_hi, W_lo, sn_hi, sn_lo;  // float-float timestep, faultwidth, nstress
  float lndt_hi, lndt_lo;  // ln timestep as a float pair (-inf when timestep <= 0)
  float eps2_lo, tdeep_lo; // low words of the temperatures markers are reset to
  int sppe_nstress;   // timesum == 0 && reloadfromDP == 0 && compressiblemode == 1
  int timesum_pos;    // timesum > 0
  int timesum_zero;   // timesum == 0
};

// ----------------------------------------------------- compensated sums
// Neumaier two-sum accumulator in FP32: (s, c) carries a sum to about twice
// FP32 precision; value() rounds it once.
struct Acc {
  float s, c;
  __device__ __forceinline__ void zero() { s = 0.f; c = 0.f; }
  __device__ __forceinline__ void add(float x) {
    float t = s + x;
    float e = (fabsf(s) >= fabsf(x)) ? (s - t) + x : (x - t) + s;
    c += e;
    s = t;
  }
  __device__ __forceinline__ float value() const { return s + c; }
};

// (a w, b w), each product rounded.  Not mul.rn.f32x2: the assembler fuses a
// packed product with the packed additions that read it, so the sums below
// would take products that were never rounded.
__device__ __forceinline__ f32x2 mul_w(float a, float b, float w) {
  return pack2(__fmul_rn(a, w), __fmul_rn(b, w));
}

// Two compensated sums side by side.  The error of each addition is formed
// by Knuth's two-sum: exact as Neumaier's is, so the sums are those of Acc
// bit for bit, without the comparison and selection, in 7 packed
// instructions for both instead of 16 scalar ones.
struct Acc2 {
  f32x2 s, c;
  __device__ __forceinline__ void zero() { s = 0; c = 0; }
  __device__ __forceinline__ void add(f32x2 x) {
    const f32x2 t = add2(s, x);
    const f32x2 bb = sub2(t, s);
    const f32x2 e = add2(sub2(s, sub2(t, bb)), sub2(x, bb));
    c = add2(c, e);
    s = t;
  }
  __device__ __forceinline__ void split(Acc &lo, Acc &hi) const {
    unpack2(s, lo.s, hi.s);
    unpack2(c, lo.c, hi.c);
  }
};

// The centre-node weight factor 1 - 2|f - 1/2| of an in-cell offset f
// (interpolation.c:620-622), written as 2f below the middle and 2(1 - f)
// above it: the same value, exact in FP32 (1 - f is exact for f >= 1/2),
// where the literal form loses the low bits of a marker near the cell edge
// -- whose weight is then tiny but whose viscosity may be 1e6 times its
// neighbours' and decide the node's average.
__device__ __forceinline__ float tent(float f) { return f < 0.5f ? 2.f * f : 2.f * (1.f - f); }

// --------------------------------------------------- cell-local geometry
// Offsets of the grid lines i-1 .. i+2 relative to line i, in FP32.
struct Axis {
  int i;      // cell index along the axis
  float X;    // position relative to line i, metres
  float w;    // width of cell i
  float gm1, g1, g2;  // line offsets of i-1, i+1, i+2
  __device__ __forceinline__ float G(int k) const {
    return k <= -1 ? gm1 : (k == 0 ? 0.f : (k == 1 ? g1 : g2));
  }
};

__device__ __forceinline__ Axis make_axis(const float *w, int nc, int i, float X) {
  Axis a;
  a.i = i;
  a.X = X;
  a.w = __ldg(w + i);
  a.gm1 = (i > 0) ? -__ldg(w + i - 1) : -a.w;
  a.g1 = a.w;
  a.g2 = (i + 1 < nc) ? a.w + __ldg(w + i + 1) : 2.f * a.w;
  return a;
}

// Move a local position to the cell containing it (FP32 cell walk).  Cells
// are clamped to [0, nc-1]; returns false when more than `maxsteps` cells
// would be crossed (the caller then falls back to an FP64 search).
__device__ __forceinline__ bool relocate(const float *w, int nc, int &i, float &X,
                                         int maxsteps) {
  for (int s = 0; s < maxsteps; s++) {
    float wi = __ldg(w + i);
    if (X >= wi && i < nc - 1) {
      X -= wi;
      i++;
    } else if (X < 0.f && i > 0) {
      i--;
      X += __ldg(w + i);
    } else {
      return true;
    }
  }
  float wi = __ldg(w + i);
  return !((X >= wi && i < nc - 1) || (X < 0.f && i > 0));
}

// True only where line + u w lies strictly inside (0, size) beyond what the
// FP32 rounding of the four could hide (below 4 2^-24 of their magnitudes);
// elsewhere the FP64 position decides.  The scatters test every marker of the
// model's edge cells: in FP64 those tests, of one lane in 32, kept the FP64
// pipe 86 % busy in the 13-node scatter (433 x 187 lines: 378 -> 118 us, with the
// fields of a marker read at once).
__device__ __forceinline__ bool surely_inside(float line, float w, float u, float size) {
  const float d = u * w, x = line + d;
  const float m = 1e-6f * (fabsf(line) + fabsf(d) + size);
  return x > m && x < size - m;
}

// nxsearch (interpolation.c:1536-1554) in FP64: largest l with g[l] <= x,
// clamped to n-2.
__device__ __forceinline__ int nsearch64(const double *g, int n, double x) {
  int lo = 0, hi = n - 1;
  do {
    int c = (lo + hi) / 2;
    if (__ldg(g + c) > x) hi = c; else lo = c;
  } while (hi - lo > 1);
  return lo > n - 2 ? n - 2 : lo;
}
// The same for the assignment of every marker.  For an x without a sign bit,
// g > x is the comparison of the bit patterns as integers (a line below 0 has
// a negative pattern): twenty FP64 comparisons per marker were the whole time
// of a cell assignment.  The length of the bracket does not depend on x, so
// its bookkeeping is the warp's.  9 M markers on 1501 x 401 lines: 341 us in
// FP64, 97 with integers (see also v2c_sort_static.cu).
__device__ __forceinline__ int nsearch_bits(const double *g, int n, double x) {
  const long long xb = __double_as_longlong(x);
  if (xb < 0) return nsearch64(g, n, x);
  const long long *gb = reinterpret_cast<const long long *>(g);
  int lo = 0;
  for (int len = n - 1; len > 1;) {  // the line sought is one of lo .. lo + len - 1
    const int half = len >> 1;
    if (__ldg(gb + lo + half) <= xb) lo += half;
    len -= half;
  }
  return lo;
}

// Offset within a cell rounded to FP32 without crossing 0.5 or 1.0: the
// scatter kernels branch on u < 0.5 / u > 0.5 and the in-grid tests on
// u < 1, so the FP32 offset must land on the same side as the FP64 one.
__device__ __forceinline__ float offset32(double u) {
  float f = (float)u;
  if (u < 0.5 && f >= 0.5f) f = nextafterf(0.5f, 0.f);
  if (u > 0.5 && f <= 0.5f) f = nextafterf(0.5f, 1.f);
  if (u < 1.0 && f >= 1.0f) f = nextafterf(1.0f, 0.f);
  if (u > 1.0 && f <= 1.0f) f = nextafterf(1.0f, 2.f);
  if (u > 0.0 && f <= 0.0f) f = 1e-30f;
  if (u < 0.0 && f >= 0.0f) f = -1e-30f;
  return f;
}

// ---------------------------------------------------------- device status
// Counters read back by v2c_get_status (64-bit, integer atomics only).
enum {
  ST_OUT_OF_GRID = 0, ST_FAR_MOVES, ST_NAN, ST_NEWTON_ITERS, ST_NEWTON_FALLBACK,
  ST_NEWTON_NONCONV, ST_NEWTON_MAXRES_BITS, ST_MAX_CELL, ST_N
};

}  // namespace v2c
