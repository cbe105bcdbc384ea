// v2c_m2n.cu -- marker2nodes (interpolation.c:55-926) as a deterministic
// segmented reduction over cell-sorted markers.
//
// Tiling.  A CTA owns node rows [j0, j0+TY) and node columns [i0, i0+TX).
// It sweeps cell columns ci = i0-1 .. i0+TX-1.  For each column it stages the
// column's markers of cell rows j0-1 .. j0+TY-1 (one contiguous run of the
// sorted order) in shared memory.  Then lane jl of each warp accumulates, for
// node row j = j0+jl, its warp's sums over the contributions of cells
// (ci, j-1) and (ci, j), which are all the cells of that column that reach
// node (ci, j) and (ci+1, j) under the interpolationmod=2 stencil
// (interpolation.c:539-628):
//   * basic node (ci, j) gets the left-half quadrants of those two cells,
//     basic node (ci+1, j) the right-half ones;
//   * vx node (ci, j) gets cell (ci, j) if u < 0.5, vx node (ci+1, j) if
//     u > 0.5 (carry);
//   * vy node (ci, j) gets cell (ci, j-1) if v > 0.5 and cell (ci, j) if
//     v < 0.5;
//   * the centre node (ci+1, j+1) gets cell (ci, j) only.
// The per-marker physics ran before, in marker order (v2c_phys.cu); staging
// only reads the marker fields and those results.
// Each node is summed by exactly one thread, in sorted-marker order, with
// FP32 two-sum compensation; the node tail (normalisation, antidiffusion
// correction, interpolation.c:714-824) runs in the same thread on the
// compensated sums, rounding each result once to FP32.
// No float atomics; the result does not depend on scheduling.
//
// Eight warps share a staged column (lanes = node rows).  Warps 0, 1: the
// basic nodes' stress/state group of even and of odd node columns; a node
// column takes the right halves of one cell column and then the left halves
// of the next, so a warp runs one list of markers per cell column and keeps
// one set of sums, and no sums are carried between warps.  Warps 2, 3: the
// same for the thermal group.  Warp 4: centre nodes, viscosities; warp 5:
// centre nodes, stress, strain rate, pressure; warp 6: vx; warp 7: vy.
#include <math.h>

#include "v2c_ff.cuh"
#include "v2c_kernels.h"
#include "v2c_internal.cuh"

namespace v2c {

namespace {

constexpr int TY = 32;
constexpr int NTH = 8 * 32;
// Markers staged at once.  A column segment (33 cells) that does not fit
// splits into chunks, and the lanes whose cells lie in the other chunk idle:
// at 20 markers per cell 384-marker chunks left 18.6 of 32 lanes busy.  780
// holds 33 cells of 23 markers, in the 56 KB that four resident CTAs leave
// each other (64 registers x 256 threads x 4 fill the register file).
constexpr int CHUNK = 780;

// staged fields, in pairs that one 8-byte shared-memory read brings straight
// into the operand pair of a packed FP32 instruction; warp k stages pair k
enum { S_UV = 0, S_NUE, S_SXYEXY, S_COHPHI, S_KTTK, S_SXXEXX, S_PRO, S_VXVY, S_N };

// The marker at position p of a chunk is staged in slot p + p / 16: the lanes
// read consecutive cells in lockstep, and with a free slot in every 17 the
// runs of 16 or 20 markers of a fresh uniform seeding start in different
// banks instead of a few.
constexpr int SLOTS = CHUNK + CHUNK / 16;
__device__ __forceinline__ int slot_of(int p) { return p + (p >> 4); }
struct Smem {
  float2 p[S_N][SLOTS];
  int32_t idx[CHUNK];  // array indices of the markers, copied a chunk ahead
  uint8_t type[CHUNK];
};

// 4-byte asynchronous copy global -> shared (no register holds the value)
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// The two marker fields this warp stages (no second one for P without
// per-marker densities)
struct Source {
  const float *x, *y;
};
__device__ __forceinline__ Source stage_source(const M2NArgs &a, int warp) {
  const Markers &m = a.m;
  switch (warp) {
    case S_UV: return {m.u_in, m.v_in};
    case S_NUE: return {m.mnu, m.e};
    case S_SXYEXY: return {m.sxy, m.exy};
    case S_COHPHI: return {m.coh, m.phi};
    case S_KTTK: return {m.mkt, m.tk};
    case S_SXXEXX: return {m.sxx, m.exx};
    case S_PRO: return {m.p, a.S.p.densimod ? m.mro : nullptr};
    default: return {m.vx, m.vy};
  }
}

// Copy this warp's pair of fields of the chunk's n markers (indices in
// sm.idx) into their slots (asynchronous copies: all in flight at once, no register
// holds a field), the CTA's threads the types, and wait for the copies.
// Warp 0 then replaces u of a marker not strictly inside the model
// (interpolation.c:219) by NaN, which fails every weight test below.
__device__ __forceinline__ void stage_fields(const M2NArgs &a, Smem &sm, int n, int ci, bool edge,
                                             const Source &src, int warp, int lane) {
  float2 *dst = sm.p[warp];
#pragma unroll 8
  for (int p = lane; p < n; p += 32) {
    const int i = sm.idx[p];
    cp_async4(&dst[slot_of(p)].x, src.x + i);
    if (src.y) cp_async4(&dst[slot_of(p)].y, src.y + i);
  }
#pragma unroll 4
  for (int p = warp * 32 + lane; p < n; p += NTH) sm.type[p] = (uint8_t)a.m.type[sm.idx[p]];
  cp_async_wait_all();
  const Grid &g = a.g;
  if (edge && warp == S_UV) {
    const bool ex = ci == 0 || ci == g.ncx - 1;
#pragma unroll 1
    for (int p = lane; p < n; p += 32) {
      const int iy = a.m.cell_in[sm.idx[p]] - ci * g.ncy;
      const bool ey = iy == 0 || iy == g.ncy - 1;
      if (!ex && !ey) continue;
      float2 *uv = &sm.p[S_UV][slot_of(p)];
      bool act = true;
      if (ex && !surely_inside(__ldg(a.gxf + ci), __ldg(g.wx + ci), uv->x, g.xsf)) {
        double x = g.gx[ci] + (double)uv->x * (g.gx[ci + 1] - g.gx[ci]);
        act = act && x > 0 && x < g.xsize;
      }
      if (ey && !surely_inside(__ldg(a.gyf + iy), __ldg(g.wy + iy), uv->y, g.ysf)) {
        double y = g.gy[iy] + (double)uv->y * (g.gy[iy + 1] - g.gy[iy]);
        act = act && y > 0 && y < g.ysize;
      }
      if (!act) uv->x = __int_as_float(0x7fc00000);
    }
  }
}

// Ahead of the chunk at sorted positions [b, e): start copying its sort
// indices (waited for before it is staged), and ask L2 for its markers'
// fields at the array indices b .. e - 1.  The arrays were stored in sorted
// order at the upload and markers move a fraction of a cell per step, so
// these are nearly the right lines.
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}
__device__ __forceinline__ void start_chunk(const M2NArgs &a, Smem &sm, const Source &src, int b,
                                            int e, int warp, int lane) {
#pragma unroll 1
  for (int s = b + warp * 32 + lane; s < e; s += NTH) cp_async4(&sm.idx[s - b], a.perm + s);
  const int s = b + 32 * lane;
  if (s >= e) return;
  prefetch_l2(src.x + s);
  if (src.y) prefetch_l2(src.y + s);
  if (warp == 0 && (lane & 3) == 0) prefetch_l2(a.m.type + s);
}

// calc_frictionpara_nodes (calc_RSF.c:298-350), FP64; out of line, taken
// only for nodes within 1 m of the frictional band (see node_friction)
__device__ __noinline__ void friction_node(const v2c_params &p, double x, double y, double &mu,
                                           double &a, double &b, double &L, double &V0) {
  double d = y - (p.fault_y + p.fault_slope * x);
  double radius = d >= 0 ? d : -d;
  if (radius <= p.fault_hw) {
    if (x > p.end_updip && x < p.start_downdip) {
      a = p.a_vw; b = p.b_vw; L = p.L_vw; V0 = p.V0_vw;
    } else if (x >= p.start_updip && x <= p.end_updip && p.half_range > 0) {
      double f = (x - (p.start_updip)) / (2 * p.half_range);
      a = p.a_vs + f * (p.a_vw - p.a_vs); b = p.b_vs + f * (p.b_vw - p.b_vs);
      L = p.L_vs + f * (p.L_vw - p.L_vs); V0 = p.V0_vs + f * (p.V0_vw - p.V0_vs);
    } else if (x >= p.start_downdip && x < p.end_downdip && p.half_range > 0) {
      double f = (x - (p.start_downdip)) / (2 * p.half_range);
      a = p.a_vw - f * (p.a_vw - p.a_vs); b = p.b_vw - f * (p.b_vw - p.b_vs);
      L = p.L_vw - f * (p.L_vw - p.L_vs); V0 = p.V0_vw - f * (p.V0_vw - p.V0_vs);
    } else {
      a = p.a_vs; b = p.b_vs; L = p.L_vs; V0 = p.V0_vs;
    }
    mu = 0.2;
  } else {
    mu = 0.6; a = p.a_hr; b = p.b_hr; L = p.L_hr; V0 = p.V0_hr;
  }
}

// Friction parameters of node (ci, j): outside the band (the FP32 distance
// clears the half-width by more than 1 m, far above its rounding) they are
// the constants of the far field; near the band the FP64 rule decides.
__device__ __forceinline__ void node_friction(const M2NArgs &a, int ci, int j, float &mu,
                                              float &fa, float &fb, float &fL, float &fV0) {
  const v2c_params &p = a.S.p;
  const Scal &S = a.S;
  const float xf = __ldg(a.gxf + ci), yf = __ldg(a.gyf + j);
  const float rad = fabsf(yf - (S.fault_y_f + S.fault_slope_f * xf));
  if (rad > S.fault_hw1_f) {
    mu = 0.6f; fa = S.a_hr_f; fb = S.b_hr_f; fL = S.L_hr_f; fV0 = S.V0_hr_f;
    return;
  }
  double dmu, da, db, dL, dV0;
  friction_node(p, a.g.gx[ci], a.g.gy[j], dmu, da, db, dL, dV0);
  mu = (float)dmu; fa = (float)da; fb = (float)db; fL = (float)dL; fV0 = (float)dV0;
}

// A compensated sum as a float pair.
__device__ __forceinline__ ff acc_ff(const Acc &a) {
  ff r;
  r.hi = two_sum(a.s, a.c, r.lo);
  return r;
}
__device__ __forceinline__ float acc_round(const Acc &a) { return ff_round(acc_ff(a)); }

// The node averages, num / den of two compensated sums as a float pair.  Out
// of line with the two stores built on it: the tail of one node is 17 such
// quotients, and as inline copies their code alone outgrew the instruction
// caches of the eight warps that run different tails (6.7 stalled cycles per
// issue waiting for instructions, of 20).
__device__ __forceinline__ ff quot(const Acc &num, const Acc &den) {
  return ff_div_fast(acc_ff(num), acc_ff(den));
}
struct NodeRef {
  float *base;  // node fields at this node
  long nn;
  __device__ __forceinline__ float &operator()(int f) const { return base[f * nn]; }
};
// field f = num / den, rounded once
static __device__ __noinline__ void put_ratio(NodeRef n, int f, Acc num, Acc den) {
  n(f) = ff_round(quot(num, den));
}
// field fn = num / den and field fo = the antidiffusion form cur + (n - prev)
// of the average n (interpolation.c:730-736, 758-763, 784-806), or the
// average itself without antidiffusion: cur and prev are consecutive states of one field that agree in their leading digits, so
// cur - prev is formed exactly and the sum is rounded once.
static __device__ __noinline__ void put_antid(NodeRef n, int fn, int fo, bool antid, float cur,
                                              float prev, Acc num, Acc den) {
  const ff avg = quot(num, den);
  const float r = ff_round(avg);
  n(fn) = r;
  n(fo) = antid ? ff_round(ff_add(avg, ff_diff(cur, prev))) : r;
}
static __device__ __noinline__ void put_zeros(NodeRef n, int first, int count) {
#pragma unroll 1
  for (int f = first; f < first + count; f++) n(f) = 0.f;
}

// The node tail of marker2nodes (interpolation.c:714-824) for node row j
// of column ci, from the compensated sums of one group: basic node (ci, j)
// stress/state group (cur[0..7]: nu, nu/G, e, sxy, exy, C, phi, w) or
// thermal group (cur[0..6]: ro, et, ht, cp, kt, tk, w); the viscosities
// (cur[0..2]: nu, nu/G, w) or the stresses (cur[0..3]: sxx, exx, p, w) of
// the centre node (ci+1, j+1) of cell (ci, j), with the centre fields of
// (ci, j) when no cell feeds it; vx or vy node (ci, j) (cur[0..2]: v*ro, ro,
// w).  The averages are float-pair quotients of the float-pair sums, rounded
// once to FP32.
enum { T_STRESS = 0, T_THERMAL, T_CENTRE_NU, T_CENTRE_S, T_VX, T_VY };
// the fields cleared together are neighbours in the node block
static_assert(V2C_NF_MRY0 - V2C_NF_PHISUM == 14 && V2C_NF_ND - V2C_NF_NU == 1 &&
                  V2C_NF_V0S - V2C_NF_MUS_S == 4 && V2C_NF_TK - V2C_NF_RO == 5,
              "node field order");
template <int GROUP>
__device__ __forceinline__ void node_tail(const M2NArgs &a, int ci, int j, const Acc *cur) {
  const Grid &g = a.g;
  const int ncy = g.ncy;
  const long m3 = (long)ci * g.yn + j;
  const NodeRef n{a.N.base + m3, a.N.nn};
  const bool antid = a.S.antid;
  if (GROUP == T_STRESS) {
    const Acc w = cur[7];
    const bool interior = ci >= 1 && j >= 1 && ci < g.xn - 1 && j < g.yn - 1;
    if (acc_round(w) != 0.f && interior) {
      // all read at once, before the calls
      const float c0 = n(V2C_NF_PHIS_IT), p0 = n(V2C_NF_PHIE), c1 = n(V2C_NF_SXY);
      const float p1 = n(V2C_NF_SXYEE), c2 = n(V2C_NF_EXY), p2 = n(V2C_NF_EXYEE);
      const float c3 = n(V2C_NF_PES), p3 = n(V2C_NF_PEE);
      put_antid(n, V2C_NF_PHIN, V2C_NF_PHIS, antid, c0, p0, cur[6], w);
      put_antid(n, V2C_NF_SXYEN, V2C_NF_SXYE, antid, c1, p1, cur[3], w);
      put_antid(n, V2C_NF_EXYEN, V2C_NF_EXYE, antid, c2, p2, cur[4], w);
      put_antid(n, V2C_NF_PEN, V2C_NF_PE, antid, c3, p3, cur[2], w);
      if (n(V2C_NF_PE) < 0.f) n(V2C_NF_PE) = 0.f;
      put_ratio(n, V2C_NF_COHESION, cur[5], w);
      put_ratio(n, V2C_NF_NU_M2C, cur[0], w);
      // nu_m2c / (sum nu/G w / sum w) = sum nu w / sum nu/G w
      put_ratio(n, V2C_NF_GG, cur[0], cur[1]);
    } else {
      n(V2C_NF_PHIN) = 0; n(V2C_NF_SXYEN) = 0; n(V2C_NF_EXYEN) = 0;
      n(V2C_NF_PHIS) = 0; n(V2C_NF_SXYE) = 0; n(V2C_NF_EXYE) = 0;
      n(V2C_NF_COHESION) = 0; n(V2C_NF_GG) = 0;
    }
  } else if (GROUP == T_THERMAL) {
    const Acc w = cur[6];
    const bool any = acc_round(w) != 0.f;
    const bool interior = ci >= 1 && j >= 1 && ci < g.xn - 1 && j < g.yn - 1;
    if (any && interior) {
      float mu, fa, fb, fL, fV0;
      node_friction(a, ci, j, mu, fa, fb, fL, fV0);
      n(V2C_NF_MUS_S) = mu; n(V2C_NF_AS) = fa; n(V2C_NF_BS) = fb;
      n(V2C_NF_LS) = fL; n(V2C_NF_V0S) = fV0;
    } else {
      put_zeros(n, V2C_NF_MUS_S, 5);
    }
    if (any) {
      put_ratio(n, V2C_NF_RO, cur[0], w);
      put_ratio(n, V2C_NF_ET, cur[1], w);
      put_ratio(n, V2C_NF_HT, cur[2], w);
      put_ratio(n, V2C_NF_CP, cur[3], w);
      put_ratio(n, V2C_NF_KT, cur[4], w);
      put_ratio(n, V2C_NF_TK, cur[5], w);
    } else {
      put_zeros(n, V2C_NF_RO, 6);
    }
    // arrays the reference zeroes at the start (interpolation.c:58-153)
    // and that marker2nodes itself does not fill
    put_zeros(n, V2C_NF_NU, 2);
    put_zeros(n, V2C_NF_PHISUM, 15);
  } else if (GROUP == T_CENTRE_NU) {
    if (ci < g.ncx && j < ncy) {
      const NodeRef c{n.base + g.yn + 1, n.nn};
      if (acc_round(cur[2]) != 0.f) {
        put_ratio(c, V2C_NF_ND_M2C, cur[0], cur[2]);
        put_ratio(c, V2C_NF_GD, cur[0], cur[1]);
        c(V2C_NF_BM) = 50e9f;
      } else {
        c(V2C_NF_GD) = 0; c(V2C_NF_BM) = 0;
      }
      c(V2C_NF_DRO) = 0; c(V2C_NF_DRP) = 0;
    }
    // centre fields of nodes no cell feeds (first column / first row)
    if (ci == 0 || j == 0) {
      n(V2C_NF_GD) = 0; n(V2C_NF_BM) = 0; n(V2C_NF_DRO) = 0; n(V2C_NF_DRP) = 0;
    }
  } else if (GROUP == T_CENTRE_S) {
    if (ci < g.ncx && j < ncy) {
      const NodeRef c{n.base + g.yn + 1, n.nn};
      const Acc w = cur[3];
      if (acc_round(w) != 0.f) {
        const float c0 = c(V2C_NF_SXX), p0 = c(V2C_NF_SXXEE), c1 = c(V2C_NF_PR);
        const float p1 = c(V2C_NF_SPPEE), c2 = c(V2C_NF_EXX), p2 = c(V2C_NF_EXXEE);
        put_antid(c, V2C_NF_SXXEN, V2C_NF_SXXE, antid, c0, p0, cur[0], w);
        put_antid(c, V2C_NF_SPPEN, V2C_NF_SPPE, antid, c1, p1, cur[2], w);
        put_antid(c, V2C_NF_EXXEN, V2C_NF_EXXE, antid, c2, p2, cur[1], w);
        if (a.S.sppe_nstress) c(V2C_NF_SPPE) = a.S.nstress_f;
      } else {
        c(V2C_NF_SXXEN) = 0; c(V2C_NF_SPPEN) = 0; c(V2C_NF_EXXEN) = 0;
        c(V2C_NF_SXXE) = 0; c(V2C_NF_SPPE) = 0; c(V2C_NF_EXXE) = 0;
      }
    }
    if (ci == 0 || j == 0) {
      n(V2C_NF_SXXEN) = 0; n(V2C_NF_SPPEN) = 0; n(V2C_NF_EXXEN) = 0;
      n(V2C_NF_SXXE) = 0; n(V2C_NF_SPPE) = 0; n(V2C_NF_EXXE) = 0;
    }
  } else {
    constexpr bool X = GROUP == T_VX;
    const int mv = X ? V2C_NF_MVX : V2C_NF_MVY, mr = X ? V2C_NF_MRX : V2C_NF_MRY;
    if (acc_round(cur[2]) != 0.f) {
      put_antid(n, X ? V2C_NF_MVXN : V2C_NF_MVYN, mv, antid, n(X ? V2C_NF_VX : V2C_NF_VY),
                n(X ? V2C_NF_MVXE : V2C_NF_MVYE), cur[0], cur[1]);
      // the boundary correction (vxvy_boundarycorrection) leaves the vx
      // ghost row and the vy ghost column at zero; only the 13-node stencil
      // gives them weight
      if (X ? j == g.yn - 1 : ci == g.xn - 1) n(mv) = 0;
      put_ratio(n, mr, cur[1], cur[2]);
    } else {
      n(mv) = 0; n(mr) = 0;
    }
  }
}

// Two runs of one lane's markers in the staged chunk, walked as one list:
// the warp's time goes with the longest of its 32 lists, and one list of two
// runs is shorter than the two runs' longest in turn.
struct Runs {
  int p, n1, n, jump;  // first position, markers of run 1, of both, positions skipped between them
};
// sorted positions [b1, e1), then [b2, e2), clipped to the chunk [cs, ce)
__device__ __forceinline__ Runs two_runs(int cs, int ce, int b1, int e1, int b2, int e2) {
  b1 = max(b1, cs); e1 = min(e1, ce); b2 = max(b2, cs); e2 = min(e2, ce);
  Runs r;
  r.n1 = max(e1 - b1, 0);
  r.n = r.n1 + max(e2 - b2, 0);
  r.p = b1 - cs;
  r.jump = (b2 - cs) - (r.p + r.n1);
  return r;
}
#define FOR_RUNS(R)                                                          \
  _Pragma("unroll 1") for (int i_ = 0, p = (R).p; i_ < (R).n; ++i_, ++p)     \
    if (p += (i_ == (R).n1) ? (R).jump : 0; true)

// what a warp of the sweep sums per marker
struct Column {
  int cs, ce;            // the staged chunk
  int4 ql, qu;           // quarter class starts of cells (ci, j-1) and (ci, j)
  int lo_e, up_e;        // their ends
  float s1lo, s1up;      // 1 / cell area
};

__device__ __forceinline__ float marker_ro(const M2NArgs &a, const Smem &sm, int p, int q) {
  return a.S.p.densimod ? sm.p[S_PRO][q].y : a.R(RK_RO, sm.type[p]);
}

// Basic nodes: one list of the halves (left: of node column ci; right: of
// ci+1) of cells (ci, j-1), bottom quarter, and (ci, j), top quarter.  The
// weight s (1-2u)(2v-1) etc. of the four quarters is written (+-s)(2u-1)(2v-1)
// -- the same roundings -- and is positive exactly for a marker strictly
// inside the quarter (exact halves belong to no basic node, u = NaN to none).
template <bool THERMAL>
__device__ __forceinline__ void sum_basic(const M2NArgs &a, const Smem &sm, const Column &C,
                                          bool left, Acc2 (&acc)[4], Acc &wt) {
  const Runs R = left ? two_runs(C.cs, C.ce, C.ql.z, C.ql.w, C.qu.x, C.qu.y)
                      : two_runs(C.cs, C.ce, C.ql.w, C.lo_e, C.qu.y, C.qu.z);
  const float s1 = left ? -C.s1lo : C.s1lo, s2 = left ? C.s1up : -C.s1up;
  FOR_RUNS(R) {
    const int q = slot_of(p);
    const float2 uv = sm.p[S_UV][q];
    const int t = sm.type[p];
    const float w = (i_ < R.n1 ? s1 : s2) * fmaf(2.f, uv.x, -1.f) * fmaf(2.f, uv.y, -1.f);
    const float2 ne = sm.p[S_NUE][q], cp = sm.p[S_COHPHI][q], se = sm.p[S_SXYEXY][q];
    const float2 kt = sm.p[S_KTTK][q];
    if (w > 0.f) {
      if (!THERMAL) {
        acc[0].add(mul_w(ne.x, __fmul_rn(ne.x, a.R(RK_INV_GG, t)), w));
        acc[1].add(mul_w(ne.y, se.x, w));
        acc[2].add(mul_w(se.y, cp.x, w));
        acc[3].add(pack2(__fmul_rn(cp.y, w), w));
      } else {
        const float bb = a.R(RK_BB, t);
        // dencalcomp adiabatic term
        const float et = fdiv_normal(bb, 1.f - bb * (kt.y - 298.15f));
        acc[0].add(mul_w(marker_ro(a, sm, p, q), et, w));
        acc[1].add(mul_w(a.R(RK_HT, t), a.R(RK_CP, t), w));
        acc[2].add(mul_w(kt.x, kt.y, w));
        wt.add(w);
      }
    }
  }
}

// C4 (80 M markers, 20 per cell): 4.96 -> 2.98 ms against four warps of
// 384-marker chunks with scalar two-sums; a 1001 x 401-line model of 20 (16)
// per cell 0.582 -> 0.382 (0.499 -> 0.316) ms, 301 x 101 lines 77 -> 48 us.
// Bound by instruction issue (30 warp instructions per marker, 54 % issue
// active at 4 CTAs) and the two waits of each chunk; staging alone takes
// 1.3 ms at C4, 5.1 TB/s.  What each part gave there: whole columns in one
// chunk and one list per warp (18.6 -> 29 active lanes), packed two-sums,
// the loops kept rolled and the tail's quotients out of line (instruction
// fetch was the largest stall: 6.7 cycles per issue), indices and L2
// prefetches a chunk ahead (3.63 -> 3.15 ms), the tail's inputs read at once
// (3.15 -> 2.98 ms).  Copying through registers instead of asynchronously
// was slower (0.47 against 0.44 ms on the smaller model).
__global__ void __launch_bounds__(NTH, 4) k_m2n(M2NArgs a) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  const Grid &g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, jl = tid & 31;
  const int i0 = blockIdx.x * a.TX, j0 = blockIdx.y * TY;
  const int j = j0 + jl;
  const bool jvalid = j < g.yn;
  const int ncy = g.ncy;
  const int ci_end = min(i0 + a.TX, g.xn);
  const int jlo = max(j0 - 1, 0), jhi = min(j0 + TY - 1, ncy - 1);
  const Source src = stage_source(a, warp);
  const int c_end = min(ci_end, g.ncx);
  const int c0 = max(i0 - 1, 0);
  if (c0 < c_end) {
    const int b = __ldg(a.start + (long)c0 * ncy + jlo);
    start_chunk(a, sm, src, b, min(b + CHUNK, __ldg(a.start + (long)c0 * ncy + jhi + 1)), warp, jl);
  }

  // warps 0, 1: nu, nu/G | e, sxy | exy, C | phi, w
  // warps 2, 3: ro, et | ht, cp | kt, tk and w      warp 4: nu, nu/G and w
  // warp 5: sxx, exx | p, w     warps 6, 7: v*ro, ro and w (vx: [1] the carry)
  Acc2 acc[4];
  Acc wt, wt1;
#pragma unroll
  for (int q = 0; q < 4; q++) acc[q].zero();
  wt.zero(); wt1.zero();

  for (int ci = c0; ci < ci_end; ++ci) {
    // owned: this CTA finishes node column ci; next: it finishes column ci+1
    const bool owned = ci >= i0, next = ci + 1 < ci_end;
    const bool mine = ((ci ^ warp) & 1) == 0;  // warps 0..3: node column ci is this warp's
    if (ci < g.ncx) {
      const long cb = (long)ci * ncy;
      const int seg_b = __ldg(a.start + cb + jlo), seg_e = __ldg(a.start + cb + jhi + 1);
      const int nseg_b = ci + 1 < c_end ? __ldg(a.start + cb + ncy + jlo) : 0;
      const int nseg_e = ci + 1 < c_end ? __ldg(a.start + cb + ncy + jhi + 1) : 0;
      const bool edge = ci == 0 || ci == g.ncx - 1 || jlo == 0 || jhi == ncy - 1;
      Column C;
      C.ql = make_int4(0, 0, 0, 0); C.qu = make_int4(0, 0, 0, 0);
      C.lo_e = 0; C.up_e = 0;
      C.s1lo = 0.f; C.s1up = 0.f;
      const float iwx = 1.f / __ldg(g.wx + ci);
      if (jvalid && j - 1 >= 0 && j - 1 <= ncy - 1) {
        C.ql = __ldg(a.qstart + cb + j - 1);
        C.lo_e = __ldg(a.start + cb + j);
        C.s1lo = iwx / __ldg(g.wy + j - 1);
      }
      if (jvalid && j <= ncy - 1) {
        C.qu = __ldg(a.qstart + cb + j);
        C.up_e = __ldg(a.start + cb + j + 1);
        C.s1up = iwx / __ldg(g.wy + j);
      }
      if (seg_b == seg_e)
        start_chunk(a, sm, src, nseg_b, min(nseg_b + CHUNK, nseg_e), warp, jl);
      for (int cs = seg_b; cs < seg_e; cs += CHUNK) {
        const int ce = min(cs + CHUNK, seg_e);
        C.cs = cs; C.ce = ce;
        cp_async_wait_all();
        __syncthreads();  // the indices are there, the previous chunk is summed
        stage_fields(a, sm, ce - cs, ci, edge, src, warp, jl);
        __syncthreads();
        const int nb = ce == seg_e ? nseg_b : ce;
        start_chunk(a, sm, src, nb, min(nb + CHUNK, ce == seg_e ? nseg_e : seg_e), warp, jl);
        if (warp < 4) {
          if (mine ? owned : next) {
            if (warp < 2) sum_basic<false>(a, sm, C, mine, acc, wt);
            else sum_basic<true>(a, sm, C, mine, acc, wt);
          }
        } else if (warp < 6) {
          // the whole cell (ci, j) to its centre node
          if (owned) {
            const Runs R = two_runs(cs, ce, C.qu.x, C.up_e, 0, 0);
#pragma unroll 1
            for (int i = 0, p = R.p; i < R.n; ++i, ++p) {
              const int q = slot_of(p);
              const float2 uv = sm.p[S_UV][q];
              const float w = C.s1up * tent(uv.x) * tent(uv.y);
              if (w >= 0.f) {
                if (warp == 4) {
                  const float nu = sm.p[S_NUE][q].x;
                  acc[0].add(mul_w(nu, __fmul_rn(nu, a.R(RK_INV_GG, sm.type[p])), w));
                  wt.add(w);
                } else {
                  const float2 se = sm.p[S_SXXEXX][q];
                  acc[0].add(mul_w(se.x, se.y, w));
                  acc[1].add(pack2(__fmul_rn(sm.p[S_PRO][q].x, w), w));
                }
              }
            }
          }
        } else if (warp == 6) {
          // vx node (ci, j) from u < 1/2 of cell (ci, j) (classes 0, 2), then
          // vx node (ci+1, j) from u > 1/2 (classes 1, 3)
          if (owned) {
            const Runs R = two_runs(cs, ce, C.qu.x, C.qu.y, C.qu.z, C.qu.w);
            FOR_RUNS(R) {
              const int q = slot_of(p);
              const float2 uv = sm.p[S_UV][q];
              if (uv.x < 0.5f) {
                const float w = C.s1up * (1.f - uv.x) * (1.f - fabsf(uv.y - 0.5f));
                const float ro = marker_ro(a, sm, p, q);
                acc[0].add(mul_w(__fmul_rn(sm.p[S_VXVY][q].x, ro), ro, w));
                wt.add(w);
              }
            }
          }
          if (next) {
            const Runs R = two_runs(cs, ce, C.qu.y, C.qu.z, C.qu.w, C.up_e);
            FOR_RUNS(R) {
              const int q = slot_of(p);
              const float2 uv = sm.p[S_UV][q];
              const float w = C.s1up * uv.x * (1.f - fabsf(uv.y - 0.5f));
              if (w >= 0.f) {
                const float ro = marker_ro(a, sm, p, q);
                acc[1].add(mul_w(__fmul_rn(sm.p[S_VXVY][q].x, ro), ro, w));
                wt1.add(w);
              }
            }
          }
        } else if (owned) {
          // vy node (ci, j) from the bottom halves of cell (ci, j-1) (classes
          // 2, 3) and the top halves of cell (ci, j) (classes 0, 1)
          const Runs R = two_runs(cs, ce, C.ql.z, C.lo_e, C.qu.x, C.qu.z);
          FOR_RUNS(R) {
            const int q = slot_of(p);
            const float2 uv = sm.p[S_UV][q];
            const bool lo = i_ < R.n1;
            if (lo || uv.y < 0.5f) {
              const float w = (lo ? C.s1lo : C.s1up) * (1.f - fabsf(uv.x - 0.5f)) *
                              (lo ? uv.y : 1.f - uv.y);
              if (w >= 0.f) {
                const float ro = marker_ro(a, sm, p, q);
                acc[0].add(mul_w(__fmul_rn(sm.p[S_VXVY][q].y, ro), ro, w));
                wt.add(w);
              }
            }
          }
        }
      }
    }

    // ------------------------------------------------------ node tail
    if (warp < 4 && !mine) continue;
    if (owned && jvalid) {
      Acc c[8];
#pragma unroll
      for (int q = 0; q < 4; q++) acc[q].split(c[2 * q], c[2 * q + 1]);
      if (warp < 2) {
        node_tail<T_STRESS>(a, ci, j, c);
      } else if (warp < 4) {
        c[6] = wt;
        node_tail<T_THERMAL>(a, ci, j, c);
      } else if (warp == 4) {
        c[2] = wt;
        node_tail<T_CENTRE_NU>(a, ci, j, c);
      } else if (warp == 5) {
        node_tail<T_CENTRE_S>(a, ci, j, c);
      } else {
        c[2] = wt;
        if (warp == 6) node_tail<T_VX>(a, ci, j, c);
        else node_tail<T_VY>(a, ci, j, c);
      }
    }
    if (warp == 6) {
      acc[0] = acc[1];
      wt = wt1;
    } else {
      acc[0].zero();
      wt.zero();
    }
#pragma unroll
    for (int q = 1; q < 4; q++) acc[q].zero();
    wt1.zero();
  }
}

// ------------------------------------------------ interpolationmod 1
// The 13-node stencil (interpolation.c:258-538) as a gather: one thread per
// node and role sums, in sorted-marker order cell by cell, the markers of
// the cells whose stencil reaches the node, with that stencil's weight
// (bilinear on basic nodes; the staggered vx, vy and centre stencils with
// their half-cell conditions), then runs the same node tail as the tile
// sweep.  A marker in cell (cx, cy) at offsets (u, v) reaches
//   basic (cx + a, cy + b), a, b in {0, 1}:  (a ? u : 1-u) (b ? v : 1-v)
//   vx (cx + a, cy + b), b in {-1, 0, 1}:    (a ? u : 1-u) times 1-|v-1/2|
//       (b = 0), v-1/2 if v > 1/2 (b = 1), 1/2-v if v < 1/2 (b = -1)
//   vy likewise with the axes exchanged (a in {-1, 0, 1}, b in {0, 1})
//   centre (cx + a, cy + b), a, b in {0, 1, 2}: the product of the axis
//       factors 1/2-u if u < 1/2 (a = 0), 1-|u-1/2| (a = 1), u-1/2 if
//       u > 1/2 (a = 2), and the same in v.
// Contributions the reference sends past the last node row (its node
// index wraps into the next column's first row, a centre node that is
// never normalised) have no effect and are not formed.
struct Mk {
  int idx, t;
  float u, v;
};

__device__ __forceinline__ bool marker_active(const M2NArgs &a, int cx, int cy, float u, float v) {
  const Grid &g = a.g;
  bool act = true;
  if ((cx == 0 || cx == g.ncx - 1) &&
      !surely_inside(__ldg(a.gxf + cx), __ldg(g.wx + cx), u, g.xsf)) {
    double x = g.gx[cx] + (double)u * (g.gx[cx + 1] - g.gx[cx]);
    act = act && x > 0 && x < g.xsize;
  }
  if ((cy == 0 || cy == g.ncy - 1) &&
      !surely_inside(__ldg(a.gyf + cy), __ldg(g.wy + cy), v, g.ysf)) {
    double y = g.gy[cy] + (double)v * (g.gy[cy + 1] - g.gy[cy]);
    act = act && y > 0 && y < g.ysize;
  }
  return act;
}

// axis factor of a staggered (half-cell) stencil: k = 0 below the cell's
// middle, 1 across it, 2 above it; 0 where the stencil does not reach
__device__ __forceinline__ float half_factor(int k, float f) {
  if (k == 0) return f < 0.5f ? 1.f - f - 0.5f : 0.f;
  if (k == 1) return 1.f - fabsf(f - 0.5f);
  return f > 0.5f ? f - 0.5f : 0.f;
}

template <int ROLE>
__device__ __forceinline__ void mode1_node(const M2NArgs &a) {
  const Grid &g = a.g;
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= g.nn) return;
  const int ix = (int)(t / g.yn), iy = (int)(t - (long)ix * g.yn);
  const int ncy = g.ncy;
  Acc cur[8], vy3[3];
#pragma unroll
  for (int q = 0; q < 8; q++) cur[q].zero();
#pragma unroll
  for (int q = 0; q < 3; q++) vy3[q].zero();
  // cells that can reach this node: dx, dy offsets of the cell from the node
  const int dx0 = ROLE == 2 ? -2 : -1, dx1 = ROLE == 3 ? 1 : 0;
  const int dy0 = ROLE == 2 ? -2 : -1, dy1 = ROLE == 3 ? 1 : 0;
  for (int dx = dx0; dx <= dx1; dx++) {
    const int cx = ix + dx;
    if (cx < 0 || cx >= g.ncx) continue;
    const float iwx = 1.f / __ldg(g.wx + cx);
    for (int dy = dy0; dy <= dy1; dy++) {
      const int cy = iy + dy;
      if (cy < 0 || cy >= ncy) continue;
      // stencil position of the node relative to the cell: a = -dx, b = -dy
      const int ax = -dx, by = -dy;
      if (ROLE == 3 && ax < 0 && by < 0) continue;  // (1, 1): no stencil reaches
      const float s1 = iwx / __ldg(g.wy + cy);
      const long c = (long)cx * ncy + cy;
      // quarter classes (2 (v > 1/2) + (u > 1/2)) that can have weight:
      // a half-cell factor k = 0 needs the lower half, k = 2 the upper
      auto ux = [](int k) { return 0xaf5 >> (4 * k) & 0xf; };
      auto vy = [](int k) { return 0xcf3 >> (4 * k) & 0xf; };
      int mask = 0xf;
      if (ROLE == 2) mask = ux(ax) & vy(by);
      if (ROLE == 3) mask = (ax >= 0 ? vy(by + 1) : 0) | (by >= 0 ? ux(ax + 1) : 0);
      const int4 qs = __ldg(a.qstart + c);
      const int qe = __ldg(a.start + c + 1);
      auto qb = [&](int q) { return q == 0 ? qs.x : q == 1 ? qs.y : q == 2 ? qs.z : q == 3 ? qs.w : qe; };
      // runs of classes with weight (one for the basic nodes, at most two)
#pragma unroll 1
      for (int q = 0; q < 4; q++) {
        if (!((mask >> q) & 1)) continue;
        const int b = qb(q);
        while (q < 3 && ((mask >> (q + 1)) & 1)) q++;
        const int e = qb(q + 1);
        if (b >= e) continue;
        // the index of the marker after next is read while this one is summed,
        // and every field of a marker at once, also of those without weight:
        // one round of memory latency per marker instead of three
        int idx1 = __ldg(a.perm + b);
#pragma unroll 1
        for (int s = b; s < e; s++) {
          const int idx = idx1;
          if (s + 1 < e) idx1 = __ldg(a.perm + s + 1);
          const float u = a.m.u_in[idx], v = a.m.v_in[idx];
          const int tt = a.m.type[idx];
          if (ROLE == 0) {
            const float mnu = a.m.mnu[idx], me = a.m.e[idx], sxy = a.m.sxy[idx];
            const float exy = a.m.exy[idx], coh = a.m.coh[idx], phi = a.m.phi[idx];
            const float ig = a.R(RK_INV_GG, tt);
            if (!marker_active(a, cx, cy, u, v)) continue;
            const float w = s1 * (ax ? u : 1.f - u) * (by ? v : 1.f - v);
            cur[0].add(mnu * w); cur[1].add(mnu * ig * w);
            cur[2].add(me * w); cur[3].add(sxy * w);
            cur[4].add(exy * w); cur[5].add(coh * w);
            cur[6].add(phi * w); cur[7].add(w);
          } else if (ROLE == 1) {
            const float T = a.m.tk[idx], kt = a.m.mkt[idx];
            const float mro = a.S.p.densimod ? a.m.mro[idx] : 0.f;
            const float bb = a.R(RK_BB, tt);
            const float ro = a.S.p.densimod ? mro : a.R(RK_RO, tt);
            if (!marker_active(a, cx, cy, u, v)) continue;
            const float w = s1 * (ax ? u : 1.f - u) * (by ? v : 1.f - v);
            cur[0].add(ro * w);
            cur[1].add(fdiv_normal(bb, 1.f - bb * (T - 298.15f)) * w);
            cur[2].add(a.R(RK_HT, tt) * w); cur[3].add(a.R(RK_CP, tt) * w);
            cur[4].add(kt * w); cur[5].add(T * w); cur[6].add(w);
          } else if (ROLE == 2) {
            const float mnu = a.m.mnu[idx], sxx = a.m.sxx[idx], exx = a.m.exx[idx];
            const float mp = a.m.p[idx], ig = a.R(RK_INV_GG, tt);
            if (!marker_active(a, cx, cy, u, v)) continue;
            const float w = s1 * half_factor(ax, u) * half_factor(by, v);
            if (w != 0.f) {
              cur[0].add(mnu * w); cur[1].add(mnu * ig * w);
              cur[2].add(sxx * w); cur[3].add(exx * w);
              cur[4].add(mp * w); cur[5].add(w);
            }
          } else {
            const float vx = a.m.vx[idx], vy = a.m.vy[idx];
            const float ro = a.S.p.densimod ? a.m.mro[idx] : a.R(RK_RO, tt);
            if (!marker_active(a, cx, cy, u, v)) continue;
            // vx node: x bilinear (ax in {0, 1}), y staggered (by + 1 in {0, 1, 2})
            if (ax >= 0) {
              const float w = s1 * (ax ? u : 1.f - u) * half_factor(by + 1, v);
              if (w != 0.f) {
                cur[0].add(vx * ro * w); cur[1].add(ro * w); cur[2].add(w);
              }
            }
            // vy node: x staggered (ax + 1), y bilinear (by in {0, 1})
            if (by >= 0) {
              const float w = s1 * half_factor(ax + 1, u) * (by ? v : 1.f - v);
              if (w != 0.f) {
                vy3[0].add(vy * ro * w); vy3[1].add(ro * w); vy3[2].add(w);
              }
            }
          }
        }
      }
    }
  }
  if (ROLE == 0) {
    node_tail<T_STRESS>(a, ix, iy, cur);
  } else if (ROLE == 1) {
    node_tail<T_THERMAL>(a, ix, iy, cur);
  } else if (ROLE == 3) {
    node_tail<T_VX>(a, ix, iy, cur);
    node_tail<T_VY>(a, ix, iy, vy3);
  } else if (ix >= 1 && iy >= 1) {  // writes centre node (ix, iy)
    const Acc nu[3] = {cur[0], cur[1], cur[5]};
    node_tail<T_CENTRE_NU>(a, ix - 1, iy - 1, nu);
    node_tail<T_CENTRE_S>(a, ix - 1, iy - 1, cur + 2);
  } else {
    // a centre node no cell has (first column or row)
    const Nodes &N = a.N;
    const long m3 = t;
    N.f(V2C_NF_SXXEN)[m3] = 0; N.f(V2C_NF_SPPEN)[m3] = 0; N.f(V2C_NF_EXXEN)[m3] = 0;
    N.f(V2C_NF_SXXE)[m3] = 0; N.f(V2C_NF_SPPE)[m3] = 0; N.f(V2C_NF_EXXE)[m3] = 0;
    N.f(V2C_NF_GD)[m3] = 0; N.f(V2C_NF_BM)[m3] = 0;
    N.f(V2C_NF_DRO)[m3] = 0; N.f(V2C_NF_DRP)[m3] = 0;
  }
}

// The four node groups in one launch, a row of blocks each: a thread walks
// its node's markers one after the other, so the kernel is latency, and the
// groups fill each other's gaps.  433 x 187 lines, 0.84 M markers: 488 us in
// four launches, 378 in one, 346 with each marker's fields read at once and
// the next one's index ahead, 118 with the edge cells' tests in FP32 where
// they are sure (surely_inside).
__global__ void __launch_bounds__(128) k_m2n_mode1(M2NArgs a) {
  after_previous();
  switch (blockIdx.y) {
    case 0: mode1_node<2>(a); break;  // most cells per node: first
    case 1: mode1_node<3>(a); break;
    case 2: mode1_node<0>(a); break;
    default: mode1_node<1>(a); break;
  }
}

// ghost copy of the state when it diffuses, interpolation.c:827-859
__global__ void k_dphis(Grid g, float *phis) {
  after_previous();
  long m3 = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (m3 >= g.nn) return;
  const int yn = g.yn, xn = g.xn;
  int m22 = (int)(m3 % yn), m11 = (int)(m3 / yn);
  float v;
  if (m11 == 0 && m22 >= 1 && m22 <= yn - 2) v = phis[m3 + yn];
  else if (m11 == xn - 1 && m22 >= 1 && m22 <= yn - 2) v = phis[m3 - yn];
  else if (m22 == 0 && m11 >= 1 && m11 <= xn - 2) v = phis[m3 + 1];
  else if (m22 == yn - 1 && m11 > 0 && m11 <= xn - 2) v = phis[m3 - 1];
  else if ((m11 == 0 || m11 == xn - 1) && (m22 == 0 || m22 == yn - 1)) v = 0.f;
  else return;
  // boundary values only read interior ones: no read-after-write hazard
  phis[m3] = v;
}

}  // namespace

cudaError_t m2n_init() {
  return cudaFuncSetAttribute(k_m2n, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(Smem));
}

void launch_m2n(const M2NArgs &a, cudaStream_t st) {
  if (a.S.p.interpolationmod == 1) {
    const unsigned nb = (unsigned)((a.g.nn + 127) / 128);
    launch_after(k_m2n_mode1, dim3(nb, 4), 128, 0, st, a);
    return;
  }
  dim3 grid((a.g.xn + a.TX - 1) / a.TX, (a.g.yn + TY - 1) / TY);
  launch_after(k_m2n, grid, NTH, sizeof(Smem), st, a);
}

void launch_dphis(const Grid &g, const Nodes &N, cudaStream_t st) {
  launch_after(k_dphis, (unsigned)((g.nn + 255) / 256), 256, 0, st, g, N.f(V2C_NF_PHIS));
}

}  // namespace v2c
