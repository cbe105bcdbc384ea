// v2c_n2m.cu -- nodes2markers (interpolation.c:929-1490) and
// moveandrotatemarkers (moveandrotatemarkers.c:1-178).
//
// nodes2markers with antidiffusion and interpolationmod 2 (k_n2m): same
// tiling as the marker2nodes sweep (see v2c_m2n.cu).  A thread gathers a
// marker's nine node fields from the four staggered stencils of
// interpolate_mechanical, updates the marker where its tile owns it, and
// leaves the quantities the antidiffusion correction scatters back (PHIS,
// SXY, EXY, ES to basic nodes, PR, SXX, EXX to the centre node, VX*MRO,
// VY*MRO and MRO to vx/vy nodes) in shared memory, where one lane per node
// row sums them per node, in sorted marker order with two-sum compensation,
// exactly as in marker2nodes.  The other settings gather without the sweep
// (k_gather): no back-scatter without antidiffusion, per-node kernels for
// the full stencils of interpolationmod 1.
//
// moveandrotatemarkers: one thread per marker, Euler or RK4 through four
// allinteri evaluations (interpolation.c:1688-1758) from per-quarter
// bilinear forms, stress rotation; new positions go to the second position
// buffer.
#include <math.h>

#include "v2c_kernels.h"
#include "v2c_rheology.cuh"

namespace v2c {

namespace {

struct Pos {
  int ix, iy;
  float X, Y;  // metres from gx[ix], gy[iy]
};

// put a position back in the cell that contains it; FP64 search if it
// crossed more than four cells
__device__ __forceinline__ void settle(const Grid &g, Pos &p, unsigned long long *stat) {
  int ix0 = p.ix, iy0 = p.iy;
  float X0 = p.X, Y0 = p.Y;
  if (!relocate(g.wx, g.ncx, p.ix, p.X, 4)) {
    double x = g.gx[ix0] + (double)X0;
    p.ix = nsearch64(g.gx, g.xn, x);
    p.X = (float)(x - g.gx[p.ix]);
    atomicAdd(stat + ST_FAR_MOVES, 1ull);
  }
  if (!relocate(g.wy, g.ncy, p.iy, p.Y, 4)) {
    double y = g.gy[iy0] + (double)Y0;
    p.iy = nsearch64(g.gy, g.yn, y);
    p.Y = (float)(y - g.gy[p.iy]);
    atomicAdd(stat + ST_FAR_MOVES, 1ull);
  }
}

// allinteri (interpolation.c:1688-1758) inside one quarter of a cell is a
// bilinear function of the position: each stencil it reads (basic nodes for
// the spin, pressure nodes for the velocities averaged in pairs, vx and vy
// nodes for the staggered velocities) keeps its nodes across the quarter,
// its weights are affine in X and Y, and the blend weight xrat is constant
// there.  k_vel_quads writes, per quarter and per quantity (VX, VY, ESP),
// the coefficients of f = c0 + c1 dX + c2 dY + c3 dX dY, with dX, dY in
// metres from the quarter's lower corner; vel_at evaluates them.  Quarter
// qx = 1 holds X >= wx/2 (allinteri: xrat and the vy stencil switch at
// X < wx/2, the pressure stencil at X > wx/2, where it is continuous).

// affine weight w = (X - A) / B of one stencil axis at the quarter's corner
// X0: w = e0 + s (X - X0)
struct Lin {
  float e0, s;
};
__device__ __forceinline__ Lin lin_w(float X0, float A, float B) {
  const float r = rcp_normal(B);
  return Lin{__fmul_rn(X0 - A, r), r};
}

// bilinear interpolation of f over nodes m3, m3+1, m3+yn, m3+yn+1 as
// c0 + c1 dX + c2 dY + c3 dX dY
__device__ __forceinline__ float4 bil_form(const float *f, long m3, long yn, Lin ex, Lin ny) {
  const float f0 = __ldg(f + m3), f1 = __ldg(f + m3 + 1), f2 = __ldg(f + m3 + yn),
              f3 = __ldg(f + m3 + yn + 1);
  const float d20 = f2 - f0, d10 = f1 - f0, D = (f3 - f2) - d10;
  float4 c;
  c.x = f0 + ex.e0 * d20 + ny.e0 * (d10 + ex.e0 * D);
  c.y = (d20 + ny.e0 * D) * ex.s;
  c.z = (d10 + ex.e0 * D) * ny.s;
  c.w = D * ex.s * ny.s;
  return c;
}

// the pair sums of allinteri (interpolation.c:1730-1745) at pressure node
// m (m has ix >= 1 and iy >= 1 on every pressure stencil)
__device__ __forceinline__ float4 bil_form_pairs(const float *v, long o1, long o2, long m3,
                                                 long yn, Lin ex, Lin ny) {
  auto P = [&](long m) { return 0.5f * (__ldg(v + m - o1) + __ldg(v + m - o2)); };
  const float f0 = P(m3), f1 = P(m3 + 1), f2 = P(m3 + yn), f3 = P(m3 + yn + 1);
  const float d20 = f2 - f0, d10 = f1 - f0, D = (f3 - f2) - d10;
  float4 c;
  c.x = f0 + ex.e0 * d20 + ny.e0 * (d10 + ex.e0 * D);
  c.y = (d20 + ny.e0 * D) * ex.s;
  c.z = (d10 + ex.e0 * D) * ny.s;
  c.w = D * ex.s * ny.s;
  return c;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ float4 blend(float4 p, float4 s, float xrat) {
  const float r = 1.f - xrat;
  return make_float4(p.x * r + s.x * xrat, p.y * r + s.y * xrat, p.z * r + s.z * xrat,
                     p.w * r + s.w * xrat);
}

// one thread per cell quarter t = 4 cell + 2 qy + qx; stencils as in
// stencil_basic / stencil_centre / stencil_vx / stencil_vy
__global__ void k_vel_quads(Grid g, Nodes N, float4 *Q) {
  after_previous();
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= (long)g.ncx * g.ncy * 4) return;
  const long c = t >> 2;
  const int qx = (int)(t & 1), qy = (int)((t >> 1) & 1);
  const int ix = (int)(c / g.ncy), iy = (int)(c - (long)ix * g.ncy);
  const Axis ax = make_axis(g.wx, g.ncx, ix, 0.f), ay = make_axis(g.wy, g.ncy, iy, 0.f);
  const float X0 = qx ? 0.5f * ax.w : 0.f, Y0 = qy ? 0.5f * ay.w : 0.f;
  const long yn = g.yn;
  // spin at basic nodes
  int mx = clampi(ix, 1, g.xn - 3), my = clampi(iy, 1, g.yn - 3);
  int kx = mx - ix, ky = my - iy;
  const float4 cE = bil_form(N.f(V2C_NF_ESP), (long)mx * yn + my, yn,
                             lin_w(X0, ax.G(kx), ax.G(kx + 1) - ax.G(kx)),
                             lin_w(Y0, ay.G(ky), ay.G(ky + 1) - ay.G(ky)));
  // velocities averaged to pressure nodes
  mx = clampi(ix + qx, 1, g.xn - 2); my = clampi(iy + qy, 1, g.yn - 2);
  kx = mx - ix; ky = my - iy;
  Lin ex = lin_w(X0, (ax.G(kx - 1) + ax.G(kx)) * 0.5f, (ax.G(kx + 1) - ax.G(kx - 1)) * 0.5f);
  Lin ny = lin_w(Y0, (ay.G(ky - 1) + ay.G(ky)) * 0.5f, (ay.G(ky + 1) - ay.G(ky - 1)) * 0.5f);
  const long mc = (long)mx * yn + my;
  const float4 cPX = bil_form_pairs(N.f(V2C_NF_VX), 1, yn + 1, mc, yn, ex, ny);
  const float4 cPY = bil_form_pairs(N.f(V2C_NF_VY), yn, yn + 1, mc, yn, ex, ny);
  // vx nodes
  mx = clampi(ix, 0, g.xn - 2); my = clampi(iy - (qy ? 0 : 1), 0, g.yn - 3);
  kx = mx - ix; ky = my - iy;
  const float4 cVX = bil_form(N.f(V2C_NF_VX), (long)mx * yn + my, yn,
                              lin_w(X0, ax.G(kx), ax.G(kx + 1) - ax.G(kx)),
                              lin_w(Y0, (ay.G(ky) + ay.G(ky + 1)) * 0.5f,
                                    (ay.G(ky + 2) - ay.G(ky)) * 0.5f));
  // vy nodes
  mx = clampi(ix - (qx ? 0 : 1), 0, g.xn - 3); my = clampi(iy, 0, g.yn - 2);
  kx = mx - ix; ky = my - iy;
  const float4 cVY = bil_form(N.f(V2C_NF_VY), (long)mx * yn + my, yn,
                              lin_w(X0, (ax.G(kx) + ax.G(kx + 1)) * 0.5f,
                                    (ax.G(kx + 2) - ax.G(kx)) * 0.5f),
                              lin_w(Y0, ay.G(ky), ay.G(ky + 1) - ay.G(ky)));
  // staggered weight: 2/3, or 1 in the outer half of a boundary cell
  float xrat = 2.f / 3.f;
  if ((ix == 0 && !qx) || (ix == g.ncx - 1 && qx) || (iy == 0 && !qy) ||
      (iy == g.ncy - 1 && qy))
    xrat = 1.f;
  float4 *o = Q + t * 3;
  o[0] = blend(cPX, cVX, xrat);
  o[1] = blend(cPY, cVY, xrat);
  o[2] = cE;
}

// allinteri at a cell-local position: velocity and spin from the quarter's
// forms (positions outside the model are clamped onto its boundary first)
__device__ __forceinline__ void vel_at(const Grid &g, const float4 *Q, Pos p, float &VX,
                                       float &VY, float &ESP) {
  const float wx = __ldg(g.wx + p.ix), wy = __ldg(g.wy + p.iy);
  if (p.ix == 0 && p.X < 0.f) p.X = 0.f;
  if (p.ix == g.ncx - 1 && p.X > wx) p.X = wx;
  if (p.iy == 0 && p.Y < 0.f) p.Y = 0.f;
  if (p.iy == g.ncy - 1 && p.Y > wy) p.Y = wy;
  const float hx = 0.5f * wx, hy = 0.5f * wy;
  const int qx = p.X >= hx, qy = p.Y >= hy;
  const float dX = qx ? p.X - hx : p.X, dY = qy ? p.Y - hy : p.Y;
  const float4 *c = Q + (((long)p.ix * g.ncy + p.iy) * 4 + qy * 2 + qx) * 3;
  const float4 a = __ldg(c), b = __ldg(c + 1), e = __ldg(c + 2);
  VX = fmaf(dY, fmaf(a.w, dX, a.z), fmaf(a.y, dX, a.x));
  VY = fmaf(dY, fmaf(b.w, dX, b.z), fmaf(b.y, dX, b.x));
  ESP = fmaf(dY, fmaf(e.w, dX, e.z), fmaf(e.y, dX, e.x));
}

// Marker values without antidiffusion (interpolation.c:985-1011): the previous
// node fields interpolated for a marker's first values, afterwards the change
// of the node fields since then, interpolated as one field of node differences
// -- the same bilinear form, so the same value in exact arithmetic, but the
// FP32 node differences of two states that agree in their leading digits are
// exact where the separate interpolations would each round at the size of the
// field.
struct Plain {
  float phi, exx, exy, sxx, sxy, p, vx, vy, e;
};
// a marker that has just come in: the previous node values themselves
__device__ __forceinline__ void plain_values(const Grid &g, const Nodes &N, Axis ax, Axis ay,
                                             float uc, float vc, Plain &o) {
  const long yn = g.yn;
  float e, n;
  long m3 = stencil_basic(g, ax, ay, e, n);
  o.exy = bil(N.f(V2C_NF_EXYE), m3, yn, e, n);
  o.sxy = bil(N.f(V2C_NF_SXYE), m3, yn, e, n);
  o.e = bil(N.f(V2C_NF_PE), m3, yn, e, n);
  o.phi = bil(N.f(V2C_NF_PHIS), m3, yn, e, n);
  m3 = stencil_centre(g, ax, ay, uc > 0.5f, vc > 0.5f, e, n);
  o.exx = bil(N.f(V2C_NF_EXXE), m3, yn, e, n);
  o.sxx = bil(N.f(V2C_NF_SXXE), m3, yn, e, n);
  o.p = bil(N.f(V2C_NF_SPPE), m3, yn, e, n);
  m3 = stencil_vx(g, ax, ay, vc < 0.5f, g.xn - 2, e, n);
  o.vx = bil(N.f(V2C_NF_MVX), m3, yn, e, n);
  m3 = stencil_vy(g, ax, ay, uc < 0.5f, g.yn - 2, e, n);
  o.vy = bil(N.f(V2C_NF_MVY), m3, yn, e, n);
}

// The nine differences of a node side by side: a marker's change is then 16
// reads instead of 72.  811 x 309 lines, 4.5 M markers: 215 -> 151 us, this
// pass over the nodes included; 301 x 101: 26 and 26, 51 x 21: 11.2 and 11.6.
struct PlainNode {
  float4 basic;   // EXY, SXY, PES, PHIS_IT, each minus its previous value
  float4 centre;  // EXX, SXX, PR
  float2 vel;     // VX, VY
  float2 pad;
};
static_assert(sizeof(PlainNode) * 16 <= sizeof(float4) * QUAD_FLOAT4 * 9,
              "the differences of the smallest grid's nodes fit its cells' forms");
__global__ void __launch_bounds__(256) k_plain_nodes(Nodes N, long nn, PlainNode *D) {
  after_previous();
  const long m = blockIdx.x * 256l + threadIdx.x;
  if (m >= nn) return;
  auto d = [&](int f, int g) { return N.f(f)[m] - N.f(g)[m]; };
  D[m].basic = make_float4(d(V2C_NF_EXY, V2C_NF_EXYE), d(V2C_NF_SXY, V2C_NF_SXYE),
                           d(V2C_NF_PES, V2C_NF_PE), d(V2C_NF_PHIS_IT, V2C_NF_PHIS));
  D[m].centre = make_float4(d(V2C_NF_EXX, V2C_NF_EXXE), d(V2C_NF_SXX, V2C_NF_SXXE),
                            d(V2C_NF_PR, V2C_NF_SPPE), 0.f);
  D[m].vel = make_float2(d(V2C_NF_VX, V2C_NF_MVX), d(V2C_NF_VY, V2C_NF_MVY));
}
__device__ __forceinline__ void plain_change(const Grid &g, const PlainNode *D, Axis ax, Axis ay,
                                             float uc, float vc, Plain &o) {
  const long yn = g.yn;
  float e, n;
  auto mix = [&](float a, float b, float c, float d) {
    const float d0 = (1.f - e) * (1.f - n), d1 = (1.f - e) * n, d2 = e * (1.f - n), d3 = e * n;
    return d0 * a + d1 * b + d2 * c + d3 * d;
  };
  auto mix4 = [&](const float4 &a, const float4 &b, const float4 &c, const float4 &d) {
    return make_float4(mix(a.x, b.x, c.x, d.x), mix(a.y, b.y, c.y, d.y), mix(a.z, b.z, c.z, d.z),
                       mix(a.w, b.w, c.w, d.w));
  };
  const PlainNode *p = D + stencil_basic(g, ax, ay, e, n);
  const float4 B = mix4(__ldg(&p[0].basic), __ldg(&p[1].basic), __ldg(&p[yn].basic),
                        __ldg(&p[yn + 1].basic));
  o.exy = B.x; o.sxy = B.y; o.e = B.z; o.phi = B.w;
  p = D + stencil_centre(g, ax, ay, uc > 0.5f, vc > 0.5f, e, n);
  const float4 C = mix4(__ldg(&p[0].centre), __ldg(&p[1].centre), __ldg(&p[yn].centre),
                        __ldg(&p[yn + 1].centre));
  o.exx = C.x; o.sxx = C.y; o.p = C.z;
  p = D + stencil_vx(g, ax, ay, vc < 0.5f, g.xn - 2, e, n);
  o.vx = mix(__ldg(&p[0].vel.x), __ldg(&p[1].vel.x), __ldg(&p[yn].vel.x), __ldg(&p[yn + 1].vel.x));
  p = D + stencil_vy(g, ax, ay, uc < 0.5f, g.yn - 2, e, n);
  o.vy = mix(__ldg(&p[0].vel.y), __ldg(&p[1].vel.y), __ldg(&p[yn].vel.y), __ldg(&p[yn + 1].vel.y));
}

// ------------------------------------------------------------ the sweep
constexpr int TY = 32;
constexpr int NTH = 8 * 32;
// markers staged at once: 33 cells of 23, in the 56 KB that four resident
// CTAs leave each other
constexpr int CHUNK = 768;
constexpr int SLOTS = CHUNK + CHUNK / 16;
// the marker at position p of a chunk, in slot p + p / 16 (see v2c_m2n.cu)
__device__ __forceinline__ int slot_of(int p) { return p + (p >> 4); }

// staged quantities, in pairs for packed FP32 sums
enum { Q_UV = 0, Q_PHSXY, Q_EXYES, Q_PRSXX, Q_EXXMRO, Q_VXVY, Q_N };

// The node columns ci-1 .. ci+2 that the markers of cell column ci read, in
// a ring of five (the fifth arrives for the next column while this one is
// gathered), rows j0-2 .. j0+33.
constexpr int RING = 5, ROWS = TY + 4;
struct NodeColumn {
  float4 basic[ROWS];   // PHIS_IT, SXY, EXY, PES
  float4 centre[ROWS];  // PR, SXX, EXX
  float2 vel[ROWS];     // VX, VY
};
// One axis of a stencil: the weight (position - a) r of its second line, and
// where its lines are: in y, the first line relative to the marker's cell
// row; in x, the byte offsets of the two node columns in the ring.
struct Side {
  float a, r;
  int o0, o1;
};
enum { S_BASIC = 0, S_CLO, S_CHI, S_LINE, S_HALF, S_HALFLO, S_N };
struct Smem {
  float2 q[Q_N][SLOTS];
  int32_t idx[CHUNK];
  NodeColumn ring[RING];
  Side x[2][S_N], y[TY + 1][S_N];  // x: this column's and the next's
};

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// The weights of one axis for a marker in cell i of it, by stencil: basic
// nodes, pressure nodes with the marker in the lower or upper half, lines
// (vx in x, vy in y), half lines (vy in x, vx in y) with the marker in the
// upper or lower half -- the four stencils of stencil_basic, stencil_centre,
// stencil_vx and stencil_vy, whose first line and divisor depend on the cell
// and the half only.
__device__ __forceinline__ void axis_side(const float *w, int nc, int n, int i, int which,
                                          bool x, Side &s) {
  const Axis ax = make_axis(w, nc, i, 0.f);
  int m;
  float A, B;
  if (which == S_BASIC || which == S_LINE) {
    m = which == S_BASIC ? min(max(i, 1), n - 3) : i;
    const int q = m - i;
    A = ax.G(q);
    B = ax.G(q + 1) - ax.G(q);
  } else if (which == S_CLO || which == S_CHI) {
    m = max(min(i + (which == S_CHI), n - 2), 1);
    const int q = m - i;
    A = (ax.G(q - 1) + ax.G(q)) * 0.5f;
    B = (ax.G(q + 1) - ax.G(q - 1)) * 0.5f;
  } else {
    m = min(max(i - (which == S_HALFLO), 0), n - 3);
    const int q = m - i;
    A = (ax.G(q) + ax.G(q + 1)) * 0.5f;
    B = (ax.G(q + 2) - ax.G(q)) * 0.5f;
  }
  s.a = A;
  s.r = __fdividef(1.f, B);
  s.o0 = x ? m % RING * (int)sizeof(NodeColumn) : m - i;
  s.o1 = x ? (m + 1) % RING * (int)sizeof(NodeColumn) : 0;
}

// Start copying node column c (rows r0 .. r0+ROWS-1) to its place in the ring
__device__ __forceinline__ void load_column(const N2MArgs &a, Smem &sm, int c, int r0, int tid) {
  if (c < 0 || c >= a.g.xn) return;
  NodeColumn &R = sm.ring[c % RING];
  const long m0 = (long)c * a.g.yn + r0;
  const Nodes &N = a.N;
#pragma unroll 1
  for (int t = tid; t < ROWS * 9; t += NTH) {
    const int f = t / ROWS, r = t - f * ROWS;
    if (r0 + r < 0 || r0 + r >= a.g.yn) continue;
    static const int field[9] = {V2C_NF_PHIS_IT, V2C_NF_SXY, V2C_NF_EXY, V2C_NF_PES, V2C_NF_PR,
                                 V2C_NF_SXX, V2C_NF_EXX, V2C_NF_VX, V2C_NF_VY};
    float *dst = f < 4 ? &R.basic[r].x + f : f < 7 ? &R.centre[r].x + (f - 4) : &R.vel[r].x + (f - 7);
    cp_async4(dst, N.f(field[f]) + m0 + r);
  }
}

// Ahead of the chunk at sorted positions [b, e): its sort indices, and the
// L2 lines of what the gather reads of its markers
__device__ __forceinline__ void start_chunk(const N2MArgs &a, Smem &sm, int b, int e, int tid) {
#pragma unroll 1
  for (int s = b + tid; s < e; s += NTH) cp_async4(&sm.idx[s - b], a.perm + s);
  const int s = b + 32 * (tid & 31);
  if (s >= e) return;
  switch (tid >> 5) {
    case 0: prefetch_l2(a.m.cell_in + s); break;
    case 1: prefetch_l2(a.m.u_in + s); break;
    case 2: prefetch_l2(a.m.v_in + s); break;
    case 3: prefetch_l2(a.m.tk + s); break;
    case 4: if ((tid & 3) == 0) prefetch_l2(a.m.type + s); break;
  }
}

// bilinear interpolation from node values (v2c_rheology.cuh's bil)
__device__ __forceinline__ float bil_of(const float (&d)[4], float f0, float f1, float f2,
                                        float f3) {
  return d[0] * f0 + d[1] * f1 + d[2] * f2 + d[3] * f3;
}
__device__ __forceinline__ void weights_of(float e, float n, float (&d)[4]) {
  d[0] = (1.f - e) * (1.f - n); d[1] = (1.f - e) * n; d[2] = e * (1.f - n); d[3] = e * n;
}

// Gather of the chunk's marker at position p (array index i) of cell column
// ci: interpolate_mechanical and the marker update of nodes2markers
// (interpolation.c:943-984); what the back-scatter sums goes to its slot.
__device__ __forceinline__ void gather_marker(const N2MArgs &a, Smem &sm, int ci, int jlo, int r0,
                                              int i0, int j0, int p, int i, int c, float u,
                                              float v, int t, float tk) {
  const Grid &g = a.g;
  const int iy = c - ci * g.ncy;
  const bool owned = ci >= i0 && iy >= j0;
  // of the halo column only the right halves reach a node of this tile, of
  // the halo row only the bottom halves
  if ((ci < i0 && !(u > 0.5f)) || (iy < j0 && !(v > 0.5f))) return;
  // interpolate_mechanical clamps the point into the model first
  float uc = u, vc = v;
  if (ci == 0 && uc < 0.f) uc = 0.f;
  if (ci == g.ncx - 1 && uc > 1.f) uc = 1.f;
  if (iy == 0 && vc < 0.f) vc = 0.f;
  if (iy == g.ncy - 1 && vc > 1.f) vc = 1.f;
  const float X = __fmul_rn(uc, __ldg(g.wx + ci)), Y = __fmul_rn(vc, __ldg(g.wy + iy));
  const Side *sx = sm.x[ci & 1], *sy = sm.y[iy - jlo];
  const char *ring = reinterpret_cast<const char *>(sm.ring);
  const int row = iy - r0;
  float d[4];
  // the weights of a stencil, and its first node row in its two columns
  auto corner = [&](int hx, int hy, const NodeColumn *&c0, const NodeColumn *&c1) {
    const Side A = sx[hx], B = sy[hy];
    weights_of((X - A.a) * A.r, (Y - B.a) * B.r, d);
    c0 = reinterpret_cast<const NodeColumn *>(ring + A.o0);
    c1 = reinterpret_cast<const NodeColumn *>(ring + A.o1);
    return row + B.o0;
  };
  const NodeColumn *c0, *c1;
  int r = corner(S_BASIC, S_BASIC, c0, c1);
  float4 f0 = c0->basic[r], f1 = c0->basic[r + 1], f2 = c1->basic[r], f3 = c1->basic[r + 1];
  const float PHIS = bil_of(d, f0.x, f1.x, f2.x, f3.x), SXY = bil_of(d, f0.y, f1.y, f2.y, f3.y);
  const float EXY = bil_of(d, f0.z, f1.z, f2.z, f3.z), ES = bil_of(d, f0.w, f1.w, f2.w, f3.w);
  r = corner(uc > 0.5f ? S_CHI : S_CLO, vc > 0.5f ? S_CHI : S_CLO, c0, c1);
  f0 = c0->centre[r]; f1 = c0->centre[r + 1]; f2 = c1->centre[r]; f3 = c1->centre[r + 1];
  const float PR = bil_of(d, f0.x, f1.x, f2.x, f3.x), SXX = bil_of(d, f0.y, f1.y, f2.y, f3.y);
  const float EXX = bil_of(d, f0.z, f1.z, f2.z, f3.z);
  r = corner(S_LINE, vc < 0.5f ? S_HALFLO : S_HALF, c0, c1);
  const float VX = bil_of(d, c0->vel[r].x, c0->vel[r + 1].x, c1->vel[r].x, c1->vel[r + 1].x);
  r = corner(uc < 0.5f ? S_HALFLO : S_HALF, S_LINE, c0, c1);
  const float VY = bil_of(d, c0->vel[r].y, c0->vel[r + 1].y, c1->vel[r].y, c1->vel[r + 1].y);
  const int q = slot_of(p);
  sm.q[Q_UV][q] = make_float2(uc, vc);
  sm.q[Q_PHSXY][q] = make_float2(PHIS, SXY);
  sm.q[Q_EXYES][q] = make_float2(EXY, ES);
  sm.q[Q_PRSXX][q] = make_float2(PR, SXX);
  sm.q[Q_EXXMRO][q] = make_float2(EXX, a.R(RK_RO, t));
  sm.q[Q_VXVY][q] = make_float2(VX, VY);
  if (!owned || t >= 50) return;
  // marker update: strictly inside with no temperature yet, or in the grid
  const bool in_strict = (ci > 0 || u > 0.f) && (ci < g.ncx - 1 || u < 1.f) &&
                         (iy > 0 || v > 0.f) && (iy < g.ncy - 1 || v < 1.f);
  const bool in_grid = (ci > 0 || u >= 0.f) && (ci < g.ncx - 1 || u <= 1.f) &&
                       (iy > 0 || v >= 0.f) && (iy < g.ncy - 1 || v <= 1.f);
  if (tk <= 0.f ? in_strict : (in_grid && tk > 0.f)) {
    a.m.phi[i] = PHIS; a.m.exx[i] = EXX; a.m.exy[i] = EXY;
    a.m.sxx[i] = SXX; a.m.sxy[i] = SXY; a.m.p[i] = PR;
    a.m.vx[i] = VX; a.m.vy[i] = VY; a.m.e[i] = ES;
    if (tk <= 0.f && !a.S.p.tempmod) {
      a.m.tk[i] = a.S.eps2_f;
      a.m.tk_lo[i] = a.S.eps2_lo;
    }
  }
}

// Back-scatter lists of one lane: two runs of sorted positions, walked as
// one list (see v2c_m2n.cu)
struct Runs {
  int p, n1, n, jump;
};
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

// Warps 0, 1 sum the basic nodes of even and odd node columns, warp 2 the
// centre nodes, warp 3 vy, warps 4, 5 vx of even and odd node columns; all
// eight gather.
// C4 (80 M markers, 20 per cell): 4.77 -> 2.37 ms against four warps of
// 384-marker chunks gathering through L1; a 1001 x 401-line model of 20 (16)
// per cell 0.606 -> 0.277 (0.589 -> 0.237) ms, 301 x 101 lines 98 -> 33 us,
// 51 x 21 lines 52 -> 16 us.  Bound by instruction issue (64 % active, 28
// warp instructions per marker) and shared-memory reads.  The node values
// come from shared memory (16 reads per marker instead of 36 through L1), a
// stencil's line offsets and reciprocals from tables per cell row and
// column, and the temperature is written only where it changes.  Halo
// markers that reach no node of the tile are not gathered.
__global__ void __launch_bounds__(NTH, 4) k_n2m(N2MArgs a) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  const Grid &g = a.g;
  const Nodes &N = a.N;
  const int tid = threadIdx.x, warp = tid >> 5, jl = tid & 31;
  const int i0 = blockIdx.x * a.TX, j0 = blockIdx.y * TY;
  const int j = j0 + jl;
  const bool jvalid = j < g.yn;
  const int ncy = g.ncy;
  const int ci_end = min(i0 + a.TX, g.xn);
  const int jlo = max(j0 - 1, 0), jhi = min(j0 + TY - 1, ncy - 1), r0 = jlo - 1;
  const int c_end = min(ci_end, g.ncx), c0 = max(i0 - 1, 0);

  // row weights, the first columns' nodes, column weights and chunk
  for (int t = tid; t < (jhi - jlo + 1) * S_N; t += NTH)
    axis_side(g.wy, ncy, g.yn, jlo + t / S_N, t % S_N, false, sm.y[t / S_N][t % S_N]);
  if (c0 < c_end) {
    for (int c = c0 - 1; c <= c0 + 2; c++) load_column(a, sm, c, r0, tid);
    if (tid < S_N) axis_side(g.wx, g.ncx, g.xn, c0, tid, true, sm.x[c0 & 1][tid]);
    const int b = __ldg(a.start + (long)c0 * ncy + jlo);
    start_chunk(a, sm, b, min(b + CHUNK, __ldg(a.start + (long)c0 * ncy + jhi + 1)), tid);
  }

  // basic: PHIS, SXY | EXY, ES and w   centre: PR, SXX | EXX, w
  // vx, vy: v*MRO, MRO and w
  Acc2 acc[2];
  Acc wt;
  acc[0].zero(); acc[1].zero(); wt.zero();

  for (int ci = c0; ci < ci_end; ++ci) {
    const bool owned = ci >= i0, next = ci + 1 < ci_end;
    // warps 0, 1, 4, 5: node column ci is this warp's
    const bool mine = ((ci ^ warp) & 1) == 0;
    if (ci < g.ncx) {
      const long cb = (long)ci * ncy;
      const int seg_b = __ldg(a.start + cb + jlo), seg_e = __ldg(a.start + cb + jhi + 1);
      const int nseg_b = ci + 1 < c_end ? __ldg(a.start + cb + ncy + jlo) : 0;
      const int nseg_e = ci + 1 < c_end ? __ldg(a.start + cb + ncy + jhi + 1) : 0;
      // quarter class starts of cells (ci, j-1) (lower) and (ci, j) (upper)
      int4 ql = make_int4(0, 0, 0, 0), qu = make_int4(0, 0, 0, 0);
      int lo_e = 0, up_e = 0;
      float s1lo = 0.f, s1up = 0.f;
      if (warp < 6) {
        const float iwx = 1.f / __ldg(g.wx + ci);
        if (jvalid && j - 1 >= 0 && j - 1 <= ncy - 1) {
          ql = __ldg(a.qstart + cb + j - 1);
          lo_e = __ldg(a.start + cb + j);
          s1lo = iwx / __ldg(g.wy + j - 1);
        }
        if (jvalid && j <= ncy - 1) {
          qu = __ldg(a.qstart + cb + j);
          up_e = __ldg(a.start + cb + j + 1);
          s1up = iwx / __ldg(g.wy + j);
        }
      }
      if (seg_b == seg_e) start_chunk(a, sm, nseg_b, min(nseg_b + CHUNK, nseg_e), tid);
      for (int cs = seg_b; cs < seg_e; cs += CHUNK) {
        const int ce = min(cs + CHUNK, seg_e);
        cp_async_wait_all();
        __syncthreads();  // indices and nodes are there, the previous chunk is summed
        {
          // each thread's next marker is read while the current one is gathered
          int p = tid, i = 0, c = 0, t = 0;
          float u = 0.f, v = 0.f, tk = 0.f;
          auto read = [&]() {
            if (p >= ce - cs) return;
            i = sm.idx[p];
            c = a.m.cell_in[i]; u = a.m.u_in[i]; v = a.m.v_in[i];
            t = a.m.type[i]; tk = a.m.tk[i];
          };
          read();
#pragma unroll 1
          while (p < ce - cs) {
            const int p_ = p, i_ = i, c_ = c, t_ = t;
            const float u_ = u, v_ = v, tk_ = tk;
            p += NTH;
            read();
            gather_marker(a, sm, ci, jlo, r0, i0, j0, p_, i_, c_, u_, v_, t_, tk_);
          }
        }
        __syncthreads();
        {
          const int nb = ce == seg_e ? nseg_b : ce;
          start_chunk(a, sm, nb, min(nb + CHUNK, ce == seg_e ? nseg_e : seg_e), tid);
        }
        if (warp < 2) {
          // left halves (of node column ci), right halves (of ci+1) of cell
          // (ci, j-1), bottom quarter, and cell (ci, j), top quarter
          if (mine ? owned : next) {
            const Runs R = mine ? two_runs(cs, ce, ql.z, ql.w, qu.x, qu.y)
                                : two_runs(cs, ce, ql.w, lo_e, qu.y, qu.z);
            const float s1 = mine ? -s1lo : s1lo, s2 = mine ? s1up : -s1up;
            FOR_RUNS(R) {
              const int q = slot_of(p);
              const float2 uv = sm.q[Q_UV][q], f = sm.q[Q_PHSXY][q], h = sm.q[Q_EXYES][q];
              const float w = (i_ < R.n1 ? s1 : s2) * fmaf(2.f, uv.x, -1.f) * fmaf(2.f, uv.y, -1.f);
              if (w > 0.f) {
                acc[0].add(mul_w(f.x, f.y, w));
                acc[1].add(mul_w(h.x, h.y, w));
                wt.add(w);
              }
            }
          }
        } else if (warp == 2) {
          // the whole cell (ci, j) to its centre node
          if (owned) {
            const Runs R = two_runs(cs, ce, qu.x, up_e, 0, 0);
#pragma unroll 1
            for (int k = 0, p = R.p; k < R.n; ++k, ++p) {
              const int q = slot_of(p);
              const float2 uv = sm.q[Q_UV][q], f = sm.q[Q_PRSXX][q];
              const float ex = sm.q[Q_EXXMRO][q].x;
              const float w = s1up * tent(uv.x) * tent(uv.y);
              acc[0].add(mul_w(f.x, f.y, w));
              acc[1].add(pack2(__fmul_rn(ex, w), w));
            }
          }
        } else if (warp == 3) {
          // vy node (ci, j) from v > 1/2 of cell (ci, j-1) (classes 2, 3) and
          // v < 1/2 of cell (ci, j) (classes 0, 1)
          if (owned) {
            const Runs R = two_runs(cs, ce, ql.z, lo_e, qu.x, qu.z);
            FOR_RUNS(R) {
              const int q = slot_of(p);
              const float2 uv = sm.q[Q_UV][q];
              const float vy = sm.q[Q_VXVY][q].y, mro = sm.q[Q_EXXMRO][q].y;
              const bool lo = i_ < R.n1;
              if (lo || uv.y < 0.5f) {
                const float w = (lo ? s1lo : s1up) * (1.f - fabsf(uv.x - 0.5f)) *
                                (lo ? uv.y : 1.f - uv.y);
                acc[0].add(mul_w(__fmul_rn(vy, mro), mro, w));
                wt.add(w);
              }
            }
          }
        } else if (warp == 4 || warp == 5) {
          // vx node (ci, j) from u < 1/2 (classes 0, 2), (ci+1, j) from
          // u > 1/2 (classes 1, 3)
          if (mine ? owned : next) {
            const Runs R = mine ? two_runs(cs, ce, qu.x, qu.y, qu.z, qu.w)
                                : two_runs(cs, ce, qu.y, qu.z, qu.w, up_e);
            FOR_RUNS(R) {
              const int q = slot_of(p);
              const float2 uv = sm.q[Q_UV][q];
              const float vx = sm.q[Q_VXVY][q].x, mro = sm.q[Q_EXXMRO][q].y;
              if (!mine || uv.x < 0.5f) {
                const float w = s1up * (mine ? 1.f - uv.x : uv.x) * (1.f - fabsf(uv.y - 0.5f));
                acc[0].add(mul_w(__fmul_rn(vx, mro), mro, w));
                wt.add(w);
              }
            }
          }
        }
      }
      // for the next column: its weights and the node column it adds
      if (ci + 1 < c_end) {
        if (warp == 7 && jl < S_N)
          axis_side(g.wx, g.ncx, g.xn, ci + 1, jl, true, sm.x[(ci + 1) & 1][jl]);
        load_column(a, sm, ci + 3, r0, tid);
      }
    }

    // ----------------------------------------------- sums and normalisation
    if ((warp < 2 || warp >= 4) && !mine) continue;
    if (owned && jvalid && warp < 6) {
      const long m3 = (long)ci * g.yn + j;
      Acc x, y, z, w;
      acc[0].split(x, y);
      if (warp < 2) {
        acc[1].split(z, w);
        const float ph = x.value(), sy = y.value(), ey = z.value(), es = w.value();
        const float sw = wt.value();
        N.f(V2C_NF_PHISUM)[m3] = ph; N.f(V2C_NF_SXYSUM)[m3] = sy;
        N.f(V2C_NF_EXYSUM)[m3] = ey; N.f(V2C_NF_ESUM)[m3] = es; N.f(V2C_NF_WTPHISUM)[m3] = sw;
        if (sw != 0.f && ci >= 1 && j >= 1 && ci < g.xn - 1 && j < g.yn - 1) {
          N.f(V2C_NF_PHIE)[m3] = __fdividef(ph, sw); N.f(V2C_NF_SXYEE)[m3] = __fdividef(sy, sw);
          N.f(V2C_NF_EXYEE)[m3] = __fdividef(ey, sw); N.f(V2C_NF_PEE)[m3] = __fdividef(es, sw);
        }
      } else if (warp == 2) {
        acc[1].split(z, w);
        if (ci < g.ncx && j < ncy) {
          const long mc = m3 + g.yn + 1;
          const float ps = x.value(), sx = y.value(), ex = z.value(), sw = w.value();
          N.f(V2C_NF_PSUM)[mc] = ps; N.f(V2C_NF_SXXSUM)[mc] = sx;
          N.f(V2C_NF_EXXSUM)[mc] = ex; N.f(V2C_NF_WTSXXSUM)[mc] = sw;
          if (sw != 0.f) {
            N.f(V2C_NF_SPPEE)[mc] = __fdividef(ps, sw); N.f(V2C_NF_SXXEE)[mc] = __fdividef(sx, sw);
            N.f(V2C_NF_EXXEE)[mc] = __fdividef(ex, sw);
          }
        }
        if (ci == 0 || j == 0) {
          N.f(V2C_NF_PSUM)[m3] = 0; N.f(V2C_NF_SXXSUM)[m3] = 0;
          N.f(V2C_NF_EXXSUM)[m3] = 0; N.f(V2C_NF_WTSXXSUM)[m3] = 0;
        }
      } else {
        const bool X = warp != 3;
        const float vs = x.value(), mr = y.value(), sw = wt.value();
        N.f(X ? V2C_NF_VXSUM : V2C_NF_VYSUM)[m3] = vs;
        N.f(X ? V2C_NF_MRX0 : V2C_NF_MRY0)[m3] = mr;
        N.f(X ? V2C_NF_WTVXSUM : V2C_NF_WTVYSUM)[m3] = sw;
        if (sw != 0.f) N.f(X ? V2C_NF_MVXE : V2C_NF_MVYE)[m3] = __fdividef(vs, mr);
      }
    }
    acc[0].zero(); acc[1].zero(); wt.zero();
  }
}

// ------------------------------------------------- gather without a sweep
// nodes2markers where no tile sums are formed: PLAIN, no antidiffusion (no
// back-scatter); BS, interpolationmod 1 (each marker's back-scatter payload
// goes to a.bs for the per-node kernel below).  One thread per marker, in
// sorted order; bound by the latency of its node reads, so 6 resident CTAs
// (811 x 309 lines, 4.5 M markers, PLAIN before plain_change: 215 us, 235 at
// the registers the compiler takes by itself, 288 at 4 CTAs; BS, 433 x 187 lines: 121 -> 100
// us against the chunked sweep).
template <bool BS, bool PLAIN>
__global__ void __launch_bounds__(256, 6) k_gather(N2MArgs a) {
  after_previous();
  const Grid &g = a.g;
  const Nodes &N = a.N;
  const v2c_params &P = a.S.p;
  const long yn = g.yn;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  const int idx = __ldg(a.perm + s);
  const int c = a.m.cell_in[idx];
  int ix, iy;
  g.cell_at(c, ix, iy);
  const float u = a.m.u_in[idx], v = a.m.v_in[idx];
  const int t = a.m.type[idx];
  // interpolate_mechanical clamps the point into the model first
  float uc = u, vc = v;
  if (ix == 0 && uc < 0.f) uc = 0.f;
  if (ix == g.ncx - 1 && uc > 1.f) uc = 1.f;
  if (iy == 0 && vc < 0.f) vc = 0.f;
  if (iy == g.ncy - 1 && vc > 1.f) vc = 1.f;
  const float wxc = __ldg(g.wx + ix), wyc = __ldg(g.wy + iy);
  const Axis ax = make_axis(g.wx, g.ncx, ix, uc * wxc);
  const Axis ay = make_axis(g.wy, g.ncy, iy, vc * wyc);
  float EXY = 0.f, SXY = 0.f, ES = 0.f, PHIS = 0.f, EXX = 0.f, SXX = 0.f, PR = 0.f;
  float VX = 0.f, VY = 0.f;
  if (!PLAIN) {
    float eb, nb, ec, ncc, e, n;
    const long mb = stencil_basic(g, ax, ay, eb, nb);
    EXY = bil(N.f(V2C_NF_EXY), mb, yn, eb, nb);
    SXY = bil(N.f(V2C_NF_SXY), mb, yn, eb, nb);
    ES = bil(N.f(V2C_NF_PES), mb, yn, eb, nb);
    PHIS = bil(N.f(V2C_NF_PHIS_IT), mb, yn, eb, nb);
    const long mc = stencil_centre(g, ax, ay, uc > 0.5f, vc > 0.5f, ec, ncc);
    EXX = bil(N.f(V2C_NF_EXX), mc, yn, ec, ncc);
    SXX = bil(N.f(V2C_NF_SXX), mc, yn, ec, ncc);
    PR = bil(N.f(V2C_NF_PR), mc, yn, ec, ncc);
    long m3 = stencil_vx(g, ax, ay, vc < 0.5f, g.xn - 2, e, n);
    VX = bil(N.f(V2C_NF_VX), m3, yn, e, n);
    m3 = stencil_vy(g, ax, ay, uc < 0.5f, g.yn - 2, e, n);
    VY = bil(N.f(V2C_NF_VY), m3, yn, e, n);
  }
  if (BS) {
    const long n = a.n;
    a.bs[BS_U * n + s] = uc; a.bs[BS_V * n + s] = vc;
    a.bs[BS_PHIS * n + s] = PHIS; a.bs[BS_SXY * n + s] = SXY;
    a.bs[BS_EXY * n + s] = EXY; a.bs[BS_ES * n + s] = ES;
    a.bs[BS_PR * n + s] = PR; a.bs[BS_SXX * n + s] = SXX;
    a.bs[BS_EXX * n + s] = EXX;
  }
  // ------------------------------------- marker update (:943-1011)
  if (t >= 50) return;
  const bool in_strict = (ix > 0 || u > 0.f) && (ix < g.ncx - 1 || u < 1.f) &&
                         (iy > 0 || v > 0.f) && (iy < g.ncy - 1 || v < 1.f);
  const bool in_grid = (ix > 0 || u >= 0.f) && (ix < g.ncx - 1 || u <= 1.f) &&
                       (iy > 0 || v >= 0.f) && (iy < g.ncy - 1 || v <= 1.f);
  float tk = a.m.tk[idx];
  // PLAIN: the marker's own values plus the change of the node fields; with
  // antidiffusion an updated marker takes all nine from the nodes
  float phi = PHIS, mexx = EXX, mexy = EXY, msxx = SXX, msxy = SXY, mp = PR, mvx = VX, mvy = VY;
  float me = ES;
  if (PLAIN) {
    phi = a.m.phi[idx]; mexx = a.m.exx[idx]; mexy = a.m.exy[idx];
    msxx = a.m.sxx[idx]; msxy = a.m.sxy[idx]; mp = a.m.p[idx];
    mvx = a.m.vx[idx]; mvy = a.m.vy[idx]; me = a.m.e[idx];
  }
  bool changed = false;
  if (in_strict && tk <= 0.f) {
    if (PLAIN) {
      Plain o;
      plain_values(g, N, ax, ay, uc, vc, o);
      msxx = o.sxx; msxy = o.sxy; mp = o.p; mexx = o.exx; mexy = o.exy;
      mvx = o.vx; mvy = o.vy; phi = o.phi; me = o.e;
    }
    if (!P.tempmod) {
      tk = a.S.eps2_f;
      a.m.tk[idx] = tk;
      a.m.tk_lo[idx] = a.S.eps2_lo;
    }
    changed = true;
  }
  if (in_grid && tk > 0.f) {
    if (PLAIN) {
      Plain o;
      plain_change(g, reinterpret_cast<const PlainNode *>(a.quad), ax, ay, uc, vc, o);
      phi += o.phi; mexx += o.exx; mexy += o.exy;
      msxx += o.sxx; msxy += o.sxy; mp += o.p;
      mvx += o.vx; mvy += o.vy; me += o.e;
    }
    changed = true;
  }
  if (changed) {
    a.m.phi[idx] = phi; a.m.exx[idx] = mexx; a.m.exy[idx] = mexy;
    a.m.sxx[idx] = msxx; a.m.sxy[idx] = msxy; a.m.p[idx] = mp;
    a.m.vx[idx] = mvx; a.m.vy[idx] = mvy; a.m.e[idx] = me;
  }
}

// ------------------------------------------------ interpolationmod 1
// The back-scatter of interpolate_mechanical (interpolation.c:1104-1158 and
// 1249-1358) with the full stencils, as a gather: one thread per node sums,
// cell by cell in sorted order, the payload k_gather left per marker —
// bilinear weights on basic nodes, the staggered centre stencil on pressure
// nodes (no vx/vy back-scatter in this mode) — and normalises as the tail of nodes2markers does (interpolation.c:1014-1046).  The centre
// stencil's contributions past the last node row land, as in the
// reference, in the next column's first row (a ghost node whose sums are
// kept but never normalised).
__device__ __forceinline__ float bs_half(int k, float f) {
  if (k == 0) return f < 0.5f ? 1.f - f - 0.5f : 0.f;
  if (k == 1) return 1.f - fabsf(f - 0.5f);
  return f > 0.5f ? f - 0.5f : 0.f;
}

template <int ROLE>
__device__ __forceinline__ void bs_mode1(const N2MArgs &a) {
  const Grid &g = a.g;
  const Nodes &N = a.N;
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= g.nn) return;
  const int ix = (int)(t / g.yn), iy = (int)(t - (long)ix * g.yn);
  const int ncy = g.ncy;
  const long n = a.n;
  const float *bs = a.bs;
  Acc sum[5];
#pragma unroll
  for (int q = 0; q < 5; q++) sum[q].zero();
  auto cell_sum = [&](int cx, int cy, int ax, int by) {
    if (cx < 0 || cx >= g.ncx || cy < 0 || cy >= ncy) return;
    const float s1 = (1.f / __ldg(g.wx + cx)) / __ldg(g.wy + cy);
    const long c = (long)cx * ncy + cy;
    if (ROLE == 0) {
      const int sb = __ldg(a.start + c), se = __ldg(a.start + c + 1);
#pragma unroll 2
      for (int s = sb; s < se; s++) {
        const float u = bs[BS_U * n + s], v = bs[BS_V * n + s];
        const float w = s1 * (ax ? u : 1.f - u) * (by ? v : 1.f - v);
        sum[0].add(bs[BS_PHIS * n + s] * w); sum[1].add(bs[BS_SXY * n + s] * w);
        sum[2].add(bs[BS_EXY * n + s] * w); sum[3].add(bs[BS_ES * n + s] * w);
        sum[4].add(w);
      }
      return;
    }
    // only the quarter classes (2 (v > 1/2) + (u > 1/2)) that have weight: a
    // half-cell factor k = 0 needs the lower half, k = 2 the upper; all fields
    // of a marker at once (433 x 187 lines, both groups: 57 -> 48 us)
    const int4 qs = __ldg(a.qstart + c);
    const int qe = __ldg(a.start + c + 1);
    const int mask = (0xaf5 >> (4 * ax)) & (0xcf3 >> (4 * by)) & 0xf;
    auto qb = [&](int q) { return q == 0 ? qs.x : q == 1 ? qs.y : q == 2 ? qs.z : q == 3 ? qs.w : qe; };
#pragma unroll 1
    for (int q = 0; q < 4; q++) {
      if (!((mask >> q) & 1)) continue;
      const int sb = qb(q);
      while (q < 3 && ((mask >> (q + 1)) & 1)) q++;
      const int se = qb(q + 1);
#pragma unroll 2
      for (int s = sb; s < se; s++) {
        const float u = bs[BS_U * n + s], v = bs[BS_V * n + s];
        const float pr = bs[BS_PR * n + s], sxx = bs[BS_SXX * n + s], exx = bs[BS_EXX * n + s];
        const float w = s1 * bs_half(ax, u) * bs_half(by, v);
        if (w != 0.f) {
          sum[0].add(pr * w); sum[1].add(sxx * w);
          sum[2].add(exx * w); sum[3].add(w);
        }
      }
    }
  };
  if (ROLE == 0) {
    for (int ax = 1; ax >= 0; ax--)
      for (int by = 1; by >= 0; by--) cell_sum(ix - ax, iy - by, ax, by);
    const float w = sum[4].value();
    const float ph = sum[0].value(), sy = sum[1].value(), ey = sum[2].value(), es = sum[3].value();
    N.f(V2C_NF_PHISUM)[t] = ph; N.f(V2C_NF_SXYSUM)[t] = sy;
    N.f(V2C_NF_EXYSUM)[t] = ey; N.f(V2C_NF_ESUM)[t] = es; N.f(V2C_NF_WTPHISUM)[t] = w;
    if (w != 0.f && ix >= 1 && iy >= 1 && ix < g.xn - 1 && iy < g.yn - 1) {
      N.f(V2C_NF_PHIE)[t] = __fdividef(ph, w); N.f(V2C_NF_SXYEE)[t] = __fdividef(sy, w);
      N.f(V2C_NF_EXYEE)[t] = __fdividef(ey, w); N.f(V2C_NF_PEE)[t] = __fdividef(es, w);
    }
  } else {
    for (int ax = 2; ax >= 0; ax--)
      for (int by = 2; by >= 0; by--) cell_sum(ix - ax, iy - by, ax, by);
    // the first row also gets what the last cell row sends past the end of
    // the previous columns
    if (iy == 0)
      for (int ax = 2; ax >= 0; ax--) cell_sum(ix - 1 - ax, ncy - 1, ax, 2);
    const float w = sum[3].value();
    const float ps = sum[0].value(), sx = sum[1].value(), ex = sum[2].value();
    N.f(V2C_NF_PSUM)[t] = ps; N.f(V2C_NF_SXXSUM)[t] = sx;
    N.f(V2C_NF_EXXSUM)[t] = ex; N.f(V2C_NF_WTSXXSUM)[t] = w;
    if (w != 0.f && ix >= 1 && iy >= 1) {
      N.f(V2C_NF_SPPEE)[t] = __fdividef(ps, w); N.f(V2C_NF_SXXEE)[t] = __fdividef(sx, w);
      N.f(V2C_NF_EXXEE)[t] = __fdividef(ex, w);
    }
  }
}

// both node kinds in one launch, a row of blocks each
__global__ void __launch_bounds__(128) k_n2m_bs_mode1(N2MArgs a) {
  after_previous();
  if (blockIdx.y == 0) bs_mode1<1>(a);
  else bs_mode1<0>(a);
}

// ----------------------------------------------------------- the move
// moveandrotatemarkers (moveandrotatemarkers.c:1-178), one thread per
// marker: Euler or RK4 through allinteri, stress rotation, markers from
// depth, out-of-grid reset.  New positions go to the second position buffer.
// In array order, which stays near cell order (the markers of a warp share
// their cells' forms in L1): the sort's order would make ten marker arrays
// follow the permutation.  Bound by the latency of the integration's chain
// of form reads, so six resident CTAs, and the stresses, which are rotated
// after it, are asked for at the start.  4001 x 1001 lines, 60 M markers,
// with the quarters' forms: 1725 -> 1525 us (1616 in array order alone, 1566
// with the stresses asked for).
__global__ void __launch_bounds__(256, 6) k_move(N2MArgs a) {
  after_previous();
  const Grid &g = a.g;
  const v2c_params &P = a.S.p;
  const int ncy = g.ncy;
  const float dt = a.S.dt;
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= a.n) return;
  const int c = a.m.cell_in[idx];
  int ix, iy;
  g.cell_at(c, ix, iy);
  const float u = a.m.u_in[idx], v = a.m.v_in[idx];
  const int t = a.m.type[idx];
  asm volatile("prefetch.global.L2 [%0];" ::"l"(a.m.sxx + idx));
  asm volatile("prefetch.global.L2 [%0];" ::"l"(a.m.sxy + idx));
  float tk = a.m.tk[idx];
  const bool in_grid = (ix > 0 || u >= 0.f) && (ix < g.ncx - 1 || u <= 1.f) &&
                       (iy > 0 || v >= 0.f) && (iy < g.ncy - 1 || v <= 1.f);
  int nix = ix, niy = iy;
  float nu_ = u, nv_ = v;
  if (!a.R(RK_IM, t) && (in_grid || P.outgrid != 1)) {
    const float wxc = __ldg(g.wx + ix), wyc = __ldg(g.wy + iy);
    const Pos p0{ix, iy, u * wxc, v * wyc};
    float vx0, vy0, sp0, vx1, vy1, sp1;
    vel_at(g, a.quad, p0, vx1, vy1, sp1);
    if (P.markmod == 1) {
      vx0 = vx1; vy0 = vy1; sp0 = sp1;
    } else {
      float vx2, vy2, sp2, vx3, vy3, sp3, vx4, vy4, sp4;
      Pos p = p0;
      p.X += vx1 * dt / 2.f; p.Y += vy1 * dt / 2.f;
      settle(g, p, a.stat);
      vel_at(g, a.quad, p, vx2, vy2, sp2);
      p = p0;
      p.X += vx2 * dt / 2.f; p.Y += vy2 * dt / 2.f;
      settle(g, p, a.stat);
      vel_at(g, a.quad, p, vx3, vy3, sp3);
      p = p0;
      p.X += vx3 * dt; p.Y += vy3 * dt;
      settle(g, p, a.stat);
      vel_at(g, a.quad, p, vx4, vy4, sp4);
      vx0 = (vx1 + 2.f * vx2 + 2.f * vx3 + vx4) / 6.f;
      vy0 = (vy1 + 2.f * vy2 + 2.f * vy3 + vy4) / 6.f;
      sp0 = (P.markmod == 2) ? (sp1 + 2.f * sp2 + 2.f * sp3 + sp4) / 6.f : sp1;
    }
    if (P.outgrid == 2) {
      if ((ix == 0 && u < 0.f) || (ix == g.ncx - 1 && u > 1.f)) vy0 = 0.f;
      if ((iy == 0 && v < 0.f) || (iy == g.ncy - 1 && v > 1.f)) vx0 = 0.f;
    }
    // new position: in offset space while the marker stays in its cell
    // (one FP32 rounding of u), else walked in metres
    nu_ = u + dt * vx0 / wxc;
    nv_ = v + dt * vy0 / wyc;
    const bool interior_x = ix > 0 && ix < g.ncx - 1, interior_y = iy > 0 && iy < g.ncy - 1;
    if (!(nu_ >= 0.f && nu_ < 1.f && (interior_x || (u >= 0.f && u <= 1.f)))) {
      Pos p{ix, 0, nu_ * wxc, 0.f};
      settle(g, p, a.stat);
      nix = p.ix;
      const float nwx = __ldg(g.wx + nix);
      nu_ = p.X / nwx;
      if (p.X < nwx && nu_ >= 1.f) nu_ = nextafterf(1.f, 0.f);
      if (p.X < 0.5f * nwx && nu_ >= 0.5f) nu_ = nextafterf(0.5f, 0.f);
      if (p.X > 0.5f * nwx && nu_ <= 0.5f) nu_ = nextafterf(0.5f, 1.f);
      if (p.X > nwx && nu_ <= 1.f) nu_ = nextafterf(1.f, 2.f);
    }
    if (!(nv_ >= 0.f && nv_ < 1.f && (interior_y || (v >= 0.f && v <= 1.f)))) {
      Pos p{0, iy, 0.f, nv_ * wyc};
      settle(g, p, a.stat);
      niy = p.iy;
      const float nwy = __ldg(g.wy + niy);
      nv_ = p.Y / nwy;
      if (p.Y < nwy && nv_ >= 1.f) nv_ = nextafterf(1.f, 0.f);
      if (p.Y < 0.5f * nwy && nv_ >= 0.5f) nv_ = nextafterf(0.5f, 0.f);
      if (p.Y > 0.5f * nwy && nv_ <= 0.5f) nv_ = nextafterf(0.5f, 1.f);
      if (p.Y > nwy && nv_ <= 1.f) nv_ = nextafterf(1.f, 2.f);
    }
    if (t >= 100) {
      // immobile marker (moveandrotatemarkers.c:88-135): inside the model
      // it spawns a mobile marker there and goes back to its anchor
      // (markk, markv), as it does when it strays more than ystpy from it
      const bool inside = (nix > 0 || nu_ >= 0.f) && (nix < g.ncx - 1 || nu_ <= 1.f) &&
                          (niy > 0 || nv_ >= 0.f) && (niy < g.ncy - 1 || nv_ <= 1.f);
      const double ax = (double)tk + (double)a.m.tk_lo[idx];
      const double ay = (double)a.m.mv[idx] + (double)a.m.mv_lo[idx];
      double x = g.gx[nix] + (double)nu_ * (g.gx[nix + 1] - g.gx[nix]);
      double y = g.gy[niy] + (double)nv_ * (g.gy[niy + 1] - g.gy[niy]);
      if (inside && a.has_imm) {
        const int id = a.m.id[idx];
        a.imm.spawn[id] = 1;
        a.imm.sp_cell[id] = nix * ncy + niy;
        a.imm.sp_u[id] = nu_;
        a.imm.sp_v[id] = nv_;
        x = ax;
        y = ay;
      }
      const double dx = x - ax, dy = y - ay;
      if (x == ax && y == ay || sqrt(dx * dx + dy * dy) > P.ystpy) {
        nix = nsearch64(g.gx, g.xn, ax);
        niy = nsearch64(g.gy, g.yn, ay);
        nu_ = offset32((ax - g.gx[nix]) / (g.gx[nix + 1] - g.gx[nix]));
        nv_ = offset32((ay - g.gy[niy]) / (g.gy[niy + 1] - g.gy[niy]));
      }
    } else {
    // stress rotation, moveandrotatemarkers.c:58-76
    float msxx = a.m.sxx[idx], msxy = a.m.sxy[idx];
    sp0 *= dt;
    if (P.stoksmod == 1) {
      float sn, cs;
      sincosf(sp0, &sn, &cs);
      const float s2 = 2.f * sn * cs, c2 = cs * cs - sn * sn;  // sin, cos of 2 sp0
      const float r1 = msxx * cs * cs - msxx * sn * sn + msxy * s2;
      const float r3 = 0.5f * (-msxx - msxx) * s2 + msxy * c2;
      msxx = r1; msxy = r3;
    } else if (P.stoksmod == 2) {
      const float r1 = msxx + msxy * 2.f * sp0;
      const float r3 = msxy + 0.5f * (-msxx - msxx) * 2.f * sp0;
      msxx = r1; msxy = r3;
    }
    a.m.sxx[idx] = msxx;
    a.m.sxy[idx] = msxy;
    // markers coming from depth, out-of-grid reset (:79-87); the FP64
    // position only when the FP32 one is within 1 m of zdeep
    // (the temperature pair's high word decides tk < tdeep; the two can
    // differ only for a temperature within half an FP32 ulp of tdeep, where
    // resetting or not leaves the same temperature to that half ulp)
    float tk_lo = 0.f;
    bool reset = false;
    if (vy0 < 0.f && tk < a.S.tdeep_f &&
        __ldg(a.gyf + niy) + nv_ * __ldg(g.wy + niy) > a.S.zdeep_lo_f) {
      const double ynew = g.gy[niy] + (double)nv_ * (g.gy[niy + 1] - g.gy[niy]);
      if (ynew > P.zdeep) {
        tk = a.S.tdeep_f;
        tk_lo = a.S.tdeep_lo;
        reset = true;
      }
    }
    const bool out = (nix == 0 && nu_ < 0.f) || (nix == g.ncx - 1 && nu_ > 1.f) ||
                     (niy == 0 && nv_ < 0.f) || (niy == g.ncy - 1 && nv_ > 1.f);
    if (out) {
      tk = 0.f;
      tk_lo = 0.f;
      reset = true;
      a.m.e[idx] = 0.f;
      a.m.flags[idx] |= MFLAG_RESET;
      atomicAdd(a.stat + ST_OUT_OF_GRID, 1ull);
    }
    if (reset) {
      a.m.tk[idx] = tk;
      a.m.tk_lo[idx] = tk_lo;
    }
    }
  }
  // mobile markers outside the model after the move: the slots that
  // markers spawned by immobile ones refill (moveandrotatemarkers.c:141-171)
  if (a.has_imm && t < 100 &&
      !((nix > 0 || nu_ >= 0.f) && (nix < g.ncx - 1 || nu_ <= 1.f) &&
        (niy > 0 || nv_ >= 0.f) && (niy < g.ncy - 1 || nv_ <= 1.f)))
    a.imm.out[a.m.id[idx]] = 1;
  a.m.cell_out[idx] = nix * ncy + niy;
  a.m.u_out[idx] = nu_;
  a.m.v_out[idx] = nv_;
}

}  // namespace

cudaError_t n2m_init() {
  return cudaFuncSetAttribute(k_n2m, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(Smem));
}

void launch_n2m(const N2MArgs &a, cudaStream_t st) {
  const unsigned mb = (unsigned)((a.n + 255) / 256);
  if (a.bs) {
    if (a.n > 0) launch_after(k_gather<true, false>, mb, 256, 0, st, a);
    const unsigned nb = (unsigned)((a.g.nn + 127) / 128);
    launch_after(k_n2m_bs_mode1, dim3(nb, 2), 128, 0, st, a);
  } else if (a.S.p.antidiffinter == 1) {
    dim3 grid((a.g.xn + a.TX - 1) / a.TX, (a.g.yn + TY - 1) / TY);
    launch_after(k_n2m, grid, NTH, sizeof(Smem), st, a);
  } else if (a.n > 0) {
    // the markers take the node fields without antidiffusion
    // (the node differences borrow the room of the move's velocity forms)
    launch_after(k_plain_nodes, (unsigned)((a.g.nn + 255) / 256), 256, 0, st, a.N, a.g.nn,
                 reinterpret_cast<PlainNode *>(a.quad));
    launch_after(k_gather<false, true>, mb, 256, 0, st, a);
  }
}

void launch_move(const N2MArgs &a, cudaStream_t st) {
  const long quarters = (long)a.g.ncx * a.g.ncy * 4;
  launch_after(k_vel_quads, (unsigned)((quarters + 255) / 256), 256, 0, st, a.g, a.N, a.quad);
  if (a.n <= 0) return;
  launch_after(k_move, (unsigned)((a.n + 255) / 256), 256, 0, st, a);
}

}  // namespace v2c
