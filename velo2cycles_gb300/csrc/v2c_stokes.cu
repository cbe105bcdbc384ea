// v2c_stokes.cu -- the Stokes matrix of the staggered grid on the device:
// preparematrix (momentum_continuity_addmatrix_checkerror.c:22-213) with its
// equation builders and gausmat4_add's CSR layout (gausevps.c:137-214).
//
// One thread per equation (3 per node: pressure/continuity, vx, vy), the
// threads of a block all of one kind, so that a warp runs one equation
// builder.  The thread forms the CSR row: columns in increasing order, the
// terms of one column summed in the reference's order starting from zero,
// zero sums left out.  Which columns a momentum or continuity equation can
// have, and their order, is known (at least 3 node rows), so each term is
// added to its column's register as it is formed, and no row is sorted; a
// boundary equation's few terms are.  Two passes: the first counts each
// row's coefficients (and writes the right-hand side), a scan turns counts
// into row starts, the second writes columns and values; when the caller
// gives room for the coefficients the first pass also keeps each row and the
// second only moves it.
//
// 301 x 101 nodes (91 203 rows), the count pass: 204 us with rows of all
// kinds in each warp, whose terms were listed and sorted in local memory,
// 55 us now, bound by the FP64 divisions.
//
// FP64 throughout, in the reference's evaluation order, and this file is
// compiled without multiply-add contraction, so a coefficient is the
// correctly rounded result of the same operations the reference performs.
#include "v2c_kernels.h"

namespace v2c {

namespace {

enum { ERR_OUTSIDE = 1, ERR_BOUNDARY = 2 };

// A row whose N columns are known: their sums so far, in column order.
template <int N>
struct Row {
  double c = 0.0;  // right-hand side
  double s[N] = {};
};

// A boundary equation: at most 4 terms in any column order.
struct Eq {
  double c;
  int n;
  long col[4];
  double w[4];
  __device__ __forceinline__ void add(long k, double v) {
    col[n] = k;
    w[n] = v;
    n++;
  }
};

struct Ctx {
  const StokesArgs &a;
  long yn, xn, nn;
  __device__ double N(int f, long m) const { return (double)a.N.f(f)[m]; }
  __device__ double gx(long i) const { return a.g.gx[i]; }
  __device__ double gy(long j) const { return a.g.gy[j]; }
};

// nueffcalc (momentum_continuity_addmatrix_checkerror.c:380-393)
__device__ __forceinline__ double nueff_of(const StokesArgs &a, double nvp, double gge,
                                           double &Z) {
  Z = gge * a.dt / (gge * a.dt + nvp);
  double nueff = Z * nvp;
  if (nueff < a.nubeg) nueff = a.nubeg;
  return nueff;
}

// sxxcalc_prepare (:395-443): the normal-stress terms of node (m1, m2)
// scaled by yv, into the sums I0 to I3
template <int I0, int I1, int I2, int I3, int N>
__device__ __forceinline__ void sxx_terms(const Ctx &C, Row<N> &E, long m1, long m2, double yv) {
  const long v3 = m1 * C.yn + m2;
  const double se = C.N(V2C_NF_SXXE, v3);
  double Z;
  const double nueff = nueff_of(C.a, C.N(V2C_NF_ND, v3), C.N(V2C_NF_GD, v3), Z);
  const double dx = C.gx(m1) - C.gx(m1 - 1), dy = C.gy(m2) - C.gy(m2 - 1);
  const double px = yv * nueff / dx, py = yv * nueff / dy;
  E.s[I0] += -px;  // vx (m1 - 1, m2 - 1)
  E.s[I1] += px;   // vx (m1, m2 - 1)
  E.s[I2] += py;   // vy (m1 - 1, m2 - 1)
  E.s[I3] += -py;  // vy (m1 - 1, m2)
  E.c -= (1.0 - Z) * yv * se;
}

// sxycalc_prepare (:483-525): the shear-stress terms of node (m1, m2)
template <int I0, int I1, int I2, int I3, int N>
__device__ __forceinline__ void sxy_terms(const Ctx &C, Row<N> &E, long m1, long m2, double yv) {
  const long v3 = m1 * C.yn + m2;
  const double se = C.N(V2C_NF_SXYE, v3);
  double Z;
  const double nueff = nueff_of(C.a, C.N(V2C_NF_NU, v3), C.N(V2C_NF_GG, v3), Z);
  const double ddy = C.gy(m2 + 1) - C.gy(m2 - 1), ddx = C.gx(m1 + 1) - C.gx(m1 - 1);
  const double py = yv * 2.0 * nueff / ddy, px = yv * 2.0 * nueff / ddx;
  E.s[I0] += -py;  // vx (m1, m2 - 1)
  E.s[I1] += py;   // vx (m1, m2)
  E.s[I2] += -px;  // vy (m1 - 1, m2)
  E.s[I3] += px;   // vy (m1, m2)
  E.c -= (1.0 - Z) * yv * se;
}

// contadd (:932-998): div v of the cell whose pressure node is (m1, m2).
// Columns: vx (-1,-1), vy (-1,-1), vy (-1,0), vx (0,-1), P (0,0).
__device__ __forceinline__ void cont_eq(const Ctx &C, Row<5> &E, long m1, long m2) {
  const StokesArgs &a = C.a;
  const long v3 = m1 * C.yn + m2;
  E.c = a.compressible ? C.N(V2C_NF_SPPE, v3) / C.N(V2C_NF_BM, v3) / a.timestep : 0.0;
  const double dx = C.gx(m1) - C.gx(m1 - 1), dy = C.gy(m2) - C.gy(m2 - 1);
  const double rx = 1.0 / dx, ry = 1.0 / dy;
  E.s[0] = -rx;
  E.s[3] = rx;
  E.s[1] = -ry;
  E.s[2] = ry;
  if (a.compressible) E.s[4] = 1.0 / C.N(V2C_NF_BM, v3) / a.timestep;
}

// bondadd (:192-211): the boundary equation of unknown r
__device__ void bond_eq(const Ctx &C, Eq &E, long r, int &bad) {
  const StokesArgs &a = C.a;
  const long B = a.bondm[r];
  E.n = 0;
  E.c = a.bondv[B * 4 + 0];
  E.add(r, 1.0);
  for (int k = 0; k < 3; k++) {
    const long bn = a.bondn[B * 3 + k];
    if (bn) {
      if (bn - 1 < 0 || bn - 1 >= 3 * C.nn) bad |= ERR_BOUNDARY;
      E.add(bn - 1, -a.bondv[B * 4 + k + 1]);
    }
  }
}

// xstoksadd (:642-731): x momentum at vx node (m1, m2).  Columns:
// 0 vx (-1,0), 1 vy (-1,0), 2 vy (-1,1), 3 vx (0,-1), 4 vx (0,0), 5 vy (0,0),
// 6 P (0,1), 7 vx (0,1), 8 vy (0,1), 9 vx (1,0), 10 P (1,1).
__device__ __forceinline__ void xstokes_eq(const Ctx &C, Row<11> &E, long m1, long m2) {
  const StokesArgs &a = C.a;
  const long yn = C.yn;
  const long v0 = m1 * yn + m2, v1 = v0 + 1, v2 = v0 + yn, v3 = v2 + 1;
  const double xkf = (C.gx(m1 + 1) - C.gx(m1 - 1)) / 2.0, ykf = C.gy(m2 + 1) - C.gy(m2);
  const double mrx = C.N(V2C_NF_MRX, v0);
  const double rx = 1.0 / xkf, ry = 1.0 / ykf;
  E.c = (-a.gxkoef - a.inertyn * C.N(V2C_NF_MVX, v0) / a.dt) * mrx;
  E.s[6] += rx;
  E.s[10] += -rx;
  E.s[4] += -a.inertyn * mrx / a.dt;
  sxx_terms<0, 4, 1, 2>(C, E, m1, m2 + 1, -rx);
  sxx_terms<4, 9, 5, 8>(C, E, m1 + 1, m2 + 1, rx);
  sxy_terms<3, 4, 1, 5>(C, E, m1, m2, -ry);
  sxy_terms<4, 7, 2, 8>(C, E, m1, m2 + 1, ry);
  if (a.drunkensailor == 1) {
    const double dt = a.dt, G = a.gxkoef;
    const double ro0 = C.N(V2C_NF_RO, v0), ro1 = C.N(V2C_NF_RO, v1);
    const double ro2 = C.N(V2C_NF_RO, v2), ro3 = C.N(V2C_NF_RO, v3);
    const double rol0 = C.N(V2C_NF_RO, v0 - yn), rol1 = C.N(V2C_NF_RO, v1 - yn);
    const double dxx = C.gx(m1 + 1) - C.gx(m1 - 1), dyy = C.gy(m2 + 1) - C.gy(m2);
    const double fl = C.gx(m1) - C.gx(m1 - 1), fr = C.gx(m1 + 1) - C.gx(m1);
    E.s[4] += -dt / 2.0 * G * (ro2 + ro3 - rol0 - rol1) / dxx / 2.0;
    const double wl = -dt / 2.0 * G * fl / dxx / 2.0 * (ro1 - ro0) / dyy;
    E.s[5] += wl;
    E.s[8] += wl;
    const double wr = -dt / 2.0 * G * fr / dxx / 2.0 * (ro1 - ro0) / dyy;
    E.s[1] += wr;
    E.s[2] += wr;
  }
}

// ystoksadd (:794-877): y momentum at vy node (m1, m2).  Columns:
// 0 vy (-1,0), 1 vx (0,-1), 2 vy (0,-1), 3 vx (0,0), 4 vy (0,0), 5 vy (0,1),
// 6 vx (1,-1), 7 P (1,0), 8 vx (1,0), 9 vy (1,0), 10 P (1,1).
__device__ __forceinline__ void ystokes_eq(const Ctx &C, Row<11> &E, long m1, long m2) {
  const StokesArgs &a = C.a;
  const long yn = C.yn;
  const long v0 = m1 * yn + m2, v1 = v0 + 1, v2 = v0 + yn, v3 = v2 + 1;
  const double xkf = C.gx(m1 + 1) - C.gx(m1), ykf = (C.gy(m2 + 1) - C.gy(m2 - 1)) / 2.0;
  const double mry = C.N(V2C_NF_MRY, v0);
  const double rx = 1.0 / xkf, ry = 1.0 / ykf;
  E.c = (-a.gykoef - a.inertyn * C.N(V2C_NF_MVY, v0) / a.dt) * mry;
  E.s[7] += ry;
  E.s[10] += -ry;
  E.s[4] += -a.inertyn * mry / a.dt;
  sxx_terms<1, 6, 2, 4>(C, E, m1 + 1, m2, ry);
  sxx_terms<3, 8, 4, 5>(C, E, m1 + 1, m2 + 1, -ry);
  sxy_terms<1, 3, 0, 4>(C, E, m1, m2, -rx);
  sxy_terms<6, 8, 4, 9>(C, E, m1 + 1, m2, rx);
  if (a.drunkensailor == 1) {
    const double dt = a.dt, G = a.gykoef;
    const double ro0 = C.N(V2C_NF_RO, v0), ro1 = C.N(V2C_NF_RO, v1);
    const double ro2 = C.N(V2C_NF_RO, v2), ro3 = C.N(V2C_NF_RO, v3);
    const double rob0 = C.N(V2C_NF_RO, v0 - 1), rob2 = C.N(V2C_NF_RO, v2 - 1);
    const double dyy = C.gy(m2 + 1) - C.gy(m2 - 1), dxx = C.gx(m1 + 1) - C.gx(m1);
    const double fu = C.gy(m2) - C.gy(m2 - 1), fd = C.gy(m2 + 1) - C.gy(m2);
    E.s[4] += -dt / 2.0 * G * (ro1 + ro3 - rob0 - rob2) / dyy / 2.0;
    const double wu = -dt / 2.0 * G * fu / dyy / 2.0 * (ro2 - ro0) / dxx;
    E.s[3] += wu;
    E.s[8] += wu;
    const double wd = -dt / 2.0 * G * fd / dyy / 2.0 * (ro2 - ro0) / dxx;
    E.s[1] += wd;
    E.s[6] += wd;
  }
}

// a vx or vy boundary given as a continuity equation (addvx :92-108,
// addvy :150-166): the cell of the referenced pressure; the reference
// checks that the pressure unknown k below the referenced one (k = 2 for
// vx, 3 for vy) has a boundary equation
__device__ bool cont_boundary(const Ctx &C, long r, long &m1, long &m2, int k, int &bad) {
  const StokesArgs &a = C.a;
  const long B = a.bondm[r];
  const long ref = a.bondn[B * 3 + 0];
  const long d = (ref - 1 - r) / 3;  // C division: truncates toward zero
  long dm1 = 0, dm2 = 0;
  if (d >= C.yn) dm1 = 1;
  if (d == 1 || d > C.yn) dm2 = 1;
  const long chk = ref - k;
  if (d < 0 || d > C.yn + 1 || !(m1 + dm1) || !(m2 + dm2) || chk < 0 || chk >= 4 * C.nn ||
      !a.bondm[chk]) {
    bad |= ERR_BOUNDARY;
    return false;
  }
  if (m1 + dm1 > C.xn - 1 || m2 + dm2 > C.yn - 1) {
    bad |= ERR_OUTSIDE;
    return false;
  }
  m1 += dm1;
  m2 += dm2;
  return true;
}

// gausmat4_add's row: sort the nonzero terms by column (stable, so the
// terms of one column keep their order) and sum each column from zero
__device__ int form_row(Eq &E) {
  int m = 0;
  for (int i = 0; i < E.n; i++)
    if (E.w[i] != 0.0) {
      E.col[m] = E.col[i];
      E.w[m] = E.w[i];
      m++;
    }
  for (int i = 1; i < m; i++) {
    const long k = E.col[i];
    const double v = E.w[i];
    int j = i - 1;
    while (j >= 0 && E.col[j] > k) {
      E.col[j + 1] = E.col[j];
      E.w[j + 1] = E.w[j];
      j--;
    }
    E.col[j + 1] = k;
    E.w[j + 1] = v;
  }
  int out = 0;
  for (int i = 0; i < m;) {
    double s = 0.0;
    const long k = E.col[i];
    for (; i < m && E.col[i] == k; i++) s += E.w[i];
    if (s != 0.0) {
      E.col[out] = k;
      E.w[out] = s;
      out++;
    }
  }
  return out;
}

// Where a row goes: its count, its right-hand side and, when the rows are
// kept, its entries (entry i of all rows of a kind side by side).
struct Out {
  const StokesArgs &a;
  long nn, m3, r;
  int kind, n = 0;
  __device__ __forceinline__ void put(long col, double w) {
    if (a.ell_col) {
      const long at = ((long)kind * STOKES_ROW_MAX + n) * nn + m3;
      a.ell_col[at] = (int32_t)(col + 1);
      a.ell_val[at] = w;
    }
    n++;
  }
  __device__ __forceinline__ void done(double c) {
    a.cnt[r] = n;
    if (a.b) a.b[r] = c;
  }
};
// the row's nonzero sums; column i is unknown K[i] of the node D1[i] columns
// and D2[i] rows from node (m1, m2)
template <int N>
__device__ __forceinline__ void put_row(Out &O, const Row<N> &E, long node, long yn,
                                        const int (&D1)[N], const int (&D2)[N],
                                        const int (&K)[N]) {
#pragma unroll
  for (int i = 0; i < N; i++)
    if (E.s[i] != 0.0) O.put((node + D1[i] * yn + D2[i]) * 3 + K[i], E.s[i]);
}

// kinds of row: none, the unknown itself (ghost), a boundary equation, a
// continuity equation, a momentum equation
enum { ROW_EMPTY, ROW_ONE, ROW_BOND, ROW_CONT, ROW_STOKES };

// The equation of unknown 3 m3 + KIND as preparematrix builds it; empty where
// the reference stops or would leave the grid.  Ghost, boundary and
// continuity rows are scaled by mukoef term by term, right side too.
template <int KIND>
__device__ __forceinline__ void build_row(const Ctx &C, Out &O, long m1, long m2, int &bad) {
  const StokesArgs &a = C.a;
  const long xn = C.xn, yn = C.yn, r = O.r;
  int row;
  if (KIND == 0) {  // addcont (:40-71)
    row = !(m1 && m2) ? ROW_ONE : !a.bondm[r] || a.compressible == 1 ? ROW_CONT : ROW_BOND;
  } else if (KIND == 1) {  // addvx (:73-129)
    if (!(m2 < yn - 1)) row = ROW_ONE;
    else if (!a.bondm[r] ||
             (a.timesum > a.timebond && m1 > 2 && m2 > 2 && m1 < xn - 4 && m2 < yn - 3)) {
      row = ROW_STOKES;
      if (m1 < 1 || m1 > xn - 2 || m2 < 1 || m2 > yn - 3) { bad |= ERR_OUTSIDE; row = ROW_EMPTY; }
    } else row = a.bondv[a.bondm[r] * 4 + 1] > 1e+30 ? ROW_CONT : ROW_BOND;
  } else {  // addvy (:131-190)
    if (!(m1 < xn - 1)) row = ROW_ONE;
    else if (!a.bondm[r]) {
      row = ROW_STOKES;
      if (m1 < 1 || m1 > xn - 3 || m2 < 1 || m2 > yn - 2) { bad |= ERR_OUTSIDE; row = ROW_EMPTY; }
    } else row = a.bondv[a.bondm[r] * 4 + 1] > 1e+30 ? ROW_CONT : ROW_BOND;
  }
  double c = 0.0;
  if (KIND != 0 && row == ROW_STOKES) {
    Row<11> E;
    if (KIND == 1) {
      xstokes_eq(C, E, m1, m2);
      constexpr int D1[11] = {-1, -1, -1, 0, 0, 0, 0, 0, 0, 1, 1};
      constexpr int D2[11] = {0, 0, 1, -1, 0, 0, 1, 1, 1, 0, 1};
      constexpr int K[11] = {1, 2, 2, 1, 1, 2, 0, 1, 2, 1, 0};
      put_row(O, E, O.m3, yn, D1, D2, K);
    } else {
      ystokes_eq(C, E, m1, m2);
      constexpr int D1[11] = {-1, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1};
      constexpr int D2[11] = {0, -1, -1, 0, 0, 1, -1, 0, 0, 0, 1};
      constexpr int K[11] = {2, 1, 2, 1, 2, 2, 1, 0, 1, 2, 0};
      put_row(O, E, O.m3, yn, D1, D2, K);
    }
    O.done(E.c);
    return;
  }
  if (row == ROW_CONT && (KIND == 0 || cont_boundary(C, r, m1, m2, KIND + 1, bad))) {
    Row<5> E;
    cont_eq(C, E, m1, m2);
#pragma unroll
    for (int i = 0; i < 5; i++) E.s[i] *= a.mukoef;
    constexpr int D1[5] = {-1, -1, -1, 0, 0}, D2[5] = {-1, -1, 0, -1, 0}, K[5] = {1, 2, 2, 1, 0};
    put_row(O, E, m1 * yn + m2, yn, D1, D2, K);
    c = E.c * a.mukoef;
  } else if (row == ROW_BOND) {
    Eq E;
    bond_eq(C, E, r, bad);
    for (int i = 0; i < E.n; i++) E.w[i] *= a.mukoef;
    const int n = form_row(E);
    for (int i = 0; i < n; i++) O.put(E.col[i], E.w[i]);
    c = E.c * a.mukoef;
  } else if (row == ROW_ONE) {
    const double w = 1.0 * a.mukoef;
    if (w != 0.0) O.put(r, w);
    c = 0.0 * a.mukoef;
  }
  O.done(c);
}

__global__ void __launch_bounds__(128) k_stokes_count(StokesArgs a) {
  after_previous();
  const long nn = a.g.nn, m3 = blockIdx.x * 128l + threadIdx.x;
  if (m3 >= nn) return;
  const Ctx C{a, a.g.yn, a.g.xn, nn};
  const int kind = blockIdx.y;
  const long m1 = m3 / C.yn, m2 = m3 - m1 * C.yn;
  Out O{a, nn, m3, 3 * m3 + kind, kind};
  int bad = 0;
  if (kind == 0) build_row<0>(C, O, m1, m2, bad);
  else if (kind == 1) build_row<1>(C, O, m1, m2, bad);
  else build_row<2>(C, O, m1, m2, bad);
  if (bad) atomicOr(a.err, bad);
}

// the rows the count pass kept, moved to their CSR positions
__global__ void __launch_bounds__(256) k_stokes_move(StokesArgs a) {
  after_previous();
  const long nn = a.g.nn, m3 = blockIdx.x * 256l + threadIdx.x;
  if (m3 >= nn) return;
  const int kind = blockIdx.y;
  const long r = 3 * m3 + kind;
  const long s = a.cnt[r], n = a.cnt[r + 1] - s;
  const long at = (long)kind * STOKES_ROW_MAX * nn + m3;
  for (int i = 0; i < n; i++) {
    a.ja[s + i] = a.ell_col[at + i * nn];
    a.a[s + i] = a.ell_val[at + i * nn];
  }
}

inline unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void launch_stokes_count(const StokesArgs &a, cudaStream_t st) {
  if (a.g.nn > 0) launch_after(k_stokes_count, dim3(nblk(a.g.nn, 128), 3), 128, 0, st, a);
}

void launch_stokes_fill(const StokesArgs &a, cudaStream_t st) {
  if (a.g.nn > 0) launch_after(k_stokes_move, dim3(nblk(a.g.nn, 256), 3), 256, 0, st, a);
}

}  // namespace v2c
