// v2c_timestep.cu -- the adaptive time step calc_timestep (calc_RSF.c:
// 352-572) over the device node fields.
//
// Per interior node: the visco-plastic Maxwell limit tcnvp*eta_vp/G, the
// displacement limit tcd/max(|vx|/dx, |vy|/dy), and with RSFmode 1 the
// Lapusta et al. (2000) slip-length limit lambda*L/V and the state limit
// tcphih/(V0/L e^-phi); the maximum slip rate; the stress and viscosity
// statistics over sticky01 == 1 / == 2 nodes.  Per-node arithmetic in FP32
// (the node fields are FP32), sums in FP64.
//
// Two sequential rules of the reference are kept by folding in node order:
// a node with b <= 0 resets the state and slip-length limits to maxtmstep
// (calc_RSF.c:497-501), so those minima run over the nodes after the last
// such node; and lambda carries over from the previous node where chi is
// NaN (no branch of calc_RSF.c:466-481 taken).  Each warp owns a contiguous
// node range and walks it in 32-node slices; segment states combine with
//   (A then B): reset = A.reset | B.reset, all = min(A.all, B.all),
//               after = B.reset ? B.after : min(A.after, B.all),
// which is associative, so the warp ranges fold in order in a tree (lanes,
// warps of a block, blocks: adjacent pairs at every level).  The
// lambda carry crosses slices but not warp ranges: a NaN-chi node at the
// start of a range takes 1/5 (MINV(NaN, 1/5) in the reference's order).
// chi == 0 (where the reference stops) sets an error flag.
#include <math.h>

#include "v2c_ff.cuh"
#include "v2c_kernels.h"

namespace v2c {

namespace {

enum {
  TS_DTNVP = 0, TS_DTD, TS_MAXVX, TS_MAXVEL,
  TS_PHI_ALL, TS_L_ALL, TS_PHI_AFTER, TS_L_AFTER, TS_RESET,
  TS_NR0, TS_MAXS0, TS_MINS0, TS_SUMS0, TS_SUM2S0, TS_MAXV0, TS_MINV0, TS_SUMV0, TS_SUM2V0,
  TS_NR1, TS_MAXS1, TS_MINS1, TS_SUMS1, TS_SUM2S1, TS_MAXV1, TS_MINV1, TS_SUMV1, TS_SUM2V1,
  TS_N
};
// extra output slots after the folded partial
enum { TS_P1S = TS_N, TS_P2S, TS_P1V, TS_P2V, TS_CHI0, TS_OUT_N };

constexpr int TW = 8;  // warps per block of the node pass

__device__ __forceinline__ int ts_kind(int k) {  // 0 min, 1 max, 2 sum, 3 ordered
  switch (k) {
    case TS_DTNVP: case TS_DTD: case TS_MINS0: case TS_MINV0: case TS_MINS1: case TS_MINV1:
      return 0;
    case TS_MAXVX: case TS_MAXVEL: case TS_MAXS0: case TS_MAXV0: case TS_MAXS1: case TS_MAXV1:
      return 1;
    case TS_PHI_ALL: case TS_L_ALL: case TS_PHI_AFTER: case TS_L_AFTER: case TS_RESET:
      return 3;
    default:
      return 2;
  }
}

// b <= a by the bit patterns, as integers (no entry is a NaN: the states
// start from numbers, and a NaN replaces none)
__device__ __forceinline__ bool ts_le(double b, double a) {
  auto key = [](double v) {
    const long long t = __double_as_longlong(v);
    return t ^ (t >> 63 & 0x7fffffffffffffffll);
  };
  return key(b) <= key(a);
}
// Entry k of "A then B" (B follows A in node order).  Only the sums are FP64
// arithmetic: a fold is one block, and its SM issues two FP64 operations a
// cycle, so FP64 comparisons of the other entries took most of its time.
__device__ __forceinline__ double ts_combined(int k, const double *a, const double *b) {
  const int kind = ts_kind(k);
  const double x = a[k], y = b[k];
  if (kind == 2) return x + y;
  const bool br = __double_as_longlong(b[TS_RESET]) != 0;
  if (k == TS_RESET) return br ? y : x;  // (0 or 1)
  double z = y;
  if (k == TS_PHI_AFTER || k == TS_L_AFTER) {
    if (br) return y;
    z = b[k == TS_PHI_AFTER ? TS_PHI_ALL : TS_L_ALL];
  }
  return (kind == 1 ? ts_le(x, z) : ts_le(z, x)) ? z : x;
}

// Fold n partials in order, pairs (2i, 2i+1) at each level, a warp per pair
// and a lane per entry; the result is partial 0.  All threads of the block.
__device__ __forceinline__ void ts_fold(double (*p)[TS_N], long n, int warp, int warps, int lane) {
  for (long step = 1; step < n; step <<= 1) {
    for (long i = warp; 2 * i * step + step < n; i += warps) {
      double *A = p[2 * i * step];
      const double *B = p[2 * i * step + step];
      const double v = lane < TS_N ? ts_combined(lane, A, B) : 0.0;
      __syncwarp();
      if (lane < TS_N) A[lane] = v;
    }
    __syncthreads();
  }
}

// One warp's running state.  The minima and maxima are FP32 values (the node
// arithmetic is FP32), kept and folded as such: FP64 compares run at 1/64 of
// the rate.  Their FP64 initial value 1e30 is put back at the end.
enum {
  F_DTNVP = 0, F_DTD, F_MINS0, F_MINV0, F_MINS1, F_MINV1,              // minima
  F_MAXVX, F_MAXVEL, F_MAXS0, F_MAXV0, F_MAXS1, F_MAXV1,               // maxima
  F_N,
  D_NR0 = 0, D_SUMS0, D_SUM2S0, D_SUMV0, D_SUM2V0, D_NR1, D_SUMS1, D_SUM2S1, D_SUMV1, D_SUM2V1,
  D_N
};
constexpr int F_MINS = F_MAXVX;
struct TsState {
  float f[F_N];
  double d[D_N];
  float all[2], after[2];  // state limit, slip-length limit
  bool reset;
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int k = 0; k < F_N; k++) f[k] = k < F_MINS ? INFINITY : 0.f;
#pragma unroll
    for (int k = 0; k < D_N; k++) d[k] = 0.0;
    all[0] = all[1] = after[0] = after[1] = INFINITY;
    reset = false;
  }
};
__device__ __forceinline__ float ts_min(float a, float b) { return b <= a ? b : a; }
__device__ __forceinline__ float ts_max(float a, float b) { return b >= a ? b : a; }

// fold the warp's lanes in order (adjacent pairs, lower lane first); the
// statistics of sticky01 == 1 and == 2 nodes only where a lane has some
__device__ __forceinline__ void ts_fold_lanes(TsState &s, bool any0, bool any1, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const bool take = (lane & (2 * o - 1)) == 0;
    auto stat = [&](int fmin, int fmax, int d0) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const float mn = __shfl_down_sync(V2C_FULL, s.f[fmin + k], o);
        const float mx = __shfl_down_sync(V2C_FULL, s.f[fmax + k], o);
        if (take) { s.f[fmin + k] = ts_min(s.f[fmin + k], mn); s.f[fmax + k] = ts_max(s.f[fmax + k], mx); }
      }
#pragma unroll
      for (int k = 0; k < 5; k++) {
        const double v = __shfl_down_sync(V2C_FULL, s.d[d0 + k], o);
        if (take) s.d[d0 + k] += v;
      }
    };
    if (any0) stat(F_MINS0, F_MAXS0, D_NR0);
    if (any1) stat(F_MINS1, F_MAXS1, D_NR1);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const float mn = __shfl_down_sync(V2C_FULL, s.f[F_DTNVP + k], o);
      const float mx = __shfl_down_sync(V2C_FULL, s.f[F_MAXVX + k], o);
      if (take) { s.f[F_DTNVP + k] = ts_min(s.f[F_DTNVP + k], mn); s.f[F_MAXVX + k] = ts_max(s.f[F_MAXVX + k], mx); }
    }
    const bool br = __shfl_down_sync(V2C_FULL, (int)s.reset, o);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const float ball = __shfl_down_sync(V2C_FULL, s.all[k], o);
      const float baft = __shfl_down_sync(V2C_FULL, s.after[k], o);
      if (take) {
        s.after[k] = br ? baft : ts_min(s.after[k], ball);
        s.all[k] = ts_min(s.all[k], ball);
      }
    }
    if (take) s.reset = s.reset || br;
  }
}
// a := a then b (sums: b has statistics)
__device__ __forceinline__ void ts_append(TsState &a, const TsState &b, bool sums) {
#pragma unroll
  for (int k = 0; k < F_N; k++) a.f[k] = k < F_MINS ? ts_min(a.f[k], b.f[k]) : ts_max(a.f[k], b.f[k]);
  if (sums) {
#pragma unroll
    for (int k = 0; k < D_N; k++) a.d[k] += b.d[k];
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    a.after[k] = b.reset ? b.after[k] : ts_min(a.after[k], b.all[k]);
    a.all[k] = ts_min(a.all[k], b.all[k]);
  }
  a.reset = a.reset || b.reset;
}
__device__ __forceinline__ void ts_store(const TsState &s, double *p) {
  // (1e30f is the first float above 1e30)
  auto lim = [](float v) { return v < 1e30f ? widen<true>(v) : 1e30; };
  p[TS_DTNVP] = lim(s.f[F_DTNVP]); p[TS_DTD] = lim(s.f[F_DTD]);
  p[TS_MAXVX] = widen<true>(s.f[F_MAXVX]); p[TS_MAXVEL] = widen<true>(s.f[F_MAXVEL]);
  p[TS_PHI_ALL] = lim(s.all[0]); p[TS_L_ALL] = lim(s.all[1]);
  p[TS_PHI_AFTER] = lim(s.after[0]); p[TS_L_AFTER] = lim(s.after[1]);
  p[TS_RESET] = s.reset ? 1.0 : 0.0;
  p[TS_NR0] = s.d[D_NR0]; p[TS_MAXS0] = widen<true>(s.f[F_MAXS0]); p[TS_MINS0] = lim(s.f[F_MINS0]);
  p[TS_SUMS0] = s.d[D_SUMS0]; p[TS_SUM2S0] = s.d[D_SUM2S0]; p[TS_MAXV0] = widen<true>(s.f[F_MAXV0]);
  p[TS_MINV0] = lim(s.f[F_MINV0]); p[TS_SUMV0] = s.d[D_SUMV0]; p[TS_SUM2V0] = s.d[D_SUM2V0];
  p[TS_NR1] = s.d[D_NR1]; p[TS_MAXS1] = widen<true>(s.f[F_MAXS1]); p[TS_MINS1] = lim(s.f[F_MINS1]);
  p[TS_SUMS1] = s.d[D_SUMS1]; p[TS_SUM2S1] = s.d[D_SUM2S1]; p[TS_MAXV1] = widen<true>(s.f[F_MAXV1]);
  p[TS_MINV1] = lim(s.f[F_MINV1]); p[TS_SUMV1] = s.d[D_SUMV1]; p[TS_SUM2V1] = s.d[D_SUM2V1];
}

struct TsArgs {
  Grid g;
  Nodes N;
  Scal S;
  v2c_timestep_ctl c;
  int oldornew;
  long per_warp;   // nodes per warp range (a multiple of 32)
  double *part;    // [blocks][TS_N]
  double *out;     // [TS_OUT_N]
};

// node pass: one warp per contiguous range, the block's warps folded at its
// end (301 x 101 lines: 22 us with FP64 minima and a serial fold per lane,
// 16 with FP32 ones, 14 with the limits and empty sums out of the FP64 pipe)
__global__ void __launch_bounds__(TW * 32) k_ts_nodes(TsArgs a) {
  after_previous();
  const Grid &g = a.g;
  const Nodes &N = a.N;
  const v2c_params &P = a.S.p;
  const int lane = threadIdx.x & 31;
  const long warp = (long)blockIdx.x * TW + (threadIdx.x >> 5);
  const long lo = warp * a.per_warp, hi = min(lo + a.per_warp, g.nn);
  const long yn = g.yn;
  __shared__ double part[TW][TS_N];
  TsState s;
  s.init();
  float lam_carry = __int_as_float(0x7fc00000);  // NaN: none yet
  for (long b0 = lo; b0 < hi; b0 += 32) {
    const long m3 = b0 + lane;
    const long m2 = m3 % yn, m1 = (m3 - m2) / yn;
    const bool interior = m3 < hi && m1 >= 1 && m2 >= 1 && m1 < g.xn - 1 && m2 < yn - 1;
    TsState d;
    d.init();
    bool rsf_node = false, chi_ok = false, reset = false, has_phi = false;
    float lam_raw = 0.f, LoV = 0.f, dtphi = 0.f, st = 0.f;
    if (interior) {
      const float dx = __ldg(g.wx + m1), dy = __ldg(g.wy + m2);
      const float faultwidth = 2.f * 0.5f * (dx + dy);
      const float nu_m2c = N.f(V2C_NF_NU_M2C)[m3], gg = N.f(V2C_NF_GG)[m3];
      float NUVP;
      if (a.oldornew == 0) {
        if (nu_m2c > 1.00e+26f) {
          const float sx = N.f(V2C_NF_SXXES)[m3], sy = N.f(V2C_NF_SXYE)[m3];
          const float sg = sqrtf(sx * sx + sy * sy);
          const float V = N.f(V2C_NF_RK_SLIPRS_FINAL)[m3];
          NUVP = (sg > 0.f && V > 0.f) ? nu_m2c * sg / (2.f * nu_m2c * V / faultwidth + sg) : nu_m2c;
        } else {
          NUVP = 5.00e+26f;
        }
      } else {
        NUVP = (nu_m2c > 1.00e+26f) ? N.f(V2C_NF_NU)[m3] : 5.00e+26f;
      }
      d.f[F_DTNVP] = (float)a.c.tcnvp * NUVP / gg;
      const float VXn = a.oldornew == 1 ? N.f(V2C_NF_VX)[m3] : N.f(V2C_NF_MVX)[m3];
      const float VYn = a.oldornew == 1 ? N.f(V2C_NF_VY)[m3] : N.f(V2C_NF_MVY)[m3];
      if (VXn != 0.f && VYn != 0.f) {
        const float ax = fabsf(VXn), ay = fabsf(VYn);
        d.f[F_MAXVX] = ax >= ay ? ax : ay;
        const float rx = fabsf(VXn / dx), ry = fabsf(VYn / dy);
        d.f[F_DTD] = (float)a.c.tcd * 1.f / (rx >= ry ? rx : ry);
      }
      if (P.RSFmode == 1) {
        rsf_node = true;
        float nps = 0.f;
        if (P.pmode == 0) nps = (float)P.nstress;
        else if (P.pmode == 1) nps = a.oldornew == 0 ? N.f(V2C_NF_SPPES)[m3] : N.f(V2C_NF_PRS)[m3];
        const float bm = N.f(V2C_NF_BM)[m3];
        const float as = N.f(V2C_NF_AS)[m3], bs = N.f(V2C_NF_BS)[m3], Ls = N.f(V2C_NF_LS)[m3];
        const float v = (3.f * bm - 2.f * gg) / (2.f * (3.f * bm + gg));
        const float k = 2.f / 3.14f * (gg / (1.f - v)) / (float)P.xstpx;
        const float q = k * Ls / (as * nps);
        const float h = q - (bs - as) / as;
        const float chi = 0.25f * h * h - q;
        if (chi > 0.f) { lam_raw = as * nps / (k * Ls - (bs - as) * nps); chi_ok = true; }
        else if (chi < 0.f) { lam_raw = 1.f - (bs - as) * nps / (k * Ls); chi_ok = true; }
        else if (chi == 0.f) a.out[TS_CHI0] = 1.0;
        reset = !(bs > 0.f);
        if (!reset) {
          const float Vf = N.f(V2C_NF_RK_SLIPRS_FINAL)[m3], Vs = N.f(V2C_NF_RK_SLIPRS_SOLVED)[m3];
          if (a.oldornew == 0 && Vf > 0.f) {
            dtphi = (float)a.c.tcphih * 1.f / (N.f(V2C_NF_V0S)[m3] / Ls * expf(-N.f(V2C_NF_PHIS)[m3]));
            LoV = Ls / Vf;
            has_phi = true;
          } else if (a.oldornew == 1 && Vs > 0.f) {
            dtphi = (float)a.c.tcphih * 1.f / (N.f(V2C_NF_V0S)[m3] / Ls * expf(-N.f(V2C_NF_PHIS_IT)[m3]));
            LoV = Ls / Vs;
            has_phi = true;
          }
        }
      }
      const float sx = N.f(V2C_NF_SXXS)[m3], sy = N.f(V2C_NF_SXY)[m3];
      const float sgf = sqrtf(sx * sx + sy * sy), nvf = N.f(V2C_NF_NU)[m3];
      st = N.f(V2C_NF_STICKY01)[m3];
      if (st == 1.f || st == 2.f) {
        const double sg = sgf, l = log10((double)nvf);
        if (st == 2.f) {
          d.f[F_MINS1] = d.f[F_MAXS1] = sgf; d.f[F_MINV1] = d.f[F_MAXV1] = nvf;
          d.d[D_NR1] = 1; d.d[D_SUMS1] = sg; d.d[D_SUM2S1] = sg * sg;
          d.d[D_SUMV1] = l; d.d[D_SUM2V1] = l * l;
        } else {
          d.f[F_MINS0] = d.f[F_MAXS0] = sgf; d.f[F_MINV0] = d.f[F_MAXV0] = nvf;
          d.d[D_NR0] = 1; d.d[D_SUMS0] = sg; d.d[D_SUM2S0] = sg * sg;
          d.d[D_SUMV0] = l; d.d[D_SUM2V0] = l * l;
          if (m1 == 50 && m2 == 50) { a.out[TS_P1S] = sg; a.out[TS_P1V] = nvf; }
          if (m1 == 500 && m2 == 50) { a.out[TS_P2S] = sg; a.out[TS_P2V] = nvf; }
        }
      }
      const float V = a.oldornew == 0 ? N.f(V2C_NF_RK_SLIPRS_FINAL)[m3] : N.f(V2C_NF_RK_SLIPRS_SOLVED)[m3];
      if (V > 0.f) d.f[F_MAXVEL] = V;
    }
    // lambda: the node's own, or that of the last earlier node with a
    // defined chi (within the slice, else carried from earlier slices)
    const unsigned okm = __ballot_sync(V2C_FULL, rsf_node && chi_ok);
    const unsigned below = okm & ((lane == 31) ? 0xffffffffu : ((2u << lane) - 1u));
    const int src = below ? 31 - __clz(below) : -1;
    const float lam_from = __shfl_sync(V2C_FULL, lam_raw, src < 0 ? 0 : src);
    const float lam = src >= 0 ? lam_from : lam_carry;
    if (okm) lam_carry = __shfl_sync(V2C_FULL, lam_raw, 31 - __clz(okm));
    if (rsf_node) {
      if (reset) {
        d.reset = true;
      } else if (has_phi) {
        const float lamc = lam <= 0.2f ? lam : 0.2f;  // MINV(lambda, 1/5)
        d.all[0] = d.after[0] = dtphi;
        d.all[1] = d.after[1] = lamc * LoV;
      }
    }
    const bool any0 = __any_sync(V2C_FULL, st == 1.f), any1 = __any_sync(V2C_FULL, st == 2.f);
    ts_fold_lanes(d, any0, any1, lane);
    if (lane == 0) ts_append(s, d, any0 || any1);
  }
  const int wl = threadIdx.x >> 5;
  if (lane == 0) ts_store(s, part[wl]);
  __syncthreads();
  ts_fold(part, TW, wl, TW, lane);
  if (threadIdx.x < TS_N) a.part[(long)blockIdx.x * TS_N + threadIdx.x] = part[0][threadIdx.x];
}

// fold the block partials in order, in shared memory (301 x 101 lines: 68 us
// as a tree in global memory with a thread per pair, 17 in shared memory, 10
// with integer comparisons)
constexpr int TF = 16;  // warps
// The results go to the host's memory, and the slots that the node pass sets
// by hand are zero again for the next call.
__global__ void __launch_bounds__(TF * 32) k_ts_fold(const double *part, int nb, double *out,
                                                     double *result) {
  after_previous();
  extern __shared__ double p[][TS_N];
  for (int i = threadIdx.x; i < nb * TS_N; i += TF * 32) p[i / TS_N][i % TS_N] = part[i];
  __syncthreads();
  ts_fold(p, nb, threadIdx.x >> 5, TF, threadIdx.x & 31);
  const int t = threadIdx.x;
  if (t < TS_OUT_N) {
    result[t] = t < TS_N ? p[0][t] : out[t];
    out[t] = 0.0;
  }
}
static_assert(TS_OUT_N <= RESULT_DOUBLES, "result buffer");
constexpr long TS_MAX_WARPS = 152 * 4 * TW;

}  // namespace

cudaError_t timestep_init() {
  return cudaFuncSetAttribute(k_ts_fold, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(sizeof(double) * TS_N * (TS_MAX_WARPS / TW)));
}

int calc_timestep_device(const Grid &g, const Nodes &N, const Scal &S, const v2c_timestep_ctl &c,
                         int oldornew, double *scratch, long scratch_doubles,
                         double *result, v2c_timestep_info *info, cudaStream_t st) {
  long per_warp = (g.nn + TS_MAX_WARPS - 1) / TS_MAX_WARPS;
  per_warp = (per_warp + 31) / 32 * 32;
  const long warps = (g.nn + per_warp - 1) / per_warp;
  if ((warps + 1) * TS_N + TS_OUT_N > scratch_doubles) return V2C_ERR_CAPACITY;
  TsArgs a;
  a.g = g; a.N = N; a.S = S; a.c = c; a.oldornew = oldornew; a.per_warp = per_warp;
  a.out = scratch;
  a.part = scratch + TS_OUT_N;
  const long blocks = (warps + TW - 1) / TW;
  // warps past the node range write empty partials
  launch_after(k_ts_nodes, (unsigned)blocks, TW * 32, 0, st, a);
  launch_after(k_ts_fold, 1, TF * 32, sizeof(double) * TS_N * blocks, st, a.part, (int)blocks,
               a.out, result);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess)
    return V2C_ERR_CUDA;
  const double *h = result;
  if (h[TS_CHI0] != 0.0) return V2C_ERR_TIMESTEP;
  const double dtphi = h[TS_RESET] != 0.0 ? (h[TS_PHI_AFTER] <= c.maxtmstep ? h[TS_PHI_AFTER] : c.maxtmstep)
                                          : h[TS_PHI_ALL];
  const double dtL = h[TS_RESET] != 0.0 ? (h[TS_L_AFTER] <= c.maxtmstep ? h[TS_L_AFTER] : c.maxtmstep)
                                        : h[TS_L_ALL];
  auto minv = [](double x, double y) { return x <= y ? x : y; };
  info->dt_f = c.dtfactor * minv(c.maxtmstep, minv(dtphi, minv(minv(dtL, h[TS_DTNVP]), h[TS_DTD])));
  info->maxvel = h[TS_MAXVEL];
  info->maxVx = h[TS_MAXVX];
  info->dtnvp = h[TS_DTNVP]; info->dtd = h[TS_DTD]; info->dtphi = dtphi; info->dtL = dtL;
  info->nr_0 = (long)h[TS_NR0]; info->nr_1 = (long)h[TS_NR1];
  info->max_sigin_0 = h[TS_MAXS0]; info->min_sigin_0 = h[TS_MINS0];
  info->sum_sigin_0 = h[TS_SUMS0]; info->sum2_sigin_0 = h[TS_SUM2S0];
  info->max_visc_0 = h[TS_MAXV0]; info->min_visc_0 = h[TS_MINV0];
  info->sum_visc_0 = h[TS_SUMV0]; info->sum2_visc_0 = h[TS_SUM2V0];
  info->max_sigin_1 = h[TS_MAXS1]; info->min_sigin_1 = h[TS_MINS1];
  info->sum_sigin_1 = h[TS_SUMS1]; info->sum2_sigin_1 = h[TS_SUM2S1];
  info->max_visc_1 = h[TS_MAXV1]; info->min_visc_1 = h[TS_MINV1];
  info->sum_visc_1 = h[TS_SUMV1]; info->sum2_visc_1 = h[TS_SUM2V1];
  info->sigin_P1 = h[TS_P1S]; info->sigin_P2 = h[TS_P2S];
  info->visco_P1 = h[TS_P1V]; info->visco_P2 = h[TS_P2V];
  return V2C_OK;
}

}  // namespace v2c
