// CloverLeaf 3D: the hydro cycle's loops fused by hand, queued by the app
// driver (apps_clover3d.cpp) in place of runs of the reference's loops, as
// kernels_clover_fused.cu does in 2D: volumes, node masses, node fluxes,
// energy and momentum fluxes stay in registers, and a step moves 1090 B per
// cell in 12 launches (and 57 B in boundary copies) instead of 2565 B in some
// 60. Every value is computed by the reference's expressions in the reference's
// order, so fields and dt are the same bits; the summary's sums are taken in
// another order. Measured at 256^3: 12.4 -> 5.65 ms of kernels a step, copies
// included, a 4-step run with its set-up 58.9 -> 30.5 ms (36.9 before every
// march's loads were issued one row ahead of their use: Raw, Row below).
//
// Each warp marches along y or z with one column of x per lane: the marched
// axis's neighbours are kept from row to row, x neighbours come by shuffles,
// the third axis's neighbouring line is loaded as well (the next warp of the
// CTA works on it, so it hits L1). The reference's eight-corner loops load
// every corner of every field at every point; a march loads two values.
#include <algorithm>
#include <cstddef>

#include "clover3d_common.h"
#include "clover_flux.cuh"
#include "march_grid.h"
#include "runtime.h"

namespace opsb {
namespace clover3d {
namespace fused {

using clover::advec_cell_face;
using clover::advec_mom_face;

__constant__ Consts c3;

using D = ACC3<double>;

#define C3_LOOP(NAME) static constexpr const char *kname = "cloverleaf3d/" #NAME

constexpr int kWarps = 4;  // warps per CTA: neighbouring lines of the third axis
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ double from_left(double v) { return __shfl_up_sync(kAll, v, 1); }
__device__ __forceinline__ double from_left2(double v) { return __shfl_up_sync(kAll, v, 2); }
__device__ __forceinline__ double from_right(double v) { return __shfl_down_sync(kAll, v, 1); }
__device__ __forceinline__ double from_right2(double v) { return __shfl_down_sync(kAll, v, 2); }

// One argument at the lane's column X.
struct Fld {
  double *p;
  int pitch, plane;
  __device__ __forceinline__ Fld(const ArgView &a, int X)
      : p(reinterpret_cast<double *>(a.ptr) + X), pitch(a.ay), plane(a.az) {}
  __device__ __forceinline__ double *at(int y, int z) const {
    return p + ((long long)y * pitch + (long long)z * plane);
  }
  __device__ __forceinline__ double operator()(int y, int z) const { return __ldg(at(y, z)); }
  __device__ __forceinline__ double right(int y, int z) const { return __ldg(at(y, z) + 1); }
  __device__ __forceinline__ void put(int y, int z, double v) const { *at(y, z) = v; }
};

// A one-dimensional argument along axis AX (cell and vertex widths).
template <int AX>
struct Widths {
  const double *p;
  int s;
  __device__ __forceinline__ Widths(const ArgView &a)
      : p(reinterpret_cast<const double *>(a.ptr)), s(AX == 0 ? a.sx : AX == 1 ? a.sy : a.sz) {}
  __device__ __forceinline__ double operator()(int i) const { return __ldg(p + (long long)i * s); }
};

// A warp's part of the range: its lane's column X (EDGE lanes before the
// strip's first owned column, OWN owned), one line of the third axis and rows
// [m0, m1) of the marched axis M (1: y, 2: z).
template <int OWN, int EDGE, int M>
struct March {
  int X, o, m0, m1;
  bool own, live;
  __device__ __forceinline__ March(const LoopParams &lp, int rows)
      : March(lp, rows, blockIdx.x * kWarps + (threadIdx.x >> 5)) {}
  __device__ __forceinline__ March(const LoopParams &lp, int rows, int w) {
    constexpr int O = M == 1 ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const int ncol = (lp.end[0] - lp.start[0] + OWN - 1) / OWN, lines = lp.end[O] - lp.start[O];
    const int rest = w / lines, c = rest % ncol;
    o = lp.start[O] + w % lines;
    X = lp.start[0] + c * OWN + lane - EDGE;
    m0 = lp.start[M] + (rest / ncol) * rows;
    m1 = min(m0 + rows, lp.end[M]);
    live = m0 < lp.end[M];
    own = live && lane >= EDGE && lane < EDGE + OWN && X < lp.end[0];
  }
};

// HALO: rows a march reads beyond its own.
template <int OWN, int M, int HALO, auto kernel>
void launch_march(const LoopParams &lp, cudaStream_t s) {
  static int per_sm = 0;  // resident CTAs, this kernel's
  if (!per_sm) {
    int n = 0;
    OPSB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 32 * kWarps, 0));
    per_sm = std::max(n, 1);
  }
  constexpr int O = M == 1 ? 2 : 1;
  const long long nx = lp.end[0] - lp.start[0], no = lp.end[O] - lp.start[O];
  const int nm = lp.end[M] - lp.start[M];
  const long long columns = (nx + OWN - 1) / OWN * no;
  const int rows = march_rows(columns, nm, HALO, 148LL * per_sm * kWarps, (long long)Runtime::kMaxRedBlocks * kWarps);
  long long blocks = (columns * ((nm + rows - 1) / rows) + kWarps - 1) / kWarps;
  // a kernel that reduces goes over its parts with the grid's stride
  if (lp.nred > 0) blocks = std::min<long long>(blocks, Runtime::kMaxRedBlocks);
  kernel<<<(unsigned)blocks, 32 * kWarps, 0, s>>>(lp, rows);
}

// The grid's reductions: `v[k]` belongs to argument first + k (every thread
// of the CTA takes part).
template <int N>
__device__ __forceinline__ void reduce_grid(const LoopParams &lp, int first, const double (&v)[N]) {
  __shared__ double smem[32];
  __shared__ int last;
  const int nblocks = gridDim.x;
#pragma unroll
  for (int k = 0; k < N; k++) {
    const ArgView &a = lp.a[first + k];
    const double b = block_reduce<double>(v[k], a.acc, smem);
    if (threadIdx.x == 0)
      reinterpret_cast<double *>(lp.red_scratch)[((size_t)a.red_index * nblocks + blockIdx.x) * OPSB_MAX_RED_DIM] = b;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(lp.red_counter, 1u) == (unsigned)(nblocks - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < N; k++) finish_grid_reduction<double>(lp.a[first + k], lp, nblocks, smem);
  if (threadIdx.x == 0) *lp.red_counter = 0u;
}

// A velocity on one plane: the node (x, y) and its right, upper and upper
// right neighbours.
struct Quad {
  double v00, v10, v01, v11;
  __device__ __forceinline__ Quad(double a, double b) : v00(a), v10(from_right(a)), v01(b), v11(from_right(b)) {}
  __device__ __forceinline__ Quad(const Fld &f, int y, int z) : Quad(f(y, z), f(y + 1, z)) {}
};

// ideal_gas_kernel then field_summary_kernel. A node's kinetic term is the
// same product at each of the eight cells around it.
__global__ void __launch_bounds__(32 * kWarps, 5) summary_kernel(const __grid_constant__ LoopParams lp, int rows) {
  double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  // one part a warp, but more columns than kMaxRedBlocks CTAs have warps (2880 x 2880 x 8, say) take several
  for (int w = blockIdx.x * kWarps + (threadIdx.x >> 5);; w += gridDim.x * kWarps) {
    const March<31, 0, 2> m(lp, rows, w);
    if (!m.live) break;
    const int X = min(m.X, lp.end[0]);
    const Fld density0(lp.a[0], X), energy0(lp.a[1], X), pressure(lp.a[2], X), soundspeed(lp.a[3], X),
        volume(lp.a[4], X), xvel0(lp.a[5], X), yvel0(lp.a[6], X), zvel0(lp.a[7], X);
    const int y = m.o;
    auto kin = [](double a, double b, double c) { return 0.125 * (a * a + b * b + c * c); };
    struct Raw {  // velocities of plane z + 1 at rows y and y + 1, cell values of plane z
      double u0, u1, v0, v1, w0, w1, d, e, vol;
    };
    auto load = [&](int z) {
      return Raw{xvel0(y, z + 1), xvel0(y + 1, z + 1), yvel0(y, z + 1), yvel0(y + 1, z + 1), zvel0(y, z + 1),
                 zvel0(y + 1, z + 1), density0(y, z), energy0(y, z), volume(y, z)};
    };
    double k0 = kin(xvel0(y, m.m0), yvel0(y, m.m0), zvel0(y, m.m0));
    double k1 = kin(xvel0(y + 1, m.m0), yvel0(y + 1, m.m0), zvel0(y + 1, m.m0));
    double k0r = from_right(k0), k1r = from_right(k1);
    Raw c = load(m.m0);
    for (int z = m.m0; z < m.m1; z++) {
      const Raw n = load(min(z + 1, m.m1 - 1));
      const double n0 = kin(c.u0, c.v0, c.w0), n1 = kin(c.u1, c.v1, c.w1);
      const double n0r = from_right(n0), n1r = from_right(n1);
      if (m.own) {
        const double d = c.d, e = c.e, cell_vol = c.vol;
        const double v = 1.0 / d;
        const double p = (1.4 - 1.0) * d * e;
        pressure.put(y, z, p);
        const double pressurebyenergy = (1.4 - 1.0) * d;
        const double pressurebyvolume = -1.0 * d * p;
        const double sound_speed_squared = v * v * (p * pressurebyenergy - pressurebyvolume);
        soundspeed.put(y, z, sqrt(sound_speed_squared));
        double vsqrd = 0.0;
        vsqrd += k0;
        vsqrd += k0r;
        vsqrd += k1;
        vsqrd += k1r;
        vsqrd += n0;
        vsqrd += n0r;
        vsqrd += n1;
        vsqrd += n1r;
        const double cell_mass = cell_vol * d;
        sum[0] = sum[0] + cell_vol;
        sum[1] = sum[1] + cell_mass;
        sum[2] = sum[2] + cell_mass * e;
        sum[3] = sum[3] + cell_mass * 0.5 * vsqrd;
        sum[4] = sum[4] + cell_vol * p;
      }
      k0 = n0;
      k1 = n1;
      k0r = n0r;
      k1r = n1r;
      c = n;
    }
  }
  reduce_grid<5>(lp, 8, sum);
}

struct ideal_gas_summary {
  C3_LOOP(ideal_gas_summary);
  static constexpr bool red_mirror = true;
  __device__ void operator()(const D &density0, const D &energy0, D &pressure, D &soundspeed, const D &volume,
                             const D &xvel0, const D &yvel0, const D &zvel0, RED<double> &vol, RED<double> &mass,
                             RED<double> &ie, RED<double> &ke, RED<double> &press) const;
  static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_march<31, 2, 1, summary_kernel>(lp, s); }
};

// calc_dt_kernel with calc_dt_kernel_min folded in. Point by point: the six
// divisions and the square root of a cell want the many warps that the plain
// executor keeps resident, so a z march gained nothing (0.49 ms at 256^3
// against 0.50 ms; viscosity_kernel as a march took 0.66 ms against 0.47 ms
// and stays the reference's loop).
struct calc_dt_fused {
  C3_LOOP(calc_dt_fused);
  static constexpr int min_blocks = 4;
  __device__ void operator()(const D &celldx, const D &celldy, const D &soundspeed, const D &viscosity,
                             const D &density0, const D &xvel0, const D &xarea, const D &volume, const D &yvel0,
                             const D &yarea, RED<double> &dt_min, const D &celldz, const D &zvel0,
                             const D &zarea) const {
    double div, ds, dtut, dtvt, dtct, dtwt, dtdivt, cc, dv1, dv2, du1, du2, dw1, dw2;
    ds = op_min(op_min(celldx(0, 0, 0), celldy(0, 0, 0)), celldz(0, 0, 0));
    ds = 1.0 / (ds * ds);
    cc = soundspeed(0, 0, 0) * soundspeed(0, 0, 0);
    cc = cc + qdiv(2.0 * viscosity(0, 0, 0), density0(0, 0, 0));
    dtct = ds * cc;
    dtct = c3.dtc_safe * 1.0 / op_max(sqrt(dtct), c3.g_small);
    du1 = (xvel0(0, 0, 0) + xvel0(0, 1, 0) + xvel0(0, 0, 1) + xvel0(0, 1, 1)) * xarea(0, 0, 0);
    du2 = (xvel0(1, 0, 0) + xvel0(1, 1, 0) + xvel0(1, 0, 1) + xvel0(1, 1, 1)) * xarea(0, 0, 0);
    dtut = c3.dtu_safe * 4.0 * volume(0, 0, 0) / op_max(op_max(fabs(du1), fabs(du2)), 1.0e-5 * volume(0, 0, 0));
    dv1 = (yvel0(0, 0, 0) + yvel0(1, 0, 0) + yvel0(0, 0, 1) + yvel0(1, 0, 1)) * yarea(0, 0, 0);
    dv2 = (yvel0(0, 1, 0) + yvel0(1, 1, 0) + yvel0(0, 1, 1) + yvel0(1, 1, 1)) * yarea(0, 0, 0);
    dtvt = c3.dtv_safe * 4.0 * volume(0, 0, 0) / op_max(op_max(fabs(dv1), fabs(dv2)), 1.0e-5 * volume(0, 0, 0));
    dw1 = (zvel0(0, 0, 0) + zvel0(0, 1, 0) + zvel0(1, 0, 0) + zvel0(1, 1, 0)) * zarea(0, 0, 0);
    dw2 = (zvel0(0, 0, 1) + zvel0(0, 1, 1) + zvel0(1, 0, 1) + zvel0(1, 1, 1)) * zarea(0, 0, 0);
    dtwt = c3.dtw_safe * 4.0 * volume(0, 0, 0) / op_max(op_max(fabs(dw1), fabs(dw2)), 1.0e-5 * volume(0, 0, 0));
    div = du2 - du1 + dv2 - dv1 + dw2 - dw1;
    dtdivt = c3.dtdiv_safe * 4.0 * (volume(0, 0, 0)) / op_max(volume(0, 0, 0) * 1.0e-05, fabs(div));
    *dt_min = op_min(*dt_min, op_min(op_min(op_min(dtct, dtut), op_min(dtvt, dtdivt)), dtwt));
  }
};

// PdV_kernel_predict then the ideal gas pressure of the predicted state; the
// predicted density and energy are nothing else's inputs (revert_kernel
// restores them and PdV_kernel_nopredict overwrites them unread).
__global__ void __launch_bounds__(32 * kWarps, 4) predict_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<31, 0, 2> m(lp, rows);
  if (!m.live) return;
  const int X = min(m.X, lp.end[0]), y = m.o;
  const Fld xarea(lp.a[0], X), xvel0(lp.a[1], X), yarea(lp.a[2], X), yvel0(lp.a[3], X), zarea(lp.a[4], X),
      zvel0(lp.a[5], X), volume(lp.a[6], X), pressure(lp.a[7], X), density0(lp.a[8], X), viscosity(lp.a[9], X),
      energy0(lp.a[10], X);
  const double dt = c3.dt;
  struct Raw {  // plane z + 1: velocities at rows y and y + 1, z area; plane z: the rest
    double u0, u1, v0, v1, w0, w1, za, xa, ya, yt, vol, p, d, q, e;
  };
  auto load = [&](int z) {
    return Raw{xvel0(y, z + 1),     xvel0(y + 1, z + 1), yvel0(y, z + 1), yvel0(y + 1, z + 1), zvel0(y, z + 1),
               zvel0(y + 1, z + 1), zarea(y, z + 1),     xarea(y, z),     yarea(y, z),         yarea(y + 1, z),
               volume(y, z),        *pressure.at(y, z),  density0(y, z),  viscosity(y, z),     energy0(y, z)};
  };
  double u0 = xvel0(y, m.m0), u1 = xvel0(y + 1, m.m0);
  Quad v(yvel0, y, m.m0);
  auto zflux = [&](const Quad &q, double za) {
    return (za * (q.v00 + q.v10 + q.v01 + q.v11 + q.v00 + q.v10 + q.v01 + q.v11)) * 0.125 * dt * 0.5;
  };
  double back_flux = zflux(Quad(zvel0, y, m.m0), zarea(y, m.m0));
  Raw c = load(m.m0);
  for (int z = m.m0; z < m.m1; z++) {
    const Raw n = load(min(z + 1, m.m1 - 1));
    const double u0n = c.u0, u1n = c.u1;
    const Quad vn(c.v0, c.v1);
    const double left_flux = (c.xa * (u0 + u1 + u0n + u1n + u0 + u1 + u0n + u1n)) * 0.125 * dt * 0.5;
    const double right_flux = from_right(left_flux);
    const double front_flux = zflux(Quad(c.w0, c.w1), c.za);
    if (m.own) {
      const double bottom_flux =
          (c.ya * (v.v00 + v.v10 + vn.v00 + vn.v10 + v.v00 + v.v10 + vn.v00 + vn.v10)) * 0.125 * dt * 0.5;
      const double top_flux =
          (c.yt * (v.v01 + v.v11 + vn.v01 + vn.v11 + v.v01 + v.v11 + vn.v01 + vn.v11)) * 0.125 * dt * 0.5;
      const double total_flux = right_flux - left_flux + top_flux - bottom_flux + front_flux - back_flux;
      const double volume_change = (c.vol) / (c.vol + total_flux);
      const double recip_volume = 1.0 / c.vol;
      const double energy_change = (c.p / c.d + qdiv(c.q, c.d)) * total_flux * recip_volume;
      const double energy1 = c.e - energy_change;
      const double density1 = c.d * volume_change;
      pressure.put(y, z, (1.4 - 1.0) * density1 * energy1);
    }
    u0 = u0n;
    u1 = u1n;
    v = vn;
    back_flux = front_flux;
    c = n;
  }
}

struct PdV_predict_pressure {
  C3_LOOP(PdV_predict_pressure);
  __device__ void operator()(const D &xarea, const D &xvel0, const D &yarea, const D &yvel0, const D &zarea,
                             const D &zvel0, const D &volume, D &pressure, const D &density0, const D &viscosity,
                             const D &energy0) const;
  static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_march<31, 2, 1, predict_march>(lp, s); }
};

// accelerate_kernel. A plane's share of a node's mass and forces is computed
// once and kept for the node above.
__global__ void __launch_bounds__(32 * kWarps, 3) accelerate_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<31, 1, 2> m(lp, rows);
  if (!m.live) return;
  const int X = min(m.X, lp.end[0] - 1), y = m.o;
  const Fld density0(lp.a[0], X), volume(lp.a[1], X), pressure(lp.a[2], X), viscosity(lp.a[3], X), xarea(lp.a[4], X),
      yarea(lp.a[5], X), zarea(lp.a[6], X), xvel0(lp.a[7], X), yvel0(lp.a[8], X), zvel0(lp.a[9], X), xvel1(lp.a[10], X),
      yvel1(lp.a[11], X), zvel1(lp.a[12], X);
  const double qdt = 0.25 * c3.dt;
  struct Plane {
    double m0, m1, m0l, m1l;          // density x volume at rows y, y - 1, and left of them
    double p0, p1, q0, q1;            // pressure and viscosity at rows y, y - 1
    double xp0, xp1, xq0, xq1;        // x forces of rows y, y - 1
    double yp, ypl, yq, yql;          // y forces at the column and left of it
  };
  struct Raw {  // the plane's own values at rows y and y - 1
    double d0, d1, v0, v1, p0, p1, q0, q1, xa0, xa1, ya, za0, za1, xv, yv, zv;
  };
  auto load = [&](int z) {
    return Raw{density0(y, z),  density0(y - 1, z),  volume(y, z),  volume(y - 1, z), pressure(y, z), pressure(y - 1, z),
               viscosity(y, z), viscosity(y - 1, z), xarea(y, z),   xarea(y - 1, z),  yarea(y, z),    zarea(y, z),
               zarea(y - 1, z), xvel0(y, z),         yvel0(y, z),   zvel0(y, z)};
  };
  auto plane = [&](const Raw &w) {
    Plane r;
    r.m0 = w.d0 * w.v0;
    r.m1 = w.d1 * w.v1;
    r.m0l = from_left(r.m0);
    r.m1l = from_left(r.m1);
    r.p0 = w.p0;
    r.p1 = w.p1;
    r.q0 = w.q0;
    r.q1 = w.q1;
    r.xp0 = w.xa0 * (r.p0 - from_left(r.p0));
    r.xp1 = w.xa1 * (r.p1 - from_left(r.p1));
    r.xq0 = w.xa0 * (r.q0 - from_left(r.q0));
    r.xq1 = w.xa1 * (r.q1 - from_left(r.q1));
    r.yp = w.ya * (r.p0 - r.p1);
    r.yq = w.ya * (r.q0 - r.q1);
    r.ypl = from_left(r.yp);
    r.yql = from_left(r.yq);
    return r;
  };
  Raw w = load(m.m0);
  Plane b = plane(load(m.m0 - 1));
  for (int z = m.m0; z < m.m1; z++) {
    const Raw n = load(min(z + 1, m.m1 - 1));
    const Plane c = plane(w);
    const double za0 = w.za0, za1 = w.za1;
    const double zp0 = za0 * (c.p0 - b.p0), zp1 = za1 * (c.p1 - b.p1);
    const double zq0 = za0 * (c.q0 - b.q0), zq1 = za1 * (c.q1 - b.q1);
    const double zp0l = from_left(zp0), zp1l = from_left(zp1), zq0l = from_left(zq0), zq1l = from_left(zq1);
    if (m.own) {
      const double nodal_mass = (c.m1l + c.m1 + c.m0 + c.m0l + b.m1l + b.m1 + b.m0 + b.m0l) * 0.125;
      const double stepbymass = qdt / nodal_mass;
      double xv = w.xv - stepbymass * (c.xp0 + c.xp1 + b.xp0 + b.xp1);
      double yv = w.yv - stepbymass * (c.yp + c.ypl + b.yp + b.ypl);
      double zv = w.zv - stepbymass * (zp0 + zp1 + zp0l + zp1l);
      xv = xv - stepbymass * (c.xq0 + c.xq1 + b.xq0 + b.xq1);
      yv = yv - stepbymass * (c.yq + c.yql + b.yq + b.yql);
      zv = zv - stepbymass * (zq0 + zq1 + zq0l + zq1l);
      xvel1.put(y, z, xv);
      yvel1.put(y, z, yv);
      zvel1.put(y, z, zv);
    }
    b = c;
    w = n;
  }
}

struct accelerate_fused {
  C3_LOOP(accelerate_fused);
  __device__ void operator()(const D &density0, const D &volume, const D &pressure, const D &viscosity,
                             const D &xarea, const D &yarea, const D &zarea, const D &xvel0, const D &yvel0,
                             const D &zvel0, D &xvel1, D &yvel1, D &zvel1) const;
  static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_march<31, 2, 1, accelerate_march>(lp, s); }
};

// PdV_kernel_nopredict and flux_calc_kernel{x,y,z} over the nodes; each
// flux stops one short of the nodes in the directions across its face.
__global__ void __launch_bounds__(32 * kWarps, 3) pdv_flux_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<31, 0, 2> m(lp, rows);
  if (!m.live) return;
  const int X = min(m.X, lp.end[0]), y = m.o;
  const Fld xarea(lp.a[0], X), yarea(lp.a[1], X), zarea(lp.a[2], X), xvel0(lp.a[3], X), xvel1(lp.a[4], X),
      yvel0(lp.a[5], X), yvel1(lp.a[6], X), zvel0(lp.a[7], X), zvel1(lp.a[8], X), volume(lp.a[9], X),
      pressure(lp.a[10], X), density0(lp.a[11], X), viscosity(lp.a[12], X), energy0(lp.a[13], X), density1(lp.a[14], X),
      energy1(lp.a[15], X), vol_flux_x(lp.a[16], X), vol_flux_y(lp.a[17], X), vol_flux_z(lp.a[18], X);
  const double dt = c3.dt, edt = 0.125 * c3.dt;
  const int zcell = lp.end[2] - 1;
  const bool cx = m.own && m.X < lp.end[0] - 1, cy = y < lp.end[1] - 1;
  struct Raw {  // plane z + 1: both velocities at rows y and y + 1, z area; plane z: the rest
    double u0, u1, t0, t1, v0, v1, s0, s1, w0, w1, r0, r1, za, xa, ya, yt, vol, p, d, q, e;
  };
  auto load = [&](int z) {
    return Raw{xvel0(y, z + 1), xvel0(y + 1, z + 1), xvel1(y, z + 1), xvel1(y + 1, z + 1), yvel0(y, z + 1),
               yvel0(y + 1, z + 1), yvel1(y, z + 1), yvel1(y + 1, z + 1), zvel0(y, z + 1), zvel0(y + 1, z + 1),
               zvel1(y, z + 1), zvel1(y + 1, z + 1), zarea(y, z + 1), xarea(y, z), yarea(y, z), yarea(y + 1, z),
               volume(y, z), pressure(y, z), density0(y, z), viscosity(y, z), energy0(y, z)};
  };
  double u0 = xvel0(y, m.m0), u1 = xvel0(y + 1, m.m0), t0 = xvel1(y, m.m0), t1 = xvel1(y + 1, m.m0);
  Quad v(yvel0, y, m.m0), s(yvel1, y, m.m0);
  // the z face of plane z: its flux of volume (the reference's flux_calc reads
  // zvel0(1,0,0) twice) and the PdV flux through it
  auto zface = [&](const Quad &w, const Quad &r, double za, double &flux, double &vflux) {
    flux = (za * (w.v00 + w.v10 + w.v01 + w.v11 + r.v00 + r.v10 + r.v01 + r.v11)) * 0.125 * dt;
    vflux = edt * za * (w.v00 + w.v10 + w.v10 + w.v11 + r.v00 + r.v10 + r.v01 + r.v11);
  };
  double back_flux, vfz;
  zface(Quad(zvel0, y, m.m0), Quad(zvel1, y, m.m0), zarea(y, m.m0), back_flux, vfz);
  const int zlast = min(m.m1, zcell) - 1;  // the last plane with cells
  Raw c = load(min(m.m0, zcell - 1));
  for (int z = m.m0; z < m.m1; z++) {
    if (cx && cy) vol_flux_z.put(y, z, vfz);
    if (z == zcell) break;
    const Raw n = load(min(z + 1, zlast));
    const double u0n = c.u0, u1n = c.u1, t0n = c.t0, t1n = c.t1;
    const Quad vn(c.v0, c.v1), sn(c.s0, c.s1);
    double front_flux;
    zface(Quad(c.w0, c.w1), Quad(c.r0, c.r1), c.za, front_flux, vfz);
    const double xa = c.xa, ya = c.ya;
    const double xsum = u0 + u1 + u0n + u1n + t0 + t1 + t0n + t1n;
    const double ysum = v.v00 + v.v10 + vn.v00 + vn.v10 + s.v00 + s.v10 + sn.v00 + sn.v10;
    const double left_flux = (xa * xsum) * 0.125 * dt;
    const double right_flux = from_right(left_flux);
    if (m.own && cy) vol_flux_x.put(y, z, edt * xa * xsum);
    if (cx) {
      vol_flux_y.put(y, z, edt * ya * ysum);
      if (cy) {
        const double bottom_flux = (ya * ysum) * 0.125 * dt;
        const double top_flux =
            (c.yt * (v.v01 + v.v11 + vn.v01 + vn.v11 + s.v01 + s.v11 + sn.v01 + sn.v11)) * 0.125 * dt;
        const double total_flux = right_flux - left_flux + top_flux - bottom_flux + front_flux - back_flux;
        const double volume_change = (c.vol) / (c.vol + total_flux);
        const double recip_volume = 1.0 / c.vol;
        const double energy_change = (c.p / c.d + qdiv(c.q, c.d)) * total_flux * recip_volume;
        energy1.put(y, z, c.e - energy_change);
        density1.put(y, z, c.d * volume_change);
      }
    }
    u0 = u0n;
    u1 = u1n;
    t0 = t0n;
    t1 = t1n;
    v = vn;
    s = sn;
    back_flux = front_flux;
    c = n;
  }
}

struct PdV_flux {
  C3_LOOP(PdV_flux);
  __device__ void operator()(const D &xarea, const D &yarea, const D &zarea, const D &xvel0, const D &xvel1,
                             const D &yvel0, const D &yvel1, const D &zvel0, const D &zvel1, const D &volume,
                             const D &pressure, const D &density0, const D &viscosity, const D &energy0, D &density1,
                             D &energy1, D &vol_flux_x, D &vol_flux_y, D &vol_flux_z) const;
  static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_march<31, 2, 1, pdv_flux_march>(lp, s); }
};

// ---- advection -------------------------------------------------------------------

// Which fluxes a sweep's volumes hold: all three (the step's first sweep),
// y and z (second, x first), y and x (second, z first), or the sweep's own
// (third). The cell sweep's pre-advection volume and the momentum sweep's
// post-advection volume (which lacks the sweep's own flux) follow from it.
enum { VOL_FIRST = 0, VOL_YZ = 1, VOL_YX = 2, VOL_LAST = 3 };

// advec_cell_kernel{1,2}_{x,y,z}dir's pre_vol at (y, z) of the lane's column.
template <int DIR, int VOL>
__device__ __forceinline__ double pre_volume(const Fld &vol, const Fld &vfx, const Fld &vfy, const Fld &vfz, int y,
                                             int z) {
  const double v = vol(y, z);
  if (VOL == VOL_FIRST)
    return v + (vfx.right(y, z) - vfx(y, z) + vfy(y + 1, z) - vfy(y, z) + vfz(y, z + 1) - vfz(y, z));
  if (VOL == VOL_YZ) return v + vfy(y + 1, z) - vfy(y, z) + vfz(y, z + 1) - vfz(y, z);
  if (VOL == VOL_YX) return v + vfy(y + 1, z) - vfy(y, z) + vfx.right(y, z) - vfx(y, z);
  return DIR == 0 ? v + vfx.right(y, z) - vfx(y, z) : v + vfz(y, z + 1) - vfz(y, z);
}

// advec_mom_kernel_{x1,z1,x2,y2,x3,z3}'s post_vol.
template <int DIR, int VOL>
__device__ __forceinline__ double post_volume(const Fld &vol, const Fld &vfx, const Fld &vfy, const Fld &vfz, int y,
                                              int z) {
  const double v = vol(y, z);
  if (VOL == VOL_FIRST && DIR == 0) return v + vfy(y + 1, z) - vfy(y, z) + vfz(y, z + 1) - vfz(y, z);
  if (VOL == VOL_FIRST) return v + vfx.right(y, z) - vfx(y, z) + vfy(y + 1, z) - vfy(y, z);
  if (VOL == VOL_YZ) return v + vfz(y, z + 1) - vfz(y, z);
  if (VOL == VOL_YX) return v + vfx.right(y, z) - vfx(y, z);
  return v;
}

// advec_cell_kernel{1,2}, 3 and 4 of one sweep; the range is the mass flux's,
// two cells longer than the cells along the sweep. Density and energy go to
// other dats than they came from; the step's last sweep writes the energy to
// energy0 and the density to density0 too (reset_field_kernel1).
// Arguments: volume, vol_flux_{x,y,z}, vertexd, density, energy, mass_flux,
// density out, energy out, [density0].
template <int VOL>
__global__ void __launch_bounds__(32 * kWarps, 5) advec_cell_x_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<28, 2, 1> m(lp, rows);
  if (!m.live) return;
  const int X = min(m.X, lp.end[0] + 1), z = m.o;
  const Fld volume(lp.a[0], X), vfx(lp.a[1], X), vfy(lp.a[2], X), vfz(lp.a[3], X), density(lp.a[5], X),
      energy(lp.a[6], X), mass_flux(lp.a[7], X), dout(lp.a[8], X), eout(lp.a[9], X),
      d0out(lp.a[VOL == VOL_LAST ? 10 : 8], X);
  const Widths<0> vd(lp.a[4]);
  const double w0 = vd(X);
  const double wm = qratio(w0, vd(X - 1)), wp = qratio(w0, vd(X + 1)), wc = qratio(w0, w0);
  const bool cell_max_test = m.X - 1 < c3.field.x_max;
  const bool cell = m.own && m.X < lp.end[0] - 2;
  struct Row {
    double f, v, d, e;  // v: the pre-advection volume
  };
  auto load = [&](int y) {
    return Row{vfx(y, z), pre_volume<0, VOL>(volume, vfx, vfy, vfz, y, z), density(y, z), energy(y, z)};
  };
  Row c = load(m.m0);
  for (int y = m.m0; y < m.m1; y++) {
    const Row n = load(min(y + 1, m.m1 - 1));
    const double f1 = from_right(c.f);
    const double pv = c.v, pvl = from_left(pv);
    const double d1 = from_right(c.d), dl = from_left(c.d), dll = from_left2(c.d);
    const double e1 = from_right(c.e), el = from_left(c.e), ell = from_left2(c.e);
    const bool pos = c.f > 0.0;
    double mf, ef;
    advec_cell_face(c.f, pos ? pvl : pv, pos ? wm : cell_max_test ? wp : wc, pos ? dl : c.d,
                    pos ? dll : cell_max_test ? d1 : c.d, pos ? c.d : dl, pos ? el : c.e,
                    pos ? ell : cell_max_test ? e1 : c.e, pos ? c.e : el, mf, ef);
    const double mf1 = from_right(mf), ef1 = from_right(ef);
    if (m.own) mass_flux.put(y, z, mf);
    if (cell) {
      const double pre_mass = c.d * pv;
      const double post_mass = pre_mass + mf - mf1;
      const double post_ener = (c.e * pre_mass + ef - ef1) / post_mass;
      const double advec_vol = pv + c.f - f1;
      const double dn = post_mass / advec_vol;
      dout.put(y, z, dn);
      eout.put(y, z, post_ener);
      if (VOL == VOL_LAST) d0out.put(y, z, dn);
    }
    c = n;
  }
}

// The same along y (DIR 1) or z (DIR 2): every lane owns its column.
template <int DIR, int VOL>
__global__ void __launch_bounds__(32 * kWarps, 5) advec_cell_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<32, 0, DIR> m(lp, rows);
  if (!m.own) return;
  const int X = m.X;
  const Fld volume(lp.a[0], X), vfx(lp.a[1], X), vfy(lp.a[2], X), vfz(lp.a[3], X), density(lp.a[5], X),
      energy(lp.a[6], X), mass_flux(lp.a[7], X), dout(lp.a[8], X), eout(lp.a[9], X),
      d0out(lp.a[VOL == VOL_LAST ? 10 : 8], X);
  const Fld &vf = DIR == 1 ? vfy : vfz;
  const Widths<DIR> vd(lp.a[4]);
  const int cmax = DIR == 1 ? c3.field.y_max : c3.field.z_max;
  auto yy = [&](int r) { return DIR == 1 ? r : m.o; };
  auto zz = [&](int r) { return DIR == 1 ? m.o : r; };
  // the y sweep's mass flux range also runs two cells beyond z's cells
  // (advec_cell.cpp:55): there is no cell to update there
  const bool line_cells = DIR == 2 || m.o < lp.end[2] - 2;
  const int last = lp.end[DIR] - 1, mend = min(m.m1, last);
  struct Row {  // row r: volume; density, energy and flux of row r + 1
    double v, d, e, f;
  };
  auto load = [&](int r) {
    return Row{pre_volume<DIR, VOL>(volume, vfx, vfy, vfz, yy(r), zz(r)), density(yy(r + 1), zz(r + 1)),
               energy(yy(r + 1), zz(r + 1)), vf(yy(r + 1), zz(r + 1))};
  };
  double dll = density(yy(m.m0 - 2), zz(m.m0 - 2)), ell = energy(yy(m.m0 - 2), zz(m.m0 - 2));
  double dl = density(yy(m.m0 - 1), zz(m.m0 - 1)), el = energy(yy(m.m0 - 1), zz(m.m0 - 1));
  Row c = load(m.m0 - 1);
  double pvl = c.v, dc = c.d, ec = c.e, f = c.f;
  double mfl = 0.0, efl = 0.0, fl = 0.0;
  c = load(m.m0);
  for (int r = m.m0; r <= mend; r++) {
    const Row n = load(min(r + 1, mend));
    const double dn = c.d, en = c.e, f1 = c.f, pv = c.v;
    const double w0 = vd(r);
    const bool pos = f > 0.0, cell_max_test = r - 1 < cmax;
    const double width = qratio(w0, pos ? vd(r - 1) : cell_max_test ? vd(r + 1) : w0);
    double mf, ef;
    advec_cell_face(f, pos ? pvl : pv, width, pos ? dl : dc, pos ? dll : cell_max_test ? dn : dc, pos ? dc : dl,
                    pos ? el : ec, pos ? ell : cell_max_test ? en : ec, pos ? ec : el, mf, ef);
    if (r < m.m1) mass_flux.put(yy(r), zz(r), mf);
    if (r > m.m0 && r - 1 < lp.end[DIR] - 2 && line_cells) {
      const double pre_mass = dl * pvl;
      const double post_mass = pre_mass + mfl - mf;
      const double post_ener = (el * pre_mass + efl - ef) / post_mass;
      const double advec_vol = pvl + fl - f;
      const double dnew = post_mass / advec_vol;
      dout.put(yy(r - 1), zz(r - 1), dnew);
      eout.put(yy(r - 1), zz(r - 1), post_ener);
      if (VOL == VOL_LAST) d0out.put(yy(r - 1), zz(r - 1), dnew);
    }
    dll = dl;
    ell = el;
    dl = dc;
    el = ec;
    dc = dn;
    ec = en;
    pvl = pv;
    mfl = mf;
    efl = ef;
    fl = f;
    f = f1;
    c = n;
  }
}

#define ADVEC_CELL(NAME, LAUNCH)                                                                                    \
  struct NAME {                                                                                                     \
    C3_LOOP(NAME);                                                                                                  \
    __device__ void operator()(const D &volume, const D &vol_flux_x, const D &vol_flux_y, const D &vol_flux_z,      \
                               const D &vertexd, const D &density, const D &energy, D &mass_flux, D &dout, D &eout) \
        const;                                                                                                      \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { LAUNCH; }                                \
  };
#define ADVEC_CELL_LAST(NAME, LAUNCH)                                                                               \
  struct NAME {                                                                                                     \
    C3_LOOP(NAME);                                                                                                  \
    __device__ void operator()(const D &volume, const D &vol_flux_x, const D &vol_flux_y, const D &vol_flux_z,      \
                               const D &vertexd, const D &density, const D &energy, D &mass_flux, D &dout, D &eout, \
                               D &density0) const;                                                                  \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { LAUNCH; }                                \
  };
ADVEC_CELL(advec_cell_fused_x1, (launch_march<28, 1, 0, advec_cell_x_march<VOL_FIRST>>(lp, s)))
ADVEC_CELL(advec_cell_fused_z1, (launch_march<32, 2, 3, advec_cell_march<2, VOL_FIRST>>(lp, s)))
ADVEC_CELL(advec_cell_fused_y2x, (launch_march<32, 1, 3, advec_cell_march<1, VOL_YZ>>(lp, s)))
ADVEC_CELL(advec_cell_fused_y2z, (launch_march<32, 1, 3, advec_cell_march<1, VOL_YX>>(lp, s)))
ADVEC_CELL_LAST(advec_cell_fused_x3, (launch_march<28, 1, 0, advec_cell_x_march<VOL_LAST>>(lp, s)))
ADVEC_CELL_LAST(advec_cell_fused_z3, (launch_march<32, 2, 3, advec_cell_march<2, VOL_LAST>>(lp, s)))

// One momentum sweep of the three velocities: node fluxes and masses (alike
// for all three), momentum fluxes and updates, into other dats than the
// velocities came from (in the last sweep the next step's xvel0, yvel0 and
// zvel0: reset_field_kernel2).
// Arguments: volume, vol_flux_{x,y,z}, celld, mass_flux, density1, xvel,
// yvel, zvel, xvel out, yvel out, zvel out.
//
// The x sweep marches along y: a row's sums of the two z lines it touches.
template <int VOL>
__global__ void __launch_bounds__(32 * kWarps, 4) advec_mom_x_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<28, 2, 1> m(lp, rows);
  if (!m.live) return;
  const int X = min(m.X, lp.end[0] + 1), z = m.o;
  const Fld volume(lp.a[0], X), vfx(lp.a[1], X), vfy(lp.a[2], X), vfz(lp.a[3], X), mflux(lp.a[5], X),
      density(lp.a[6], X);
  const Widths<0> cd(lp.a[4]);
  const double w0 = cd(X), wl = cd(X - 1), wr = cd(X + 1);
  const Fld xvel(lp.a[7], X), yvel(lp.a[8], X), zvel(lp.a[9], X);
  struct Row {  // mass flux and density x volume on lines z and z - 1; velocities
    double m0, m1, v0, v1, vel[3];
  };
  auto load = [&](int y) {
    Row r;
    r.m0 = mflux(y, z);
    r.m1 = mflux(y, z - 1);
    r.v0 = density(y, z) * post_volume<0, VOL>(volume, vfx, vfy, vfz, y, z);
    r.v1 = density(y, z - 1) * post_volume<0, VOL>(volume, vfx, vfy, vfz, y, z - 1);
    r.vel[0] = xvel(y, z);
    r.vel[1] = yvel(y, z);
    r.vel[2] = zvel(y, z);
    return r;
  };
  Row b = load(m.m0 - 1);
  double bm0r = from_right(b.m0), bm1r = from_right(b.m1), bv0l = from_left(b.v0), bv1l = from_left(b.v1);
  Row c = load(m.m0);
  for (int y = m.m0; y < m.m1; y++) {
    const Row n = load(min(y + 1, m.m1 - 1));
    const double m0r = from_right(c.m0), m1r = from_right(c.m1), v0l = from_left(c.v0), v1l = from_left(c.v1);
    const double nf = 0.125 * (b.m0 + c.m0 + bm0r + m0r + b.m1 + c.m1 + bm1r + m1r);
    const double mass_post = 0.125 * (b.v0 + c.v0 + bv0l + v0l + b.v1 + c.v1 + bv1l + v1l);
    const double mass_pre = mass_post - from_left(nf) + nf;
    const double mass_pre1 = from_right(mass_pre);
    const bool neg = nf < 0.0;
    const double sigma = qdiv(fabs(nf), neg ? mass_pre1 : mass_pre);
    const double wdif = neg ? wr : wl;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const Fld out(lp.a[10 + k], X);
      const double v = c.vel[k];
      const double vr = from_right(v), vrr = from_right2(v), vl = from_left(v);
      const double mom = advec_mom_face(nf, sigma, w0, wdif, neg ? vr : v, neg ? vrr : vl, neg ? v : vr);
      const double moml = from_left(mom);
      if (m.own) out.put(y, z, qdiv(v * mass_pre + moml - mom, mass_post));
    }
    b = c;
    bm0r = m0r;
    bm1r = m1r;
    bv0l = v0l;
    bv1l = v1l;
    c = n;
  }
}

// The y (DIR 1) and z (DIR 2) sweeps march along the sweep; the other of the
// two axes and x reach one line back.
template <int DIR, int VOL>
__global__ void __launch_bounds__(32 * kWarps, 3) advec_mom_march(const __grid_constant__ LoopParams lp, int rows) {
  const March<31, 1, DIR> m(lp, rows);
  if (!m.live) return;
  const int X = min(m.X, lp.end[0] - 1);
  const Fld volume(lp.a[0], X), vfx(lp.a[1], X), vfy(lp.a[2], X), vfz(lp.a[3], X), mflux(lp.a[5], X),
      density(lp.a[6], X), xvel(lp.a[7], X), yvel(lp.a[8], X), zvel(lp.a[9], X), xout(lp.a[10], X), yout(lp.a[11], X),
      zout(lp.a[12], X);
  const Widths<DIR> cd(lp.a[4]);
  // row r of the sweep on this line (back 0) or the line before it (back 1)
  auto yy = [&](int r, int back) { return DIR == 1 ? r : m.o - back; };
  auto zz = [&](int r, int back) { return DIR == 1 ? m.o - back : r; };
  struct Flux {  // mass flux of one row: this line and the one before, and left of them
    double a, al, b, bl;
  };
  auto pair = [](double a, double b) { return Flux{a, from_left(a), b, from_left(b)}; };
  auto flux = [&](int r) { return pair(mflux(yy(r, 0), zz(r, 0)), mflux(yy(r, 1), zz(r, 1))); };
  // (-1,0) + (0,0) + (-1,1) + (0,1) along (x, sweep), then the line before
  auto node_flux = [&](const Flux &p, const Flux &q) {
    return 0.125 * (p.al + p.a + q.al + q.a + p.bl + p.b + q.bl + q.b);
  };
  auto dvol = [&](int r, int back) {
    const int y = yy(r, back), z = zz(r, back);
    return density(y, z) * post_volume<DIR, VOL>(volume, vfx, vfy, vfz, y, z);
  };
  auto mass = [&](int r) { return pair(dvol(r, 0), dvol(r, 1)); };
  // (x, y, z) order of the reference: (0,-1,0) (0,0,0) (-1,-1,0) (-1,0,0),
  // then the same at z - 1; p is the row before q
  auto node_mass = [&](const Flux &p, const Flux &q) {
    return DIR == 1 ? 0.125 * (p.a + q.a + p.al + q.al + p.b + q.b + p.bl + q.bl)
                    : 0.125 * (q.b + q.a + q.bl + q.al + p.b + p.a + p.bl + p.al);
  };
  auto vel3 = [&](int r, double (&v)[3]) {
    v[0] = xvel(yy(r, 0), zz(r, 0));
    v[1] = yvel(yy(r, 0), zz(r, 0));
    v[2] = zvel(yy(r, 0), zz(r, 0));
  };
  const int r0 = m.m0 - 1;
  Flux f0 = flux(r0), f1 = flux(r0 + 1);
  double nf_b = node_flux(flux(r0 - 1), f0), nf = node_flux(f0, f1);
  Flux ms = mass(r0);
  double mass_post = node_mass(mass(r0 - 1), ms);
  double mass_pre = mass_post - nf_b + nf;
  double vb[3], vc[3], vn[3], ml[3] = {0.0, 0.0, 0.0};
  vel3(r0 - 1, vb);
  vel3(r0, vc);
  vel3(r0 + 1, vn);
  struct Row {  // row r + 2's velocities and mass fluxes, row r + 1's density x volume (this line, the one before)
    double v[3], fa, fb, ma, mb;
  };
  auto load = [&](int r) {
    Row w;
    vel3(r + 2, w.v);
    w.fa = mflux(yy(r + 2, 0), zz(r + 2, 0));
    w.fb = mflux(yy(r + 2, 1), zz(r + 2, 1));
    w.ma = dvol(r + 1, 0);
    w.mb = dvol(r + 1, 1);
    return w;
  };
  Row c = load(r0);
  for (int r = r0; r < m.m1; r++) {
    const Row n = load(min(r + 1, m.m1 - 1));
    const double *vnn = c.v;
    const Flux f2 = pair(c.fa, c.fb), ms1 = pair(c.ma, c.mb);
    const double nf1 = node_flux(f1, f2);
    const double mass_post1 = node_mass(ms, ms1);
    const double mass_pre1 = mass_post1 - nf + nf1;
    const bool neg = nf < 0.0;
    const double sigma = qdiv(fabs(nf), neg ? mass_pre1 : mass_pre);
    const double w0 = cd(r), wdif = neg ? cd(r + 1) : cd(r - 1);
    const bool put = m.own && r >= m.m0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double mom =
          advec_mom_face(nf, sigma, w0, wdif, neg ? vn[k] : vc[k], neg ? vnn[k] : vb[k], neg ? vc[k] : vn[k]);
      if (put)
        (k == 0 ? xout : k == 1 ? yout : zout)
            .put(yy(r, 0), zz(r, 0), qdiv(vc[k] * mass_pre + ml[k] - mom, mass_post));
      ml[k] = mom;
      vb[k] = vc[k];
      vc[k] = vn[k];
      vn[k] = vnn[k];
    }
    f1 = f2;
    ms = ms1;
    nf = nf1;
    mass_post = mass_post1;
    mass_pre = mass_pre1;
    c = n;
  }
}

#define ADVEC_MOM(NAME, LAUNCH)                                                                                     \
  struct NAME {                                                                                                     \
    C3_LOOP(NAME);                                                                                                  \
    __device__ void operator()(const D &volume, const D &vol_flux_x, const D &vol_flux_y, const D &vol_flux_z,      \
                               const D &celld, const D &mass_flux, const D &density, const D &xvel, const D &yvel,  \
                               const D &zvel, D &xout, D &yout, D &zout) const;                                     \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { LAUNCH; }                                \
  };
ADVEC_MOM(advec_mom_fused_x1, (launch_march<28, 1, 1, advec_mom_x_march<VOL_FIRST>>(lp, s)))
ADVEC_MOM(advec_mom_fused_x3, (launch_march<28, 1, 1, advec_mom_x_march<VOL_LAST>>(lp, s)))
ADVEC_MOM(advec_mom_fused_y2x, (launch_march<31, 1, 3, advec_mom_march<1, VOL_YZ>>(lp, s)))
ADVEC_MOM(advec_mom_fused_y2z, (launch_march<31, 1, 3, advec_mom_march<1, VOL_YX>>(lp, s)))
ADVEC_MOM(advec_mom_fused_z1, (launch_march<31, 2, 3, advec_mom_march<2, VOL_FIRST>>(lp, s)))
ADVEC_MOM(advec_mom_fused_z3, (launch_march<31, 2, 3, advec_mom_march<2, VOL_LAST>>(lp, s)))

#define REG(K) OPSB_REGISTER_LOOP(K);
REG(ideal_gas_summary) REG(calc_dt_fused) REG(PdV_predict_pressure) REG(accelerate_fused)
REG(PdV_flux) REG(advec_cell_fused_x1) REG(advec_cell_fused_x3) REG(advec_cell_fused_y2x) REG(advec_cell_fused_y2z)
REG(advec_cell_fused_z1) REG(advec_cell_fused_z3) REG(advec_mom_fused_x1) REG(advec_mom_fused_x3)
REG(advec_mom_fused_y2x) REG(advec_mom_fused_y2z) REG(advec_mom_fused_z1) REG(advec_mom_fused_z3)

struct ConstReg {
  ConstReg() {
#define C(name, member) \
  Runtime::register_const("cloverleaf3d/" name, &c3, offsetof(Consts, member), sizeof(Consts::member))
    C("g_small", g_small); C("g_big", g_big); C("dtc_safe", dtc_safe); C("dtu_safe", dtu_safe);
    C("dtv_safe", dtv_safe); C("dtw_safe", dtw_safe); C("dtdiv_safe", dtdiv_safe); C("dt", dt); C("field", field);
#undef C
  }
};
static ConstReg const_reg;

}  // namespace fused
}  // namespace clover3d
}  // namespace opsb
