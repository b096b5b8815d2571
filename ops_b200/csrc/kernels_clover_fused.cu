// CloverLeaf 2D: the hydro cycle's loops fused by hand, queued by the app
// driver (apps_clover.cpp) in place of runs of the reference's loops.
//
// The reference's loops pass every intermediate through HBM: volumes before
// and after advection, node masses and fluxes, energy and momentum fluxes,
// 1595 B per cell and step in 43 launches. None of those outlive the step, so
// each kernel here computes them in registers and moves only the fields that
// the next kernel needs: 608 B per cell and step in 9 launches plus the
// boundary copies. Measured at 3840^2: 4.75 -> 2.28 ms of kernels a step, copies
// included, a whole 10-step run with its set-up 59.0 -> 25.8 ms (250 x 187:
// 14.2 -> 3.5 ms, half the launches, and a queue the planner passes over). Every
// value is computed by the reference's expressions in the reference's order
// (clover_flux.cuh, --fmad=false), so fields and dt are the same bits.
// The sweeps wait for their loads: 70 to 102 registers a thread leave 24 to 39 %
// of an SM's warps, which issue in 32 to 52 % of the cycles, the FP64 pipe 14 to
// 28 % busy.
//
// The stencil loops march up columns. A warp owns a strip of columns, one per
// lane, and keeps the rows it needs in registers: values of other rows come
// from earlier iterations, values of other columns from the neighbouring lanes
// by shuffles, so a row of a field is loaded once. The lanes at the strip's
// edges lack a neighbour and own no column (30 of 32 lanes own one in the
// Lagrangian kernel, 28 in the x sweeps, 31 in the y momentum sweep, all in
// the y cell sweep); their loads are the neighbouring strips' and hit L1. The
// next row's loads are issued before the current row is worked on.
#include <algorithm>
#include <cstddef>

#include "clover_common.h"
#include "clover_flux.cuh"
#include "march_grid.h"
#include "runtime.h"

namespace opsb {
namespace clover {
namespace fused {

__constant__ Consts cc;

using D = ACC2<double>;

#define CL_LOOP(NAME) static constexpr const char *kname = "cloverleaf/" #NAME

// ---- single-point loops -----------------------------------------------------

// ideal_gas_kernel then field_summary_kernel (field_summary.cpp:44-110).
struct ideal_gas_summary {
  CL_LOOP(ideal_gas_summary);
  static constexpr bool touch_next_row = true;
  static constexpr int min_blocks = 6;
  __device__ void operator()(const D &density0, const D &energy0, D &pressure, D &soundspeed, const D &volume,
                             const D &xvel0, const D &yvel0, RED<double> &vol, RED<double> &mass, RED<double> &ie,
                             RED<double> &ke, RED<double> &press) const {
    const double d = density0(0, 0), e = energy0(0, 0);
    double v = 1.0 / d;
    double p = (1.4 - 1.0) * d * e;
    pressure(0, 0) = p;
    double pressurebyenergy = (1.4 - 1.0) * d;
    double pressurebyvolume = -1 * d * p;
    double sound_speed_squared = v * v * (p * pressurebyenergy - pressurebyvolume);
    soundspeed(0, 0) = sqrt(sound_speed_squared);
    double vsqrd = 0.0;
    vsqrd = vsqrd + 0.25 * (xvel0(0, 0) * xvel0(0, 0) + yvel0(0, 0) * yvel0(0, 0));
    vsqrd = vsqrd + 0.25 * (xvel0(1, 0) * xvel0(1, 0) + yvel0(1, 0) * yvel0(1, 0));
    vsqrd = vsqrd + 0.25 * (xvel0(0, 1) * xvel0(0, 1) + yvel0(0, 1) * yvel0(0, 1));
    vsqrd = vsqrd + 0.25 * (xvel0(1, 1) * xvel0(1, 1) + yvel0(1, 1) * yvel0(1, 1));
    double cell_vol = volume(0, 0);
    double cell_mass = cell_vol * d;
    *vol = *vol + cell_vol;
    *mass = *mass + cell_mass;
    *ie = *ie + cell_mass * e;
    *ke = *ke + cell_mass * 0.5 * vsqrd;
    *press = *press + cell_vol * p;
  }
};

// calc_dt_kernel with calc_dt_kernel_min folded in (calc_dt.cpp:37-131).
struct calc_dt_fused {
  CL_LOOP(calc_dt_fused);
  __device__ void operator()(const D &celldx, const D &celldy, const D &soundspeed, const D &viscosity,
                             const D &density0, const D &xvel0, const D &xarea, const D &volume, const D &yvel0,
                             const D &yarea, RED<double> &dt_min) const {
    double dsx = celldx(0, 0);
    double dsy = celldy(0, 0);
    double cc2 = soundspeed(0, 0) * soundspeed(0, 0);
    cc2 = cc2 + qdiv(2.0 * viscosity(0, 0), density0(0, 0));
    cc2 = op_max(sqrt(cc2), cc.g_small);
    double dtct = cc.dtc_safe * op_min(dsx, dsy) / cc2;
    double div = 0.0;
    double dv1 = (xvel0(0, 0) + xvel0(0, 1)) * xarea(0, 0);
    double dv2 = (xvel0(1, 0) + xvel0(1, 1)) * xarea(1, 0);
    div = div + dv2 - dv1;
    double dtut = cc.dtu_safe * 2.0 * volume(0, 0) / op_max(op_max(fabs(dv1), fabs(dv2)), cc.g_small * volume(0, 0));
    dv1 = (yvel0(0, 0) + yvel0(1, 0)) * yarea(0, 0);
    dv2 = (yvel0(0, 1) + yvel0(1, 1)) * yarea(0, 1);
    div = div + dv2 - dv1;
    double dtvt = cc.dtv_safe * 2.0 * volume(0, 0) / op_max(op_max(fabs(dv1), fabs(dv2)), cc.g_small * volume(0, 0));
    div = qdiv(div, 2.0 * volume(0, 0));
    double dtdivt;
    if (div < -cc.g_small)
      dtdivt = cc.dtdiv_safe * (-1.0 / div);
    else
      dtdivt = cc.g_big;
    *dt_min = op_min(*dt_min, op_min(op_min(dtct, dtut), op_min(dtvt, dtdivt)));
  }
};

// PdV_kernel_predict then the ideal gas pressure of the predicted state
// (PdV.cpp:41-117). The predicted density and energy are only that pressure's
// inputs: revert_kernel puts density0 and energy0 back and PdV_kernel_nopredict
// overwrites them before anything reads them; the sound speed is recomputed
// before its next reader too.
struct PdV_predict_pressure {
  CL_LOOP(PdV_predict_pressure);
  static constexpr int min_blocks = 6;
  __device__ void operator()(const D &xarea, const D &xvel0, const D &yarea, const D &yvel0, const D &volume,
                             D &pressure, const D &density0, const D &viscosity, const D &energy0) const {
    const double dt = cc.dt;
    double left_flux = (xarea(0, 0) * (xvel0(0, 0) + xvel0(0, 1) + xvel0(0, 0) + xvel0(0, 1))) * 0.25 * dt * 0.5;
    double right_flux = (xarea(1, 0) * (xvel0(1, 0) + xvel0(1, 1) + xvel0(1, 0) + xvel0(1, 1))) * 0.25 * dt * 0.5;
    double bottom_flux = (yarea(0, 0) * (yvel0(0, 0) + yvel0(1, 0) + yvel0(0, 0) + yvel0(1, 0))) * 0.25 * dt * 0.5;
    double top_flux = (yarea(0, 1) * (yvel0(0, 1) + yvel0(1, 1) + yvel0(0, 1) + yvel0(1, 1))) * 0.25 * dt * 0.5;
    double total_flux = right_flux - left_flux + top_flux - bottom_flux;
    const double vol = volume(0, 0), d0 = density0(0, 0);
    double volume_change = vol / (vol + total_flux);
    double recip_volume = 1.0 / vol;
    double energy_change = (pressure(0, 0) / d0 + qdiv(viscosity(0, 0), d0)) * total_flux * recip_volume;
    double energy1 = energy0(0, 0) - energy_change;
    double density1 = d0 * volume_change;
    pressure(0, 0) = (1.4 - 1.0) * density1 * energy1;
  }
};

// ---- column marches -----------------------------------------------------------

constexpr int kWarps = 4;  // warps per CTA
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ double from_left(double v) { return __shfl_up_sync(kAll, v, 1); }
__device__ __forceinline__ double from_left2(double v) { return __shfl_up_sync(kAll, v, 2); }
__device__ __forceinline__ double from_right(double v) { return __shfl_down_sync(kAll, v, 1); }
__device__ __forceinline__ double from_right2(double v) { return __shfl_down_sync(kAll, v, 2); }

// One argument at the warp's column: element (X, y) is p[y * pitch].
struct Col {
  double *p;
  int pitch;
  __device__ __forceinline__ Col(const ArgView &a, int X) : p(reinterpret_cast<double *>(a.ptr) + X), pitch(a.ay) {}
  __device__ __forceinline__ double operator()(int y) const { return __ldg(p + (long long)y * pitch); }
  __device__ __forceinline__ void put(int y, double v) const { p[(long long)y * pitch] = v; }
};

// The strip of a warp: its lane's column X (kEdge lanes before the strip's
// first owned column) and rows [y0, y1) of the range.
template <int OWN, int EDGE>
struct Strip {
  int X, y0, y1;
  bool own, live;
  __device__ __forceinline__ Strip(const LoopParams &lp, int rows) {
    const int w = blockIdx.x * kWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int nx = lp.end[0] - lp.start[0], ncol = (nx + OWN - 1) / OWN;
    const int c = w % ncol;
    X = lp.start[0] + c * OWN + lane - EDGE;
    y0 = lp.start[1] + (w / ncol) * rows;
    y1 = min(y0 + rows, lp.end[1]);
    live = y0 < lp.end[1];
    own = lane >= EDGE && lane < EDGE + OWN && X < lp.end[0];
  }
};

// HALO: rows a strip reads beyond its own.
template <int OWN, int HALO, auto kernel>
void launch_strips(const LoopParams &lp, cudaStream_t s) {
  static int per_sm = 0;  // resident CTAs, per kernel
  if (!per_sm) {
    int n = 0;
    OPSB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 32 * kWarps, 0));
    per_sm = std::max(n, 1);
  }
  const int nx = lp.end[0] - lp.start[0], ny = lp.end[1] - lp.start[1];
  const long long ncol = (nx + OWN - 1) / OWN;
  const int rows = march_rows(ncol, ny, HALO, 148LL * per_sm * kWarps);
  const long long warps = ncol * ((ny + rows - 1) / rows);
  kernel<<<(unsigned)((warps + kWarps - 1) / kWarps), 32 * kWarps, 0, s>>>(lp, rows);
}

// accelerate_kernel, PdV_kernel_nopredict and flux_calc_kernel{x,y}
// (accelerate.cpp:39-63, PdV.cpp:41-117, flux_calc.cpp:38-64) over the nodes
// [x_min, x_max + 1) x [y_min, y_max + 1); cells stop one short of the
// nodes in each direction. The flux through a cell's right (top) face is the
// left (bottom) face flux of the next column (row), the same expression.
__global__ void __launch_bounds__(32 * kWarps, 4) lagrange_kernel(const __grid_constant__ LoopParams lp, int rows) {
  const Strip<30, 1> st(lp, rows);
  if (!st.live) return;
  const int X = min(st.X, lp.end[0]);  // the column right of the last node is the last one read
  const Col density0(lp.a[0], X), volume(lp.a[1], X), pressure(lp.a[2], X), viscosity(lp.a[3], X), xvel0(lp.a[4], X),
      yvel0(lp.a[5], X), xarea(lp.a[6], X), yarea(lp.a[7], X), energy0(lp.a[8], X);
  const Col xvel1(lp.a[9], X), yvel1(lp.a[10], X), density1(lp.a[11], X), energy1(lp.a[12], X), vol_flux_x(lp.a[13], X),
      vol_flux_y(lp.a[14], X);
  const double dt = cc.dt;
  const int xcell = lp.end[0] - 1, ycell = lp.end[1] - 1;  // end of the cells
  const bool cell_x = st.own && st.X < xcell;
  struct Row {
    double d, v, p, q, xv, yv, xa, ya;
  };
  auto load = [&](int y) {
    return Row{density0(y), volume(y), pressure(y), viscosity(y), xvel0(y), yvel0(y), xarea(y), yarea(y)};
  };
  // rows j - 1 and j of what a node needs
  double dv_m, dvl_m, dpx_m, dqx_m, p_m, q_m, xa_m;
  {
    const int y = st.y0 - 1;
    p_m = pressure(y);
    q_m = viscosity(y);
    xa_m = xarea(y);
    dv_m = density0(y) * volume(y);
    dvl_m = from_left(dv_m);
    dpx_m = p_m - from_left(p_m);
    dqx_m = q_m - from_left(q_m);
  }
  // the node of row y (its lane must have a left neighbour)
  auto node = [&](const Row &r, double &xv1, double &yv1) {
    const double dv = r.d * r.v, dvl = from_left(dv);
    const double dpx = r.p - from_left(r.p), dqx = r.q - from_left(r.q);
    const double typ = r.ya * (r.p - p_m), tyq = r.ya * (r.q - q_m);
    const double typl = from_left(typ), tyql = from_left(tyq);
    const double nodal_mass = (dvl_m + dv_m + dv + dvl) * 0.25;
    const double stepbymass = 0.5 * dt / nodal_mass;
    xv1 = r.xv - stepbymass * (r.xa * dpx + xa_m * dpx_m);
    yv1 = r.yv - stepbymass * (typ + typl);
    xv1 = xv1 - stepbymass * (r.xa * dqx + xa_m * dqx_m);
    yv1 = yv1 - stepbymass * (tyq + tyql);
    dv_m = dv;
    dvl_m = dvl;
    dpx_m = dpx;
    dqx_m = dqx;
    p_m = r.p;
    q_m = r.q;
    xa_m = r.xa;
  };
  Row c = load(st.y0);
  Row n = load(st.y0 + 1);
  double xv1, yv1;
  node(c, xv1, yv1);
  double ysum = c.yv + from_right(c.yv) + yv1 + from_right(yv1);
  double bottom = (c.ya * ysum) * 0.25 * dt;
  for (int j = st.y0; j < st.y1; j++) {
    if (st.own) {
      xvel1.put(j, xv1);
      yvel1.put(j, yv1);
      if (cell_x) vol_flux_y.put(j, 0.25 * dt * c.ya * ysum);
    }
    if (j == ycell) break;  // the last node row has no cells
    const double e = energy0(j);
    const Row nn = j + 1 < st.y1 ? load(min(j + 2, lp.end[1])) : n;
    double xn, yn;
    node(n, xn, yn);
    const double xsum = c.xv + n.xv + xv1 + xn;
    const double left = (c.xa * xsum) * 0.25 * dt;
    const double right = from_right(left);
    const double ysum_n = n.yv + from_right(n.yv) + yn + from_right(yn);
    const double top = (n.ya * ysum_n) * 0.25 * dt;
    if (st.own) {
      vol_flux_x.put(j, 0.25 * dt * c.xa * xsum);
      if (cell_x) {
        const double total_flux = right - left + top - bottom;
        const double volume_change = c.v / (c.v + total_flux);
        const double recip_volume = 1.0 / c.v;
        const double energy_change = (c.p / c.d + qdiv(c.q, c.d)) * total_flux * recip_volume;
        energy1.put(j, e - energy_change);
        density1.put(j, c.d * volume_change);
      }
    }
    bottom = top;
    ysum = ysum_n;
    xv1 = xn;
    yv1 = yn;
    c = n;
    n = nn;
  }
}

struct lagrange {
  CL_LOOP(lagrange);
  __device__ void operator()(const D &density0, const D &volume, const D &pressure, const D &viscosity,
                             const D &xvel0, const D &yvel0, const D &xarea, const D &yarea, const D &energy0,
                             D &xvel1, D &yvel1, D &density1, D &energy1, D &vol_flux_x, D &vol_flux_y) const;
  static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_strips<30, 2, lagrange_kernel>(lp, s); }
};

// advec_cell_kernel{1,2}, 3 and 4 of an x sweep (advec_cell.cpp:38-147). The
// range is the mass flux's, two columns beyond the cells. FIRST: the first
// sweep of the step (volumes from both flux directions). The updated density
// and energy go to other dats than they came from (neighbouring strips still
// read the old ones); the second sweep also writes the next step's density0
// and energy0 (reset_field_kernel1) and leaves energy1, which nothing reads
// before it is written again.
// Arguments: vol_flux_x, volume, vertexdx, density, energy, [vol_flux_y,]
// then mass_flux_x, density out, energy out, [density0 out].
template <bool FIRST>
__global__ void __launch_bounds__(32 * kWarps, 5) advec_cell_x_kernel(const __grid_constant__ LoopParams lp, int rows) {
  const Strip<28, 2> st(lp, rows);
  if (!st.live) return;
  const int X = min(st.X, lp.end[0] + 1);
  const Col vfx(lp.a[0], X), volume(lp.a[1], X), density(lp.a[3], X), energy(lp.a[4], X);
  constexpr int O = FIRST ? 6 : 5;
  const Col vfy(lp.a[FIRST ? 5 : 0], X), mass_flux(lp.a[O], X), dout(lp.a[O + 1], X), eout(lp.a[O + 2], X),
      d0out(lp.a[FIRST ? O + 1 : O + 3], X);
  const double *vdx = reinterpret_cast<const double *>(lp.a[2].ptr);
  const double w0 = vdx[X];
  const double wm = qratio(w0, vdx[X - 1]), wp = qratio(w0, vdx[X + 1]), wc = qratio(w0, w0);
  const bool cell_max_test = st.X - 1 < cc.field.x_max;
  const bool cell = st.own && st.X < lp.end[0] - 2;
  struct Row {
    double f, v, d, e, g;  // g: vol_flux_y of the next row
  };
  auto load = [&](int y) { return Row{vfx(y), volume(y), density(y), energy(y), FIRST ? vfy(y + 1) : 0.0}; };
  double g0 = FIRST ? vfy(st.y0) : 0.0;
  Row c = load(st.y0);
  for (int j = st.y0; j < st.y1; j++) {
    const Row n = load(min(j + 1, st.y1 - 1));
    const double f1 = from_right(c.f);
    const double pv = FIRST ? c.v + (f1 - c.f + c.g - g0) : c.v + f1 - c.f;
    const double pvl = from_left(pv);
    const double d1 = from_right(c.d), dl = from_left(c.d), dll = from_left2(c.d);
    const double e1 = from_right(c.e), el = from_left(c.e), ell = from_left2(c.e);
    const bool pos = c.f > 0.0;
    double mf, ef;
    advec_cell_face(c.f, pos ? pvl : pv, pos ? wm : cell_max_test ? wp : wc, pos ? dl : c.d,
                    pos ? dll : cell_max_test ? d1 : c.d, pos ? c.d : dl, pos ? el : c.e,
                    pos ? ell : cell_max_test ? e1 : c.e, pos ? c.e : el, mf, ef);
    const double mf1 = from_right(mf), ef1 = from_right(ef);
    if (st.own) mass_flux.put(j, mf);
    if (cell) {
      const double pre_mass = c.d * pv;
      const double post_mass = pre_mass + mf - mf1;
      const double post_ener = (c.e * pre_mass + ef - ef1) / post_mass;
      const double advec_vol = pv + c.f - f1;
      const double dn = post_mass / advec_vol;
      dout.put(j, dn);
      eout.put(j, post_ener);
      if (!FIRST) d0out.put(j, dn);
    }
    g0 = c.g;
    c = n;
  }
}

// The same for a y sweep: every lane owns its column; a strip's rows start
// with the face below its first cell, whose flux the strip below computes too.
// Arguments: vol_flux_y, volume, vertexdy, density, energy, [vol_flux_x,]
// then mass_flux_y, density out, energy out, [density0 out].
template <bool FIRST>
__global__ void __launch_bounds__(32 * kWarps, 5) advec_cell_y_kernel(const __grid_constant__ LoopParams lp, int rows) {
  const Strip<32, 0> st(lp, rows);
  if (!st.live || !st.own) return;
  const int X = st.X;
  const Col vfy(lp.a[0], X), volume(lp.a[1], X), density(lp.a[3], X), energy(lp.a[4], X);
  constexpr int O = FIRST ? 6 : 5;
  const Col vfx(lp.a[FIRST ? 5 : 0], X), mass_flux(lp.a[O], X), dout(lp.a[O + 1], X), eout(lp.a[O + 2], X),
      d0out(lp.a[FIRST ? O + 1 : O + 3], X);
  const double *vdy = reinterpret_cast<const double *>(lp.a[2].ptr);
  const int wp = lp.a[2].ay;
  const int ylast = lp.end[1] - 1;  // last face row; cells stop two rows before the end
  const int yend = min(st.y1, ylast);
  struct Row {  // row y: volume, x fluxes; density, energy and flux of row y + 1
    double v, x0, x1, d, e, f;
  };
  auto load = [&](int y) {
    return Row{volume(y), FIRST ? vfx(y) : 0.0, FIRST ? __ldg(vfx.p + (long long)y * vfx.pitch + 1) : 0.0,
               density(y + 1), energy(y + 1), vfy(y + 1)};
  };
  auto prevol = [&](const Row &r, double f) {
    return FIRST ? r.v + (r.f - f + r.x1 - r.x0) : r.v + r.f - f;
  };
  double dll = density(st.y0 - 2), ell = energy(st.y0 - 2);
  double dl = density(st.y0 - 1), el = energy(st.y0 - 1);
  Row c = load(st.y0 - 1);
  double pvl = prevol(c, vfy(st.y0 - 1));
  double dc = c.d, ec = c.e, f = c.f;
  double mfl = 0.0, efl = 0.0, fl = 0.0;
  c = load(st.y0);
  // face rows y0 .. yend; the cell below each face but the first
  for (int j = st.y0; j <= yend; j++) {
    const Row n = load(min(j + 1, yend));
    const double dn = c.d, en = c.e, f1 = c.f;
    const double pv = prevol(c, f);
    const double w0 = vdy[j * wp];
    const bool pos = f > 0.0, cell_max_test = j - 1 < cc.field.y_max;
    const double width = qratio(w0, pos ? vdy[(j - 1) * wp] : cell_max_test ? vdy[(j + 1) * wp] : w0);
    double mf, ef;
    advec_cell_face(f, pos ? pvl : pv, width, pos ? dl : dc, pos ? dll : cell_max_test ? dn : dc, pos ? dc : dl,
                    pos ? el : ec, pos ? ell : cell_max_test ? en : ec, pos ? ec : el, mf, ef);
    if (j < st.y1) mass_flux.put(j, mf);
    if (j > st.y0 && j - 1 < lp.end[1] - 2) {
      const double pre_mass = dl * pvl;
      const double post_mass = pre_mass + mfl - mf;
      const double post_ener = (el * pre_mass + efl - ef) / post_mass;
      const double advec_vol = pvl + fl - f;
      const double dnew = post_mass / advec_vol;
      dout.put(j - 1, dnew);
      eout.put(j - 1, post_ener);
      if (!FIRST) d0out.put(j - 1, dnew);
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

#define ADVEC_CELL(NAME, OWN, HALO, KERNEL)                                                                          \
  struct NAME##1 {                                                                                             \
    CL_LOOP(NAME##1);                                                                                          \
    __device__ void operator()(const D &vol_flux, const D &volume, const D &vertexd, const D &density,         \
                               const D &energy, const D &vol_flux_t, D &mass_flux, D &dout, D &eout) const;    \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_strips<OWN, HALO, KERNEL<true>>(lp, s); }  \
  };                                                                                                           \
  struct NAME##2 {                                                                                             \
    CL_LOOP(NAME##2);                                                                                          \
    __device__ void operator()(const D &vol_flux, const D &volume, const D &vertexd, const D &density,         \
                               const D &energy, D &mass_flux, D &dout, D &eout, D &d0out) const;               \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_strips<OWN, HALO, KERNEL<false>>(lp, s); } \
  };
ADVEC_CELL(advec_cell_fused_x, 28, 0, advec_cell_x_kernel)
ADVEC_CELL(advec_cell_fused_y, 32, 3, advec_cell_y_kernel)

// The x momentum sweep of both velocities (advec_mom.cpp:40-163): node
// fluxes and masses, the two momentum fluxes and the updates; the node
// fluxes, masses and sigma are the two velocities' alike. The updated
// velocities go to other dats (in the second sweep to the next step's xvel0
// and yvel0: reset_field_kernel2).
// Arguments: mass_flux_x, volume, celldx, density1, xvel, yvel, xvel out,
// yvel out, [vol_flux_y].
template <bool FIRST>
__global__ void __launch_bounds__(32 * kWarps, 4) advec_mom_x_kernel(const __grid_constant__ LoopParams lp, int rows) {
  const Strip<28, 2> st(lp, rows);
  if (!st.live) return;
  const int X = min(st.X, lp.end[0] + 1);
  const Col mfx(lp.a[0], X), volume(lp.a[1], X), density(lp.a[3], X), xvel(lp.a[4], X), yvel(lp.a[5], X),
      xout(lp.a[6], X), yout(lp.a[7], X), vfy(lp.a[FIRST ? 8 : 0], X);
  const double *cdx = reinterpret_cast<const double *>(lp.a[2].ptr);
  const double w0 = cdx[X], wl = cdx[X - 1], wr = cdx[X + 1];
  struct Row {
    double m, v, d, xv, yv, g;
  };
  auto load = [&](int y) { return Row{mfx(y), volume(y), density(y), xvel(y), yvel(y), FIRST ? vfy(y + 1) : 0.0}; };
  double g0 = 0.0;
  auto post_vol = [&](double v, double g) { return FIRST ? v + g - g0 : v; };
  double m_b, m1_b, dv_b, dvl_b;
  {
    const int y = st.y0 - 1;
    m_b = mfx(y);
    m1_b = from_right(m_b);
    double g = 0.0;
    if (FIRST) {
      g0 = vfy(y);
      g = vfy(y + 1);
    }
    dv_b = density(y) * post_vol(volume(y), g);
    dvl_b = from_left(dv_b);
    g0 = g;
  }
  Row c = load(st.y0);
  for (int j = st.y0; j < st.y1; j++) {
    const Row n = load(min(j + 1, st.y1 - 1));
    const double m1 = from_right(c.m);
    const double nf = 0.25 * (m_b + c.m + m1_b + m1);
    const double dv = c.d * post_vol(c.v, c.g), dvl = from_left(dv);
    const double mass_post = 0.25 * (dv_b + dv + dvl_b + dvl);
    const double mass_pre = mass_post - from_left(nf) + nf;
    const double mass_pre1 = from_right(mass_pre);
    const bool neg = nf < 0.0;
    const double sigma = qdiv(fabs(nf), neg ? mass_pre1 : mass_pre);
    const double wdif = neg ? wr : wl;
    const double x1 = from_right(c.xv), x2 = from_right2(c.xv), xl = from_left(c.xv);
    const double y1 = from_right(c.yv), y2 = from_right2(c.yv), yl = from_left(c.yv);
    const double xm = advec_mom_face(nf, sigma, w0, wdif, neg ? x1 : c.xv, neg ? x2 : xl, neg ? c.xv : x1);
    const double ym = advec_mom_face(nf, sigma, w0, wdif, neg ? y1 : c.yv, neg ? y2 : yl, neg ? c.yv : y1);
    const double xml = from_left(xm), yml = from_left(ym);
    if (st.own) {
      xout.put(j, qdiv(c.xv * mass_pre + xml - xm, mass_post));
      yout.put(j, qdiv(c.yv * mass_pre + yml - ym, mass_post));
    }
    m_b = c.m;
    m1_b = m1;
    dv_b = dv;
    dvl_b = dvl;
    g0 = c.g;
    c = n;
  }
}

// The y momentum sweep; only the node masses and fluxes reach across columns.
// Arguments: mass_flux_y, volume, celldy, density1, xvel, yvel, xvel out,
// yvel out, [vol_flux_x].
template <bool FIRST>
__global__ void __launch_bounds__(32 * kWarps, 4) advec_mom_y_kernel(const __grid_constant__ LoopParams lp, int rows) {
  const Strip<31, 1> st(lp, rows);
  if (!st.live) return;
  const int X = min(st.X, lp.end[0]);
  const Col mfy(lp.a[0], X), volume(lp.a[1], X), density(lp.a[3], X), xvel(lp.a[4], X), yvel(lp.a[5], X),
      xout(lp.a[6], X), yout(lp.a[7], X), vfx(lp.a[FIRST ? 8 : 0], X);
  const double *cdy = reinterpret_cast<const double *>(lp.a[2].ptr);
  const int wp = lp.a[2].ay;
  struct Row {  // row y: mass flux of row y + 1, density x post volume, velocities of row y + 1
    double m, dv, xv, yv;
  };
  auto dvol = [&](int y) {
    const double v = volume(y);
    const double pv = FIRST ? v + __ldg(vfx.p + (long long)y * vfx.pitch + 1) - vfx(y) : v;
    return density(y) * pv;
  };
  auto load = [&](int y) { return Row{mfy(y + 1), dvol(y), xvel(y + 1), yvel(y + 1)}; };
  // node flux of row y from mass fluxes of rows y and y + 1:
  // 0.25 * (m(-1, y) + m(0, y) + m(-1, y + 1) + m(0, y + 1))
  const int yb = st.y0 - 1;
  double mm = mfy(yb - 1), m0 = mfy(yb);
  double mml = from_left(mm), m0l = from_left(m0);
  double nf_b = 0.25 * (mml + mm + m0l + m0);  // row y0 - 2
  double m1 = mfy(yb + 1), m1l = from_left(m1);
  double nf = 0.25 * (m0l + m0 + m1l + m1);  // row y0 - 1
  double dv_b = dvol(yb - 1), dvl_b = from_left(dv_b);
  double dv = dvol(yb), dvl = from_left(dv);
  double mass_post = 0.25 * (dv_b + dv + dvl_b + dvl);
  double mass_pre = mass_post - nf_b + nf;
  double xb = xvel(yb - 1), xc = xvel(yb), xn = xvel(yb + 1);
  double yb_ = yvel(yb - 1), yc = yvel(yb), yn = yvel(yb + 1);
  double xml = 0.0, yml = 0.0;
  Row c = load(yb + 1);
  // node row j: its mass flux, then its update (j >= y0) with the flux below
  for (int j = yb; j < st.y1; j++) {
    const Row n = load(min(j + 2, st.y1));
    // row j + 1
    const double m2 = c.m, m2l = from_left(m2);
    const double nf1 = 0.25 * (m1l + m1 + m2l + m2);
    const double dv1 = c.dv, dvl1 = from_left(dv1);
    const double mass_post1 = 0.25 * (dv + dv1 + dvl + dvl1);
    const double mass_pre1 = mass_post1 - nf + nf1;
    const double xnn = c.xv, ynn = c.yv;
    const bool neg = nf < 0.0;
    const double sigma = qdiv(fabs(nf), neg ? mass_pre1 : mass_pre);
    const double w0 = cdy[j * wp], wdif = neg ? cdy[(j + 1) * wp] : cdy[(j - 1) * wp];
    const double xm = advec_mom_face(nf, sigma, w0, wdif, neg ? xn : xc, neg ? xnn : xb, neg ? xc : xn);
    const double ym = advec_mom_face(nf, sigma, w0, wdif, neg ? yn : yc, neg ? ynn : yb_, neg ? yc : yn);
    if (st.own && j >= st.y0) {
      xout.put(j, qdiv(xc * mass_pre + xml - xm, mass_post));
      yout.put(j, qdiv(yc * mass_pre + yml - ym, mass_post));
    }
    xml = xm;
    yml = ym;
    m1 = m2;
    m1l = m2l;
    nf = nf1;
    dv = dv1;
    dvl = dvl1;
    mass_post = mass_post1;
    mass_pre = mass_pre1;
    xb = xc;
    xc = xn;
    xn = xnn;
    yb_ = yc;
    yc = yn;
    yn = ynn;
    c = n;
  }
}

#define ADVEC_MOM(NAME, OWN, HALO, KERNEL)                                                                             \
  struct NAME##1 {                                                                                               \
    CL_LOOP(NAME##1);                                                                                            \
    __device__ void operator()(const D &mass_flux, const D &volume, const D &celld, const D &density,            \
                               const D &xvel, const D &yvel, D &xout, D &yout, const D &vol_flux_t) const;       \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_strips<OWN, HALO, KERNEL<true>>(lp, s); }    \
  };                                                                                                             \
  struct NAME##2 {                                                                                               \
    CL_LOOP(NAME##2);                                                                                            \
    __device__ void operator()(const D &mass_flux, const D &volume, const D &celld, const D &density,            \
                               const D &xvel, const D &yvel, D &xout, D &yout) const;                            \
    static void launch(const LoopParams &lp, dim3, dim3, cudaStream_t s) { launch_strips<OWN, HALO, KERNEL<false>>(lp, s); }   \
  };
ADVEC_MOM(advec_mom_fused_x, 28, 1, advec_mom_x_kernel)
ADVEC_MOM(advec_mom_fused_y, 31, 3, advec_mom_y_kernel)

#define REG(K) OPSB_REGISTER_LOOP(K);
REG(ideal_gas_summary) REG(calc_dt_fused) REG(PdV_predict_pressure) REG(lagrange)
REG(advec_cell_fused_x1) REG(advec_cell_fused_x2) REG(advec_cell_fused_y1) REG(advec_cell_fused_y2)
REG(advec_mom_fused_x1) REG(advec_mom_fused_x2) REG(advec_mom_fused_y1) REG(advec_mom_fused_y2)

struct ConstReg {
  ConstReg() {
#define C(name, member) Runtime::register_const("cloverleaf/" name, &cc, offsetof(Consts, member), sizeof(Consts::member))
    C("g_small", g_small); C("g_big", g_big); C("dtc_safe", dtc_safe); C("dtu_safe", dtu_safe);
    C("dtv_safe", dtv_safe); C("dtdiv_safe", dtdiv_safe); C("dt", dt); C("field", field);
#undef C
  }
};
static ConstReg const_reg;

}  // namespace fused
}  // namespace clover
}  // namespace opsb
