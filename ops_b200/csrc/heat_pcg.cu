// Device-resident Jacobi-PCG for the TeaLeaf 2D heat operator; interface and
// algorithm notes in heat_pcg.h.
//
// Per iteration (tea_leaf_cg.cpp:103-214) two kernels, each one pass:
//   k_pw  p = beta p + z, w = A p, pw = p.w, and u += alpha p for the
//         previous iteration's direction and step -> last block: alpha = rro / pw
//   k_r   r -= alpha w, rz = r.(Mi r)       -> last block: beta, rro, stop test
// and after the loop k_flush, the last iteration's u update. The reference's
// sequence (w; u, r, z; p) passes p through HBM three times and z and u twice
// as often: 120 B per cell and iteration in FP64, 96 B here (u, p, w, r once
// in and once out, the faces once in k_pw, Mi once in k_r). The new direction
// goes to a second buffer, since a cell's neighbours still read the old one;
// `iters` says which of the two is current.
// The arithmetic of every cell is the reference's, in its order (this file
// builds without FMA contraction). Grid sums finish in a fixed order (each
// block's partial, then the last block to arrive adds the partials by block
// index), so a solve is bit-reproducible run to run. Once the stop test has
// fired every later kernel returns at entry, so a chunk of iterations that
// runs past convergence costs only its launch latency.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "heat_pcg.h"
#include "march_grid.h"
#include "runtime.h"

namespace opsb {
namespace heat {

namespace {

constexpr int BX = 128, BY = 2, NT = BX * BY, kWarps = NT / 32;
constexpr int kMaxBlocks = 4096;
constexpr int kChunk = 16;          // iterations per replayed graph
// Grids are one wave of kResident blocks per SM; every kernel is held to the
// registers that let kResident blocks stay resident (a kernel over budget
// would run its grid in 1 1/3 waves).
constexpr int kResident = 8;
constexpr int kTargetBlocks = 148 * kResident;

struct Scalars {
  double rro, rro_prev, pw, alpha, beta;
  double err, stop, ref, rr, rr0;
  int done;       // 0 running, 1 converged, 2 iteration limit, 3 reliable update due,
                  // 4 FCG lost positive curvature, 5 FCG restart (||r|| not halved over the window)
  int iters;
  int max_iters;
  int first;
  int pend;  // u += alpha p of the last k_pw is still to be made
  int restart;  // FCG: the next direction is z itself
  // FCG restart test on the device (replayed chunks): ||r|| of the last
  // iterations since the last (re)start, `window` 0 when the test is off
  int window, hcount;
  double hist[64];
};

// Stopping quantity of k_r.
enum { STOP_TEALEAF = 0,  // sqrt|r.z| < eps ||r0|| (tea_solve.cpp:349-355)
       STOP_TRUE = 1,     // ||r|| < eps ||r0||
       STOP_RELIABLE = 2  // inner FP32 loop: estimate test, or a decade of decrease since the last update
};

struct Geom {
  int nx, ny;
  long long pitch;
};

__device__ __forceinline__ int tid_() { return threadIdx.x + threadIdx.y * BX; }

// Sum over the block; the result is valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *sm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int t = tid_(), lane = t & 31, wid = t >> 5;
  __syncthreads();
  if (lane == 0) sm[wid] = v;
  __syncthreads();
  v = 0.0;
  if (wid == 0) {
    v = lane < kWarps ? sm[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// Stores the block's partials (NV values, part[NV * block + k]); true in
// every thread of the last block to arrive.
template <int NV>
__device__ __forceinline__ bool publish(const double (&v)[NV], double *part, unsigned *cnt, double *sm, int *last) {
  const int nb = gridDim.x * gridDim.y, bid = blockIdx.x + blockIdx.y * gridDim.x;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    const double b = block_sum(v[k], sm);
    if (tid_() == 0) part[NV * bid + k] = b;
  }
  if (tid_() == 0) {
    __threadfence();
    const unsigned t = atomicAdd(cnt, 1u);
    *last = (t == (unsigned)(nb - 1));
  }
  __syncthreads();
  return *last != 0;
}

// Last block only: partial k of every block added in block order; valid in
// thread 0. The caller resets the arrival counter once all totals are taken.
template <int NV>
__device__ __forceinline__ double grid_total(const double *part, int k, double *sm) {
  __threadfence();
  const int nb = gridDim.x * gridDim.y;
  double v = 0.0;
  for (int b = tid_(); b < nb; b += NT) v += __ldcg(part + NV * b + k);
  return block_sum(v, sm);
}

// tea_leaf_common_kernels.h (the 5-point operator shared by the CG kernels).
template <class T>
__device__ __forceinline__ T smvp(const T *__restrict__ Kx, const T *__restrict__ Ky, const T *__restrict__ u,
                                  long long i, long long P, T rx, T ry) {
  const T kx0 = Kx[i], kx1 = Kx[i + 1], ky0 = Ky[i], ky1 = Ky[i + P];
  return (T(1) + ry * (ky1 + ky0) + rx * (kx1 + kx0)) * u[i] - ry * (ky1 * u[i + P] + ky0 * u[i - P]) -
         rx * (kx1 * u[i + 1] + kx0 * u[i - 1]);
}

#define HEAT_CELLS(g)                                                                          \
  for (int y = blockIdx.y * BY + threadIdx.y; y < (g).ny; y += gridDim.y * BY)                 \
    for (int x = blockIdx.x * BX + threadIdx.x; x < (g).nx; x += gridDim.x * BX)

// How k_pw gets z: the residual itself, Mi r with Mi read, or Mi r with
// Mi = 1 / diag(A) computed from the faces it holds anyway (FP64: the same
// bits as tea_leaf_common_init_diag_init_kernel's Mi, 8 B a cell less).
// Z_FCG: the flexible CG's z itself in `r`, and the residual in `Mi`.
enum { Z_R = 0, Z_MI = 1, Z_DIAG = 2, Z_FCG = 3 };

// tea_leaf_axpby_kernel (p = beta p + z), tea_leaf_cg_calc_w_reduce_kernel
// (w = A p, p.w; tea_leaf_cg_kernels.h:8) and the previous iteration's
// tea_leaf_axpy_kernel on u; then alpha = rro / pw. A warp marches up a strip
// of 32 columns, one per lane, 30 of them its own: p of the rows below and
// above stays in registers, p of the columns beside comes by shuffles. The
// ring's p never changes and is read from the first buffer.
// A row's loads are issued two rows ahead; FP32 rows are half the bytes, so
// four CTAs an SM there, three in FP64.
// Z_FCG (Notay 2000, FCG with one-step truncation): alpha = p.r / p.w, p = z
// after a restart, and a non-positive p.w (the preconditioned direction lost
// positive curvature) stops with done = 4.
template <class T>
constexpr int kPwBlocks = sizeof(T) == 4 ? 4 : 3;
template <class T, int Z>
__global__ void __launch_bounds__(NT, kPwBlocks<T>) k_pw(Geom g, const T *__restrict__ Kx, const T *__restrict__ Ky, T *pa, T *pb,
                                              const T *__restrict__ r, const T *__restrict__ Mi, T *__restrict__ u,
                                              T *__restrict__ w, T rx, T ry, int rows, Scalars *s, double *part,
                                              unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  if (s->done) return;
  const int odd = s->iters & 1;
  const T *pin = odd ? pb : pa;
  T *pout = odd ? pa : pb;
  const bool first = Z == Z_FCG ? s->restart != 0 : s->iters == 0 && !s->pend, pend = s->pend != 0;
  const T alpha = (T)s->alpha, beta = (T)s->beta;
  constexpr int NV = Z == Z_FCG ? 2 : 1;
  const int ncol = (g.nx + 29) / 30, nst = (g.ny + rows - 1) / rows;
  const int wi = blockIdx.x * kWarps + (tid_() >> 5), lane = tid_() & 31;
  double acc[NV] = {};
  if (wi < ncol * nst) {
    const int x = (wi % ncol) * 30 + lane - 1, y0 = (wi / ncol) * rows, y1 = min(y0 + rows, g.ny);
    const bool in = x >= 0 && x < g.nx, own = in && lane >= 1 && lane <= 30, ring = x == -1 || x == g.nx;
    const long long P = g.pitch;
    struct Row {
      T kx0, kx1, ky1, r, p, m, u;
    };
    auto load = [&](int y) {
      Row v{};
      const long long i = (long long)y * P + x;
      if (in && y >= 0 && y < g.ny) {
        v.kx0 = Kx[i];
        if (lane == 31) v.kx1 = Kx[i + 1];  // the other lanes' comes from their neighbour
        v.ky1 = Ky[i + P];
        v.r = r[i];
        v.p = pin[i];
        if (Z == Z_MI || (Z == Z_FCG && own && y >= y0 && y < y1)) v.m = Mi[i];
        if (pend && own && y >= y0 && y < y1) v.u = u[i];
      } else if (in || (ring && y >= 0 && y < g.ny)) {
        v.p = pa[i];
        if (x == g.nx) v.kx0 = Kx[i];  // the last column's right face
      }
      return v;
    };
    // the new direction at row y; d is the diagonal of A there
    auto dir = [&](Row &v, int y, T ky0, T &d) {
      const T kr = __shfl_down_sync(0xffffffffu, v.kx0, 1);
      if (lane < 31) v.kx1 = kr;
      d = T(1) + ry * (v.ky1 + ky0) + rx * (v.kx1 + v.kx0);
      if (!in || y < 0 || y >= g.ny) return v.p;
      const T z = Z == Z_R || Z == Z_FCG ? v.r : Z == Z_MI ? v.m * v.r : (T(1) / d) * v.r;
      return first ? z : beta * v.p + z;
    };
    auto face = [&](int y) { return in && y >= 0 && y < g.ny ? Ky[(long long)y * P + x] : T(0); };
    Row b = load(y0 - 1);
    T d;
    T pm = dir(b, y0 - 1, face(y0 - 1), d);
    T ky0 = face(y0);
    Row c = load(y0), n = load(y0 + 1);
    T pc = dir(c, y0, ky0, d);
    for (int y = y0; y < y1; y++) {
      const Row nn = load(min(y + 2, y1));
      const T ky1 = c.ky1;
      T dn;
      const T pn = dir(n, y + 1, ky1, dn);
      const T pl = __shfl_up_sync(0xffffffffu, pc, 1), pr = __shfl_down_sync(0xffffffffu, pc, 1);
      if (own) {
        const long long i = (long long)y * P + x;
        const T wv = d * pc - ry * (ky1 * pn + ky0 * pm) - rx * (c.kx1 * pr + c.kx0 * pl);
        w[i] = wv;
        pout[i] = pc;
        if (pend) u[i] = c.u + alpha * c.p;
        acc[0] = acc[0] + (double)wv * (double)pc;
        if (Z == Z_FCG) acc[NV - 1] = acc[NV - 1] + (double)pc * (double)c.m;
      }
      pm = pc;
      pc = pn;
      d = dn;
      ky0 = ky1;
      c = n;
      n = nn;
    }
  }
  if (publish<NV>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<NV>(part, 0, sm);
    const double pr = Z == Z_FCG ? grid_total<NV>(part, NV - 1, sm) : 0.0;
    if (tid_() == 0) {
      s->pw = t;
      if (Z == Z_FCG) {
        s->restart = 0;
        s->pend = t > 0.0;
        if (t > 0.0) s->alpha = pr / t;
        else s->done = 4;
      } else {
        s->alpha = s->rro / t;
        s->pend = 1;
      }
      *cnt = 0u;
    }
  }
}

// The last block's part of k_r: beta = rrn / rro and the stop test.
template <int NV, int STOP>
__device__ __forceinline__ void finish_r(const double (&acc)[NV], Scalars *s, double *part, unsigned *cnt, double *sm,
                                         int *last) {
  if (publish<NV>(acc, part, cnt, sm, last)) {
    const double t = grid_total<NV>(part, 0, sm);
    const double rr = NV == 2 ? grid_total<NV>(part, NV - 1, sm) : t;
    if (tid_() == 0) {
      s->rro_prev = s->rro;
      s->beta = t / s->rro;
      s->rro = t;
      s->iters = s->iters + 1;
      const double err = STOP == STOP_TRUE ? sqrt(fabs(rr)) : sqrt(fabs(t));
      s->err = err;
      if (fabs(err) < s->stop) s->done = 1;
      else if (STOP == STOP_RELIABLE && err < s->ref) s->done = 3;
      else if (s->iters >= s->max_iters) s->done = 2;
      *cnt = 0u;
    }
  }
}

// tea_leaf_axpy_kernel on r, tea_leaf_zeqxty_kernel (z = Mi r) and
// tea_leaf_dot_kernel (r.z), or tea_leaf_cg_calc_ur_r_reduce_kernel's r.r
// without preconditioner.
template <class T, bool PREC, int STOP>
__global__ void __launch_bounds__(NT, kResident) k_r(Geom g, T *__restrict__ r, const T *__restrict__ w,
                                                     const T *__restrict__ Mi, Scalars *s, double *part,
                                                     unsigned *cnt) {
  constexpr int NV = (STOP == STOP_TRUE && PREC) ? 2 : 1;
  __shared__ double sm[kWarps];
  __shared__ int last;
  if (s->done) return;
  const T alpha = (T)s->alpha;
  double acc[NV] = {};
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const T rv = r[i] - alpha * w[i];
    r[i] = rv;
    const T zv = PREC ? Mi[i] * rv : rv;
    acc[0] = acc[0] + (double)rv * (double)zv;
    if (NV == 2) acc[NV - 1] = acc[NV - 1] + (double)rv * (double)rv;
  }
  finish_r<NV, STOP>(acc, s, part, cnt, sm, &last);
}

// After the loop: the pending u += alpha p, the current direction back in the
// first buffer and, when `z` is wanted, z = Mi r.
template <class T>
__global__ void __launch_bounds__(NT, kResident) k_flush(Geom g, T *__restrict__ u, T *pa, const T *pb,
                                                         const T *__restrict__ r, const T *__restrict__ Mi, T *z,
                                                         const Scalars *s) {
  if (!s->pend) return;
  const T alpha = (T)s->alpha;
  const bool odd = s->iters & 1;
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const T p = odd ? pb[i] : pa[i];
    u[i] = u[i] + alpha * p;
    if (odd) pa[i] = p;
    if (z) z[i] = Mi[i] * r[i];
  }
}

// tea_leaf_common_residual_kernel + tea_leaf_norm2_kernel (tea_leaf_common.cpp:160-211):
// r = u0 - A u, rr = r.r. The first call of a solve fixes ||r0|| and the
// stop threshold eps * ||r0|| (tea_solve.cpp:105-114); later calls test against it.
__global__ void __launch_bounds__(NT, kResident) k_resid(Geom g, const double *__restrict__ Kx, const double *__restrict__ Ky,
                                              const double *__restrict__ u, const double *__restrict__ u0,
                                              double *__restrict__ r, double rx, double ry, double eps, Scalars *s,
                                              double *part, unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  double acc[1] = {0.0};
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const double smv = smvp(Kx, Ky, u, i, g.pitch, rx, ry);
    const double rv = u0[i] - smv;
    r[i] = rv;
    acc[0] = acc[0] + rv * rv;
  }
  if (publish<1>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<1>(part, 0, sm);
    if (tid_() == 0) {
      s->rr = t;
      const double nrm = sqrt(fabs(t));
      if (s->first) {
        s->rr0 = t;
        s->stop = eps * nrm;
        s->first = 0;
      }
      s->err = nrm;
      s->done = (fabs(nrm) < s->stop) ? 1 : 0;
      *cnt = 0u;
    }
  }
}

// cg_init (tea_leaf_cg.cpp:53-101): z = Mi r (or none), p = z (or r), rro = r.p.
template <bool PREC>
__global__ void __launch_bounds__(NT, kResident) k_init(Geom g, const double *__restrict__ r, const double *__restrict__ Mi,
                                             double *__restrict__ z, double *__restrict__ p, int max_iters,
                                             Scalars *s, double *part, unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  double acc[1] = {0.0};
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const double rv = r[i];
    double pv = rv;
    if (PREC) {
      pv = Mi[i] * rv;
      z[i] = pv;
    }
    p[i] = pv;
    acc[0] = acc[0] + rv * pv;
  }
  if (publish<1>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<1>(part, 0, sm);
    if (tid_() == 0) {
      s->rro = t;
      s->iters = 0;
      s->max_iters = max_iters;
      s->done = 0;
      s->pend = 0;
      *cnt = 0u;
    }
  }
}

// Reliable update of the FP32 loop (Sleijpen and van der Vorst 1996, "Reliable
// updated residuals in hybrid Bi-CG methods"): the recursive FP32 residual is
// replaced by the FP64 residual r64 = u0 - A u, z32 = Mi32 r32, and the search
// direction is kept: beta = rz_new / rz_prev, which the next k_pw applies. The
// first call starts the loop (no direction yet, so p = z) and fixes the estimate
// threshold eps * sqrt(rz0); `scale` tightens it after an estimate that the
// FP64 check did not confirm. The next update is due once sqrt(rz) has fallen
// by `delta`.
template <bool PREC>
__global__ void __launch_bounds__(NT, kResident) k_reinit32(Geom g, Geom g32, const double *__restrict__ r64,
                                                 float *__restrict__ r, const float *__restrict__ Mi, int first,
                                                 double eps, double scale,
                                                 double delta, int max_iters, Scalars *s, double *part,
                                                 unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  double acc[1] = {0.0};
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const long long j = (long long)y * g32.pitch + x;
    const float rv = (float)r64[i];
    r[j] = rv;
    const float zv = PREC ? Mi[j] * rv : rv;
    acc[0] = acc[0] + (double)rv * (double)zv;
  }
  if (publish<1>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<1>(part, 0, sm);
    if (tid_() == 0) {
      if (first) {
        s->rr0 = t;
        s->iters = 0;
        s->max_iters = max_iters;
        s->beta = 0.0;
      } else {
        s->beta = t / s->rro_prev;
      }
      s->stop = eps * scale * sqrt(fabs(s->rr0));
      s->ref = delta * sqrt(fabs(t));
      s->rro = t;
      s->done = 0;
      s->pend = 0;
      *cnt = 0u;
    }
  }
}

// Reliable update, FP64 side: e += alpha p (the last iteration's), u += e, e = 0.
__global__ void __launch_bounds__(NT, kResident) k_update(Geom g, Geom g32, double *__restrict__ u,
                                                          float *__restrict__ e, const float *__restrict__ pa,
                                                          const float *__restrict__ pb, const Scalars *s) {
  const float alpha = (float)s->alpha;
  const float *p = s->iters & 1 ? pb : pa;
  const bool pend = s->pend != 0;
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const long long j = (long long)y * g32.pitch + x;
    const float ev = pend ? e[j] + alpha * p[j] : e[j];
    u[i] = u[i] + (double)ev;
    e[j] = 0.0f;
  }
}

// FP32 copies of Kx, Ky, Mi over the interior and its one-cell ring.
__global__ void __launch_bounds__(NT, kResident) k_to_float(Geom g, Geom g32, const double *__restrict__ a,
                                                 const double *__restrict__ b, const double *__restrict__ c,
                                                 float *__restrict__ fa, float *__restrict__ fb,
                                                 float *__restrict__ fc) {
  for (int y = blockIdx.y * BY + threadIdx.y - 1; y < g.ny + 1; y += gridDim.y * BY)
    for (int x = blockIdx.x * BX + threadIdx.x - 1; x < g.nx + 1; x += gridDim.x * BX) {
      const long long i = (long long)y * g.pitch + x, j = (long long)y * g32.pitch + x;
      fa[j] = (float)a[i];
      fb[j] = (float)b[i];
      if (c) fc[j] = x >= 0 && x < g.nx && y >= 0 && y < g.ny ? (float)c[i] : 0.0f;  // Mi: zero on the ring
    }
}


// ---- the whole loop in one kernel, for grids that fit the registers ---------
// On small grids an iteration of the two kernels above is launch and drain
// latency: 14 us at 128^2, 17 us at 512^2. Grids of up to kTargetBlocks blocks of
// 128 x 2 cells that fit one CTA an SM, 8 to a CTA (on 148 SMs up to 512^2 or 1024
// x 288), take one kernel. Here a CTA keeps K such blocks, one above the other: its cells' r,
// u and coefficients stay in registers, the direction p in shared memory with a
// one-cell halo, for the whole loop. CTAs exchange only z along their edges
// and the partial sums (a neighbour's p is beta p + z, tracked in the halo):
// 64^2 14.1 -> 3.7 us an iteration, 128^2 14.0 -> 4.5, 256^2 14.2 -> 5.4, 512^2
// 17.3 -> 10.8 (FP64; 128^2 took 3.5 us on one B200 and 5.2 on another, 500 x 511
// 8.0 and 11.4).
// Each block's partial is its own, and the totals are taken, in the order that
// the launched kernels use (publish, grid_total), so alpha, beta and every
// iterate are the same bits as an iteration of single-cell threads gave.
//
// A value travels as two 64-bit words, each with half of it and the number of
// the exchange, so a reader knows a whole value without a fence or a counter;
// two slots alternate, since a CTA can be one exchange ahead of another. The
// CTAs wait for one another, so the launch is cooperative, and a wait ends with
// an error after the limit given (option heat_wait_ms; at 0 nothing is published
// and every wait runs out). A thread takes no further value of a sum then, so its
// CTA stops within four limits, and leaves u, r and p as they were.

__device__ __forceinline__ void ll_put(ulonglong2 *slot, double v, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(t | (b & 0xffffffffull)), "l"(t | (b >> 32))
               : "memory");
}
// The value tagged `tag`; false when it did not arrive in time. (How often the
// loop polls decides how soon values travel: 128^2 to 550^2 moved by up to 25 %
// with the shape of this loop and its callers, on the same machine. This one and
// a compile-time limit measure the same; a flag to leave early costs 5 to 10 %.)
__device__ __forceinline__ bool ll_get(const ulonglong2 *slot, unsigned tag, double *v, unsigned long long wait_ns) {
  unsigned long long t0 = 0;
  for (unsigned i = 0;; i++) {
    unsigned long long a, b;
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(slot) : "memory");
    if ((unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag) {
      *v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
      return true;
    }
    if ((i & 255u) == 255u) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (!t0) t0 = now;
      else if (now - t0 > wait_ns) return false;
    }
  }
}

template <class T, int Z, int STOP, int K>
__global__ void __launch_bounds__(NT, 1) k_pcg_resident(Geom g, const T *__restrict__ Kx, const T *__restrict__ Ky,
                                                        T *__restrict__ p, T *__restrict__ r, const T *__restrict__ Mi,
                                                        T *__restrict__ u, T *__restrict__ zout, T rx, T ry, int gx,
                                                        Scalars *s, ulonglong2 *slots, unsigned long long wait_ns,
                                                        int *err) {
  constexpr int NV = (STOP == STOP_TRUE && Z != Z_R) ? 2 : 1;
  __shared__ T ps[2 * K + 2][BX + 2];
  __shared__ double ws[NV * K][kWarps], sm[kWarps], tot[2];
  __shared__ int expired;
  if (s->done) return;
  const int tx = threadIdx.x, ty = threadIdx.y, t = tid_(), lane = t & 31, warp = t >> 5;
  const int bx = blockIdx.x % gx, by = blockIdx.x / gx, y0 = by * 2 * K, x = bx * BX + tx;
  const int gy = (g.ny + BY - 1) / BY, nb = gx * gy;  // the launched kernels' blocks
  const int put_rows = wait_ns ? gy : 0;  // with no time to wait, nothing is published
  const long long P = g.pitch;
  const bool first = s->iters == 0;
  double rro = s->rro, rro_prev = s->rro_prev, alpha = s->alpha, beta = s->beta, pw = s->pw, e = s->err;
  int iters = s->iters;
  const int max_iters = s->max_iters;
  const double stop = s->stop, ref = s->ref;
  if (t == 0) expired = 0;

  T kx0[K], kx1[K], ky0[K], ky1[K], d[K], mi[K], rv[K], uv[K], pv[K], zv[K], wv[K];
  auto row = [&](int k) { return y0 + 2 * k + ty; };
  auto cell = [&](int xx, int yy) { return xx >= 0 && xx < g.nx && yy >= 0 && yy < g.ny; };
  // a ring cell beside the interior holds a constant direction
  auto ring = [&](int xx, int yy) {
    return ((xx == -1 || xx == g.nx) && yy >= 0 && yy < g.ny) || ((yy == -1 || yy == g.ny) && xx >= 0 && xx < g.nx);
  };
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int y = row(k);
    const long long i = (long long)y * P + x;
    kx0[k] = kx1[k] = ky0[k] = ky1[k] = d[k] = mi[k] = rv[k] = uv[k] = pv[k] = zv[k] = T(0);
    if (cell(x, y)) {
      kx0[k] = Kx[i];
      kx1[k] = Kx[i + 1];
      ky0[k] = Ky[i];
      ky1[k] = Ky[i + P];
      d[k] = T(1) + ry * (ky1[k] + ky0[k]) + rx * (kx1[k] + kx0[k]);
      mi[k] = Z == Z_R ? T(1) : Mi[i];
      rv[k] = r[i];
      uv[k] = u[i];
      if (!first) pv[k] = p[i];
      zv[k] = Z == Z_R ? rv[k] : mi[k] * rv[k];
    } else {
      ps[1 + 2 * k + ty][1 + tx] = ring(x, y) ? p[i] : T(0);
    }
  }
  // z on a CTA's edges: its first row, last row, first column, last column,
  // in one of two buffers
  constexpr int kEdge = 2 * BX + 4 * K;
  ulonglong2 *edges = slots + 4 * kTargetBlocks;
  auto edge = [&](int cx, int cy, int at, unsigned buf) {
    return edges + ((size_t)(cx + cy * gx) * 2 + buf) * kEdge + at;
  };
  // this thread's halo cells: above or below its column, and one at the side
  struct Halo {
    T *at;  // its place in ps
    const ulonglong2 *from;  // its CTA's edge slot, first buffer
    bool live;  // an interior cell of another CTA
    T p, z;
  };
  auto halo = [&](int xx, int yy, int cx, int cy, int slot) {
    const long long i = (long long)yy * P + xx;
    Halo h{&ps[yy - y0 + 1][xx - bx * BX + 1], nullptr, cell(xx, yy), T(0), T(0)};
    if (h.live) {
      h.from = edge(cx, cy, slot, 0);
      h.z = Z == Z_R ? r[i] : Mi[i] * r[i];
      if (!first) h.p = p[i];
    } else {
      *h.at = ring(xx, yy) ? p[i] : T(0);
    }
    return h;
  };
  Halo hv = ty ? halo(x, y0 + 2 * K, bx, by + 1, tx) : halo(x, y0 - 1, bx, by - 1, BX + tx), hs{};
  if (t < 2 * K) hs = halo(bx * BX - 1, y0 + t, bx - 1, by, 2 * BX + 2 * K + t);
  else if (t < 4 * K) hs = halo(bx * BX + BX, y0 + t - 2 * K, bx + 1, by, 2 * BX + t - 2 * K);

  // the grid's sums of acc[v * K + k], block k of this CTA; `meanwhile` runs
  // between this CTA's share and the wait for the others'
  auto total = [&](auto &acc, auto nv, unsigned tag, auto meanwhile) {
    constexpr int N = decltype(nv)::value;
#pragma unroll
    for (int q = 0; q < N * K; q++) {
      double v = acc[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) ws[q][warp] = v;
    }
    __syncthreads();
    ulonglong2 *buf = slots + (size_t)(tag & 1u) * 2 * kTargetBlocks;
    for (int q = warp; q < N * K; q += kWarps) {
      double v = lane < kWarps ? ws[q][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      const int k = q % K, vb = y0 / 2 + k;
      if (lane == 0 && vb < put_rows) ll_put(buf + (size_t)(q / K) * kTargetBlocks + bx + vb * gx, v, tag);
    }
    meanwhile();
#pragma unroll
    for (int n = 0; n < N; n++) {
      double v = 0.0;
      for (int b = t; b < nb; b += NT) {
        double q = 0.0;
        if (!ll_get(buf + (size_t)n * kTargetBlocks + b, tag, &q, wait_ns)) {
          expired = 1;
          break;
        }
        v += q;
      }
      v = block_sum(v, sm);
      if (t == 0) tot[n] = v;
    }
    __syncthreads();
  };

  unsigned tag = 0;
  int done = 0;
  bool fresh = first;
  while (true) {
    const T bt = (T)beta;
#pragma unroll
    for (int k = 0; k < K; k++) {
      pv[k] = fresh ? zv[k] : bt * pv[k] + zv[k];
      if (cell(x, row(k))) ps[1 + 2 * k + ty][1 + tx] = pv[k];
    }
    if (hv.live) *hv.at = hv.p = fresh ? hv.z : bt * hv.p + hv.z;
    if (hs.live) *hs.at = hs.p = fresh ? hs.z : bt * hs.p + hs.z;
    fresh = false;
    __syncthreads();
    {
      double acc[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int yy = 1 + 2 * k + ty, xx = 1 + tx;
        wv[k] = d[k] * pv[k] - ry * (ky1[k] * ps[yy + 1][xx] + ky0[k] * ps[yy - 1][xx]) -
                rx * (kx1[k] * ps[yy][xx + 1] + kx0[k] * ps[yy][xx - 1]);
        acc[k] = (double)wv[k] * (double)pv[k];
      }
      total(acc, std::integral_constant<int, 1>{}, ++tag, [] {});
    }
    if (expired) break;
    pw = tot[0];
    alpha = rro / pw;
    const T al = (T)alpha;
    {
      double acc[NV * K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        uv[k] = uv[k] + al * pv[k];
        rv[k] = rv[k] - al * wv[k];
        zv[k] = Z == Z_R ? rv[k] : mi[k] * rv[k];
        acc[k] = (double)rv[k] * (double)zv[k];
        if (NV == 2) acc[(NV - 1) * K + k] = (double)rv[k] * (double)rv[k];
      }
      ++tag;
      const unsigned buf = (tag >> 1) & 1u;
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (!cell(x, row(k))) continue;
        const int q = 2 * k + ty;
        const double zd = (double)zv[k];
        if (q == 0) ll_put(edge(bx, by, tx, buf), zd, tag);
        if (q == 2 * K - 1) ll_put(edge(bx, by, BX + tx, buf), zd, tag);
        if (tx == 0) ll_put(edge(bx, by, 2 * BX + q, buf), zd, tag);
        if (tx == BX - 1) ll_put(edge(bx, by, 2 * BX + 2 * K + q, buf), zd, tag);
      }
      total(acc, std::integral_constant<int, NV>{}, tag, [&] {
        double z = 0.0;
        if (hv.live) {
          if (!ll_get(hv.from + (size_t)buf * kEdge, tag, &z, wait_ns)) expired = 1;
          hv.z = (T)z;
        }
        if (hs.live) {
          if (!ll_get(hs.from + (size_t)buf * kEdge, tag, &z, wait_ns)) expired = 1;
          hs.z = (T)z;
        }
      });
    }
    if (expired) break;
    const double rz = tot[0], rr = tot[NV - 1];
    rro_prev = rro;
    beta = rz / rro;
    rro = rz;
    iters++;
    e = STOP == STOP_TRUE ? sqrt(fabs(rr)) : sqrt(fabs(rz));
    if (fabs(e) < stop) done = 1;
    else if (STOP == STOP_RELIABLE && e < ref) done = 3;
    else if (iters >= max_iters) done = 2;
    if (done) break;
  }
#pragma unroll
  for (int k = 0; k < K; k++) {
    if (!cell(x, row(k)) || expired) continue;
    const long long i = (long long)row(k) * P + x;
    u[i] = uv[k];
    r[i] = rv[k];
    p[i] = pv[k];
    if (zout) zout[i] = zv[k];
  }
  if (blockIdx.x == 0 && t == 0 && !expired) {
    s->rro = rro;
    s->rro_prev = rro_prev;
    s->alpha = alpha;
    s->beta = beta;
    s->pw = pw;
    s->err = e;
    s->iters = iters;
    s->done = done;
  }
  if (t == 0 && expired) *err = 1;
}

// ---- flexible CG -----------------------------------------------------------
// An iteration is k_pw<Z_FCG> (direction, w = A p and the previous step of u;
// they were three passes of 112 B a cell, now one of 72), k_fr, the
// preconditioner and k_fzw.
// r -= alpha w, rr = r.r; stop when ||r|| < eps ||r0||.
__global__ void __launch_bounds__(NT, kResident) k_fr(Geom g, double *__restrict__ r, const double *__restrict__ w,
                                                      Scalars *s, double *part, unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  if (s->done) return;
  const double alpha = s->alpha;
  double acc[1] = {0.0};
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    const double rv = r[i] - alpha * w[i];
    r[i] = rv;
    acc[0] = acc[0] + rv * rv;
  }
  if (publish<1>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<1>(part, 0, sm);
    if (tid_() == 0) {
      s->rr = t;
      s->err = sqrt(t);
      s->iters = s->iters + 1;
      if (s->err < s->stop) s->done = 1;
      else if (s->iters >= s->max_iters) s->done = 2;
      if (s->done == 0 && s->window > 0) {  // the same test the host loop applies
        const int k = s->hcount;
        s->hist[k & 63] = s->err;
        s->hcount = k + 1;
        if (k + 1 > s->window && s->err > 0.5 * s->hist[(k - s->window) & 63]) s->done = 5;
      }
      *cnt = 0u;
    }
  }
}

// beta = -(z.w) / pw.
__global__ void __launch_bounds__(NT, kResident) k_fzw(Geom g, const double *__restrict__ z, const double *__restrict__ w,
                                            Scalars *s, double *part, unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  if (s->done) return;  // the solve stopped earlier in a replayed chunk
  double acc[1] = {0.0};
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    acc[0] = acc[0] + z[i] * w[i];
  }
  if (publish<1>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<1>(part, 0, sm);
    if (tid_() == 0) {
      s->beta = -t / s->pw;
      *cnt = 0u;
    }
  }
}

// z = Mi r (Jacobi).
__global__ void __launch_bounds__(NT, kResident) k_jacobi(Geom g, const double *__restrict__ Mi, const double *__restrict__ r,
                                               double *__restrict__ z) {
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    z[i] = Mi[i] * r[i];
  }
}

// tea_leaf_common_init_diag_init_kernel (tea_leaf_common_kernels.h:38):
// Mi = 1 / (1 + ry (Ky(0,1) + Ky(0,0)) + rx (Kx(1,0) + Kx(0,0))) on the interior.
__global__ void __launch_bounds__(NT, kResident) k_diag(Geom g, const double *__restrict__ Kx, const double *__restrict__ Ky,
                                             double rx, double ry, double *__restrict__ Mi) {
  HEAT_CELLS(g) {
    const long long i = (long long)y * g.pitch + x;
    Mi[i] = 1.0 / (1.0 + ry * (Ky[i + g.pitch] + Ky[i]) + rx * (Kx[i + 1] + Kx[i]));
  }
}

// ---- 3D: the 7-point heat operator ------------------------------------------
// Interior cells (x, y, z) at i = z * plane + y * pitch + x from the first
// interior cell; Kz[i] is the face between z-1 and z (as Kx, Ky in 2D).
// The pointwise CG kernels run on the padded volume as a flat array (the
// solver's own fields are zero on every halo cell), so only the operator,
// the residual and the diagonal need these.
struct Geom3 {
  int nx, ny, nz;
  long long pitch, plane;
};

#define HEAT_CELLS3(g)                                                                                        \
  for (int row = blockIdx.y * BY + threadIdx.y, y = row % (g).ny, z = row / (g).ny; row < (g).ny * (g).nz;   \
       row += gridDim.y * BY, y = row % (g).ny, z = row / (g).ny)                                            \
    for (int x = blockIdx.x * BX + threadIdx.x; x < (g).nx; x += gridDim.x * BX)

template <class T>
__device__ __forceinline__ T smvp3(const T *__restrict__ Kx, const T *__restrict__ Ky, const T *__restrict__ Kz,
                                   const T *__restrict__ u, long long i, long long P, long long Q, T rx, T ry, T rz) {
  const T kx0 = Kx[i], kx1 = Kx[i + 1], ky0 = Ky[i], ky1 = Ky[i + P], kz0 = Kz[i], kz1 = Kz[i + Q];
  return (T(1) + rz * (kz1 + kz0) + ry * (ky1 + ky0) + rx * (kx1 + kx0)) * u[i] - rz * (kz1 * u[i + Q] + kz0 * u[i - Q]) -
         ry * (ky1 * u[i + P] + ky0 * u[i - P]) - rx * (kx1 * u[i + 1] + kx0 * u[i - 1]);
}

// k_pw in 3D (FP64, or FP32 for the mixed solver's inner iterations), with z =
// Mi r. A CTA marches along z over a tile of 30 x (kTileY - 2) cells, one
// column a thread, its outermost threads computing p for their neighbours:
// p of the planes below and above stays in registers, p of the columns beside
// comes by shuffles in x and through shared memory in y (three planes, so that
// one barrier a plane is enough). Halo cells hold p = 0.
constexpr int kTileY = 16;

template <class T>
__global__ void __launch_bounds__(32 * kTileY, 2) k_pw3(Geom3 g, const T *__restrict__ Kx, const T *__restrict__ Ky,
                                                       const T *__restrict__ Kz, T *pa, T *pb,
                                                       const T *__restrict__ r, const T *__restrict__ Mi,
                                                       T *__restrict__ u, T *__restrict__ w, T rx, T ry, T rz, int tx,
                                                       int ty, int planes, Scalars *s, double *part, unsigned *cnt) {
  __shared__ double sm[kTileY];
  __shared__ T ps[3][kTileY][32];
  __shared__ int last;
  if (s->done) return;
  const int odd = s->iters & 1;
  const T *pin = odd ? pb : pa;
  T *pout = odd ? pa : pb;
  const bool first = s->iters == 0 && !s->pend, pend = s->pend != 0;
  const T alpha = (T)s->alpha, beta = (T)s->beta;
  const int lane = threadIdx.x, row = threadIdx.y;
  const int bx = blockIdx.x % tx, by = (blockIdx.x / tx) % ty, bz = blockIdx.x / (tx * ty);
  const int x = bx * 30 + lane - 1, y = by * (kTileY - 2) + row - 1;
  const int z0 = bz * planes, z1 = min(z0 + planes, g.nz);
  const bool in = x >= 0 && x < g.nx && y >= 0 && y < g.ny;
  const bool own = in && lane >= 1 && lane <= 30 && row >= 1 && row <= kTileY - 2;
  const long long P = g.pitch, Q = g.plane, base = (long long)y * P + x;
  struct Raw {
    T r, p, m;
  };
  auto load = [&](int z) {
    Raw v{};
    if (in && z >= 0 && z < g.nz) {
      const long long i = base + (long long)z * Q;
      v.r = r[i];
      v.p = pin[i];
      v.m = Mi[i];
    }
    return v;
  };
  auto dir = [&](const Raw &v) {
    const T z = v.m * v.r;
    return first ? z : beta * v.p + z;
  };
  double acc = 0.0;
  const Raw b = load(z0 - 1);
  Raw c = load(z0), n = load(z0 + 1);
  T pm = dir(b), pc = dir(c);
  ps[z0 % 3][row][lane] = pc;
  T kz0 = own ? Kz[base + (long long)z0 * Q] : T(0);
  struct Face {
    T kx0, kx1, ky0, ky1, kz1, u;
  };
  auto faces = [&](int z) {
    Face f{};
    if (own) {
      const long long i = base + (long long)z * Q;
      f.kx0 = Kx[i];
      f.kx1 = Kx[i + 1];
      f.ky0 = Ky[i];
      f.ky1 = Ky[i + P];
      f.kz1 = Kz[i + Q];
      if (pend) f.u = u[i];
    }
    return f;
  };
  // FP32 has the registers to load a plane's faces one plane ahead too
  constexpr bool kAhead = sizeof(T) == 4;
  Face f{};
  if (kAhead) f = faces(z0);
  for (int z = z0; z < z1; z++) {
    const long long i = base + (long long)z * Q;
    if (!kAhead) f = faces(z);
    const Face c_f = f;
    if (kAhead) f = faces(min(z + 1, z1 - 1));
    const Raw nn = load(min(z + 2, z1));
    const T pn = dir(n);
    ps[(z + 1) % 3][row][lane] = pn;
    __syncthreads();
    const T pl = __shfl_up_sync(0xffffffffu, pc, 1), pr = __shfl_down_sync(0xffffffffu, pc, 1);
    if (own) {
      const T kx0 = c_f.kx0, kx1 = c_f.kx1, ky0 = c_f.ky0, ky1 = c_f.ky1, kz1 = c_f.kz1;
      const T ps0 = ps[z % 3][row - 1][lane], ps1 = ps[z % 3][row + 1][lane];
      const T wv = (T(1) + rz * (kz1 + kz0) + ry * (ky1 + ky0) + rx * (kx1 + kx0)) * pc - rz * (kz1 * pn + kz0 * pm) -
                   ry * (ky1 * ps1 + ky0 * ps0) - rx * (kx1 * pr + kx0 * pl);
      w[i] = wv;
      pout[i] = pc;
      if (pend) u[i] = c_f.u + alpha * c.p;
      acc = acc + (double)wv * (double)pc;
    }
    kz0 = c_f.kz1;
    pm = pc;
    pc = pn;
    c = n;
    n = nn;
  }
  // the block's partial, then the last block's total, as publish / grid_total
  auto sum = [&](double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sm[row] = v;
    __syncthreads();
    double t = 0.0;
    if (row == 0) {
      t = lane < kTileY ? sm[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    }
    return t;
  };
  const double bs = sum(acc);
  const bool lead = lane == 0 && row == 0;
  if (lead) {
    part[blockIdx.x] = bs;
    __threadfence();
    last = atomicAdd(cnt, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0.0;
  for (int k = row * 32 + lane; k < (int)gridDim.x; k += 32 * kTileY) v += __ldcg(part + k);
  const double t = sum(v);
  if (lead) {
    s->pw = t;
    s->alpha = s->rro / t;
    s->pend = 1;
    *cnt = 0u;
  }
}

// k_r over n consecutive values (the padded volume: its halo cells hold zeros
// and stay zero), 16 bytes a load: rows of 194 values or so would leave a
// quarter of a row-wise grid idle. The fields start on 16-byte boundaries.
constexpr int kFlatBlocks = 4;  // CTAs per SM: 64 registers hold a vector of each field
template <class T, int STOP>
__global__ void __launch_bounds__(NT, kFlatBlocks) k_r_flat(T *__restrict__ r, const T *__restrict__ w,
                                                          const T *__restrict__ Mi, long long n, Scalars *s,
                                                          double *part, unsigned *cnt) {
  constexpr int NV = STOP == STOP_TRUE ? 2 : 1, V = 16 / sizeof(T);
  __shared__ double sm[kWarps];
  __shared__ int last;
  if (s->done) return;
  const T alpha = (T)s->alpha;
  double acc[NV] = {};
  struct alignas(16) Vec {
    T v[V];
  };
  auto cell = [&](T rin, T wv, T m) {
    const T rv = rin - alpha * wv;
    acc[0] = acc[0] + (double)rv * (double)(m * rv);
    if (NV == 2) acc[NV - 1] = acc[NV - 1] + (double)rv * (double)rv;
    return rv;
  };
  const long long nv = n / V, step = (long long)gridDim.x * NT;
  for (long long k = (long long)blockIdx.x * NT + tid_(); k < nv; k += step) {
    Vec a = reinterpret_cast<Vec *>(r)[k];
    const Vec b = reinterpret_cast<const Vec *>(w)[k], c = reinterpret_cast<const Vec *>(Mi)[k];
#pragma unroll
    for (int j = 0; j < V; j++) a.v[j] = cell(a.v[j], b.v[j], c.v[j]);
    reinterpret_cast<Vec *>(r)[k] = a;
  }
  if (blockIdx.x == 0)
    for (long long k = nv * V + tid_(); k < n; k += NT) r[k] = cell(r[k], w[k], Mi[k]);
  finish_r<NV, STOP>(acc, s, part, cnt, sm, &last);
}

// r = u0 - A u, rr = r.r; the first call of a solve fixes ||r0|| and the stop
// threshold (k_resid in 3D).
__global__ void __launch_bounds__(NT, kResident) k_resid3(Geom3 g, const double *__restrict__ Kx,
                                                         const double *__restrict__ Ky, const double *__restrict__ Kz,
                                                         const double *__restrict__ u, const double *__restrict__ u0,
                                                         double *__restrict__ r, double rx, double ry, double rz,
                                                         double eps, Scalars *s, double *part, unsigned *cnt) {
  __shared__ double sm[kWarps];
  __shared__ int last;
  double acc[1] = {0.0};
  HEAT_CELLS3(g) {
    const long long i = (long long)z * g.plane + (long long)y * g.pitch + x;
    const double rv = u0[i] - smvp3<double>(Kx, Ky, Kz, u, i, g.pitch, g.plane, rx, ry, rz);
    r[i] = rv;
    acc[0] = acc[0] + rv * rv;
  }
  if (publish<1>(acc, part, cnt, sm, &last)) {
    const double t = grid_total<1>(part, 0, sm);
    if (tid_() == 0) {
      s->rr = t;
      const double nrm = sqrt(fabs(t));
      if (s->first) {
        s->rr0 = t;
        s->stop = eps * nrm;
        s->first = 0;
      }
      s->err = nrm;
      s->done = (fabs(nrm) < s->stop) ? 1 : 0;
      *cnt = 0u;
    }
  }
}

// Mi = 1 / diag(A) on the interior.
__global__ void __launch_bounds__(NT, kResident) k_diag3(Geom3 g, const double *__restrict__ Kx,
                                                        const double *__restrict__ Ky, const double *__restrict__ Kz,
                                                        double rx, double ry, double rz, double *__restrict__ Mi) {
  HEAT_CELLS3(g) {
    const long long i = (long long)z * g.plane + (long long)y * g.pitch + x;
    Mi[i] = 1.0 / (1.0 + rz * (Kz[i + g.plane] + Kz[i]) + ry * (Ky[i + g.pitch] + Ky[i]) + rx * (Kx[i + 1] + Kx[i]));
  }
}

// FP32 copy of n consecutive FP64 values (a padded volume, halos included).
__global__ void __launch_bounds__(NT, kResident) k_flat_to_float(const double *__restrict__ a, float *__restrict__ fa,
                                                                long long n) {
  for (long long k = (long long)blockIdx.x * NT + tid_(); k < n; k += (long long)gridDim.x * NT) fa[k] = (float)a[k];
}

dim3 grid_for3(int nx, int rows) {
  int gx = (nx + BX - 1) / BX;
  if (gx > 1024) gx = 1024;
  int gy = kTargetBlocks / gx;
  const int r = (rows + BY - 1) / BY;
  if (gy > r) gy = r;
  if (gy < 1) gy = 1;
  return dim3(gx, gy);
}

void check_launch(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw Error(E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace

// "heat_wait_ms" option: how long a block of k_pcg_resident waits for another.
static std::atomic<int> &wait_ms() {
  static std::atomic<int> ms{2000};
  return ms;
}
void set_wait_ms(int ms) {
  if (ms < 0) throw Error(E_ARG, "heat_wait_ms must be >= 0");
  wait_ms() = ms;
}

struct Solver::Impl {
  Scalars *s64 = nullptr, *s32 = nullptr;
  double *part = nullptr;
  int part_n = 0;
  unsigned *cnt = nullptr;
  int *h_flag = nullptr;  // pinned, two slots
  cudaEvent_t ev[2] = {nullptr, nullptr};
  // FP32 mirror for the mixed solver
  float *f32 = nullptr;
  size_t f32_bytes = 0;
  long long pitch32 = 0;
  float *Kx = nullptr, *Ky = nullptr, *Mi = nullptr, *r = nullptr, *p = nullptr, *w = nullptr, *p2 = nullptr,
        *e = nullptr;
  double *p64b = nullptr;  // of `second`
  size_t p64b_n = 0;
  float *Kz = nullptr;  // 3D only
  ulonglong2 *slots = nullptr;  // k_pcg_resident's exchange, then its error word
  // 2 x 2 partials a block, and the edges of up to 256 CTAs of 16 rows
  static constexpr size_t kSlotBytes = (4 * (size_t)kTargetBlocks + 256 * 2 * (2 * BX + 32)) * sizeof(ulonglong2);
  // replayed iteration chunks, rebuilt when any argument changes
  struct Chunk {
    cudaGraphExec_t exec = nullptr;
    std::string key;
  } chunk64, chunk32;

  ~Impl() {
    for (Chunk *c : {&chunk64, &chunk32})
      if (c->exec) cudaGraphExecDestroy(c->exec);
    for (cudaEvent_t x : ev)
      if (x) cudaEventDestroy(x);
    if (h_flag) cudaFreeHost(h_flag);
    cudaFree(s64);
    cudaFree(part);
    cudaFree(cnt);
    cudaFree(f32);
    cudaFree(p64b);
    cudaFree(slots);
  }

  // The loop of one PCG run by k_pcg_resident when the grid fits it (returns
  // false otherwise): s must hold what k_init or k_reinit32 left.
  template <class T, int Z, int STOP>
  bool resident(const Geom &g, const T *Kx, const T *Ky, T *p, T *r, const T *Mi, T *u, T *zout, T rx, T ry, Scalars *s,
                cudaStream_t st) {
    const int gx = (g.nx + BX - 1) / BX, gy = (g.ny + BY - 1) / BY;
    if ((long long)gx * gy > kTargetBlocks) return false;
    int dev = 0, sms = 0, coop = 0;
    OPSB_CUDA(cudaGetDevice(&dev));
    OPSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    OPSB_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return false;
    int K = 1;
    sms = std::min(sms, 256);
    while (K <= 8 && gx * ((gy + K - 1) / K) > sms) K *= 2;
    if (K > 8) return false;
    if (!slots) OPSB_CUDA(cudaMalloc(&slots, kSlotBytes + 64));
    OPSB_CUDA(cudaMemsetAsync(slots, 0, kSlotBytes + 64, st));
    int *err = reinterpret_cast<int *>(reinterpret_cast<char *>(slots) + kSlotBytes);
    const void *f = K == 1 ? (const void *)k_pcg_resident<T, Z, STOP, 1>
                  : K == 2 ? (const void *)k_pcg_resident<T, Z, STOP, 2>
                  : K == 4 ? (const void *)k_pcg_resident<T, Z, STOP, 4>
                           : (const void *)k_pcg_resident<T, Z, STOP, 8>;
    Geom gg = g;
    int gxx = gx;
    unsigned long long wait_ns = (unsigned long long)wait_ms() * 1000000ull;
    void *args[] = {&gg, &Kx, &Ky, &p, &r, &Mi, &u, &zout, &rx, &ry, &gxx, &s, &slots, &wait_ns, &err};
    OPSB_CUDA(cudaLaunchCooperativeKernel(f, dim3(gx * ((gy + K - 1) / K)), dim3(BX, BY), args, 0, st));
    OPSB_CUDA(cudaMemcpyAsync(h_flag, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    OPSB_CUDA(cudaStreamSynchronize(st));
    if (h_flag[0]) throw Error(E_TIMEOUT, "heat solver: a wait between thread blocks expired");
    return true;
  }

  // The FP64 direction's second buffer (addressed as its field's interior).
  double *second(const Field2D &f) {
    if (f.p2) return f.p2;
    const size_t n = (size_t)f.pitch * f.ny;
    if (n > p64b_n) {
      cudaFree(p64b);
      p64b = nullptr;
      p64b_n = 0;
      OPSB_CUDA(cudaMalloc(&p64b, n * sizeof(double)));
      p64b_n = n;
    }
    return p64b;
  }

  // Partials for a grid of more than kMaxBlocks (a strip or tile is a block's
  // least: 2D rows of a million cells, 3D cross-sections of 1312^2).
  void ensure_part(int blocks) {
    if (blocks <= part_n) return;
    cudaFree(part);
    part = nullptr;
    part_n = 0;
    chunk64.key.clear();  // the captured chunks hold the old address
    chunk32.key.clear();
    OPSB_CUDA(cudaMalloc(&part, 2 * (size_t)blocks * sizeof(double)));
    part_n = blocks;
  }

  void ensure_base() {
    if (s64) return;
    OPSB_CUDA(cudaMalloc(&s64, 2 * sizeof(Scalars)));
    s32 = s64 + 1;
    ensure_part(kMaxBlocks);
    OPSB_CUDA(cudaMalloc(&cnt, 64));
    OPSB_CUDA(cudaMemset(cnt, 0, 64));
    OPSB_CUDA(cudaMallocHost(&h_flag, 2 * sizeof(int)));
    for (cudaEvent_t &x : ev) OPSB_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
  }

  // The 3D mixed solver's nine FP32 fields, each a padded volume of nf
  // values in the FP64 fields' flat layout, zero on every halo cell; each
  // field starts on a 128-byte boundary.
  void ensure_f32_flat(size_t nf, cudaStream_t st) {
    nf = (nf + 31) / 32 * 32;
    const size_t bytes = 9 * nf * sizeof(float);
    if (bytes != f32_bytes || pitch32 != -1) {
      cudaFree(f32);
      f32 = nullptr;
      OPSB_CUDA(cudaMalloc(&f32, bytes));
      f32_bytes = bytes;
      pitch32 = -1;  // the 2D layout must be rebuilt
      chunk32.key.clear();
    }
    OPSB_CUDA(cudaMemsetAsync(f32, 0, bytes, st));
    float **fields[9] = {&Kx, &Ky, &Kz, &Mi, &r, &p, &w, &p2, &e};
    for (int k = 0; k < 9; k++) *fields[k] = f32 + k * nf;
  }

  // Eight FP32 fields with a one-cell ring; x = 0 of the interior starts a
  // 128-byte line.
  void ensure_f32(int nx, int ny, cudaStream_t st) {
    long long pitch = ((32 + nx + 1 + 31) / 32) * 32;
    size_t one = (size_t)pitch * (ny + 2);
    size_t bytes = 8 * one * sizeof(float);
    if (bytes != f32_bytes || pitch != pitch32) {
      cudaFree(f32);
      f32 = nullptr;
      OPSB_CUDA(cudaMalloc(&f32, bytes));
      f32_bytes = bytes;
      pitch32 = pitch;
      chunk32.key.clear();
    }
    OPSB_CUDA(cudaMemsetAsync(f32, 0, bytes, st));
    float **fields[8] = {&Kx, &Ky, &Mi, &r, &p, &w, &p2, &e};
    for (int k = 0; k < 8; k++) *fields[k] = f32 + k * one + pitch + 32;
  }
};

Solver::Solver() : m_(new Impl) {}
Solver::~Solver() { delete m_; }

namespace {

dim3 grid_for(int nx, int ny) {
  int gx = (nx + BX - 1) / BX;
  if (gx > 1024) gx = 1024;
  int gy = kTargetBlocks / gx;
  const int rows = (ny + BY - 1) / BY;
  if (gy > rows) gy = rows;
  if (gy < 1) gy = 1;
  return dim3(gx, gy);
}

// k_pw's strips and k_pw3's tiles (two CTAs).
void pw_grid(int nx, int ny, int per_sm, int *rows, int *blocks) {
  const long long ncol = (nx + 29) / 30;
  *rows = march_rows(ncol, ny, 2, 148LL * per_sm * kWarps, (long long)kMaxBlocks * kWarps);
  *blocks = (int)((ncol * ((ny + *rows - 1) / *rows) + kWarps - 1) / kWarps);
}
struct Grid3 {
  int tx, ty, planes, blocks;
};
Grid3 pw3_grid(int nx, int ny, int nz) {
  Grid3 q;
  q.tx = (nx + 29) / 30;
  q.ty = (ny + kTileY - 3) / (kTileY - 2);
  const long long tiles = (long long)q.tx * q.ty;
  if (tiles > 0x7fffffffLL) throw Error(E_UNSUPPORTED, "heat solver 3D: cross-section too large");
  q.planes = march_rows(tiles, nz, 2, 148LL * 2, kMaxBlocks);
  q.blocks = (int)(tiles * ((nz + q.planes - 1) / q.planes));
  return q;
}

std::string key_of(std::initializer_list<const void *> ptrs, std::initializer_list<double> vals) {
  std::string k;
  for (const void *p : ptrs) k.append(reinterpret_cast<const char *>(&p), sizeof(p));
  for (double v : vals) k.append(reinterpret_cast<const char *>(&v), sizeof(v));
  return k;
}

// Launches chunks of iterations until the solver flag says done; the host
// reads the flag of chunk c while chunk c+1 runs.
long long run_chunks(cudaGraphExec_t g, const Scalars *s, int max_iters, int *h_flag, cudaEvent_t *ev,
                     cudaStream_t st, int launches_per_chunk) {
  long long launches = 0;
  const int max_chunks = max_iters / kChunk + 2;
  for (int c = 0; c < max_chunks; c++) {
    OPSB_CUDA(cudaGraphLaunch(g, st));
    launches += launches_per_chunk;
    OPSB_CUDA(cudaMemcpyAsync(&h_flag[c & 1], &s->done, sizeof(int), cudaMemcpyDeviceToHost, st));
    OPSB_CUDA(cudaEventRecord(ev[c & 1], st));
    if (c > 0) {
      OPSB_CUDA(cudaEventSynchronize(ev[(c - 1) & 1]));
      if (h_flag[(c - 1) & 1]) break;
    }
  }
  OPSB_CUDA(cudaStreamSynchronize(st));
  return launches;
}

template <class F>
cudaGraphExec_t capture(cudaStream_t st, F body) {
  cudaGraph_t graph = nullptr;
  OPSB_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  body();
  cudaError_t le = cudaGetLastError();
  OPSB_CUDA(cudaStreamEndCapture(st, &graph));
  if (le != cudaSuccess) {
    cudaGraphDestroy(graph);
    throw Error(E_CUDA, std::string("heat solver capture: ") + cudaGetErrorString(le));
  }
  cudaGraphExec_t exec = nullptr;
  cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  OPSB_CUDA(ie);
  return exec;
}

void validate(const Field2D &f) {
  if (f.nx < 1 || f.ny < 1) throw Error(E_ARG, "heat solver: empty interior");
  if (f.pitch < f.nx + 2) throw Error(E_ARG, "heat solver: pitch smaller than the row");
  if (!f.Kx || !f.Ky || !f.u0 || !f.u || !f.r || !f.w || !f.p || !f.z || !f.Mi)
    throw Error(E_ARG, "heat solver: null field");
  if ((long long)f.ny * f.pitch > (1LL << 40)) throw Error(E_ARG, "heat solver: field too large");
}

Scalars fresh(double stop) {
  Scalars h;
  memset(&h, 0, sizeof(h));
  h.first = 1;
  h.stop = stop;
  return h;
}

}  // namespace

void Solver::pcg_fp64(const Field2D &f, double rx, double ry, bool precond, bool true_stop, double eps,
                      int max_iters, cudaStream_t st, SolveStats *out) {
  validate(f);
  Impl &m = *m_;
  m.ensure_base();
  launches_ = 0;
  const Geom g{f.nx, f.ny, f.pitch};
  const dim3 grid = grid_for(f.nx, f.ny), block(BX, BY);
  Scalars h = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s64, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  // initial residual (tea_solve.cpp:105-114) and cg_init
  k_resid<<<grid, block, 0, st>>>(g, f.Kx, f.Ky, f.u, f.u0, f.r, rx, ry, eps, m.s64, m.part, m.cnt);
  if (precond)
    k_init<true><<<grid, block, 0, st>>>(g, f.r, f.Mi, f.z, f.p, max_iters, m.s64, m.part, m.cnt);
  else
    k_init<false><<<grid, block, 0, st>>>(g, f.r, f.Mi, f.z, f.p, max_iters, m.s64, m.part, m.cnt);
  check_launch("heat solver init");
  launches_ += 2;
  if (max_iters > 0) {
    // z is written before the loop and after it only (k_init, k_flush)
    double *pb = precond ? f.z : m.second(f);
    bool ran;
    if (precond && true_stop)
      ran = m.resident<double, Z_MI, STOP_TRUE>(g, f.Kx, f.Ky, f.p, f.r, f.Mi, f.u, f.z, rx, ry, m.s64, st);
    else if (precond)
      ran = m.resident<double, Z_MI, STOP_TEALEAF>(g, f.Kx, f.Ky, f.p, f.r, f.Mi, f.u, f.z, rx, ry, m.s64, st);
    else
      ran = m.resident<double, Z_R, STOP_TEALEAF>(g, f.Kx, f.Ky, f.p, f.r, f.Mi, f.u, nullptr, rx, ry, m.s64, st);
    if (ran) {
      launches_ += 1;
    } else {
      int rows, blocks;
      pw_grid(f.nx, f.ny, kPwBlocks<double>, &rows, &blocks);
      m.ensure_part(blocks);
      const std::string key = key_of({f.Kx, f.Ky, f.u, f.r, f.w, f.p, pb, f.Mi},
                                     {rx, ry, (double)f.nx, (double)f.ny, (double)f.pitch, precond ? 1.0 : 0.0,
                                      true_stop ? 1.0 : 0.0});
      if (m.chunk64.key != key) {
        if (m.chunk64.exec) cudaGraphExecDestroy(m.chunk64.exec);
        m.chunk64.exec = nullptr;
        m.chunk64.key.clear();
        m.chunk64.exec = capture(st, [&] {
          for (int it = 0; it < kChunk; it++) {
            if (precond)
              k_pw<double, Z_DIAG><<<blocks, block, 0, st>>>(g, f.Kx, f.Ky, f.p, pb, f.r, f.Mi, f.u, f.w, rx, ry, rows,
                                                             m.s64, m.part, m.cnt);
            else
              k_pw<double, Z_R><<<blocks, block, 0, st>>>(g, f.Kx, f.Ky, f.p, pb, f.r, f.Mi, f.u, f.w, rx, ry, rows,
                                                          m.s64, m.part, m.cnt);
            if (precond && true_stop)
              k_r<double, true, STOP_TRUE><<<grid, block, 0, st>>>(g, f.r, f.w, f.Mi, m.s64, m.part, m.cnt);
            else if (precond)
              k_r<double, true, STOP_TEALEAF><<<grid, block, 0, st>>>(g, f.r, f.w, f.Mi, m.s64, m.part, m.cnt);
            else
              k_r<double, false, STOP_TEALEAF><<<grid, block, 0, st>>>(g, f.r, f.w, f.Mi, m.s64, m.part, m.cnt);
          }
        });
        m.chunk64.key = key;
      }
      launches_ += run_chunks(m.chunk64.exec, m.s64, max_iters, m.h_flag, m.ev, st, 2 * kChunk);
      k_flush<double><<<grid, block, 0, st>>>(g, f.u, f.p, pb, f.r, f.Mi, precond ? f.z : nullptr, m.s64);
      check_launch("heat solver flush");
      launches_ += 1;
    }
  }
  OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  const double r0 = sqrt(fabs(h.rr0));
  out->initial_residual = r0;
  out->error = h.err;
  out->converged = h.done == 1 || (max_iters <= 0 && h.err < h.stop);
  // the reference reports n - 1: one less than the iteration that met the test
  out->iterations = h.done == 1 ? h.iters - 1 : h.iters;
  out->outer = 0;
  // true FP64 residual at exit, computed into w (which the next solve
  // overwrites before reading), so r keeps the loop's recursive residual.
  Scalars t = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s32, &t, sizeof(t), cudaMemcpyHostToDevice, st));
  k_resid<<<grid, block, 0, st>>>(g, f.Kx, f.Ky, f.u, f.u0, f.w, rx, ry, 0.0, m.s32, m.part, m.cnt);
  check_launch("heat solver residual");
  launches_ += 1;
  OPSB_CUDA(cudaMemcpyAsync(&t, m.s32, sizeof(t), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  out->true_residual = sqrt(fabs(t.rr));
}

void Solver::pcg_mixed(const Field2D &f, double rx, double ry, bool precond, double eps, double delta,
                       int max_iters, cudaStream_t st, SolveStats *out) {
  validate(f);
  if (!(delta > 0.0 && delta < 1.0)) throw Error(E_ARG, "heat solver: reliable-update delta must be in (0, 1)");
  Impl &m = *m_;
  m.ensure_base();
  m.ensure_f32(f.nx, f.ny, st);
  launches_ = 0;
  const Geom g{f.nx, f.ny, f.pitch}, g32{f.nx, f.ny, m.pitch32};
  const dim3 grid = grid_for(f.nx, f.ny), block(BX, BY);
  // a whole FP32 field: its ring and row ends hold zeros
  const long long o32 = m.pitch32 + 32, n32 = m.pitch32 * (f.ny + 2);
  const int gridr = (int)std::min<long long>((n32 / 4 + NT - 1) / NT, 148 * kFlatBlocks);
  const float rxf = (float)rx, ryf = (float)ry;
  k_to_float<<<grid_for(f.nx + 2, f.ny + 2), block, 0, st>>>(g, g32, f.Kx, f.Ky, precond ? f.Mi : nullptr, m.Kx,
                                                              m.Ky, m.Mi);
  Scalars h = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s64, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  k_resid<<<grid, block, 0, st>>>(g, f.Kx, f.Ky, f.u, f.u0, f.r, rx, ry, eps, m.s64, m.part, m.cnt);
  check_launch("heat solver init");
  launches_ += 2;
  OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  const double r0 = sqrt(fabs(h.rr0));
  out->initial_residual = r0;
  int rows, blocks;
  pw_grid(f.nx, f.ny, kPwBlocks<float>, &rows, &blocks);
  m.ensure_part(blocks);
  const std::string key = key_of({m.Kx, m.Ky, m.e, m.r, m.w, m.p, m.p2, m.Mi},
                                 {(double)rxf, (double)ryf, (double)f.nx, (double)f.ny, (double)m.pitch32,
                                  precond ? 1.0 : 0.0});
  auto capture_chunk = [&] {
    if (m.chunk32.key == key) return;
    if (m.chunk32.exec) cudaGraphExecDestroy(m.chunk32.exec);
    m.chunk32.exec = nullptr;
    m.chunk32.key.clear();
    m.chunk32.exec = capture(st, [&] {
      for (int it = 0; it < kChunk; it++) {
        if (precond) {
          k_pw<float, Z_MI><<<blocks, block, 0, st>>>(g32, m.Kx, m.Ky, m.p, m.p2, m.r, m.Mi, m.e, m.w, rxf, ryf, rows,
                                                      m.s32, m.part, m.cnt);
          k_r_flat<float, STOP_RELIABLE><<<gridr, block, 0, st>>>(m.r - o32, m.w - o32, m.Mi - o32, n32, m.s32, m.part,
                                                                  m.cnt);
        } else {
          k_pw<float, Z_R><<<blocks, block, 0, st>>>(g32, m.Kx, m.Ky, m.p, m.p2, m.r, m.Mi, m.e, m.w, rxf, ryf, rows,
                                                     m.s32, m.part, m.cnt);
          k_r<float, false, STOP_RELIABLE><<<grid, block, 0, st>>>(g32, m.r, m.w, m.Mi, m.s32, m.part, m.cnt);
        }
      }
    });
    m.chunk32.key = key;
  };
  int updates = 0, iters = 0;
  double scale = 1.0;
  bool done = h.done == 1 || r0 == 0.0;
  Scalars in;
  memset(&in, 0, sizeof(in));
  while (!done) {
    if (precond)
      k_reinit32<true><<<grid, block, 0, st>>>(g, g32, f.r, m.r, m.Mi, updates == 0, eps, scale, delta, max_iters,
                                               m.s32, m.part, m.cnt);
    else
      k_reinit32<false><<<grid, block, 0, st>>>(g, g32, f.r, m.r, m.Mi, updates == 0, eps, scale, delta, max_iters,
                                                m.s32, m.part, m.cnt);
    check_launch("heat solver reliable update");
    launches_ += 1;
    const bool ran =
        max_iters > 0 &&
        (precond ? m.resident<float, Z_MI, STOP_RELIABLE>(g32, m.Kx, m.Ky, m.p, m.r, m.Mi, m.e, nullptr, rxf, ryf, m.s32,
                                                          st)
                 : m.resident<float, Z_R, STOP_RELIABLE>(g32, m.Kx, m.Ky, m.p, m.r, m.Mi, m.e, nullptr, rxf, ryf, m.s32,
                                                         st));
    if (ran) {
      launches_ += 1;
    } else {
      capture_chunk();
      launches_ += run_chunks(m.chunk32.exec, m.s32, max_iters, m.h_flag, m.ev, st, 2 * kChunk);
    }
    OPSB_CUDA(cudaMemcpyAsync(&in, m.s32, sizeof(in), cudaMemcpyDeviceToHost, st));
    k_update<<<grid, block, 0, st>>>(g, g32, f.u, m.e, m.p, m.p2, m.s32);
    k_resid<<<grid, block, 0, st>>>(g, f.Kx, f.Ky, f.u, f.u0, f.r, rx, ry, eps, m.s64, m.part, m.cnt);
    check_launch("heat solver reliable update");
    launches_ += 2;
    OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
    OPSB_CUDA(cudaStreamSynchronize(st));
    updates++;
    iters = in.iters;
    done = h.done == 1;
    if (done || in.done == 2 || in.iters >= max_iters || updates > 10000) break;
    // the estimate said converged but the FP64 residual disagrees: tighten it
    if (in.done == 1) scale *= 0.1;
  }
  out->iterations = iters;
  out->outer = updates;
  out->converged = done;
  out->error = h.err;
  out->true_residual = h.err;
}


namespace {
void validate3(const Field3D &f) {
  if (f.nx < 1 || f.ny < 1 || f.nz < 1) throw Error(E_ARG, "heat solver 3D: empty interior");
  if (f.pitch < f.nx + 2 || f.plane != f.pitch * (f.ny + 2))
    throw Error(E_ARG, "heat solver 3D: pitch >= nx + 2 and plane == pitch * (ny + 2) required");
  if (!f.Kx || !f.Ky || !f.Kz || !f.u0 || !f.u || !f.r || !f.w || !f.p || !f.z || !f.Mi)
    throw Error(E_ARG, "heat solver 3D: null field");
  if ((long long)(f.ny + 2) * (f.nz + 2) > (1LL << 30) || f.plane * (f.nz + 2) > (1LL << 40))
    throw Error(E_ARG, "heat solver 3D: field too large");
}
}  // namespace

void Solver::diag3(const Field3D &f, double rx, double ry, double rz, cudaStream_t st) {
  validate3(f);
  k_diag3<<<grid_for3(f.nx, f.ny * f.nz), dim3(BX, BY), 0, st>>>(Geom3{f.nx, f.ny, f.nz, f.pitch, f.plane}, f.Kx,
                                                                   f.Ky, f.Kz, rx, ry, rz, f.Mi);
  check_launch("heat solver 3D diagonal");
}

void Solver::pcg3d(const Field3D &f, double rx, double ry, double rz, bool true_stop, double eps, int max_iters,
                   cudaStream_t st, SolveStats *out) {
  validate3(f);
  Impl &m = *m_;
  m.ensure_base();
  launches_ = 0;
  const Geom3 g{f.nx, f.ny, f.nz, f.pitch, f.plane};
  const dim3 grid3 = grid_for3(f.nx, f.ny * f.nz), block(BX, BY);
  // the pointwise kernels see the padded volume as rows of `pitch`
  const long long off = f.plane + f.pitch + 1;
  const int rows = (f.ny + 2) * (f.nz + 2);
  const Geom gf{(int)f.pitch, rows, f.pitch};
  const dim3 gridf = grid_for((int)f.pitch, rows);
  double *r = f.r - off, *w = f.w - off, *p = f.p - off, *z = f.z - off;
  const double *Mi = f.Mi - off;
  const long long nf = f.plane * (f.nz + 2);
  if (((uintptr_t)r | (uintptr_t)w | (uintptr_t)Mi) & 15) throw Error(E_ARG, "heat solver 3D: misaligned field");
  const Grid3 q = pw3_grid(f.nx, f.ny, f.nz);
  m.ensure_part(q.blocks);
  const int gridr = (int)std::min<long long>((nf / 2 + NT - 1) / NT, 148 * kFlatBlocks);
  Scalars h = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s64, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  k_resid3<<<grid3, block, 0, st>>>(g, f.Kx, f.Ky, f.Kz, f.u, f.u0, f.r, rx, ry, rz, eps, m.s64, m.part, m.cnt);
  k_init<true><<<gridf, block, 0, st>>>(gf, r, Mi, z, p, max_iters, m.s64, m.part, m.cnt);
  check_launch("heat solver 3D init");
  launches_ += 2;
  if (max_iters > 0) {
    const std::string key = "3d" + key_of({f.Kx, f.Ky, f.Kz, f.u, f.r, f.w, f.p, f.z, f.Mi},
                                          {rx, ry, rz, (double)f.nx, (double)f.ny, (double)f.nz, (double)f.pitch,
                                           true_stop ? 1.0 : 0.0});
    if (m.chunk64.key != key) {
      if (m.chunk64.exec) cudaGraphExecDestroy(m.chunk64.exec);
      m.chunk64.exec = nullptr;
      m.chunk64.key.clear();
      m.chunk64.exec = capture(st, [&] {
        for (int it = 0; it < kChunk; it++) {
          // f.z is the direction's second buffer
          k_pw3<double><<<q.blocks, dim3(32, kTileY), 0, st>>>(g, f.Kx, f.Ky, f.Kz, f.p, f.z, f.r, f.Mi, f.u, f.w, rx,
                                                               ry, rz, q.tx, q.ty, q.planes, m.s64, m.part, m.cnt);
          if (true_stop)
            k_r_flat<double, STOP_TRUE><<<gridr, block, 0, st>>>(r, w, Mi, nf, m.s64, m.part, m.cnt);
          else
            k_r_flat<double, STOP_TEALEAF><<<gridr, block, 0, st>>>(r, w, Mi, nf, m.s64, m.part, m.cnt);
        }
      });
      m.chunk64.key = key;
    }
    launches_ += run_chunks(m.chunk64.exec, m.s64, max_iters, m.h_flag, m.ev, st, 2 * kChunk);
    k_flush<double><<<gridf, block, 0, st>>>(gf, f.u - off, p, z, r, Mi, nullptr, m.s64);
    check_launch("heat solver 3D flush");
    launches_ += 1;
  }
  OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  out->initial_residual = sqrt(fabs(h.rr0));
  out->error = h.err;
  out->converged = h.done == 1 || (max_iters <= 0 && h.err < h.stop);
  out->iterations = h.done == 1 ? h.iters - 1 : h.iters;
  out->outer = 0;
  Scalars t = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s32, &t, sizeof(t), cudaMemcpyHostToDevice, st));
  k_resid3<<<grid3, block, 0, st>>>(g, f.Kx, f.Ky, f.Kz, f.u, f.u0, f.w, rx, ry, rz, 0.0, m.s32, m.part, m.cnt);
  check_launch("heat solver 3D residual");
  launches_ += 1;
  OPSB_CUDA(cudaMemcpyAsync(&t, m.s32, sizeof(t), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  out->true_residual = sqrt(fabs(t.rr));
}

void Solver::pcg3d_mixed(const Field3D &f, double rx, double ry, double rz, double eps, double delta, int max_iters,
                         cudaStream_t st, SolveStats *out) {
  validate3(f);
  if (!(delta > 0.0 && delta < 1.0)) throw Error(E_ARG, "heat solver: reliable-update delta must be in (0, 1)");
  Impl &m = *m_;
  m.ensure_base();
  const long long off = f.plane + f.pitch + 1;
  const size_t nf = (size_t)f.plane * (f.nz + 2);
  m.ensure_f32_flat(nf, st);
  launches_ = 0;
  const Geom3 g{f.nx, f.ny, f.nz, f.pitch, f.plane};
  const dim3 grid3 = grid_for3(f.nx, f.ny * f.nz), block(BX, BY);
  const int rows = (f.ny + 2) * (f.nz + 2);
  const Geom gf{(int)f.pitch, rows, f.pitch};
  const dim3 gridf = grid_for((int)f.pitch, rows);
  const dim3 grid1((unsigned)std::min<long long>(((long long)nf + NT - 1) / NT, 148LL * 16));
  const Grid3 q = pw3_grid(f.nx, f.ny, f.nz);
  m.ensure_part(q.blocks);
  const int gridr = (int)std::min<long long>(((long long)nf / 4 + NT - 1) / NT + 1, 148 * kFlatBlocks);
  const float rxf = (float)rx, ryf = (float)ry, rzf = (float)rz;
  k_flat_to_float<<<grid1, block, 0, st>>>(f.Kx - off, m.Kx, (long long)nf);
  k_flat_to_float<<<grid1, block, 0, st>>>(f.Ky - off, m.Ky, (long long)nf);
  k_flat_to_float<<<grid1, block, 0, st>>>(f.Kz - off, m.Kz, (long long)nf);
  k_flat_to_float<<<grid1, block, 0, st>>>(f.Mi - off, m.Mi, (long long)nf);
  Scalars h = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s64, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  k_resid3<<<grid3, block, 0, st>>>(g, f.Kx, f.Ky, f.Kz, f.u, f.u0, f.r, rx, ry, rz, eps, m.s64, m.part, m.cnt);
  check_launch("heat solver 3D init");
  launches_ += 5;
  OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  const double r0 = sqrt(fabs(h.rr0));
  out->initial_residual = r0;
  const std::string key = "3d" + key_of({m.Kx, m.Ky, m.Kz, m.e, m.r, m.w, m.p, m.p2, m.Mi},
                                        {(double)rxf, (double)ryf, (double)rzf, (double)f.nx, (double)f.ny,
                                         (double)f.nz, (double)f.pitch});
  if (m.chunk32.key != key) {
    if (m.chunk32.exec) cudaGraphExecDestroy(m.chunk32.exec);
    m.chunk32.exec = nullptr;
    m.chunk32.key.clear();
    m.chunk32.exec = capture(st, [&] {
      for (int it = 0; it < kChunk; it++) {
        k_pw3<float><<<q.blocks, dim3(32, kTileY), 0, st>>>(g, m.Kx + off, m.Ky + off, m.Kz + off, m.p + off,
                                                            m.p2 + off, m.r + off, m.Mi + off, m.e + off, m.w + off,
                                                            rxf, ryf, rzf, q.tx, q.ty, q.planes, m.s32, m.part, m.cnt);
        k_r_flat<float, STOP_RELIABLE><<<gridr, block, 0, st>>>(m.r, m.w, m.Mi, (long long)nf, m.s32, m.part, m.cnt);
      }
    });
    m.chunk32.key = key;
  }
  int updates = 0, iters = 0;
  double scale = 1.0;
  bool done = h.done == 1 || r0 == 0.0;
  Scalars in;
  memset(&in, 0, sizeof(in));
  while (!done) {
    k_reinit32<true><<<gridf, block, 0, st>>>(gf, gf, f.r - off, m.r, m.Mi, updates == 0, eps, scale, delta,
                                              max_iters, m.s32, m.part, m.cnt);
    check_launch("heat solver 3D reliable update");
    launches_ += 1;
    launches_ += run_chunks(m.chunk32.exec, m.s32, max_iters, m.h_flag, m.ev, st, 2 * kChunk);
    OPSB_CUDA(cudaMemcpyAsync(&in, m.s32, sizeof(in), cudaMemcpyDeviceToHost, st));
    k_update<<<gridf, block, 0, st>>>(gf, gf, f.u - off, m.e, m.p, m.p2, m.s32);
    k_resid3<<<grid3, block, 0, st>>>(g, f.Kx, f.Ky, f.Kz, f.u, f.u0, f.r, rx, ry, rz, eps, m.s64, m.part, m.cnt);
    check_launch("heat solver 3D reliable update");
    launches_ += 2;
    OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
    OPSB_CUDA(cudaStreamSynchronize(st));
    updates++;
    iters = in.iters;
    done = h.done == 1;
    if (done || in.done == 2 || in.iters >= max_iters || updates > 10000) break;
    if (in.done == 1) scale *= 0.1;  // the estimate said converged, the FP64 residual disagrees
  }
  out->iterations = iters;
  out->outer = updates;
  out->converged = done;
  out->error = h.err;
  out->true_residual = h.err;
}

void Solver::diag(const Field2D &f, double rx, double ry, cudaStream_t st) {
  validate(f);
  k_diag<<<grid_for(f.nx, f.ny), dim3(BX, BY), 0, st>>>(Geom{f.nx, f.ny, f.pitch}, f.Kx, f.Ky, rx, ry, f.Mi);
  check_launch("heat solver diagonal");
}

double Solver::residual(const Field2D &f, double rx, double ry, double *outp, cudaStream_t st) {
  validate(f);
  Impl &m = *m_;
  m.ensure_base();
  Scalars t = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s32, &t, sizeof(t), cudaMemcpyHostToDevice, st));
  k_resid<<<grid_for(f.nx, f.ny), dim3(BX, BY), 0, st>>>(Geom{f.nx, f.ny, f.pitch}, f.Kx, f.Ky, f.u, f.u0, outp, rx,
                                                         ry, 0.0, m.s32, m.part, m.cnt);
  check_launch("heat residual");
  OPSB_CUDA(cudaMemcpyAsync(&t, m.s32, sizeof(t), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  return sqrt(fabs(t.rr));
}

void Solver::fcg(const Field2D &f, double rx, double ry, double eps, int max_iters, const Precond &M, int window,
                 cudaStream_t st, SolveStats *out, const Precond *fallback, bool chunked) {
  validate(f);
  Impl &m = *m_;
  m.ensure_base();
  launches_ = 0;
  const Geom g{f.nx, f.ny, f.pitch};
  const dim3 grid = grid_for(f.nx, f.ny), block(BX, BY);
  Scalars h = fresh(0.0);
  h.max_iters = max_iters;
  h.restart = 1;
  OPSB_CUDA(cudaMemcpyAsync(m.s64, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  k_resid<<<grid, block, 0, st>>>(g, f.Kx, f.Ky, f.u, f.u0, f.r, rx, ry, eps, m.s64, m.part, m.cnt);
  check_launch("fcg init");
  launches_ += 1;
  bool learned = static_cast<bool>(M);
  auto precond = [&] {
    if (learned) {
      launches_ += M(f.r, f.z, st);
    } else if (fallback && *fallback) {
      launches_ += (*fallback)(f.r, f.z, st);
    } else {
      k_jacobi<<<grid, block, 0, st>>>(g, f.Mi, f.r, f.z);
      launches_ += 1;
    }
  };
  OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  const double r0 = sqrt(fabs(h.rr0));
  out->initial_residual = r0;
  out->fallbacks = 0;
  bool done = h.done == 1 || r0 == 0.0;
  double *pb = nullptr;
  if (!done) {
    // the initial residual kernel leaves done = 0 and iters = 0
    pb = m.second(f);
    precond();
  }
  int rows = 1, blocks = 1;
  pw_grid(f.nx, f.ny, kPwBlocks<double>, &rows, &blocks);
  m.ensure_part(blocks);
  auto step = [&] {
    k_pw<double, Z_FCG><<<blocks, block, 0, st>>>(g, f.Kx, f.Ky, f.p, pb, f.z, f.r, f.u, f.w, rx, ry, rows, m.s64,
                                                  m.part, m.cnt);
    k_fr<<<grid, block, 0, st>>>(g, f.r, f.w, m.s64, m.part, m.cnt);
    launches_ += 2;
  };
  auto beta = [&] {
    k_fzw<<<grid, block, 0, st>>>(g, f.z, f.w, m.s64, m.part, m.cnt);
    launches_ += 1;
  };
  auto flush = [&] {  // the pending u += alpha p
    k_flush<double><<<grid, block, 0, st>>>(g, f.u, f.p, pb, f.r, f.Mi, nullptr, m.s64);
    launches_ += 1;
  };
  // after a stop with done 4 or 5: u up to date, and the next direction z
  auto restart_from = [&] {
    flush();
    const int set[3] = {0, 0, 1};  // done; pend, restart
    OPSB_CUDA(cudaMemcpyAsync(&m.s64->done, set, sizeof(int), cudaMemcpyHostToDevice, st));
    OPSB_CUDA(cudaMemcpyAsync(&m.s64->pend, set + 1, 2 * sizeof(int), cudaMemcpyHostToDevice, st));
    precond();
  };
  bool host_loop = true;
  if (chunked && window < 64 && !done) {
    host_loop = false;
    // Replayed chunks of kFcgChunk iterations (w = A p, update, precondition,
    // beta, direction); the device stops them (done != 0) and the host reads
    // the flag one chunk behind. A restart (done 4 or 5) falls back to the
    // Jacobi (or fallback) preconditioner and continues with that chunk.
    // The graphs hold this call's pointers and are rebuilt per call.
    constexpr int kFcgChunk = 4;
    int set[2] = {learned ? window : 0, 0};
    OPSB_CUDA(cudaMemcpyAsync(&m.s64->window, set, sizeof(set), cudaMemcpyHostToDevice, st));
    cudaGraphExec_t graphs[2] = {nullptr, nullptr};  // learned, fallback
    long long per_chunk[2] = {0, 0};
    try {
      while (!done) {
        const int which = learned ? 0 : 1;
        if (!graphs[which]) {
          const long long before = launches_;
          graphs[which] = capture(st, [&] {
            for (int it = 0; it < kFcgChunk; it++) {
              step();
              precond();
              beta();
            }
          });
          per_chunk[which] = launches_ - before;
          launches_ = before;
        }
        // run_chunks stops after (its bound) / kChunk + 2 chunks at most; the
        // device stops them first (done 2 at max_iters)
        launches_ += run_chunks(graphs[which], m.s64, (max_iters / kFcgChunk + 2) * kChunk, m.h_flag, m.ev, st,
                                per_chunk[which]);
        OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
        OPSB_CUDA(cudaStreamSynchronize(st));
        if (h.done == 1 || h.done == 2 || h.done == 0) break;
        // done 4 (lost curvature) or 5 (not halved over the window): restart
        if (learned) out->fallbacks++;
        learned = false;
        const int zero2[2] = {0, 0};  // window = hcount = 0 (no restart test on the fallback)
        OPSB_CUDA(cudaMemcpyAsync(&m.s64->window, zero2, 2 * sizeof(int), cudaMemcpyHostToDevice, st));
        restart_from();
      }
    } catch (...) {
      for (cudaGraphExec_t x : graphs)
        if (x) cudaGraphExecDestroy(x);
      throw;
    }
    for (cudaGraphExec_t x : graphs)
      if (x) cudaGraphExecDestroy(x);
  }
  std::vector<double> hist;
  while (!done && host_loop) {
    step();
    check_launch("fcg iteration");
    OPSB_CUDA(cudaMemcpyAsync(&h, m.s64, sizeof(h), cudaMemcpyDeviceToHost, st));
    OPSB_CUDA(cudaStreamSynchronize(st));
    if (h.done == 1 || h.done == 2) break;
    bool restart = false;
    if (h.done == 4) {
      restart = true;  // lost positive curvature: fall back to Jacobi and restart the recursion
    } else {
      hist.push_back(h.err);
      const size_t k = hist.size();
      if (learned && window > 0 && k > (size_t)window && hist[k - 1] > 0.5 * hist[k - 1 - window]) restart = true;
    }
    if (restart) {
      if (learned) out->fallbacks++;
      learned = false;
      hist.clear();
      restart_from();
      continue;
    }
    precond();
    beta();
    check_launch("fcg direction");
  }
  if (!done) flush();
  out->iterations = h.iters;
  out->converged = h.done == 1 || done;
  out->error = h.err;
  out->outer = 0;
  // true FP64 residual at exit (into w)
  Scalars t = fresh(0.0);
  OPSB_CUDA(cudaMemcpyAsync(m.s32, &t, sizeof(t), cudaMemcpyHostToDevice, st));
  k_resid<<<grid, block, 0, st>>>(g, f.Kx, f.Ky, f.u, f.u0, f.w, rx, ry, 0.0, m.s32, m.part, m.cnt);
  check_launch("fcg residual");
  launches_ += 1;
  OPSB_CUDA(cudaMemcpyAsync(&t, m.s32, sizeof(t), cudaMemcpyDeviceToHost, st));
  OPSB_CUDA(cudaStreamSynchronize(st));
  out->true_residual = sqrt(fabs(t.rr));
}

}  // namespace heat
}  // namespace opsb
