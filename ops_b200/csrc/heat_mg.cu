// Aggregation multigrid V-cycle for the TeaLeaf 2D heat operator; the
// hierarchy and the cycle are described in heat_mg.h.
//
// Storage: every level keeps its FP32 arrays without a halo ring, rows of
// `pitch` elements (a multiple of 32, at least nx + 1 so that a row holds all
// nx + 1 x-faces); the y-face array has ny + 1 rows. Face x of a row is the
// face between cells x - 1 and x, so cell x reads faces x and x + 1 of its
// row and y-faces from its own row and the next. Neighbours outside the
// domain hold zero, so their terms are dropped while their face weights stay
// in the diagonal (as the halo of the FP64 operator does).
//
// A level above the coarsest costs two passes: k_cycle on the way down (both
// pre-sweeps, the residual and its restriction) and k_cycle on the way up
// (the correction and both post-sweeps). On level 0 that is 21 and 29 bytes a
// cell; the coarser levels add a third.
#include <algorithm>
#include <cstdint>
#include <string>

#include "heat_mg.h"
#include "march_grid.h"
#include "runtime.h"

namespace opsb {
namespace heat {

namespace {

constexpr int BX = 128, BY = 2;
constexpr int kCoarseThreads = Multigrid::kCoarsest * Multigrid::kCoarsest;

struct LV {
  int nx, ny;
  long long P;
  const float *m, *ax, *ay;
};

void check(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw Error(E_CUDA, std::string("multigrid ") + what + ": " + cudaGetErrorString(e));
}

dim3 grid_of(int nx, int ny) {
  const int gx = (nx + BX - 1) / BX;
  const int gy = std::min((ny + BY - 1) / BY, 32768);
  return dim3(gx, gy);
}

#define MG_CELLS(L)                                                                   \
  for (int y = blockIdx.y * BY + threadIdx.y; y < (L).ny; y += gridDim.y * BY)        \
    for (int x = blockIdx.x * BX + threadIdx.x; x < (L).nx; x += gridDim.x * BX)

// Diagonal of cell i: its mass plus its four face weights.
template <bool UNIT>
__device__ __forceinline__ float diag(const LV &L, long long i, float aw, float ae, float as, float an) {
  return (UNIT ? 1.0f : L.m[i]) + aw + ae + as + an;
}

// omega / c: the reciprocal approximation (1 ulp) with one Newton step (1/c =
// q + q (1 - c q)), whose error is that of a rounded reciprocal; a division
// and its range checks, two per cell and pass, were half of a pass's
// instructions.
__device__ __forceinline__ float over(float omega, float c) {
  float q;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(c));
  return omega * fmaf(q, fmaf(-c, q, 1.0f), q);
}

constexpr int kCycleWarps = 4;
constexpr int cycle_blocks(bool up) { return up ? 4 : 5; }

// One level on the way down (UP false):
//    z0 = omega r / c;  z = z0 + omega (r - A z0) / c, kept in `zmid`;
//    rc = the sum of r - A z over each aggregate (rows, then columns)
// or up: z0 = zmid + P e (each cell its aggregate's value of e), then two
// damped-Jacobi sweeps on it, the second one written out. On level 0 (R64,
// OUT64) r is read from and z written to the FP64 fields (pitch `fp`; `vec`
// says that their pairs of columns are 16-byte aligned).
// Each of the sweeps used to be a pass of its own, 106 bytes a fine cell and
// cycle. Here a warp marches up a strip of `rows` rows: a lane owns an
// aggregate's two columns (30 lanes' own, one beside on each side), rows y of
// z0, y - 1 of the first sweep and y - 2 of the second stage are in registers
// at a time, neighbours beside come by shuffles, and a row is loaded two rows
// or three ahead. Bound by memory on the fine levels (4096^2: 76 us down and
// 89 up, 4.5 and 5.4 TB/s, where the five passes took 419), by latency on the
// coarse ones (5 to 6 us a pass, launch included, below 512^2). A CTA of four
// warps, five an SM down and four up, is what holds a pass in its registers
// (with 80 registers a pass up spilled and took 134 us).
template <bool UP, bool UNIT, bool R64, bool OUT64>
__global__ void __launch_bounds__(32 * kCycleWarps, cycle_blocks(UP))
    k_cycle(LV L, const double *__restrict__ r64, long long fp, int vec, const float *__restrict__ r32, float *zmid,
            const float *__restrict__ e, long long cP, float *__restrict__ out, double *__restrict__ z64, float omega,
            int rows) {
  const int lane = threadIdx.x & 31, wi = blockIdx.x * kCycleWarps + (threadIdx.x >> 5);
  const int ncol = ((L.nx + 1) / 2 + 29) / 30, nst = (L.ny + rows - 1) / rows;
  if (wi >= ncol * nst) return;
  const int I = (wi % ncol) * 30 + lane - 1, x = 2 * I, y0 = (wi / ncol) * rows, y1 = min(y0 + rows, L.ny);
  const bool in0 = I >= 0 && x < L.nx, in1 = I >= 0 && x + 1 < L.nx, own = in0 && lane >= 1 && lane <= 30;
  const long long P = L.P;
  struct Row {
    double2 r64;
    float2 r, a, n, m, z;
    float ae, e;
  };
  // a pair's second column may be the row's padding: it is masked below
  auto pair = [](const float *q) { return *reinterpret_cast<const float2 *>(q); };
  auto load = [&](int y) {
    Row v{};
    const long long i = (long long)y * P + x;
    if (in0 && y >= -1 && y < L.ny) v.n = pair(L.ay + i + P);
    if (I >= 0 && x <= L.nx && y >= 0 && y < L.ny) {
      v.a = pair(L.ax + i);
      if (lane == 31 && x + 2 <= L.nx) v.ae = L.ax[i + 2];  // the other lanes' comes from their neighbour
      if (in0) {
        if (R64) {
          const double *q = r64 + (long long)y * fp + x;
          if (vec && in1) {
            v.r64 = *reinterpret_cast<const double2 *>(q);
          } else {
            v.r64.x = q[0];
            if (in1) v.r64.y = q[1];
          }
        } else {
          v.r = pair(r32 + i);
        }
        if (!UNIT) v.m = pair(L.m + i);
        if (UP) {
          v.z = pair(zmid + i);
          v.e = e[(long long)(y >> 1) * cP + I];
        }
      }
    }
    return v;
  };
  struct Cells {
    float2 r, c, q, a, s, n;  // r, diagonal, omega / diagonal, x-faces, y-faces below and above
    float ae;
  };
  // r - A z on a row's two columns: centre zc, rows below and above zs, zn
  auto resid = [&](const Cells &q, float2 zc, float2 zs, float2 zn) {
    const float l = __shfl_up_sync(0xffffffffu, zc.y, 1), r = __shfl_down_sync(0xffffffffu, zc.x, 1);
    float2 t;
    t.x = q.r.x - q.c.x * zc.x;
    t.x += q.a.x * l;
    t.x += q.a.y * zc.y;
    t.x += q.s.x * zs.x;
    t.x += q.n.x * zn.x;
    t.y = q.r.y - q.c.y * zc.y;
    t.y += q.a.y * zc.x;
    t.y += q.ae * r;
    t.y += q.s.y * zs.y;
    t.y += q.n.y * zn.y;
    return t;
  };
  float acc = 0.f;
  // Row y: z0 there, the first sweep on row y - 1 (cells A; z0 of y - 2, y - 1
  // in za, zb) and the second stage on row y - 2 (cells B; the first sweep's of
  // y - 3, y - 2 in va, vb), the upper row of an aggregate if ODD.
  auto step = [&](int y, const Row &cur, float2 south, const Cells &A, const Cells &B, float2 za, float2 zb, float2 va,
                  float2 vb, bool odd, Cells &C, float2 &z, float2 &v) {
    const float ae = __shfl_down_sync(0xffffffffu, cur.a.x, 1);
    C.r = R64 ? make_float2((float)cur.r64.x, (float)cur.r64.y) : cur.r;
    C.a = cur.a;
    C.ae = lane == 31 ? cur.ae : ae;
    C.s = south;
    C.n = cur.n;
    C.c.x = (UNIT ? 1.0f : cur.m.x) + C.a.x + C.a.y + C.s.x + C.n.x;
    C.c.y = (UNIT ? 1.0f : cur.m.y) + C.a.y + C.ae + C.s.y + C.n.y;
    // outside the level q is 0 (and so is all of r, faces and z): z stays 0 there
    const bool in = y >= 0 && y < L.ny;
    C.q.x = in && in0 ? over(omega, C.c.x) : 0.f;
    C.q.y = in && in1 ? over(omega, C.c.y) : 0.f;
    if (UP) {
      z.x = in && in0 ? cur.z.x + cur.e : 0.f;
      z.y = in && in1 ? cur.z.y + cur.e : 0.f;
    } else {
      z.x = C.r.x * C.q.x;
      z.y = C.r.y * C.q.y;
    }
    float2 t = resid(A, zb, za, z);
    v.x = zb.x + A.q.x * t.x;
    v.y = zb.y + A.q.y * t.y;
    if (!UP && own && y - 1 >= y0 && y - 1 < y1) {
      float *q = zmid + (long long)(y - 1) * P + x;
      if (in1) *reinterpret_cast<float2 *>(q) = v;
      else *q = v.x;
    }
    t = resid(B, vb, va, v);
    const int yo = y - 2;
    if (own && yo >= y0 && yo < y1) {
      if (UP) {
        const float2 o = make_float2(vb.x + B.q.x * t.x, vb.y + B.q.y * t.y);
        if (OUT64) {
          double *q = z64 + (long long)yo * fp + x;
          if (vec && in1) {
            *reinterpret_cast<double2 *>(q) = make_double2((double)o.x, (double)o.y);
          } else {
            q[0] = (double)o.x;
            if (in1) q[1] = (double)o.y;
          }
        } else {
          float *q = out + (long long)yo * P + x;
          if (in1) *reinterpret_cast<float2 *>(q) = o;
          else *q = o.x;
        }
      } else {
        acc = odd ? acc + t.x : t.x;
        if (in1) acc += t.y;
        if (odd || yo == L.ny - 1) out[(long long)(yo >> 1) * cP + I] = acc;
      }
    }
  };
  float2 s{};  // the faces below the current row
  if (in0 && y0 >= 2) s = pair(L.ay + (long long)(y0 - 2) * P + x);
  Row c0 = load(y0 - 2), c1 = load(y0 - 1);
  Cells A{}, B{};
  float2 za{}, zb{}, va{}, vb{};
  for (int y = y0 - 2; y < y1 + 2; y += 2) {
    const Row n0 = load(min(y + 2, y1 + 1)), n1 = load(min(y + 3, y1 + 1));
    Cells C, D;
    float2 z0, z1, v0, v1;
    step(y, c0, s, A, B, za, zb, va, vb, false, C, z0, v0);
    step(y + 1, c1, C.n, C, A, zb, z0, vb, v0, true, D, z1, v1);
    s = D.n;
    za = z0;
    zb = z1;
    va = v0;
    vb = v1;
    B = C;
    A = D;
    c0 = n0;
    c1 = n1;
  }
}

// The FP32 copy of r for a cycle whose z overlaps it.
__global__ void __launch_bounds__(BX *BY) k_copy_r(LV L, const double *__restrict__ r64, long long fp,
                                                   float *__restrict__ r32) {
  MG_CELLS(L) r32[(long long)y * L.P + x] = (float)r64[(long long)y * fp + x];
}

// The coarsest level (at most kCoarsest x kCoarsest cells, one per thread of
// one CTA): `sweeps` damped-Jacobi sweeps from z = 0 in shared memory. With
// IO64 the level is level 0: r is read from and z written to the FP64 fields.
template <bool UNIT, bool IO64>
__global__ void __launch_bounds__(kCoarseThreads) k_coarsest(LV L, const float *__restrict__ r32,
                                                             const double *__restrict__ r64, long long fp,
                                                             float *__restrict__ zout, double *__restrict__ z64,
                                                             int sweeps, float omega) {
  __shared__ float zs[2][kCoarseThreads];
  const int t = threadIdx.x, n = L.nx * L.ny;
  const bool on = t < n;
  const int x = on ? t % L.nx : 0, y = on ? t / L.nx : 0;
  const long long i = (long long)y * L.P + x;
  float aw = 0.f, ae = 0.f, as = 0.f, an = 0.f, c = 1.f, rv = 0.f;
  if (on) {
    aw = L.ax[i];
    ae = L.ax[i + 1];
    as = L.ay[i];
    an = L.ay[i + L.P];
    c = diag<UNIT>(L, i, aw, ae, as, an);
    rv = IO64 ? (float)r64[(long long)y * fp + x] : r32[i];
  }
  const float q = over(omega, c);
  float v = on ? q * rv : 0.f;
  zs[0][t] = v;
  __syncthreads();
  int cur = 0;
  for (int k = 1; k < sweeps; k++) {
    if (on) {
      const float *zc = zs[cur];
      float s = rv - c * zc[t];
      if (x > 0) s += aw * zc[t - 1];
      if (x < L.nx - 1) s += ae * zc[t + 1];
      if (y > 0) s += as * zc[t - L.nx];
      if (y < L.ny - 1) s += an * zc[t + L.nx];
      v = zc[t] + q * s;
    }
    zs[cur ^ 1][t] = v;
    __syncthreads();
    cur ^= 1;
  }
  if (on) {
    if (IO64) z64[(long long)y * fp + x] = (double)v;
    else zout[i] = v;
  }
}

// Level-0 face weights: ax(x, y) = rx Kx[y fp + x] for x in [0, nx],
// ay(x, y) = ry Ky[y fp + x] for y in [0, ny], rounded to FP32.
__global__ void k_fine_faces(int nx, int ny, long long fp, const double *__restrict__ Kx,
                             const double *__restrict__ Ky, double rx, double ry, long long P, float *__restrict__ ax,
                             float *__restrict__ ay) {
  for (int y = blockIdx.y * BY + threadIdx.y; y <= ny; y += gridDim.y * BY)
    for (int x = blockIdx.x * BX + threadIdx.x; x <= nx; x += gridDim.x * BX) {
      const long long s = (long long)y * fp + x, d = (long long)y * P + x;
      if (y < ny) ax[d] = (float)(rx * Kx[s]);
      if (x < nx) ay[d] = (float)(ry * Ky[s]);
    }
}

// Coarse level from fine level F: mass sums, and coarse face I of a row takes
// fine face min(2 I, nx_f) of the aggregate's rows (likewise in y), summed and
// scaled by `fs`.
__global__ void k_coarsen(LV F, int cnx, int cny, long long cP, float *__restrict__ m, float *__restrict__ ax,
                          float *__restrict__ ay, float fs) {
  for (int J = blockIdx.y * BY + threadIdx.y; J <= cny; J += gridDim.y * BY)
    for (int I = blockIdx.x * BX + threadIdx.x; I <= cnx; I += gridDim.x * BX) {
      const long long d = (long long)J * cP + I;
      if (I < cnx && J < cny) {
        float s = 0.f;
        for (int y = 2 * J; y < min(2 * J + 2, F.ny); y++)
          for (int x = 2 * I; x < min(2 * I + 2, F.nx); x++) s += F.m ? F.m[(long long)y * F.P + x] : 1.0f;
        m[d] = s;
      }
      if (J < cny) {
        const int fx = min(2 * I, F.nx);
        float s = 0.f;
        for (int y = 2 * J; y < min(2 * J + 2, F.ny); y++) s += F.ax[(long long)y * F.P + fx];
        ax[d] = fs * s;
      }
      if (I < cnx) {
        const int fy = min(2 * J, F.ny);
        float s = 0.f;
        for (int x = 2 * I; x < min(2 * I + 2, F.nx); x++) s += F.ay[(long long)fy * F.P + x];
        ay[d] = fs * s;
      }
    }
}

}  // namespace

Multigrid::~Multigrid() { release(); }

void Multigrid::drop_graph() {
  if (exec_) cudaGraphExecDestroy(exec_);
  exec_ = nullptr;
  g_r_ = nullptr;
  g_z_ = nullptr;
  g_s_ = nullptr;
}

void Multigrid::release() {
  drop_graph();
  cudaFree(buf_);
  buf_ = nullptr;
  buf_elems_ = 0;
  lv_.clear();
}

void Multigrid::setup(int nx, int ny, long long pitch, const double *Kx, const double *Ky, double rx, double ry,
                      cudaStream_t s) {
  if (nx < 1 || ny < 1 || pitch < nx + 2) throw Error(E_ARG, "multigrid: bad shape");
  // level shapes and storage
  std::vector<Level> lv;
  size_t elems = 0;
  for (int x = nx, y = ny;;) {
    Level L;
    L.nx = x;
    L.ny = y;
    L.pitch = ((long long)x + 1 + 31) / 32 * 32;
    lv.push_back(L);
    const size_t one = (size_t)y * L.pitch;
    elems += 6 * one + L.pitch;  // m (unused on level 0), ax, ay (+1 row), r, z0, z1
    if (x <= kCoarsest && y <= kCoarsest) break;
    x = (x + 1) / 2;
    y = (y + 1) / 2;
  }
  if (lv.size() != lv_.size() || lv[0].nx != (lv_.empty() ? -1 : lv_[0].nx) ||
      lv[0].ny != (lv_.empty() ? -1 : lv_[0].ny) || elems > buf_elems_ || pitch != fpitch_) {
    release();
    OPSB_CUDA(cudaMalloc(&buf_, elems * sizeof(float)));
    buf_elems_ = elems;
    // the cycle loads padding columns beside a row's last cell and masks what
    // it makes of them; they are zeroed once, since a product with a mask of 0
    // needs a finite factor
    OPSB_CUDA(cudaMemsetAsync(buf_, 0, elems * sizeof(float), s));
  }
  float *q = buf_;
  for (size_t l = 0; l < lv.size(); l++) {
    Level &L = lv[l];
    const size_t one = (size_t)L.ny * L.pitch;
    L.m = l ? q : nullptr;
    q += one;
    L.ax = q;
    q += one;
    L.ay = q;
    q += one + L.pitch;
    L.r = q;
    q += one;
    L.z0 = q;
    q += one;
    L.z1 = q;
    q += one;
  }
  lv_ = lv;
  fpitch_ = pitch;
  {
    const Level &L = lv_[0];
    k_fine_faces<<<grid_of(nx + 1, ny + 1), dim3(BX, BY), 0, s>>>(nx, ny, pitch, Kx, Ky, rx, ry, L.pitch, L.ax,
                                                                   L.ay);
    check("level-0 faces");
  }
  for (size_t l = 1; l < lv_.size(); l++) {
    const Level &F = lv_[l - 1], &C = lv_[l];
    const LV fv{F.nx, F.ny, F.pitch, F.m, F.ax, F.ay};
    k_coarsen<<<grid_of(C.nx + 1, C.ny + 1), dim3(BX, BY), 0, s>>>(fv, C.nx, C.ny, C.pitch, C.m, C.ax, C.ay,
                                                                    kFaceScale);
    check("coarsening");
  }
}

long long Multigrid::apply(const double *r, double *z, cudaStream_t s) {
  if (lv_.empty()) throw Error(E_STATE, "multigrid: apply before setup");
  if (exec_ && r == g_r_ && z == g_z_ && s == g_s_) {
    OPSB_CUDA(cudaGraphLaunch(exec_, s));
    return g_n_;
  }
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  OPSB_CUDA(cudaStreamIsCapturing(s, &cs));
  if (cs != cudaStreamCaptureStatusNone) return enqueue(r, z, s);  // the caller's capture records the launches
  drop_graph();
  OPSB_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  long long n = 0;
  cudaGraph_t g = nullptr;
  try {
    n = enqueue(r, z, s);
  } catch (...) {
    cudaStreamEndCapture(s, &g);
    if (g) cudaGraphDestroy(g);
    throw;
  }
  OPSB_CUDA(cudaStreamEndCapture(s, &g));
  cudaGraphExec_t ex = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
  cudaGraphDestroy(g);
  OPSB_CUDA(e);
  exec_ = ex;
  g_r_ = r;
  g_z_ = z;
  g_s_ = s;
  g_n_ = n;
  OPSB_CUDA(cudaGraphLaunch(exec_, s));
  return n;
}

long long Multigrid::enqueue(const double *r, double *z, cudaStream_t s) {
  const int nl = (int)lv_.size();
  const float w = kOmega;
  const dim3 blk(BX, BY);
  auto view = [&](int l) {
    const Level &L = lv_[l];
    return LV{L.nx, L.ny, L.pitch, L.m, L.ax, L.ay};
  };
  long long n = 0;
  if (nl == 1) {
    k_coarsest<true, true><<<1, kCoarseThreads, 0, s>>>(view(0), nullptr, r, fpitch_, nullptr, z, kCoarseSweeps, w);
    check("coarsest level");
    return 1;
  }
  static_assert(kSweeps == 2, "k_cycle makes two sweeps a side");
  // strips of whole aggregates' rows
  auto strips = [&](const Level &L, bool up, int *rows) {
    const int ncol = ((L.nx + 1) / 2 + 29) / 30, cny = (L.ny + 1) / 2;
    *rows = 2 * march_rows(ncol, cny, 2, 148LL * cycle_blocks(up) * kCycleWarps);
    const long long warps = (long long)ncol * ((L.ny + *rows - 1) / *rows);
    return (unsigned)((warps + kCycleWarps - 1) / kCycleWarps);
  };
  const int nt = 32 * kCycleWarps;
  // r and z of level 0: strips read r beside the rows they write z to, so
  // where the two overlap r is taken from a copy
  const long long span = (long long)(lv_[0].ny - 1) * fpitch_ + lv_[0].nx;
  const bool apart = z + span <= r || r + span <= z;
  auto even = [&](const double *p) { return fpitch_ % 2 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const int vr = even(r), vz = even(z);
  if (!apart) {
    k_copy_r<<<grid_of(lv_[0].nx, lv_[0].ny), blk, 0, s>>>(view(0), r, fpitch_, lv_[0].r);
    n++;
  }
  // down: smooth, then hand the residual to the next level
  for (int l = 0; l + 1 < nl; l++) {
    Level &L = lv_[l], &C = lv_[l + 1];
    const LV v = view(l);
    int rows;
    const unsigned g = strips(L, false, &rows);
    if (l == 0 && apart)
      k_cycle<false, true, true, false><<<g, nt, 0, s>>>(v, r, fpitch_, vr, nullptr, L.z0, nullptr, C.pitch, C.r,
                                                         nullptr, w, rows);
    else if (l == 0)
      k_cycle<false, true, false, false><<<g, nt, 0, s>>>(v, nullptr, 0, 0, L.r, L.z0, nullptr, C.pitch, C.r, nullptr,
                                                          w, rows);
    else
      k_cycle<false, false, false, false><<<g, nt, 0, s>>>(v, nullptr, 0, 0, L.r, L.z0, nullptr, C.pitch, C.r,
                                                           nullptr, w, rows);
    n++;
    check("pre-smoothing and restriction");
  }
  {
    Level &L = lv_[nl - 1];
    k_coarsest<false, false><<<1, kCoarseThreads, 0, s>>>(view(nl - 1), L.r, nullptr, 0, L.z1, nullptr,
                                                          kCoarseSweeps, w);
    n++;
    check("coarsest level");
  }
  // up: correct with the coarse solution, then post-smooth
  for (int l = nl - 2; l >= 0; l--) {
    Level &L = lv_[l], &C = lv_[l + 1];
    const LV v = view(l);
    int rows;
    const unsigned g = strips(L, true, &rows);
    if (l == 0 && apart)
      k_cycle<true, true, true, true><<<g, nt, 0, s>>>(v, r, fpitch_, vr && vz, nullptr, L.z0, C.z1, C.pitch, nullptr, z,
                                                       w, rows);
    else if (l == 0)
      k_cycle<true, true, false, true><<<g, nt, 0, s>>>(v, nullptr, fpitch_, vz, L.r, L.z0, C.z1, C.pitch, nullptr, z,
                                                        w, rows);
    else
      k_cycle<true, false, false, false><<<g, nt, 0, s>>>(v, nullptr, 0, 0, L.r, L.z0, C.z1, C.pitch, L.z1, nullptr, w,
                                                          rows);
    n++;
    check("prolongation and post-smoothing");
  }
  return n;
}

}  // namespace heat
}  // namespace opsb
