// Batched tridiagonal solver (ops_tridMultiDimBatch / _Inc).
//
// Reference: ops/c/src/tridiag/ops_tridiag.cpp:78-249 hands every line along
// `solvedim` of the range to the external Tridsolver library
// (trid{D,S}mtsvStridedBatch[Inc]); each line is the system
//     a_i x_{i-1} + b_i x_i + c_i x_{i+1} = d_i   (a_0, c_{n-1} unused).
// The non-Inc form overwrites d with x; the Inc form adds x to u.
//
// B200 design: one persistent launch walks a work list of line groups over
// any number of systems (blocks of different shapes solve in one launch).
// Every line is split into chunks of about 8 rows, one chunk per thread; a
// thread runs the modified Thomas elimination on its chunk, expressing each
// row through the chunk's first and last unknowns (the partition method of
// Wang 1981, as used for GPUs by Laszlo, Giles and Appleyard, ACM TOMS 42(4)
// 2016):
//   forward, rows 0 and 1 normalised, then for i >= 2
//     r = 1 / (b_i - a_i c'_{i-1}),  d'_i = r (d_i - a_i d'_{i-1}),
//     a'_i = -r a_i a'_{i-1},        c'_i = r c_i;
//   backward for i = m-3 .. 1
//     d'_i -= c'_i d'_{i+1},  a'_i -= c'_i a'_{i+1},  c'_i = -c'_i c'_{i+1};
//   row 0 folds in row 1.
// The chunks' end rows form a small tridiagonal system in shared memory,
// solved by parallel cyclic reduction; a last pass substitutes back. The lines of a work item
// are staged through shared memory, so coefficients and right-hand sides are
// read from HBM once and the solution written once: 40 bytes per FP64
// unknown (48 for _Inc).
#include <algorithm>
#include <cstdio>
#include <vector>

#include "../../include/ops_b200.h"
#include "runtime.h"

namespace opsb {
namespace trid {

struct Sys {
  const char *a, *b, *c;
  char *d, *u;
  int n;           // line length
  int nl0, nl1;    // line counts along the two non-solve dimensions (fastest first)
  long long ss;    // stride along the solve dimension (elements)
  long long s0, s1;
  // line kernel: an entry is a system's groups of `glines` lines from line lofs
  // on; its first group, and its first group's scratch
  long long line0 = 0, scr0 = 0, lofs = 0;
  int glines = 0;
};

struct Work {
  int sys, l0, l1;  // system, first line along dim 0, line index along dim 1
};

// Reciprocal: the hardware's approximation r (rcp.approx.ftz.f64, about 20 bits)
// and one third-order step of Newton's iteration for 1/x (e = 1 - x r,
// r' = r + r (e + e^2), whose error is e^3, beyond FP64). About 1 ulp, without
// the out-of-line slow path of IEEE division, whose call would force the
// per-thread coefficient arrays out of registers, and short: the reciprocal is
// most of the chain from row to row (a single-precision seed with its
// conversions, scaling and two second-order steps took twice as long). Valid
// for finite normal pivots with 2^-1000 < |x| < 2^1000; the solver's tolerance
// is relative (1e-12 in FP64), not bit-exact.
__device__ __forceinline__ float recip(float x) {
  float r = __fdividef(1.0f, x);
  const float e = fmaf(-x, r, 1.0f);
  return fmaf(r, e, r);
}
__device__ __forceinline__ double recip(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// r = 1 / x and cr = c / x by the same steps: c takes part in the correction, so
// the two are ready together.
__device__ __forceinline__ void recip_times(float x, float c, float &r, float &cr) {
  const float q = __fdividef(1.0f, x), cq = c * q, e = fmaf(-x, q, 1.0f);
  r = fmaf(q, e, q);
  cr = fmaf(cq, e, cq);
}
__device__ __forceinline__ void recip_times(double x, double c, double &r, double &cr) {
  double q;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(x));
  const double cq = c * q, e = fma(-x, q, 1.0), t = fma(e, e, e);
  r = fma(q, t, q);
  cr = fma(cq, t, cq);
}

// One work item = L neighbouring lines x n rows of one system, staged in
// shared memory: the four coefficient tiles are loaded with cp.async (rows
// of the tile along whichever dimension is contiguous in HBM, so the loads
// coalesce), each thread eliminates its chunk of about 8 rows in place in
// shared memory, the chunks' end rows form the reduced system (solved per
// line by Thomas), and the substituted solution is stored with the same
// coalesced mapping. Registers stay few, so two CTAs share an SM and one
// CTA's loads overlap the other's elimination. Tile rows are padded to
// L + 1 elements to spread the chunks over the shared-memory banks.
constexpr int kTileThreads = 256;

#ifndef TRID_CTAS_PER_SM
#define TRID_CTAS_PER_SM 2
#endif
constexpr int kCtasPerSm = TRID_CTAS_PER_SM;
// shared memory per CTA, so that kCtasPerSm CTAs share an SM (227 KB)
constexpr size_t kTileSmem = (size_t)(220 / kCtasPerSm) * 1024;

template <class T>
size_t tile_smem(int L, int n) {
  return (size_t)(4 * (L + 1) * n + 8 * (kTileThreads / L) * L) * sizeof(T);
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <class T>
__device__ __forceinline__ void cp_async(T *dst, const T *src) {
  if (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

template <class T>
__global__ void __launch_bounds__(kTileThreads, kCtasPerSm) trid_tile_kernel(const Sys *__restrict__ sys,
                                                                    const Work *__restrict__ work, int nwork, int L,
                                                                    int nmax) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int P = L + 1;  // padded tile row
  const int tile = P * nmax;
  T *ta = reinterpret_cast<T *>(smraw);
  T *tb = ta + tile, *tc = tb + tile, *td = tc + tile;
  const int K = kTileThreads / L;
  T *RA = td + tile, *RB = RA + 2 * K * L, *RC = RB + 2 * K * L, *RD = RC + 2 * K * L;
  const int tid = threadIdx.x;
  const int l = tid % L, chunk = tid / L;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const Work wk = work[w];
    const Sys s = sys[wk.sys];
    const int n = s.n;
    const int nl = min(L, s.nl0 - wk.l0);
    const long long base = (long long)wk.l0 * s.s0 + (long long)wk.l1 * s.s1;
    const T *ga = reinterpret_cast<const T *>(s.a) + base;
    const T *gb = reinterpret_cast<const T *>(s.b) + base;
    const T *gc = reinterpret_cast<const T *>(s.c) + base;
    T *gd = reinterpret_cast<T *>(s.d) + base;
    T *gu = s.u ? reinterpret_cast<T *>(s.u) + base : nullptr;
    const bool rows_contig = s.ss == 1;
    const int warp = tid >> 5, lane = tid & 31;
    // 1. stage the four tiles: along x one warp per line (lanes walk the
    // contiguous rows), otherwise thread t takes line t mod L and every
    // (256 / L)-th row from t / L, so each warp-wide copy covers L
    // neighbouring lines of 256 / L rows; no division per element
    if (rows_contig) {
      for (int ll = warp; ll < nl; ll += kTileThreads / 32) {
        const long long g0 = (long long)ll * s.s0;
        for (int i = lane; i < n; i += 32) {
          const int si = i * P + ll;
          cp_async(ta + si, ga + g0 + i);
          cp_async(tb + si, gb + g0 + i);
          cp_async(tc + si, gc + g0 + i);
          cp_async(td + si, gd + g0 + i);
        }
      }
    } else if (l < nl) {
      const long long g0 = (long long)l * s.s0;
      for (int i = chunk; i < n; i += K) {
        const long long g = g0 + (long long)i * s.ss;
        const int si = i * P + l;
        cp_async(ta + si, ga + g);
        cp_async(tb + si, gb + g);
        cp_async(tc + si, gc + g);
        cp_async(td + si, gd + g);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // 2. eliminate this thread's chunk in place (same recurrences as chunk_eliminate)
    const int kact = n >= 2 * K ? K : (n / 2 > 0 ? n / 2 : 1);
    const int r0 = chunk * n / kact, r1 = (chunk + 1) * n / kact, m = r1 - r0;
    const bool mine = l < nl && chunk < kact && n > 1;
    if (n == 1 && chunk == 0 && l < nl) td[l] = td[l] * recip(tb[l]);
    if (mine) {
      T pa = T(0), pc = T(0), pd = T(0);
      for (int i = 0; i < m; i++) {
        const int q = (r0 + i) * P + l;
        const T ai = ta[q], bi = tb[q], ci = tc[q], di = td[q];
        T na, nc, nd;
        if (i < 2) {
          const T r = recip(bi);
          na = ai * r;
          nc = ci * r;
          nd = di * r;
        } else {
          const T r = recip(bi - ai * pc);
          nd = r * (di - ai * pd);
          na = -r * ai * pa;
          nc = r * ci;
        }
        ta[q] = na;
        tc[q] = nc;
        td[q] = nd;
        pa = na;
        pc = nc;
        pd = nd;
      }
      const T la = pa, lc = pc, ld = pd;
      if (m > 3) {
        const int q1 = (r0 + m - 2) * P + l;
        T na = ta[q1], nc = tc[q1], nd = td[q1];
        for (int i = m - 3; i >= 1; i--) {
          const int q = (r0 + i) * P + l;
          const T ci = tc[q];
          nd = td[q] - ci * nd;
          na = ta[q] - ci * na;
          nc = -ci * nc;
          ta[q] = na;
          tc[q] = nc;
          td[q] = nd;
        }
      }
      const int q0 = r0 * P + l, q1 = (r0 + 1) * P + l;
      T a0 = ta[q0], c0 = tc[q0], d0 = td[q0];
      if (m > 2) {
        const T r = recip(T(1) - c0 * ta[q1]);
        d0 = r * (d0 - c0 * td[q1]);
        a0 = r * a0;
        c0 = -r * c0 * tc[q1];
        ta[q0] = a0;
        tc[q0] = c0;
        td[q0] = d0;
      }
      RA[(2 * chunk) * L + l] = chunk == 0 ? T(0) : a0;
      RB[(2 * chunk) * L + l] = T(1);
      RC[(2 * chunk) * L + l] = c0;
      RD[(2 * chunk) * L + l] = d0;
      RA[(2 * chunk + 1) * L + l] = la;
      RB[(2 * chunk + 1) * L + l] = T(1);
      RC[(2 * chunk + 1) * L + l] = chunk == kact - 1 ? T(0) : lc;
      RD[(2 * chunk + 1) * L + l] = ld;
    }
    __syncthreads();
    // 3. the reduced system (2 kact rows per line) by parallel cyclic
    // reduction (Hockney 1965): at stride h every row eliminates its
    // neighbours h above and below, log2(2 kact) steps with every chunk
    // thread taking its two rows; afterwards x_k = d_k / b_k.
    if (n > 1) {
      const int N = 2 * kact;
      const bool act = l < nl && chunk < kact;
      for (int h = 1; h < N; h *= 2) {
        T na[2], nb[2], nc[2], nd[2];
        if (act) {
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const int k = 2 * chunk + j;
            const int q = k * L + l;
            T ak = RA[q], bk = RB[q], ck = RC[q], dk = RD[q];
            if (k - h >= 0) {
              const int qm = (k - h) * L + l;
              const T al = -ak * recip(RB[qm]);
              ak = al * RA[qm];
              bk = bk + al * RC[qm];
              dk = dk + al * RD[qm];
            } else {
              ak = T(0);
            }
            if (k + h < N) {
              const int qp = (k + h) * L + l;
              const T ga = -ck * recip(RB[qp]);
              ck = ga * RC[qp];
              bk = bk + ga * RA[qp];
              dk = dk + ga * RD[qp];
            } else {
              ck = T(0);
            }
            na[j] = ak;
            nb[j] = bk;
            nc[j] = ck;
            nd[j] = dk;
          }
        }
        __syncthreads();
        if (act) {
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const int q = (2 * chunk + j) * L + l;
            RA[q] = na[j];
            RB[q] = nb[j];
            RC[q] = nc[j];
            RD[q] = nd[j];
          }
        }
        __syncthreads();
      }
      if (act) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const int q = (2 * chunk + j) * L + l;
          RD[q] = RD[q] * recip(RB[q]);
        }
      }
    }
    __syncthreads();
    // 4. substitute back into the d tile
    if (mine) {
      const T xf = RD[(2 * chunk) * L + l], xl = RD[(2 * chunk + 1) * L + l];
      for (int i = 0; i < m; i++) {
        const int q = (r0 + i) * P + l;
        td[q] = (i == 0) ? xf : (i == m - 1) ? xl : td[q] - ta[q] * xf - tc[q] * xl;
      }
    }
    __syncthreads();
    // 5. store (d = x, or u += x), with the loads' mapping
    if (rows_contig) {
      for (int ll = warp; ll < nl; ll += kTileThreads / 32) {
        const long long g0 = (long long)ll * s.s0;
        for (int i = lane; i < n; i += 32) {
          const T x = td[i * P + ll];
          if (gu) gu[g0 + i] += x;
          else gd[g0 + i] = x;
        }
      }
    } else if (l < nl) {
      const long long g0 = (long long)l * s.s0;
      for (int i = chunk; i < n; i += K) {
        const long long g = g0 + (long long)i * s.ss;
        const T x = td[i * P + l];
        if (gu) gu[g] += x;
        else gd[g] = x;
      }
    }
    __syncthreads();
  }
}

// x sweeps (lines contiguous in HBM) of up to 32 R rows, no block-wide
// barriers: a warp solves 32 / P lines at once, P lanes per line (P = 32,
// 16 or 8: the fewest lanes whose chunks of at most R rows cover a line, so
// short lines share a warp). The warp stages its lines' a, b, c, d through
// its own strip of shared memory with coalesced cp.async copies (row r at
// r + r / 8, so that lanes reading neighbouring chunks hit different
// banks), every lane eliminates its chunk in registers by the same partition
// recurrences as trid_tile_kernel, each line's 2 P chunk end rows are solved
// by parallel cyclic reduction over shuffles within its lane group, and the
// lanes substitute back and store through the strip. A warp keeps all its
// lines' 4 n loads in flight at once. Its time is its instructions (FP64 chains
// and reduction steps): with the short reciprocal and one of them a reduced row
// and step instead of two, 256^3 FP64 0.248 -> 0.168 ms, FP32 0.135 -> 0.120, the
// 64-block batch 0.837 -> 0.587 and 0.480 -> 0.402, each sweep repeated by itself.
// Right after a z sweep, as in an ADI step, 256^3 FP64 takes 0.205 ms and the FP64
// batch 0.748.
constexpr int kWarpLines = 8;  // warps per CTA

template <int R>
__host__ __device__ constexpr int warp_strip(int) { return 32 * R + 4 * R + 2; }
__device__ __forceinline__ int strip_pos(int r) { return r + (r >> 3); }
// Lanes per line for lines of n rows and chunks of at most R rows.
__host__ __device__ inline int lanes_per_line(int n, int R) {
  int p = 32;
  while (p > 8 && (p / 2) * R >= n) p /= 2;
  return p;
}

// FP32 lines hold half the registers: three CTAs per SM. FP: lanes per
// line fixed at compile time (32: every line of the launch fills a warp), or
// 0 to choose per system.
template <class T, int R, int FP>
__global__ void __launch_bounds__(32 * kWarpLines, sizeof(T) == 4 ? 3 : 2)
    trid_warp_kernel(const Sys *__restrict__ sys, const Work *__restrict__ work, int nwork) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int SW = warp_strip<R>(0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T *Sa = reinterpret_cast<T *>(smraw) + (size_t)warp * 4 * SW;
  T *Sb = Sa + SW, *Sc = Sb + SW, *Sd = Sc + SW;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const Work wk = work[w];
    const Sys s = sys[wk.sys];
    const int n = s.n;
    const int P = FP ? FP : lanes_per_line(n, R), G = 32 / P;  // lanes per line, lines per warp
    const int line0 = wk.l0 + warp * G;               // this warp's first line
    if (line0 >= s.nl0) continue;                     // the same for the whole warp
    const long long base0 = (long long)line0 * s.s0 + (long long)wk.l1 * s.s1;
    const T *ga = reinterpret_cast<const T *>(s.a) + base0;
    const T *gb = reinterpret_cast<const T *>(s.b) + base0;
    const T *gc = reinterpret_cast<const T *>(s.c) + base0;
    T *gd = reinterpret_cast<T *>(s.d) + base0;
    T *gu = s.u ? reinterpret_cast<T *>(s.u) + base0 : nullptr;
    const int nlines = min(G, s.nl0 - line0);
    // asynchronous copies, line by line over the whole warp: every load in flight at once
    for (int g = 0; g < nlines; g++) {
      const long long lo = (long long)g * s.s0;
      const int ro = g * P * R;
      for (int i = lane; i < n; i += 32) {
        const int p = strip_pos(ro + i);
        cp_async(Sa + p, ga + lo + i);
        cp_async(Sb + p, gb + lo + i);
        cp_async(Sc + p, gc + lo + i);
        cp_async(Sd + p, gd + lo + i);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    // 1. this lane's chunk of its line: forward and backward partition sweeps in registers
    const int g = lane / P, gl = lane - g * P, ro = g * P * R;
    const int kact = n >= 2 * P ? P : (n / 2 > 0 ? n / 2 : 1);
    const int r0 = ro + gl * n / kact, m = (gl + 1) * n / kact - gl * n / kact;
    const bool act = g < nlines && gl < kact && n > 1;
    T ra[R], rc[R], rd[R];
    T fa[2] = {T(0), T(0)}, fc[2] = {T(0), T(0)}, fd[2] = {T(0), T(0)};
    if (act) {
      T pa = T(0), pc = T(0), pd = T(0);
#pragma unroll
      for (int i = 0; i < R; i++) {
        if (i < m) {
          const int p = strip_pos(r0 + i);
          const T ai = Sa[p], bi = Sb[p], ci = Sc[p], di = Sd[p];
          T na, nc, nd;
          if (i < 2) {
            const T r = recip(bi);
            na = ai * r;
            nc = ci * r;
            nd = di * r;
          } else {
            const T r = recip(bi - ai * pc);
            nd = r * (di - ai * pd);
            na = -r * ai * pa;
            nc = r * ci;
          }
          ra[i] = na;
          rc[i] = nc;
          rd[i] = nd;
          pa = na;
          pc = nc;
          pd = nd;
        }
      }
      fa[1] = pa;
      fc[1] = gl == kact - 1 ? T(0) : pc;
      fd[1] = pd;
      // backward: rows m-3 .. 1 fold in row i + 1 (whose values ride in
      // na, nc, nd; rows from m-2 up pass theirs on unchanged)
      T na = T(0), nc = T(0), nd = T(0);
#pragma unroll
      for (int t = 0; t < R - 1; t++) {
        const int i = R - 1 - t;
        if (i <= m - 3) {
          const T ci = rc[i];
          nd = rd[i] - ci * nd;
          na = ra[i] - ci * na;
          nc = -ci * nc;
          ra[i] = na;
          rc[i] = nc;
          rd[i] = nd;
        } else {
          na = ra[i];
          nc = rc[i];
          nd = rd[i];
        }
      }
      T a0 = ra[0], c0 = rc[0], d0 = rd[0];
      if (m > 2) {
        const T r = recip(T(1) - c0 * ra[1]);
        d0 = r * (d0 - c0 * rd[1]);
        a0 = r * a0;
        c0 = -r * c0 * rc[1];
      }
      ra[0] = a0;
      rc[0] = c0;
      rd[0] = d0;
      fa[0] = gl == 0 ? T(0) : a0;
      fc[0] = c0;
      fd[0] = d0;
    }
    // 2. each line's 2 P chunk end rows (row 2 gl + j), parallel cyclic
    // reduction over shuffles within the line's lane group; lanes without a
    // chunk hold identity rows
    // (the rows enter with b = 1 and every step divides its row by the new b, so
    // a step takes one reciprocal a row and the solution is the last d)
    const int N = 2 * P;
    for (int h = 1; h < N; h *= 2) {
      T ma[2], mc[2], md[2], pa[2], pc[2], pd[2];
      if (h == 1) {
        ma[0] = __shfl_up_sync(0xffffffffu, fa[1], 1, P);
        mc[0] = __shfl_up_sync(0xffffffffu, fc[1], 1, P);
        md[0] = __shfl_up_sync(0xffffffffu, fd[1], 1, P);
        pa[1] = __shfl_down_sync(0xffffffffu, fa[0], 1, P);
        pc[1] = __shfl_down_sync(0xffffffffu, fc[0], 1, P);
        pd[1] = __shfl_down_sync(0xffffffffu, fd[0], 1, P);
        pa[0] = fa[1]; pc[0] = fc[1]; pd[0] = fd[1];
        ma[1] = fa[0]; mc[1] = fc[0]; md[1] = fd[0];
      } else {
        const int q = h >> 1;
#pragma unroll
        for (int j = 0; j < 2; j++) {
          ma[j] = __shfl_up_sync(0xffffffffu, fa[j], q, P);
          mc[j] = __shfl_up_sync(0xffffffffu, fc[j], q, P);
          md[j] = __shfl_up_sync(0xffffffffu, fd[j], q, P);
          pa[j] = __shfl_down_sync(0xffffffffu, fa[j], q, P);
          pc[j] = __shfl_down_sync(0xffffffffu, fc[j], q, P);
          pd[j] = __shfl_down_sync(0xffffffffu, fd[j], q, P);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int k = 2 * gl + j;
        // a row without a neighbour there has no coefficient for it either
        const T ak = k - h >= 0 ? fa[j] : T(0), ck = k + h < N ? fc[j] : T(0);
        const T r = recip(T(1) - ak * mc[j] - ck * pa[j]);
        fa[j] = -ak * ma[j] * r;
        fc[j] = -ck * pc[j] * r;
        fd[j] = (fd[j] - ak * md[j] - ck * pd[j]) * r;
      }
    }
    // 3. substitute back, then store through the strip with the loads' mapping
    if (act) {
      const T xf = fd[0], xl = fd[1];
#pragma unroll
      for (int i = 0; i < R; i++)
        if (i < m) Sd[strip_pos(r0 + i)] = (i == 0) ? xf : (i == m - 1) ? xl : rd[i] - ra[i] * xf - rc[i] * xl;
    }
    if (n == 1 && gl == 0 && g < nlines) Sd[strip_pos(ro)] = Sd[strip_pos(ro)] * recip(Sb[strip_pos(ro)]);
    __syncwarp();
    for (int gg = 0; gg < nlines; gg++) {
      const long long lo = (long long)gg * s.s0;
      const int rg = gg * P * R;
      for (int i = lane; i < n; i += 32) {
        const T x = Sd[strip_pos(rg + i)];
        if (gu) gu[lo + i] += x;
        else gd[lo + i] = x;
      }
    }
    __syncwarp();
  }
}

// ---- strided sweeps -----------------------------------------------------------
// The y and z sweeps run the textbook Thomas elimination straight from HBM:
//   c'_0 = c_0 / b_0, d'_0 = d_0 / b_0; for i >= 1, r = 1 / (b_i - a_i c'_{i-1}),
//   c'_i = c_i r, d'_i = (d_i - a_i d'_{i-1}) r; x_{n-1} = d'_{n-1},
//   x_i = d'_i - c'_i x_{i+1}.
// It needs a fraction of the partition method's instructions, but c' and d' have
// to wait for the backward pass. They go to a scratch that stays in L2: the
// grid keeps only so many lines in flight that their c' and d' fit
// (kScratchBytes; a CTA an SM at least), each warp reuses its own part group after
// group, the scratch is marked evict-last and everything else evict-first. HBM then sees the
// compulsory 40 B per FP64 unknown (48 with _Inc). With every line in flight
// the scratch went through HBM too (68 to 77 B; now 43.7 and 52.3). In an ADI step
// at 256^3 FP64: y sweep 0.213 -> 0.162 ms, z sweep (_Inc) 0.289 -> 0.209 ms; the
// 64-block FP64 batch's 0.548 -> 0.443 and 0.655 -> 0.497 ms. Limits of 60 to 400 MB
// measured within 7 % of one another, 40 MB 1.3x slower.
constexpr size_t kScratchBytes = 64ull << 20;

__device__ __forceinline__ uint64_t policy_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
template <class T>
__device__ __forceinline__ void cp_async_hint(T *dst, const T *src, uint64_t pol) {
  asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], %2, %3;" ::"r"(smem_addr(dst)), "l"(src),
               "n"((int)sizeof(T)), "l"(pol)
               : "memory");
}
__device__ __forceinline__ double ld_hint(const double *p, uint64_t pol) {
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol) : "memory");
  return v;
}
__device__ __forceinline__ float ld_hint(const float *p, uint64_t pol) {
  float v;
  asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol) : "memory");
  return v;
}
__device__ __forceinline__ void st_hint(double *p, double v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_hint(float *p, float v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
}

// The size of a value as an integer that orders like it: NaN above infinity.
__device__ __forceinline__ int magnitude(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ int magnitude(float x) { return __float_as_int(x) & 0x7fffffff; }

// Lines strided along the solve dimension and contiguous across lines (the y
// and z sweeps). A warp solves 16 neighbouring lines, two lanes each: one
// eliminates from the top, its partner (lane + 16) from the bottom with a and c
// in each other's place, they meet in the middle,
//   x_m = (d'_m - c'_m d''_{m+1}) / (1 - c'_m a''_{m+1}),
// and substitute outwards. So a line's chain is half as long and the lines
// whose c' and d' fit L2 keep twice the threads busy. The rows ahead come by
// cp.async into the thread's own column of a ring of kLineStages stages of
// U rows (no barrier: nobody else reads it); the backward pass reads c' and d' U
// rows ahead into registers.
//
// A line may have pivots from the top only (b_{n-1} = 0, say). While |c'| stays
// within kGrowth a pivot's rounding error is that of its row's entries, so the
// elimination from the bottom is as sound as the rows are; a line whose c' pass
// it (a vanished pivot leaves infinity or NaN) is solved again from the top
// alone, a lane a line, in the two lanes' scratch. Diagonally dominant rows
// have |c'| <= 1. (The maximum costs 0.1 to 0.2 % of an ADI step. Where every line
// is solved again, 256^3 FP64 takes 1.75 ms instead of 0.17; the loops' loads in
// batches of eight rows, in or out of line, cost ordinary lines 20 %.)
constexpr float kGrowth = 16.0f;
constexpr int kLineThreads = 128, kLineStages = 3;
// U is 8, which leaves an SM 2 CTAs (FP64) or 3, and 4, with 4 to 6 of them, where
// lines of up to 64 rows fill more than a wave of the former: a wave more or less
// counts for more there than the loads ahead. 300,000 lines FP64 of 24 rows 75 ->
// 62 us, of 64 rows 167 -> 159, of 128 rows 335 -> 347; 65,536 lines FP32 of 48 rows
// 26 -> 23.5.
constexpr int kFewRows = 64;

// Scratch of a group: c' and d' of its lines' halves.
__host__ __device__ inline long long group_scratch(int n, int glines) { return (n + 1) / 2 * 4ll * glines; }

template <class T, int U>
constexpr int kLineSmem = kLineStages * U * 4 * kLineThreads * (int)sizeof(T);

template <class T, int U>
__global__ void __launch_bounds__(kLineThreads) trid_line_kernel(const Sys *__restrict__ sys, int nsys,
                                                                 long long groups, T *scr) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T *ring = reinterpret_cast<T *>(smraw) + threadIdx.x;  // element (stage, row, array) every kLineThreads
  const uint64_t keep = policy_last(), pass = policy_first();
  const int lane = threadIdx.x & 31, half = lane >> 4, warps = gridDim.x * (kLineThreads / 32);
  const int first = blockIdx.x * (kLineThreads / 32) + (threadIdx.x >> 5);
  T *part = nullptr;  // the warp's scratch: its first group's, which needs the most
  for (long long g = first; g < groups; g += warps) {
    int lo = 0, hi = nsys - 1;  // last system whose first group of lines is <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sys[mid].line0 <= g) lo = mid;
      else hi = mid - 1;
    }
    const Sys &s = sys[lo];
    const long long l = s.lofs + (g - s.line0) * 16 + (lane & 15);
    const int n = s.n, len = (lane & 15) < s.glines ? (half ? n / 2 : (n + 1) / 2) : 0;
    const int width = 2 * s.glines;
    if (g == first) part = scr + s.scr0 + (g - s.line0) * group_scratch(n, s.glines);
    T *cp = part + half * s.glines + (lane & 15);  // c' of row i at [2 i width], d' at [(2 i + 1) width]
    const long long ss = half ? -s.ss : s.ss;
    const long long base = (l % s.nl0) * s.s0 + (l / s.nl0) * s.s1 + (half ? (long long)(n - 1) * s.ss : 0);
    const T *a = reinterpret_cast<const T *>(half ? s.c : s.a) + base;
    const T *b = reinterpret_cast<const T *>(s.b) + base;
    const T *c = reinterpret_cast<const T *>(half ? s.a : s.c) + base;
    T *d = reinterpret_cast<T *>(s.d) + base;
    T *u = s.u ? reinterpret_cast<T *>(s.u) + base : nullptr;
    const int nst = ((n + 1) / 2 + U - 1) / U, full = (n / 2) / U;  // stages; those that every live lane fills
    long long ahead = 0;  // offset of the next row to fetch
    auto fetch_row = [&](T *t) {
      cp_async_hint(t, a + ahead, pass);
      cp_async_hint(t + kLineThreads, b + ahead, pass);
      cp_async_hint(t + 2 * kLineThreads, c + ahead, pass);
      cp_async_hint(t + 3 * kLineThreads, (const T *)d + ahead, pass);
      ahead += ss;
    };
    auto fetch = [&](int st) {
      T *t = ring + (st % kLineStages) * (U * 4 * kLineThreads);
      if (st < full && len) {
#pragma unroll
        for (int j = 0; j < U; j++) fetch_row(t + 4 * j * kLineThreads);
      } else {
        for (int j = 0; j < min(U, len - st * U); j++) fetch_row(t + 4 * j * kLineThreads);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int st = 0; st < kLineStages - 1; st++) fetch(st);
    // the chain from row to row is one product and the reciprocal. (A product
    // a_i c_{i-1} taken ahead would be a cycle shorter but has the square of the
    // rows' scale: FP32 rows of 1e20 overflow in it.)
    T pc = T(0), pd = T(0);
    int worst = 0;  // the largest |c'|
    T *q = cp;
    auto eliminate = [&](T ai, T bi, T ci, T di) {
      T r;
      recip_times(bi - ai * pc, ci, r, pc);
      pd = (di - ai * pd) * r;
      worst = max(worst, magnitude(pc));
      st_hint(q, pc, keep);
      st_hint(q + width, pd, keep);
      q += 2 * width;
    };
    for (int st = 0; st < nst; st++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kLineStages - 2) : "memory");
      T *t = ring + (st % kLineStages) * (U * 4 * kLineThreads);
      if (st == 0) t[0] = T(0);  // the first row has no neighbour before it
      if (st < full) {
        T v[U][4];
#pragma unroll
        for (int j = 0; j < U; j++)
#pragma unroll
          for (int f = 0; f < 4; f++) v[j][f] = t[(4 * j + f) * kLineThreads];
        fetch(st + kLineStages - 1);
        if (len) {
#pragma unroll
          for (int j = 0; j < U; j++) eliminate(v[j][0], v[j][1], v[j][2], v[j][3]);
        }
      } else {
        for (int j = 0; j < min(U, len - st * U); j++) {
          const T *r = t + 4 * j * kLineThreads;
          eliminate(r[0], r[kLineThreads], r[2 * kLineThreads], r[3 * kLineThreads]);
        }
        fetch(st + kLineStages - 1);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (n == 1) pc = T(0);  // no c
    const T oc = __shfl_xor_sync(0xffffffffu, pc, 16), od = __shfl_xor_sync(0xffffffffu, pd, 16);
    const bool ill = __shfl_sync(0xffffffffu, worst, (lane & 15) + 16) > magnitude(T(kGrowth));
    if (__any_sync(0xffffffffu, ill)) {
      __syncwarp();  // the partner's scratch changes hands
      if (ill && !half) {
        // row i's c' and d': in this lane's scratch, from row len on in its partner's
        auto row = [&](int i) { return i < len ? cp + 2ll * i * width : cp + s.glines + 2ll * (i - len) * width; };
        T tc = T(0), td = T(0);
        for (int i = 0; i < n; i++) {
          const long long o = i * ss;
          const T ai = i ? a[o] : T(0), r = recip(b[o] - ai * tc);
          tc = c[o] * r;
          td = (d[o] - ai * td) * r;
          row(i)[0] = tc;
          row(i)[width] = td;
        }
        for (int i = n - 1; i >= 0; i--) {
          const long long o = i * ss;
          if (i < n - 1) td = row(i)[width] - row(i)[0] * td;
          if (u) u[o] += td;
          else d[o] = td;
        }
      }
      __syncwarp();
    }
    const int todo = ill ? 0 : len;  // rows still to substitute
    T xv = n > 1 ? (pd - pc * od) * recip(T(1) - pc * oc) : pd;
    // outwards, from the row before the middle
    long long out = (long long)(len - 1) * ss;
    auto put = [&](T ui) {
      if (u) __stcs(u + out, ui + xv);
      else __stcs(d + out, xv);
      out -= ss;
    };
    if (todo) put(u ? u[out] : T(0));
    q = cp + (long long)(len - 2) * 2 * width;
    struct Back {
      T c[U], d[U], u[U];
    };
    long long uo = out;
    auto back = [&](int i, Back &w) {  // rows i .. i - U + 1
      if (i >= U - 1) {
#pragma unroll
        for (int j = 0; j < U; j++) {
          w.c[j] = ld_hint(q, keep);
          w.d[j] = ld_hint(q + width, keep);
          q -= 2 * width;
        }
        if (u) {
#pragma unroll
          for (int j = 0; j < U; j++, uo -= ss) w.u[j] = __ldcs(u + uo);
        }
      } else {
#pragma unroll
        for (int j = 0; j < U; j++)
          if (i - j >= 0) {
            w.c[j] = ld_hint(q, keep);
            w.d[j] = ld_hint(q + width, keep);
            q -= 2 * width;
            if (u) w.u[j] = __ldcs(u + uo);
            uo -= ss;
          }
      }
    };
    auto substitute = [&](int i, const Back &w) {
#pragma unroll
      for (int j = 0; j < U; j++)
        if (i - j >= 0) {
          xv = w.d[j] - w.c[j] * xv;
          put(w.u[j]);
        }
    };
    Back w0, w1;
    back(todo - 2, w0);
    for (int i = todo - 2; i >= 0; i -= 2 * U) {
      back(i - U, w1);
      substitute(i, w0);
      back(i - 2 * U, w0);
      substitute(i - U, w1);
    }
  }
}

// Short lines in great number. A group of the line kernel costs the latency of
// its stages and exchanges however few its rows are, and an SM has few groups
// in flight. Here a thread solves a line, from the top: its 4 N coefficients are
// all loaded at once, c' and d' take their place in registers, and nothing else
// moves. 1,000,000 lines, FP64: of 3 rows 24 us against 135 in the line kernel, of
// 7 rows 61 against 163, of 16 rows 118 against 182; FP32 of 7 rows 28 against 114,
// of 32 rows 159 against 193. In FP64 20 rows no longer fit the registers (_Inc 295
// us against 257).
template <class T>
constexpr int kShortRows = sizeof(T) == 4 ? 32 : 16;
// From a line for every thread of a CTA an SM on, and any number where no line of
// the batch is longer than 8 rows; fewer lines of more rows are faster with the
// line kernel's two lanes each, and a second launch for them would cost more.
constexpr long long kShortLines = 148LL * kLineThreads;

template <class T, int N>
__global__ void __launch_bounds__(kLineThreads) trid_short_kernel(const Sys *__restrict__ sys, int nsys,
                                                                  long long lines) {
  for (long long g = (long long)blockIdx.x * kLineThreads + threadIdx.x; g < lines;
       g += (long long)gridDim.x * kLineThreads) {
    int lo = 0, hi = nsys - 1;  // last system whose first line is <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sys[mid].line0 <= g) lo = mid;
      else hi = mid - 1;
    }
    const Sys &s = sys[lo];
    const long long l = g - s.line0, base = (l % s.nl0) * s.s0 + (l / s.nl0) * s.s1, ss = s.ss;
    const int n = s.n;
    const T *a = reinterpret_cast<const T *>(s.a) + base, *b = reinterpret_cast<const T *>(s.b) + base;
    const T *c = reinterpret_cast<const T *>(s.c) + base;
    T *d = reinterpret_cast<T *>(s.d) + base;
    T *u = s.u ? reinterpret_cast<T *>(s.u) + base : nullptr;
    T v[N][4];
#pragma unroll
    for (int i = 0; i < N; i++)
      if (i < n) {
        v[i][0] = i ? __ldcs(a + i * ss) : T(0);
        v[i][1] = __ldcs(b + i * ss);
        v[i][2] = __ldcs(c + i * ss);
        v[i][3] = __ldcs((const T *)d + i * ss);
      }
    T cp[N], dp[N], x = T(0), pc = T(0);
#pragma unroll
    for (int i = 0; i < N; i++)
      if (i < n) {
        T r;
        recip_times(v[i][1] - v[i][0] * pc, v[i][2], r, pc);
        x = (v[i][3] - v[i][0] * x) * r;
        cp[i] = pc;
        dp[i] = x;
      }
    // x is the last row's
    if (!u) {
#pragma unroll
      for (int i = N - 1; i >= 0; i--) {
        if (i < n - 1) x = dp[i] - cp[i] * x;
        if (i < n) __stcs(d + i * ss, x);
      }
      continue;
    }
    T w[N];
#pragma unroll
    for (int i = 0; i < N; i++)
      if (i < n) w[i] = __ldcs(u + i * ss);
#pragma unroll
    for (int i = N - 1; i >= 0; i--) {
      if (i < n - 1) x = dp[i] - cp[i] * x;
      if (i < n) __stcs(u + i * ss, w[i] + x);
    }
  }
}

// Device copies of the work description, grown as needed.
struct Buffers {
  Sys *sys = nullptr;
  Work *work = nullptr;
  size_t sys_cap = 0, work_cap = 0;
  void *scr = nullptr;  // c' and d' of the lines in flight
  size_t scr_bytes = 0;
};
Buffers &buffers() {
  static Buffers b;
  return b;
}

// Threads of trid_line_kernel<T, U> that an SM holds.
template <class T, int U>
int line_threads() {
  static int per_sm = 0;
  if (!per_sm) {
    int k = 0;
    OPSB_CUDA(cudaFuncSetAttribute(trid_line_kernel<T, U>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kLineSmem<T, U>));
    OPSB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, trid_line_kernel<T, U>, kLineThreads,
                                                            kLineSmem<T, U>));
    per_sm = std::max(k, 1) * kLineThreads;
  }
  return per_sm;
}

// Groups of a system's entry of the line kernel.
long long groups_of(const Sys &s) { return s.glines == 16 ? (long long)s.nl0 * s.nl1 / 16 : 1ll; }

// The line kernel over `live`, whose entries are on the device.
template <class T, int U>
void launch_groups(const std::vector<Sys> &live, long long groups, int maxn, cudaStream_t stream) {
  // threads: what is resident, no more than kScratchBytes hold half lines for
  // (but a CTA an SM at least), nor than there are groups
  const int rows = (maxn + 1) / 2;
  const size_t line = 2 * sizeof(T) * (size_t)rows;
  const long long fit = (long long)(kScratchBytes / line) / 148 / kLineThreads * kLineThreads;
  long long slots = 148 * std::max<long long>(kLineThreads, std::min<long long>(line_threads<T, U>(), fit));
  slots = std::min(slots, (32 * groups + kLineThreads - 1) / kLineThreads * kLineThreads);
  long long elems = 0, left = slots / 32;  // the first group's scratch of every warp
  for (const Sys &s : live) {
    elems += std::min(left, groups_of(s)) * group_scratch(s.n, s.glines);
    left -= std::min(left, groups_of(s));
  }
  const size_t need = (size_t)elems * sizeof(T);
  Buffers &B = buffers();
  if (B.scr_bytes < need) {
    if (B.scr) cudaFree(B.scr);
    B.scr = nullptr;
    B.scr_bytes = 0;
    OPSB_CUDA(cudaMalloc(&B.scr, need));
    B.scr_bytes = need;
  }
  trid_line_kernel<T, U><<<(unsigned)(slots / kLineThreads), kLineThreads, kLineSmem<T, U>, stream>>>(
      B.sys, (int)live.size(), groups, static_cast<T *>(B.scr));
  OPSB_CUDA(cudaGetLastError());
}

// The y/z sweeps (solve dimension strided, lines contiguous) by the line kernel,
// and in great number the short ones by a launch of their own; returns false
// when some system does not have that shape.
template <class T>
bool launch_lines(const std::vector<Sys> &systems, cudaStream_t stream, long long *kernels) {
  std::vector<Sys> live, shorts;  // systems with no rows or no lines take no part
  long long short_lines = 0;
  int maxn = 0, short_n = 0;
  for (const Sys &s : systems) {
    if (s.ss == 1 || s.s0 != 1) return false;
    const long long nl = (long long)s.nl0 * s.nl1;
    if (s.n <= 0 || s.n > kShortRows<T> || nl <= 0) continue;
    shorts.push_back(s);
    shorts.back().line0 = short_lines;
    short_lines += nl;
    short_n = std::max(short_n, s.n);
  }
  bool longer = false;
  for (const Sys &s : systems) longer |= s.n > 8;
  if (short_lines < kShortLines && longer) shorts.clear();
  for (const Sys &s : systems) {
    const long long nl = (long long)s.nl0 * s.nl1;
    if (s.n <= 0 || nl <= 0 || (s.n <= kShortRows<T> && !shorts.empty())) continue;
    maxn = std::max(maxn, s.n);
    for (int lines : {16, (int)(nl % 16)}) {
      if (lines == 0 || nl < lines) continue;
      live.push_back(s);
      live.back().glines = lines;
      live.back().lofs = lines == 16 ? 0 : nl - nl % 16;
    }
  }
  if (live.empty() && shorts.empty()) return true;
  // the groups that need the most scratch first: a warp's first group then
  // sizes its part of it, so that all of it is never more than every line's c' and d'
  std::stable_sort(live.begin(), live.end(), [](const Sys &x, const Sys &y) {
    return group_scratch(x.n, x.glines) > group_scratch(y.n, y.glines);
  });
  long long groups = 0, all = 0;
  for (Sys &s : live) {
    s.line0 = groups;
    s.scr0 = all;
    groups += groups_of(s);
    all += groups_of(s) * group_scratch(s.n, s.glines);
  }
  const int nlive = (int)live.size(), nshort = (int)shorts.size();
  live.insert(live.end(), shorts.begin(), shorts.end());
  Buffers &B = buffers();
  if (B.sys_cap < live.size()) {
    if (B.sys) cudaFree(B.sys);
    B.sys = nullptr;
    B.sys_cap = 0;
    const size_t cap = std::max<size_t>(live.size(), 64);
    OPSB_CUDA(cudaMalloc(&B.sys, cap * sizeof(Sys)));
    B.sys_cap = cap;
  }
  OPSB_CUDA(cudaMemcpyAsync(B.sys, live.data(), live.size() * sizeof(Sys), cudaMemcpyHostToDevice, stream));
  live.resize(nlive);
  if (nshort) {
    const Sys *at = B.sys + nlive;
    const unsigned grid = (unsigned)std::min<long long>((short_lines + kLineThreads - 1) / kLineThreads, 1 << 20);
    if (short_n <= 2) trid_short_kernel<T, 2><<<grid, kLineThreads, 0, stream>>>(at, nshort, short_lines);
    else if (short_n <= 4) trid_short_kernel<T, 4><<<grid, kLineThreads, 0, stream>>>(at, nshort, short_lines);
    else if (short_n <= 8) trid_short_kernel<T, 8><<<grid, kLineThreads, 0, stream>>>(at, nshort, short_lines);
    else if (short_n <= 12) trid_short_kernel<T, 12><<<grid, kLineThreads, 0, stream>>>(at, nshort, short_lines);
    else if (short_n <= 16) trid_short_kernel<T, 16><<<grid, kLineThreads, 0, stream>>>(at, nshort, short_lines);
    else trid_short_kernel<T, kShortRows<T>><<<grid, kLineThreads, 0, stream>>>(at, nshort, short_lines);
    OPSB_CUDA(cudaGetLastError());
    if (kernels) (*kernels)++;
    if (!nlive) return true;
  }
  // a wave of the kernel with U = 8: line_threads<T, 8>() / 32 groups an SM
  if (maxn <= kFewRows && groups > 148LL * (line_threads<T, 8>() / 32))
    launch_groups<T, 4>(live, groups, maxn, stream);
  else
    launch_groups<T, 8>(live, groups, maxn, stream);
  if (kernels) (*kernels)++;
  return true;
}

// "trid_warp" option: -1 and 1 use the warp kernel whenever it applies, 0 never.
int &warp_mode() {
  static int m = -1;
  return m;
}
void set_warp_mode(int m) {
  if (m < -1 || m > 1) throw Error(E_ARG, "trid_warp must be -1, 0 or 1");
  warp_mode() = m;
}

template <class T, int R, int FP>
void launch_warp(const Buffers &B, int nwork, cudaStream_t stream) {
  const int smem = (int)(kWarpLines * 4 * warp_strip<R>(0) * sizeof(T));
  static int occupancy = 0;  // CTAs per SM, per instantiation
  if (occupancy == 0) {
    OPSB_CUDA(cudaFuncSetAttribute(trid_warp_kernel<T, R, FP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    OPSB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occupancy, trid_warp_kernel<T, R, FP>,
                                                            32 * kWarpLines, smem));
    occupancy = std::max(occupancy, 1);
  }
  const int grid = std::min(nwork, 148 * occupancy);
  trid_warp_kernel<T, R, FP><<<grid, 32 * kWarpLines, smem, stream>>>(B.sys, B.work, nwork);
  OPSB_CUDA(cudaGetLastError());
}

template <class T>
void launch(const std::vector<Sys> &systems, int solvedim, cudaStream_t stream, long long *kernels) {
  (void)solvedim;
  int maxn = 0;
  for (const Sys &s : systems) maxn = std::max(maxn, s.n);
  if (maxn == 0) return;
  if (launch_lines<T>(systems, stream, kernels)) return;
  bool contig = true;
  for (const Sys &s : systems) contig = contig && (s.n == 0 || s.ss == 1);
  // x sweeps of lines up to 256 rows: a warp per 1, 2 or 4 lines
  // (trid_warp_kernel); longer lines, or the option set to 0, take the tile
  // kernel
  const int wm = warp_mode();
  const bool warp_path = contig && maxn <= 256 && wm != 0;
  const int wR = maxn <= 128 ? 4 : 8;  // rows per lane of the warp kernel
  // tile kernel: lines per work item, the largest power of two (<= 64) whose tiles fit
  int L = 64;
  if (!warp_path) {
    while (L > 1 && tile_smem<T>(L, maxn) > kTileSmem) L /= 2;
    if (tile_smem<T>(L, maxn) > kTileSmem) throw Error(E_UNSUPPORTED, "tridiagonal lines longer than the tile budget");
  }
  std::vector<Work> work;
  for (int i = 0; i < (int)systems.size(); i++) {
    const Sys &s = systems[i];
    if (s.n == 0) continue;
    // warp kernel: a CTA's warps take kWarpLines x (lines per warp) lines
    const int Ls = warp_path ? kWarpLines * (32 / lanes_per_line(s.n, wR)) : L;
    for (int l1 = 0; l1 < s.nl1; l1++)
      for (int l0 = 0; l0 < s.nl0; l0 += Ls) work.push_back({i, l0, l1});
  }
  if (work.empty()) return;
  Buffers &B = buffers();
  if (B.sys_cap < systems.size()) {
    if (B.sys) cudaFree(B.sys);
    B.sys_cap = std::max<size_t>(systems.size(), 64);
    OPSB_CUDA(cudaMalloc(&B.sys, B.sys_cap * sizeof(Sys)));
  }
  if (B.work_cap < work.size()) {
    if (B.work) cudaFree(B.work);
    B.work_cap = std::max<size_t>(work.size() * 2, 4096);
    OPSB_CUDA(cudaMalloc(&B.work, B.work_cap * sizeof(Work)));
  }
  OPSB_CUDA(cudaMemcpyAsync(B.sys, systems.data(), systems.size() * sizeof(Sys), cudaMemcpyHostToDevice, stream));
  OPSB_CUDA(cudaMemcpyAsync(B.work, work.data(), work.size() * sizeof(Work), cudaMemcpyHostToDevice, stream));
  const int nwork = (int)work.size();
  if (warp_path) {
    bool full = true;  // every line needs all 32 lanes
    for (const Sys &s : systems) full = full && (s.n == 0 || lanes_per_line(s.n, wR) == 32);
    if (wR == 4)
      full ? launch_warp<T, 4, 32>(B, nwork, stream) : launch_warp<T, 4, 0>(B, nwork, stream);
    else
      full ? launch_warp<T, 8, 32>(B, nwork, stream) : launch_warp<T, 8, 0>(B, nwork, stream);
    if (kernels) (*kernels)++;
    return;
  }
  const size_t smem = tile_smem<T>(L, maxn);
  static size_t attr_set = 0;
  if (smem > attr_set) {
    OPSB_CUDA(cudaFuncSetAttribute(trid_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set = smem;
  }
  const int per_sm = std::max(1, std::min(kCtasPerSm, (int)(233472 / (smem + 1024))));
  const int grid = std::min(nwork, 148 * per_sm);
  trid_tile_kernel<T><<<grid, kTileThreads, smem, stream>>>(B.sys, B.work, nwork, L, maxn);
  OPSB_CUDA(cudaGetLastError());
  if (kernels) (*kernels)++;
}

// Line geometry of a Tridsolver-style strided array: dims (solved extents)
// and pads (allocated extents; element (i,j,k) at i + j*pads[0] + k*pads[0]*pads[1]).
Sys make_sys(const void *a, const void *b, const void *c, void *d, void *u, int ndim, int solvedim, const int *dims,
             const int *pads) {
  if (ndim < 1 || ndim > 3 || solvedim < 0 || solvedim >= ndim) throw Error(E_ARG, "bad ndim/solvedim");
  long long stride[3] = {1, 1, 1};
  for (int k = 1; k < 3; k++) stride[k] = stride[k - 1] * (k - 1 < ndim ? pads[k - 1] : 1);
  Sys s;
  s.a = (const char *)a; s.b = (const char *)b; s.c = (const char *)c;
  s.d = (char *)d; s.u = (char *)u;
  s.n = dims[solvedim];
  s.ss = stride[solvedim];
  int other[2], no = 0;
  for (int k = 0; k < ndim; k++)
    if (k != solvedim) other[no++] = k;
  s.nl0 = no > 0 ? dims[other[0]] : 1;
  s.s0 = no > 0 ? stride[other[0]] : 0;
  s.nl1 = no > 1 ? dims[other[1]] : 1;
  s.s1 = no > 1 ? stride[other[1]] : 0;
  for (int k = 0; k < ndim; k++)
    if (dims[k] < 0 || pads[k] < dims[k]) throw Error(E_ARG, "tridiagonal dims must satisfy 0 <= dims <= pads");
  return s;
}

}  // namespace trid

int capi_guard(const std::function<int()> &f);

// ops_tridMultiDimBatch(_Inc) on dats (ops/c/src/tridiag/ops_tridiag.cpp:78-249).
static int trid_dats(int ndim, int solvedim, const int *range, int a, int b, int c, int d, int u) {
  return capi_guard([&] {
    if (!Runtime::exists()) throw Error(E_STATE, "ops_b200_init has not been called");
    Runtime &r = Runtime::get();
    if (!range) throw Error(E_ARG, "range required");
    Dat &A = r.dat(a), &B = r.dat(b), &C = r.dat(c), &Dd = r.dat(d);
    Dat *U = u >= 0 ? &r.dat(u) : nullptr;
    // a line solve needs its whole line on one GPU: no partitioned dats
    if (A.split >= 0 || B.split >= 0 || C.split >= 0 || Dd.split >= 0 || (U && U->split >= 0))
      throw Error(E_UNSUPPORTED, "Tridsolver: dats partitioned across ranks are not supported");
    for (int i = 0; i < 3; i++)
      if (A.size[i] != B.size[i] || B.size[i] != C.size[i] || C.size[i] != Dd.size[i] ||
          (U && U->size[i] != A.size[i]))
        throw Error(E_ARG, "Tridsolver error: the a,b,c,d datasets all need to be the same size");
    if (A.type != B.type || B.type != C.type || C.type != Dd.type || (U && U->type != A.type))
      throw Error(E_ARG, "Tridsolver error: the a,b,c,d datasets must all be of the same type");
    if (A.type != "double" && A.type != "float")
      throw Error(E_UNSUPPORTED, "Tridsolver error: unsupported type. Dataset type must either be \"double\" or \"float\"");
    if (A.pitch != B.pitch || A.pitch != C.pitch || A.pitch != Dd.pitch || (U && U->pitch != A.pitch))
      throw Error(E_ARG, "tridiagonal dats must share one layout");
    r.execute();  // the reference takes raw pointers, which flushes the queue
    int dims[3], pads[3] = {(int)A.pitch, A.size[1], A.size[2]};
    long long offset = 0;
    for (int i = 0; i < ndim; i++) {
      dims[i] = range[2 * i + 1] - range[2 * i];
      if (dims[i] < 0) throw Error(E_ARG, "empty or inverted range");
    }
    offset = range[0] + (ndim > 1 ? (long long)range[2] * A.pitch : 0) + (ndim > 2 ? (long long)range[4] * A.plane : 0);
    const size_t es = A.elem_size;
    auto P = [&](Dat &x) { return x.origin_ptr() + offset * es; };
    std::vector<trid::Sys> sys = {trid::make_sys(P(A), P(B), P(C), P(Dd), U ? P(*U) : nullptr, ndim, solvedim, dims, pads)};
    long long k = 0;
    if (es == 8) trid::launch<double>(sys, solvedim, r.stream(), &k);
    else trid::launch<float>(sys, solvedim, r.stream(), &k);
    r.count_kernels(k);
    return 0;
  });
}

}  // namespace opsb

extern "C" int ops_b200_tridMultiDimBatch(int ndim, int solvedim, const int *range, int a, int b, int c, int d) {
  return opsb::trid_dats(ndim, solvedim, range, a, b, c, d, -1);
}

extern "C" int ops_b200_tridMultiDimBatch_Inc(int ndim, int solvedim, const int *range, int a, int b, int c, int d,
                                              int u) {
  return opsb::trid_dats(ndim, solvedim, range, a, b, c, d, u);
}

extern "C" int ops_b200_trid_batch(int elem_size, int solvedim, int nsys, const ops_b200_trid_system *systems,
                                   void *stream) {
  using namespace opsb;
  return capi_guard([&] {
    if (elem_size != 8 && elem_size != 4) throw Error(E_ARG, "elem_size must be 8 (double) or 4 (float)");
    if (nsys < 0 || (nsys > 0 && !systems)) throw Error(E_ARG, "bad system list");
    std::vector<trid::Sys> sys;
    for (int i = 0; i < nsys; i++) {
      const ops_b200_trid_system &t = systems[i];
      if (!t.a || !t.b || !t.c || !t.d) throw Error(E_ARG, "a, b, c and d are required");
      sys.push_back(trid::make_sys(t.a, t.b, t.c, t.d, t.u, t.ndim, solvedim, t.dims, t.pads));
    }
    long long k = 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (elem_size == 8) trid::launch<double>(sys, solvedim, s, &k);
    else trid::launch<float>(sys, solvedim, s, &k);
    if (Runtime::exists()) Runtime::get().count_kernels(k);
    return 0;
  });
}
