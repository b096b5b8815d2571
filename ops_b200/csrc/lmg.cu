// Learned multigrid preconditioner: network, training step and application
// (see lmg.h for the architecture). The 3x3 convolutions, forward and
// input-gradient, run on the tcgen05 kernel of conv_tc.cu; the input gradient
// of a convolution is the convolution of the output gradient with the
// weights flipped in space and transposed in channels. Everything else is
// bandwidth-bound elementwise work on CUDA cores, NHWC with 8 channels
// (16 bytes) per thread. Weight gradients are per-CTA partial sums added in
// a fixed order, so a training step is reproducible run to run.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "conv_tc.cuh"
#include "lmg.h"
#include "runtime.h"

namespace opsb {
namespace cnn {
int *error_word();
}
namespace lmg {
namespace {

struct LayerDef {
  int cin, cout;
};
constexpr LayerDef kDefs[kLayers] = {{16, 16}, {16, 32}, {32, 32}, {32, 64}, {64, 64},
                                     {64, 64}, {64, 64}, {64, 32}, {32, 16}, {16, 16}};
enum { C0 = 0, C1A, C1B, C2A, C2B, C3A, C3B, C2U, C1U, C0U };
constexpr int kFeat = 16;   // input channels (5 used)
constexpr int kT = 256;     // threads of the elementwise kernels
constexpr int kWgX = 128;   // pixel groups of the weight-gradient kernel
constexpr int kWgTile = 128;  // pixels per weight-gradient tile (16 x 8)

using bf16 = __nv_bfloat16;

struct Offsets {
  int w[kLayers], b[kLayers], wout, bout, total;
  Offsets() {
    int o = 0;
    for (int l = 0; l < kLayers; l++) {
      w[l] = o;
      o += 9 * kDefs[l].cin * kDefs[l].cout;
      b[l] = o;
      o += kDefs[l].cout;
    }
    wout = o;
    o += 16;
    bout = o;
    o += 1;
    total = o;
  }
};
const Offsets &offs() {
  static Offsets o;
  return o;
}

__device__ __forceinline__ void ld8(const bf16 *p, float *v) {
  uint4 u = *reinterpret_cast<const uint4 *>(p);
  const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    float2 f = __bfloat1622float2(h[k]);
    v[2 * k] = f.x;
    v[2 * k + 1] = f.y;
  }
}
__device__ __forceinline__ void st8(bf16 *p, const float *v) {
  uint4 u;
  __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
  for (int k = 0; k < 4; k++) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
  *reinterpret_cast<uint4 *>(p) = u;
}

__device__ __forceinline__ double block_sum_d(double v, double *sm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sm[wid] = v;
  __syncthreads();
  v = 0.0;
  if (wid == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sm[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// Face weights and diagonal of A at interior cell (x, y) of image n.
struct Coef {
  double a, b, c, d, D;
};
__device__ __forceinline__ Coef coef(const Fields &f, int n, int y, int x) {
  const long long i = n * f.image + (long long)y * f.pitch + x;
  Coef k;
  k.a = f.rx * f.Kx[i];
  k.b = f.rx * f.Kx[i + 1];
  k.c = f.ry * f.Ky[i];
  k.d = f.ry * f.Ky[i + f.pitch];
  k.D = 1.0 + k.a + k.b + k.c + k.d;
  return k;
}

// Per image, per block: partial sums of r^2.
__global__ void k_zsq(Fields f, double *part) {
  __shared__ double sm[kT / 32];
  const int n = blockIdx.y;
  const int hw = f.h * f.w;
  double acc = 0.0;
  for (int p = blockIdx.x * kT + threadIdx.x; p < hw; p += gridDim.x * kT) {
    const int y = p / f.w, x = p - y * f.w;
    const double r = f.r[n * f.image + (long long)y * f.pitch + x];
    acc += r * r;
  }
  acc = block_sum_d(acc, sm);
  if (threadIdx.x == 0) part[n * gridDim.x + blockIdx.x] = acc;
}

// s[n] = rms(r) (1 when the residual is zero), partials added in block order.
__global__ void k_scale(const double *part, int nblk, int hw, double *s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double t = 0.0;
  for (int b = 0; b < nblk; b++) t += part[i * nblk + b];
  const double v = sqrt(t / (double)hw);
  s[i] = v > 0.0 ? v : 1.0;
}

__global__ void k_features(Fields f, const double *s, bf16 *x0) {
  const long long total = (long long)f.n * f.h * f.w;
  for (long long p = (long long)blockIdx.x * kT + threadIdx.x; p < total; p += (long long)gridDim.x * kT) {
    const int n = (int)(p / ((long long)f.h * f.w));
    const int rem = (int)(p - (long long)n * f.h * f.w);
    const int y = rem / f.w, x = rem - y * f.w;
    const Coef k = coef(f, n, y, x);
    float v[16] = {0};
    v[0] = (float)(f.r[n * f.image + (long long)y * f.pitch + x] / s[n]);
    v[1] = (float)(k.a / k.D);
    v[2] = (float)(k.b / k.D);
    v[3] = (float)(k.c / k.D);
    v[4] = (float)(k.d / k.D);
    st8(x0 + p * kFeat, v);
    st8(x0 + p * kFeat + 8, v + 8);
  }
}

// 2x2 average pooling, C channels.
__global__ void k_pool(const bf16 *in, bf16 *out, int n, int h, int w, int C) {
  const int h2 = h / 2, w2 = w / 2, g = C / 8;
  const long long total = (long long)n * h2 * w2 * g;
  for (long long t = (long long)blockIdx.x * kT + threadIdx.x; t < total; t += (long long)gridDim.x * kT) {
    const int cg = (int)(t % g);
    long long p = t / g;
    const int X = (int)(p % w2);
    p /= w2;
    const int Y = (int)(p % h2);
    const int img = (int)(p / h2);
    float acc[8] = {0}, v[8];
    for (int dy = 0; dy < 2; dy++)
      for (int dx = 0; dx < 2; dx++) {
        ld8(in + (((long long)img * h + 2 * Y + dy) * w + 2 * X + dx) * C + cg * 8, v);
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] += v[k];
      }
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] *= 0.25f;
    st8(out + (((long long)img * h2 + Y) * w2 + X) * C + cg * 8, acc);
  }
}

// out = up2(coarse) + skip, fine grid n x h x w, C channels.
__global__ void k_up_add(const bf16 *coarse, const bf16 *skip, bf16 *out, int n, int h, int w, int C) {
  const int g = C / 8;
  const long long total = (long long)n * h * w * g;
  for (long long t = (long long)blockIdx.x * kT + threadIdx.x; t < total; t += (long long)gridDim.x * kT) {
    const int cg = (int)(t % g);
    long long p = t / g;
    const int x = (int)(p % w);
    p /= w;
    const int y = (int)(p % h);
    const int img = (int)(p / h);
    float a[8], b[8];
    ld8(coarse + (((long long)img * (h / 2) + y / 2) * (w / 2) + x / 2) * C + cg * 8, a);
    const long long fi = (((long long)img * h + y) * w + x) * C + cg * 8;
    ld8(skip + fi, b);
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] += b[k];
    st8(out + fi, a);
  }
}

// Gradient through up2: coarse (n, h/2, w/2) = sum of its four children,
// times (mask > 0) (the ReLU of the layer that produced the coarse tensor).
__global__ void k_upT_mask(const bf16 *fine, const bf16 *mask, bf16 *out, int n, int h, int w, int C) {
  const int h2 = h / 2, w2 = w / 2, g = C / 8;
  const long long total = (long long)n * h2 * w2 * g;
  for (long long t = (long long)blockIdx.x * kT + threadIdx.x; t < total; t += (long long)gridDim.x * kT) {
    const int cg = (int)(t % g);
    long long p = t / g;
    const int X = (int)(p % w2);
    p /= w2;
    const int Y = (int)(p % h2);
    const int img = (int)(p / h2);
    float acc[8] = {0}, v[8], m[8];
    for (int dy = 0; dy < 2; dy++)
      for (int dx = 0; dx < 2; dx++) {
        ld8(fine + (((long long)img * h + 2 * Y + dy) * w + 2 * X + dx) * C + cg * 8, v);
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] += v[k];
      }
    const long long ci = (((long long)img * h2 + Y) * w2 + X) * C + cg * 8;
    ld8(mask + ci, m);
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] = m[k] > 0.0f ? acc[k] : 0.0f;
    st8(out + ci, acc);
  }
}

// out = (a + 0.25 * up2(b)) * (mask > 0): the gradient reaching a tensor that
// feeds both a skip connection (a) and a 2x2 average pool (b, coarse).
__global__ void k_add_poolT_mask(const bf16 *a, const bf16 *b, const bf16 *mask, bf16 *out, int n, int h, int w,
                                 int C) {
  const int g = C / 8;
  const long long total = (long long)n * h * w * g;
  for (long long t = (long long)blockIdx.x * kT + threadIdx.x; t < total; t += (long long)gridDim.x * kT) {
    const int cg = (int)(t % g);
    long long p = t / g;
    const int x = (int)(p % w);
    p /= w;
    const int y = (int)(p % h);
    const int img = (int)(p / h);
    const long long fi = (((long long)img * h + y) * w + x) * C + cg * 8;
    float va[8], vb[8], m[8];
    ld8(a + fi, va);
    ld8(b + (((long long)img * (h / 2) + y / 2) * (w / 2) + x / 2) * C + cg * 8, vb);
    ld8(mask + fi, m);
#pragma unroll
    for (int k = 0; k < 8; k++) va[k] = m[k] > 0.0f ? va[k] + 0.25f * vb[k] : 0.0f;
    st8(out + fi, va);
  }
}

// Output layer: y = wout . h0 + bout; M(r) = z + s y. Writes M(r) to `out`
// (FP64, field layout) and/or the prediction to `pred` (FP32, dense n*h*w).
__global__ void k_out(Fields f, const double *s, const bf16 *h0, const float *params, int wout_off,
                      double *out, long long out_image, long long out_pitch, float *pred) {
  __shared__ float wsm[17];
  if (threadIdx.x < 17) wsm[threadIdx.x] = params[wout_off + threadIdx.x];
  __syncthreads();
  const long long total = (long long)f.n * f.h * f.w;
  for (long long p = (long long)blockIdx.x * kT + threadIdx.x; p < total; p += (long long)gridDim.x * kT) {
    const int n = (int)(p / ((long long)f.h * f.w));
    const int rem = (int)(p - (long long)n * f.h * f.w);
    const int y = rem / f.w, x = rem - y * f.w;
    float v[16];
    ld8(h0 + p * 16, v);
    ld8(h0 + p * 16 + 8, v + 8);
    float acc = wsm[16];
#pragma unroll
    for (int c = 0; c < 16; c++) acc += wsm[c] * v[c];
    const Coef k = coef(f, n, y, x);
    const double z = f.r[n * f.image + (long long)y * f.pitch + x] / k.D;
    const double m = z + s[n] * (double)acc;
    if (out) out[n * out_image + (long long)y * out_pitch + x] = m;
    if (pred) pred[p] = (float)m;
  }
}

// d = pred - e in place (FP32, dense n x h x w); per-image partials of d.d
// and e.e (the L2 loss).
__global__ void k_diff(Fields f, float *pd, const double *e, double *part) {
  __shared__ double sm[kT / 32];
  const int n = blockIdx.y, hw = f.h * f.w;
  double a = 0.0, b = 0.0;
  for (int p = blockIdx.x * kT + threadIdx.x; p < hw; p += gridDim.x * kT) {
    const int y = p / f.w, x = p - y * f.w;
    const double ev = e[n * f.image + (long long)y * f.pitch + x];
    const double d = (double)pd[(long long)n * hw + p] - ev;
    pd[(long long)n * hw + p] = (float)d;
    a += d * d;
    b += ev * ev;
  }
  a = block_sum_d(a, sm);
  b = block_sum_d(b, sm);
  if (threadIdx.x == 0) {
    part[(n * gridDim.x + blockIdx.x) * 2] = a;
    part[(n * gridDim.x + blockIdx.x) * 2 + 1] = b;
  }
}

// A-norm loss: G = A d (the heat operator on the interior, d zero outside)
// and per-image partials of d.(A d) and e.(A e).
__global__ void k_anorm(Fields f, const float *d, const double *e, float *G, double *part) {
  __shared__ double sm[kT / 32];
  const int n = blockIdx.y, hw = f.h * f.w;
  const float *dn = d + (long long)n * hw;
  double a = 0.0, b = 0.0;
  for (int p = blockIdx.x * kT + threadIdx.x; p < hw; p += gridDim.x * kT) {
    const int y = p / f.w, x = p - y * f.w;
    const Coef k = coef(f, n, y, x);
    const double dc = dn[p];
    const double dw = x > 0 ? dn[p - 1] : 0.0, de = x + 1 < f.w ? dn[p + 1] : 0.0;
    const double ds = y > 0 ? dn[p - f.w] : 0.0, dnn = y + 1 < f.h ? dn[p + f.w] : 0.0;
    const double Ad = k.D * dc - k.a * dw - k.b * de - k.c * ds - k.d * dnn;
    const long long i = n * f.image + (long long)y * f.pitch + x;
    const double Ae = k.D * e[i] - k.a * e[i - 1] - k.b * e[i + 1] - k.c * e[i - f.pitch] - k.d * e[i + f.pitch];
    G[(long long)n * hw + p] = (float)Ad;
    a += dc * Ad;
    b += e[i] * Ae;
  }
  a = block_sum_d(a, sm);
  b = block_sum_d(b, sm);
  if (threadIdx.x == 0) {
    part[(n * gridDim.x + blockIdx.x) * 2] = a;
    part[(n * gridDim.x + blockIdx.x) * 2 + 1] = b;
  }
}

// Per image: E[n] = ||e||^2 (or e.Ae); loss = mean_n d.d / E[n] (or d.Ad /
// E[n]). One block, an image a thread, its partials added in block order with
// their loads ahead (one thread for everything took 38 us of a 16 x 64^2 step);
// the images' ratios, left in `part`, are added in order too.
__global__ void k_loss_finish(double *part, int nblk, int n, double *E, double *loss) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double *p = part + (size_t)i * nblk * 2;
    double a = 0.0, b = 0.0;
#pragma unroll 8
    for (int k = 0; k < nblk; k++) {
      a += p[2 * k];
      b += p[2 * k + 1];
    }
    if (!(b > 0.0)) b = 1.0;
    E[i] = b;
    p[0] = a / b;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double L = 0.0;
#pragma unroll 4
  for (int i = 0; i < n; i++) L += part[(size_t)i * nblk * 2];
  *loss = L / (double)n;
}

// dL/dy = (2 / n) s G / E with G = pred - e (L2) or A (pred - e) (A-norm),
// then through the output layer: g0u = dy * wout * (h0 > 0); per-block
// partials of dwout = sum dy h0, dbout = sum dy.
__global__ void k_out_bwd(Fields f, const double *s, const double *E, const float *G, const bf16 *h0,
                          const float *params, int wout_off, bf16 *g0u, float *part) {
  __shared__ float wsm[16];
  __shared__ double sm[kT / 32];
  if (threadIdx.x < 16) wsm[threadIdx.x] = params[wout_off + threadIdx.x];
  __syncthreads();
  double acc[17];
#pragma unroll
  for (int c = 0; c < 17; c++) acc[c] = 0.0;
  const long long total = (long long)f.n * f.h * f.w;
  for (long long p = (long long)blockIdx.x * kT + threadIdx.x; p < total; p += (long long)gridDim.x * kT) {
    const int n = (int)(p / ((long long)f.h * f.w));
    const int rem = (int)(p - (long long)n * f.h * f.w);
    const int y = rem / f.w, x = rem - y * f.w;
    (void)y;
    (void)x;
    const double dm = 2.0 / (double)f.n * (double)G[p] / E[n];
    const float dy = (float)(dm * s[n]);
    float v[16], g[16];
    ld8(h0 + p * 16, v);
    ld8(h0 + p * 16 + 8, v + 8);
#pragma unroll
    for (int c = 0; c < 16; c++) {
      g[c] = v[c] > 0.0f ? dy * wsm[c] : 0.0f;
      acc[c] += (double)dy * (double)v[c];
    }
    acc[16] += (double)dy;
    st8(g0u + p * 16, g);
    st8(g0u + p * 16 + 8, g + 8);
  }
  for (int c = 0; c < 17; c++) {
    const double t = block_sum_d(acc[c], sm);
    if (threadIdx.x == 0) part[blockIdx.x * 17 + c] = (float)t;
  }
}

// Weight gradients of the 3x3 layers: dW[tap][co][ci] = sum_p g[p][co] x[p + tap][ci]
// (x zero outside the image), db[co] = sum_p g[p][co]. All layers run in one
// launch, a CTA per layer and share of the pixel tiles (and row of three taps
// where the layer has 2048 weights a tap or more); it sums its tiles in order
// and leaves partial[share][...] in W layout. A thread holds RO x RI outputs of
// three taps, so a pixel's values are loaded (one word each way) and converted
// once for 3 RO RI products; a small layer's three rows of taps go to three
// groups of 64 threads of one CTA for that, and its bias to the fourth. Bound
// by issue: a product is a multiplication and an addition. (One CTA a tap, one
// output a thread at a time and a launch a layer: 343 us of a 16 x 64^2 step;
// all layers in one launch with rows of taps in CTAs of their own 140 us; now
// 123 us.) Every output is still one chain over the pixels in the same order.
struct WgLayer {
  const bf16 *x, *g;
  float *partial;  // this layer's shares
  float *grad;
  int h, w, tiles, shares, len, first;  // first: this layer's first CTA
};
struct WgPlan {
  WgLayer l[kLayers];
  // the output layer's partials (k_out_bwd)
  const float *opart;
  float *ograd;
  int oparts;
};

// bf16 pairs of a word, exactly.
template <int N>
__device__ __forceinline__ void unpack(const bf16 *p, float (&o)[N]) {
  unsigned u[(N + 1) / 2];
  if constexpr (N == 1) {
    o[0] = __bfloat162float(*p);
    return;
  } else if constexpr (N == 2) {
    u[0] = *reinterpret_cast<const unsigned *>(p);
  } else {
    static_assert(N == 4, "one, two or four values");
    const uint2 v = *reinterpret_cast<const uint2 *>(p);
    u[0] = v.x;
    u[1] = v.y;
  }
#pragma unroll
  for (int k = 0; k < N / 2; k++) {
    o[2 * k] = __uint_as_float(u[k] << 16);
    o[2 * k + 1] = __uint_as_float(u[k] & 0xffff0000u);
  }
}

// Rows of taps that one CTA takes: all three where 64 threads hold a row's.
constexpr int wg_rows(int cin, int cout) { return cin * cout <= 1024 ? 3 : 1; }

template <int CIN, int COUT>
__device__ __forceinline__ void wgrad_share(const WgLayer &L, int b, uint4 *smem) {
  constexpr int ROWS = wg_rows(CIN, COUT), THR = ROWS == 3 ? 64 : kT;
  constexpr int NO = CIN * COUT, PER = NO / THR;
  constexpr int RI = PER >= 8 ? 4 : 2, RO = PER / RI;  // outputs a thread: RO co x RI ci
  static_assert(NO % THR == 0 && RO * RI == PER && RO >= 1 && RO <= 4, "wgrad tiling");
  constexpr int XW = 18, XH = ROWS == 3 ? 10 : 8;  // 16 pixels and a column either side; a row either side too
  bf16 *gs = reinterpret_cast<bf16 *>(smem), *xs = gs + kWgTile * COUT;
  const int share = ROWS == 3 ? b : b / 3, group = ROWS == 3 ? threadIdx.x / 64 : 0;
  const int dyi = ROWS == 3 ? group : b % 3;   // row of taps; group 3 takes the bias
  const int row0 = ROWS == 3 ? -1 : dyi - 1;   // x's first row in the tile, from the tile's
  const int h = L.h, w = L.w;
  const int tx = (w + 15) / 16, ty = (h + 7) / 8;
  const int q = threadIdx.x % THR, ci0 = (q % (CIN / RI)) * RI, co0 = (q / (CIN / RI)) * RO;
  const bool bias = ROWS == 3 ? group == 3 && q < COUT : dyi == 0 && q < COUT;
  float acc[3][RO][RI] = {}, bacc = 0.0f;
  for (int t = share; t < L.tiles; t += L.shares) {
    const int img = t / (tx * ty), rem = t - img * tx * ty;
    const int y0 = (rem / tx) * 8, x0 = (rem % tx) * 16;
    __syncthreads();
    for (int v = threadIdx.x; v < kWgTile * (COUT / 8); v += kT) {
      const int p = v / (COUT / 8), cg = v % (COUT / 8);
      const int y = y0 + p / 16, xx = x0 + p % 16;
      uint4 val = make_uint4(0, 0, 0, 0);
      if (y < h && xx < w)
        val = *reinterpret_cast<const uint4 *>(L.g + (((long long)img * h + y) * w + xx) * COUT + cg * 8);
      *reinterpret_cast<uint4 *>(gs + p * COUT + cg * 8) = val;
    }
    for (int v = threadIdx.x; v < XH * XW * (CIN / 8); v += kT) {
      const int p = v / (CIN / 8), cg = v % (CIN / 8);
      const int y = y0 + p / XW + row0, xx = x0 + p % XW - 1;
      uint4 val = make_uint4(0, 0, 0, 0);
      if (y >= 0 && y < h && xx >= 0 && xx < w)
        val = *reinterpret_cast<const uint4 *>(L.x + (((long long)img * h + y) * w + xx) * CIN + cg * 8);
      *reinterpret_cast<uint4 *>(xs + p * CIN + cg * 8) = val;
    }
    __syncthreads();
    if (group < 3) {
      for (int r = 0; r < 8; r++) {
        const bf16 *gr = gs + r * 16 * COUT + co0, *xr = xs + (r + (ROWS == 3 ? dyi : 0)) * XW * CIN + ci0;
        float x[3][RI];  // the columns left of, at and right of the pixel
        unpack<RI>(xr, x[0]);
        unpack<RI>(xr + CIN, x[1]);
#pragma unroll 4
        for (int p = 0; p < 16; p++) {
          unpack<RI>(xr + (p + 2) * CIN, x[2]);
          float g[RO];
          unpack<RO>(gr + p * COUT, g);
#pragma unroll
          for (int d = 0; d < 3; d++)
#pragma unroll
            for (int o = 0; o < RO; o++)
#pragma unroll
              for (int k = 0; k < RI; k++) acc[d][o][k] += g[o] * x[d][k];
#pragma unroll
          for (int k = 0; k < RI; k++) {
            x[0][k] = x[1][k];
            x[1][k] = x[2][k];
          }
        }
      }
    }
    if (bias)
#pragma unroll 8
      for (int p = 0; p < kWgTile; p++) bacc += __bfloat162float(gs[p * COUT + q]);
  }
  float *out = L.partial + (size_t)share * L.len;
  if (group < 3)
#pragma unroll
    for (int d = 0; d < 3; d++)
#pragma unroll
      for (int o = 0; o < RO; o++)
#pragma unroll
        for (int k = 0; k < RI; k++) out[(dyi * 3 + d) * NO + (co0 + o) * CIN + ci0 + k] = acc[d][o][k];
  if (bias) out[9 * NO + q] = bacc;
}

__global__ void __launch_bounds__(kT) k_wgrad(const __grid_constant__ WgPlan P) {
  __shared__ uint4 smem[(kWgTile * 64 + 8 * 18 * 64) / 8];  // 64 to 64 channels; the small layers' rows fit it
  int l = 0;
  while (l + 1 < kLayers && (int)blockIdx.x >= P.l[l + 1].first) l++;
  const WgLayer &L = P.l[l];
  const int b = blockIdx.x - L.first;
  switch (l) {
    case C0: case C0U: wgrad_share<16, 16>(L, b, smem); break;
    case C1A: wgrad_share<16, 32>(L, b, smem); break;
    case C1B: wgrad_share<32, 32>(L, b, smem); break;
    case C2A: wgrad_share<32, 64>(L, b, smem); break;
    case C2U: wgrad_share<64, 32>(L, b, smem); break;
    case C1U: wgrad_share<32, 16>(L, b, smem); break;
    default: wgrad_share<64, 64>(L, b, smem); break;
  }
}

// grad[i] = sum_k partial[k * len + i], k in order, eight loads ahead.
__device__ __forceinline__ float sum_parts(const float *p, int nparts, int len) {
  float t = 0.0f;
  int k = 0;
  for (; k + 8 <= nparts; k += 8) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __ldcg(p + (size_t)(k + j) * len);
#pragma unroll
    for (int j = 0; j < 8; j++) t += v[j];
  }
  for (; k < nparts; k++) t += __ldcg(p + (size_t)k * len);
  return t;
}
// Every layer's gradient from its partials, blockIdx.y = layer; the last is
// the output layer.
__global__ void k_sum_parts(const __grid_constant__ WgPlan P) {
  if (blockIdx.y == kLayers) {
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < 17) P.ograd[i] = sum_parts(P.opart + i, P.oparts, 17);
    return;
  }
  const WgLayer &L = P.l[blockIdx.y];
  for (int i = blockIdx.x * kT + threadIdx.x; i < L.len; i += gridDim.x * kT)
    L.grad[i] = sum_parts(L.partial + i, L.shares, L.len);
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, int np, float lr_t, float b1, float b2,
                       float eps) {
  for (int i = blockIdx.x * kT + threadIdx.x; i < np; i += gridDim.x * kT) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr_t * mi / (sqrtf(vi) + eps);
  }
}

// BF16 copies of every layer's weights (blockIdx.y = layer): forward
// [9][cout][cin] and, for the input gradient, flipped and transposed
// [9][cin][cout] with tap' = 8 - tap.
struct PrepPlan {
  const float *W[kLayers];
  bf16 *wf[kLayers], *wt[kLayers];
  int cin[kLayers], cout[kLayers];
};
__global__ void k_prep(const __grid_constant__ PrepPlan P) {
  const int l = blockIdx.y, cin = P.cin[l], cout = P.cout[l];
  const int total = 9 * cin * cout;
  for (int i = blockIdx.x * kT + threadIdx.x; i < total; i += gridDim.x * kT) {
    const int tap = i / (cin * cout), rem = i - tap * cin * cout;
    const int co = rem / cin, ci = rem - co * cin;
    const bf16 v = __float2bfloat16_rn(P.W[l][i]);
    P.wf[l][i] = v;
    P.wt[l][(8 - tap) * cin * cout + ci * cout + co] = v;
  }
}

int blocks_for(long long work) {
  long long b = (work + kT - 1) / kT;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

void check(cudaError_t e, const char *what) {
  if (e != cudaSuccess) throw Error(E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// SplitMix64 stream for the weight initialisation.
struct Rng {
  unsigned long long s;
  unsigned long long next() {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
  double u01() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
  double normal() { return sqrt(-2.0 * log(u01())) * cos(6.283185307179586 * u01()); }
};

}  // namespace

namespace {
// Level of each layer's grid (0 the finest), its pixel tiles, shares of them
// and length of a partial.
constexpr int kLevel[kLayers] = {0, 1, 1, 2, 2, 3, 3, 2, 1, 0};
int wg_tiles(int l, int n, int h, int w) {
  const int hl = h >> kLevel[l], wl = w >> kLevel[l];
  return n * ((wl + 15) / 16) * ((hl + 7) / 8);
}
int wg_shares(int l, int n, int h, int w) { return std::min(kWgX, wg_tiles(l, n, h, w)); }
int wg_len(int l) { return 9 * kDefs[l].cin * kDefs[l].cout + kDefs[l].cout; }
}  // namespace

struct Net::Impl {
  float *params = nullptr, *grads = nullptr, *am = nullptr, *av = nullptr;
  bf16 *wbuf = nullptr;
  bf16 *wf[kLayers] = {}, *wt[kLayers] = {};
  bool prepped = false;
  int step = 0;
  // activations for (an, ah, aw)
  int an = 0, ah = 0, aw = 0;
  char *act = nullptr;
  bf16 *x0, *e0, *u0, *h0, *p1, *a1, *e1, *u1, *h1, *p2, *a2, *e2, *u2, *h2, *p3, *a3, *h3;
  bf16 *g0u, *du0, *ge0, *g1u, *du1, *ge1, *ga1, *dp1, *g2u, *du2, *ge2, *ga2, *dp2, *g3b, *ga3, *dp3;
  float *pred = nullptr, *gbuf = nullptr, *wpart = nullptr, *opart = nullptr;
  double *dscal = nullptr;  // s[n], E[n], loss, partials
  int zblk = 0;

  ~Impl() {
    cudaFree(params);
    cudaFree(wbuf);
    cudaFree(act);
  }

  void ensure(int n, int h, int w) {
    if (n == an && h == ah && w == aw) return;
    if (h % 8 || w % 8 || h < 8 || w < 8 || n < 1) throw Error(E_ARG, "learned preconditioner: h and w must be multiples of 8");
    cudaFree(act);
    act = nullptr;
    const long long P0 = (long long)n * h * w, P1 = P0 / 4, P2 = P0 / 16, P3 = P0 / 64;
    struct B {
      bf16 **p;
      long long elems;
    };
    std::vector<B> list = {
        {&x0, P0 * 16}, {&e0, P0 * 16}, {&u0, P0 * 16}, {&h0, P0 * 16}, {&p1, P1 * 16}, {&a1, P1 * 32},
        {&e1, P1 * 32}, {&u1, P1 * 32}, {&h1, P1 * 16}, {&p2, P2 * 32}, {&a2, P2 * 64}, {&e2, P2 * 64},
        {&u2, P2 * 64}, {&h2, P2 * 32}, {&p3, P3 * 64}, {&a3, P3 * 64}, {&h3, P3 * 64}, {&g0u, P0 * 16},
        {&du0, P0 * 16}, {&ge0, P0 * 16}, {&g1u, P1 * 16}, {&du1, P1 * 32}, {&ge1, P1 * 32}, {&ga1, P1 * 32},
        {&dp1, P1 * 16}, {&g2u, P2 * 32}, {&du2, P2 * 64}, {&ge2, P2 * 64}, {&ga2, P2 * 64}, {&dp2, P2 * 32},
        {&g3b, P3 * 64}, {&ga3, P3 * 64}, {&dp3, P3 * 64}};
    size_t bytes = 0;
    for (auto &b : list) bytes += ((size_t)b.elems * 2 + 255) / 256 * 256;
    zblk = (int)std::max<long long>(1, std::min<long long>(std::min<long long>(1024, 148 * 8 / n),
                                                            (h * (long long)w + kT - 1) / kT));
    const size_t pred_b = ((size_t)P0 * 4 + 255) / 256 * 256;
    size_t wpart_n = 0;
    for (int l = 0; l < kLayers; l++) wpart_n += (size_t)wg_shares(l, n, h, w) * wg_len(l);
    const size_t wpart_b = (wpart_n * 4 + 255) / 256 * 256;
    const size_t opart_b = ((size_t)148 * 16 * 17 * 4 + 255) / 256 * 256;
    const size_t dscal_b = ((size_t)(2 * n + 1 + 2 * n * zblk) * 8 + 255) / 256 * 256;
    check(cudaMalloc(&act, bytes + 2 * pred_b + wpart_b + opart_b + dscal_b), "learned preconditioner buffers");
    char *c = act;
    for (auto &b : list) {
      *b.p = reinterpret_cast<bf16 *>(c);
      c += ((size_t)b.elems * 2 + 255) / 256 * 256;
    }
    pred = reinterpret_cast<float *>(c);
    c += pred_b;
    gbuf = reinterpret_cast<float *>(c);
    c += pred_b;
    wpart = reinterpret_cast<float *>(c);
    c += wpart_b;
    opart = reinterpret_cast<float *>(c);
    c += opart_b;
    dscal = reinterpret_cast<double *>(c);
    an = n;
    ah = h;
    aw = w;
  }
};

int Net::num_params() { return offs().total; }

Net::Net(unsigned long long seed) : m_(new Impl) {
  const Offsets &o = offs();
  check(cudaMalloc(&m_->params, (size_t)4 * o.total * 4), "learned preconditioner parameters");
  m_->grads = m_->params + o.total;
  m_->am = m_->grads + o.total;
  m_->av = m_->am + o.total;
  check(cudaMemset(m_->params, 0, (size_t)4 * o.total * 4), "learned preconditioner parameters");
  size_t wel = 0;
  for (int l = 0; l < kLayers; l++) wel += 9 * kDefs[l].cin * kDefs[l].cout;
  check(cudaMalloc(&m_->wbuf, wel * 2 * 2 + 512), "learned preconditioner weights");
  bf16 *p = m_->wbuf;
  for (int l = 0; l < kLayers; l++) {
    const int e = 9 * kDefs[l].cin * kDefs[l].cout;
    m_->wf[l] = p;
    p += e;
    m_->wt[l] = p;
    p += e;
  }
  // He-normal weights, zero biases, zero output layer (an untrained net is Jacobi)
  std::vector<float> h(o.total, 0.0f);
  Rng rng{seed};
  for (int l = 0; l < kLayers; l++) {
    const double sd = sqrt(2.0 / (9.0 * kDefs[l].cin));
    for (int i = 0; i < 9 * kDefs[l].cin * kDefs[l].cout; i++) h[o.w[l] + i] = (float)(sd * rng.normal());
  }
  set_params(h.data());
}

Net::~Net() { delete m_; }

void Net::get_params(float *host) const {
  check(cudaMemcpy(host, m_->params, (size_t)offs().total * 4, cudaMemcpyDeviceToHost), "get params");
}
void Net::get_grads(float *host) const {
  check(cudaMemcpy(host, m_->grads, (size_t)offs().total * 4, cudaMemcpyDeviceToHost), "get grads");
}
void Net::set_params(const float *host) {
  check(cudaMemcpy(m_->params, host, (size_t)offs().total * 4, cudaMemcpyHostToDevice), "set params");
  check(cudaMemset(m_->am, 0, (size_t)2 * offs().total * 4), "reset adam");
  m_->step = 0;
  m_->prepped = false;
}

namespace {
void conv(const bf16 *x, const bf16 *w, int n, int h, int wd, int cin, int cout, const float *bias, const bf16 *mask,
          bf16 *y, int mode, cudaStream_t s) {
  cudaError_t e = cnn::conv3x3(x, w, n, h, wd, cin, cout, bias, mask, y, mode, cnn::error_word(), s);
  check(e, "learned preconditioner conv3x3");
}
}  // namespace

// Forward pass through h0 (features, encoder, decoder). Returns nothing; the
// output layer is applied by the callers.
static void forward(Net::Impl &m, const Fields &f, cudaStream_t s, long long &launches) {
  const Offsets &o = offs();
  if (!m.prepped) {
    PrepPlan P;
    for (int l = 0; l < kLayers; l++) {
      P.W[l] = m.params + o.w[l];
      P.wf[l] = m.wf[l];
      P.wt[l] = m.wt[l];
      P.cin[l] = kDefs[l].cin;
      P.cout[l] = kDefs[l].cout;
    }
    k_prep<<<dim3(16, kLayers), kT, 0, s>>>(P);
    launches += 1;
    m.prepped = true;
  }
  const int n = f.n, h = f.h, w = f.w;
  double *spart = m.dscal + 2 * n + 1;
  k_zsq<<<dim3(m.zblk, n), kT, 0, s>>>(f, spart);
  k_scale<<<(n + 63) / 64, 64, 0, s>>>(spart, m.zblk, h * w, m.dscal, n);
  k_features<<<blocks_for((long long)n * h * w), kT, 0, s>>>(f, m.dscal, m.x0);
  auto B = [&](int l) { return m.params + o.b[l]; };
  const int h1 = h / 2, w1 = w / 2, h2 = h / 4, w2 = w / 4, h3 = h / 8, w3 = w / 8;
  conv(m.x0, m.wf[C0], n, h, w, 16, 16, B(C0), nullptr, m.e0, cnn::CONV_BIAS_RELU, s);
  k_pool<<<blocks_for((long long)n * h1 * w1 * 2), kT, 0, s>>>(m.e0, m.p1, n, h, w, 16);
  conv(m.p1, m.wf[C1A], n, h1, w1, 16, 32, B(C1A), nullptr, m.a1, cnn::CONV_BIAS_RELU, s);
  conv(m.a1, m.wf[C1B], n, h1, w1, 32, 32, B(C1B), nullptr, m.e1, cnn::CONV_BIAS_RELU, s);
  k_pool<<<blocks_for((long long)n * h2 * w2 * 4), kT, 0, s>>>(m.e1, m.p2, n, h1, w1, 32);
  conv(m.p2, m.wf[C2A], n, h2, w2, 32, 64, B(C2A), nullptr, m.a2, cnn::CONV_BIAS_RELU, s);
  conv(m.a2, m.wf[C2B], n, h2, w2, 64, 64, B(C2B), nullptr, m.e2, cnn::CONV_BIAS_RELU, s);
  k_pool<<<blocks_for((long long)n * h3 * w3 * 8), kT, 0, s>>>(m.e2, m.p3, n, h2, w2, 64);
  conv(m.p3, m.wf[C3A], n, h3, w3, 64, 64, B(C3A), nullptr, m.a3, cnn::CONV_BIAS_RELU, s);
  conv(m.a3, m.wf[C3B], n, h3, w3, 64, 64, B(C3B), nullptr, m.h3, cnn::CONV_BIAS_RELU, s);
  k_up_add<<<blocks_for((long long)n * h2 * w2 * 8), kT, 0, s>>>(m.h3, m.e2, m.u2, n, h2, w2, 64);
  conv(m.u2, m.wf[C2U], n, h2, w2, 64, 32, B(C2U), nullptr, m.h2, cnn::CONV_BIAS_RELU, s);
  k_up_add<<<blocks_for((long long)n * h1 * w1 * 4), kT, 0, s>>>(m.h2, m.e1, m.u1, n, h1, w1, 32);
  conv(m.u1, m.wf[C1U], n, h1, w1, 32, 16, B(C1U), nullptr, m.h1, cnn::CONV_BIAS_RELU, s);
  k_up_add<<<blocks_for((long long)n * h * w * 2), kT, 0, s>>>(m.h1, m.e0, m.u0, n, h, w, 16);
  conv(m.u0, m.wf[C0U], n, h, w, 16, 16, B(C0U), nullptr, m.h0, cnn::CONV_BIAS_RELU, s);
  check(cudaGetLastError(), "learned preconditioner forward");
  launches += 19;
}

void Net::apply(const Fields &f, double *out, cudaStream_t s) {
  m_->ensure(f.n, f.h, f.w);
  check(cudaMemsetAsync(cnn::error_word(), 0, sizeof(int), s), "conv error word");
  forward(*m_, f, s, launches_);
  k_out<<<blocks_for((long long)f.n * f.h * f.w), kT, 0, s>>>(f, m_->dscal, m_->h0, m_->params, offs().wout, out,
                                                              f.image, f.pitch, nullptr);
  check(cudaGetLastError(), "learned preconditioner output");
  launches_ += 1;
}

double Net::loss_and_grad(const Fields &f, const double *e, int kind, cudaStream_t s) {
  Impl &m = *m_;
  m.ensure(f.n, f.h, f.w);
  check(cudaMemsetAsync(cnn::error_word(), 0, sizeof(int), s), "conv error word");
  forward(m, f, s, launches_);
  const Offsets &o = offs();
  const int n = f.n, h = f.h, w = f.w;
  k_out<<<blocks_for((long long)n * h * w), kT, 0, s>>>(f, m.dscal, m.h0, m.params, o.wout, nullptr, 0, 0, m.pred);
  double *E = m.dscal + n, *loss = m.dscal + 2 * n, *lpart = m.dscal + 2 * n + 1;
  k_diff<<<dim3(m.zblk, n), kT, 0, s>>>(f, m.pred, e, lpart);
  const float *G = m.pred;
  if (kind == LOSS_ANORM) {
    k_anorm<<<dim3(m.zblk, n), kT, 0, s>>>(f, m.pred, e, m.gbuf, lpart);
    G = m.gbuf;
    launches_ += 1;
  }
  k_loss_finish<<<1, std::min(1024, (n + 31) / 32 * 32), 0, s>>>(lpart, m.zblk, n, E, loss);
  const int ob = blocks_for((long long)n * h * w);
  k_out_bwd<<<ob, kT, 0, s>>>(f, m.dscal, E, G, m.h0, m.params, o.wout, m.g0u, m.opart);
  launches_ += 5;
  const int h1 = h / 2, w1 = w / 2, h2 = h / 4, w2 = w / 4, h3 = h / 8, w3 = w / 8;
  // input gradients (tensor cores, flipped/transposed weights)
  conv(m.g0u, m.wt[C0U], n, h, w, 16, 16, nullptr, nullptr, m.du0, cnn::CONV_PLAIN, s);
  k_upT_mask<<<blocks_for((long long)n * h1 * w1 * 2), kT, 0, s>>>(m.du0, m.h1, m.g1u, n, h, w, 16);
  conv(m.g1u, m.wt[C1U], n, h1, w1, 16, 32, nullptr, nullptr, m.du1, cnn::CONV_PLAIN, s);
  k_upT_mask<<<blocks_for((long long)n * h2 * w2 * 4), kT, 0, s>>>(m.du1, m.h2, m.g2u, n, h1, w1, 32);
  conv(m.g2u, m.wt[C2U], n, h2, w2, 32, 64, nullptr, nullptr, m.du2, cnn::CONV_PLAIN, s);
  k_upT_mask<<<blocks_for((long long)n * h3 * w3 * 8), kT, 0, s>>>(m.du2, m.h3, m.g3b, n, h2, w2, 64);
  conv(m.g3b, m.wt[C3B], n, h3, w3, 64, 64, nullptr, m.a3, m.ga3, cnn::CONV_MASK, s);
  conv(m.ga3, m.wt[C3A], n, h3, w3, 64, 64, nullptr, nullptr, m.dp3, cnn::CONV_PLAIN, s);
  k_add_poolT_mask<<<blocks_for((long long)n * h2 * w2 * 8), kT, 0, s>>>(m.du2, m.dp3, m.e2, m.ge2, n, h2, w2, 64);
  conv(m.ge2, m.wt[C2B], n, h2, w2, 64, 64, nullptr, m.a2, m.ga2, cnn::CONV_MASK, s);
  conv(m.ga2, m.wt[C2A], n, h2, w2, 64, 32, nullptr, nullptr, m.dp2, cnn::CONV_PLAIN, s);
  k_add_poolT_mask<<<blocks_for((long long)n * h1 * w1 * 4), kT, 0, s>>>(m.du1, m.dp2, m.e1, m.ge1, n, h1, w1, 32);
  conv(m.ge1, m.wt[C1B], n, h1, w1, 32, 32, nullptr, m.a1, m.ga1, cnn::CONV_MASK, s);
  conv(m.ga1, m.wt[C1A], n, h1, w1, 32, 16, nullptr, nullptr, m.dp1, cnn::CONV_PLAIN, s);
  k_add_poolT_mask<<<blocks_for((long long)n * h * w * 2), kT, 0, s>>>(m.du0, m.dp1, m.e0, m.ge0, n, h, w, 16);
  launches_ += 16;
  // weight gradients (CUDA cores, fixed-order partial sums)
  WgPlan P;
  const bf16 *xin[kLayers] = {m.x0, m.p1, m.a1, m.p2, m.a2, m.p3, m.a3, m.u2, m.u1, m.u0};
  const bf16 *gout[kLayers] = {m.ge0, m.ga1, m.ge1, m.ga2, m.ge2, m.ga3, m.g3b, m.g2u, m.g1u, m.g0u};
  float *part = m.wpart;
  int ctas = 0;
  for (int l = 0; l < kLayers; l++) {
    WgLayer &L = P.l[l];
    L.x = xin[l];
    L.g = gout[l];
    L.partial = part;
    L.grad = m.grads + o.w[l];
    L.h = h >> kLevel[l];
    L.w = w >> kLevel[l];
    L.tiles = wg_tiles(l, n, h, w);
    L.shares = wg_shares(l, n, h, w);
    L.len = wg_len(l);
    L.first = ctas;
    ctas += wg_rows(kDefs[l].cin, kDefs[l].cout) == 3 ? L.shares : 3 * L.shares;
    part += (size_t)L.shares * L.len;
  }
  P.opart = m.opart;
  P.ograd = m.grads + o.wout;
  P.oparts = ob;
  k_wgrad<<<ctas, kT, 0, s>>>(P);
  k_sum_parts<<<dim3(148, kLayers + 1), kT, 0, s>>>(P);
  check(cudaGetLastError(), "learned preconditioner backward");
  launches_ += 2;
  double L = 0.0;
  check(cudaMemcpyAsync(&L, loss, 8, cudaMemcpyDeviceToHost, s), "loss readback");
  check(cudaStreamSynchronize(s), "learned preconditioner step");
  int err = 0;
  check(cudaMemcpy(&err, cnn::error_word(), 4, cudaMemcpyDeviceToHost), "conv error word");
  if (err) throw Error(E_TIMEOUT, "learned preconditioner: a convolution pipeline wait expired");
  return L;
}

void Net::adam(double lr, cudaStream_t s) {
  Impl &m = *m_;
  const int np = offs().total;
  m.step++;
  const double b1 = 0.9, b2 = 0.999;
  const double lr_t = lr * sqrt(1.0 - pow(b2, m.step)) / (1.0 - pow(b1, m.step));
  k_adam<<<blocks_for(np), kT, 0, s>>>(m.params, m.grads, m.am, m.av, np, (float)lr_t, (float)b1, (float)b2, 1e-8f);
  check(cudaGetLastError(), "adam");
  launches_ += 1;
  m.prepped = false;
}

}  // namespace lmg
}  // namespace opsb
