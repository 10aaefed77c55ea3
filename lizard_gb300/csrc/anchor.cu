// The anchor search on sm_103a: the registration's 7 x 7 anchors found in a batch of captured frames, the step of the
// reference's front half that the refinement of the registration starts from (liblizard/src/acquire.c:1876-2036
// anchor_find, restated from its portable build, the scalar twin of its SIMD paths). Compiled with -fmad=false: every
// float and double operation rounds once, in the reference's order, so the results are that build's bit for bit.
//
// One CTA an anchor of a frame: the window of W x W samples a template step (a / 16 modules) apart about the anchor's
// place, read through H and the lens model; its integral images of the greys and of their squares in double (each
// row's running sums by one thread a row, then each column accumulated down by one thread a column, the additions
// the reference makes); the normalised correlation with the anchor's pattern (two concentric squares) at every
// offset within three modules, from four box sums an offset; the first largest in scan order; a parabola each way.
//
// The double pipe (two lanes a cycle an SM) is the bound: forty operations an offset, 2,401 offsets of a 64 x 64 window.
// So the correlation is bounded in float first, and only the offsets whose bound reaches the best lower bound are
// worked out in double (with the parabola's neighbours): the largest and the outputs are as if all were. 3,136 anchors of
// 64 frames (span 128): 1,010 us with every offset in double and the pattern's norm before the window on one thread, 430 so.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string>
#include "lizard_gb300.h"
#include "lizg_internal.h"
#include "reg_dev.cuh"

namespace lizg {

constexpr int kAnchK = 7, kAnchTs = 16, kAnchReach = 3, kMarginM = 15;
constexpr float kAnchPeak = 0.6f;

// The window's geometry for a ring span (a = span / 64 modules a side, r steps of reach, W samples across, O offsets).
struct AnchGeom {
  int a, r, W, O;
  float hs;
};
static AnchGeom anch_geom(int span) {
  AnchGeom g;
  g.a = span / 64;
  g.hs = (float)g.a / kAnchTs;
  g.r = (int)ceilf((float)kAnchReach / g.hs);
  g.W = kAnchTs + 2 * g.r;
  g.O = 2 * g.r + 1;
  return g;
}

__device__ __forceinline__ void anchor_map(const float *h, const double *lens, float X, float Y, float *u, float *v) {
  project(h, X, Y, u, v);
  if (lens) { float dx, dy; lens_at(lens, *u, *v, &dx, &dy); *u += dx; *v += dy; }
}

// lens_at without what it need not do at every sample of a window, to the bit but a zero's sign (which the read's half
// pixel takes away): its terms of a coefficient times 0.0 (nothing, the coefficients finite), and its two divisions by R,
// the correctly rounded quotients from R's correctly rounded reciprocal and two remainders (Markstein, 1990: the first
// correction is within a unit of the quotient, the second rounds it). 1,600 to 4,096 samples an anchor, and the double
// pipe is the bound: 64 frames' second search 197 us through lens_at, 152 so. ok: the model's numbers are such that nothing overflows or underflows on the way; a place
// that is not within 1e30 pixels takes lens_at.
struct LensWindow {
  double r;
  bool ok;
  // whether number k of a model is one of those
  static __device__ __forceinline__ bool fits(int k, double v) { return k == 0 || (k == 3 ? v > 1e-30 && v < 1e30 : fabs(v) < 1e30); }
  __device__ __forceinline__ double over(double a, double b) const {
    double q = a * r;
    q = fma(fma(-b, q, a), r, q);
    return fma(fma(-b, q, a), r, q);
  }
  __device__ __forceinline__ void at(const double *l, float u, float v, float *dx, float *dy) const {
    if (!ok || !(fabsf(u) < 1e30f && fabsf(v) < 1e30f)) { lens_at(l, u, v, dx, dy); return; }
    const int K = (int)l[0];
    const double x = over(u - l[1], l[3]), y = over(v - l[2], l[3]), xx = x * x, xy = x * y, yy = y * y;
    double fx = l[4] * x + l[5] * y + l[8] - l[10] * xx - l[11] * xy, fy = l[6] * x + l[7] * y + l[9] - l[10] * xy - l[11] * yy;
    const double s = xx + yy;
    double sk = s;
    for (int k = 0; k < K; k++, sk *= s) { fx += l[12 + k] * (sk * x); fy += l[12 + k] * (sk * y); }
    *dx = (float)fx; *dy = (float)fy;
  }
};

struct AnchArgs {
  int span, w, h, frames, hstride;
  int64_t fstride;
  AnchGeom g;
  int m0[kAnchK];
  const uint8_t *luma, *skip;
  const float *H;
  const double *lens;
  const int *lens_on;       // frames: 0 where frame f searches through H alone (NULL: every frame through lens)
  const uint8_t *active;    // frames: 0 where frame f is not searched at all (NULL: every frame)
  lizg_anchor_out out;
};

__device__ __forceinline__ double abox(const double *I, int W1, int x, int y, int s) {
  return I[(y + s) * W1 + x + s] - I[y * W1 + x + s] - I[(y + s) * W1 + x] + I[y * W1 + x];
}

// How far the float sums below may lie from the double ones, u = 2^-24: greys (0..1) less 1/2, so |v| <= 0.51 and v^2 <=
// 0.261, each rounded once. A row's run of at most 16 summed and slid: 16 + 2 x 13 roundings at u 8.2 and u 4.2 and the
// values' own, 2.1e-5 and 1.1e-5; 16 rows of them added: 16 roundings at u 131 and u 67: 4.6e-4 for a sum of values, 2.4e-4
// for one of squares. Their parts in st = 2 (s25 - s6) + s1 (1 - tm), |1 - tm| <= 2: 2.8e-3; in the variance, with the
// square's 2 |s1| 4.6e-4 / 256 and the last roundings: 2.7e-4 + 3.6e-6 |s1|.
constexpr int kAnchThreads = 256, kSlide = 13;
constexpr float kErrSt = 4e-3f, kErrVar = 3.5e-4f, kErrVarS = 5e-6f, kLeastVar = 2e-5f;

__global__ void __launch_bounds__(kAnchThreads) anchor_find_kernel(AnchArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int f = blockIdx.x / (kAnchK * kAnchK), k = blockIdx.x % (kAnchK * kAnchK), i = k % kAnchK, j = k / kAnchK;
  const int64_t o = (int64_t)f * kAnchK * kAnchK + k;
  if (a.skip && a.skip[o]) return;   // found before: left as it is
  if (a.active && !a.active[f]) return;
  const AnchGeom g = a.g;
  const int r = g.r, W = g.W, O = g.O, W1 = W + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float hs = g.hs, ah = (float)g.a * 0.5f;
  // the integral images, and before them in the same place the rows' runs; the window (rows W1 apart); the bounds, the
  // offsets to work out
  double *I1 = reinterpret_cast<double *>(sm), *I2 = I1 + W1 * W1;
  float *run = reinterpret_cast<float *>(sm), *win = reinterpret_cast<float *>(I2 + W1 * W1), *hi = win + W * W1;
  uint16_t *list = reinterpret_cast<uint16_t *>(hi + O * O);
  __shared__ float s_h[9], s_tn, s_bv[kAnchThreads / 32], s_nb[4];
  __shared__ double s_lens[kLensStride];
  __shared__ LensWindow s_lw;
  __shared__ uint32_t s_light[kAnchThreads / 32], s_in[2];
  __shared__ int s_count, s_bi[kAnchThreads / 32];
  if (tid < 9) s_h[tid] = a.H[(int64_t)f * a.hstride + tid];
  const bool use_lens = a.lens && (!a.lens_on || a.lens_on[f]);
  if (use_lens && warp == 0) {
    const double v = lane < kLensStride ? a.lens[(int64_t)f * kLensStride + lane] : 0.0;
    if (lane < kLensStride) s_lens[lane] = v;
    const bool ok = __all_sync(0xffffffffu, lane >= kLensStride || LensWindow::fits(lane, v));
    if (lane == 3) { s_lw.r = 1.0 / v; s_lw.ok = ok; }
  }
  if (tid == 0) s_count = 0;
  // the pattern, a thread a point: light or dark, and its squares' ranges along an axis
  {
    static_assert(kAnchThreads == kAnchTs * kAnchTs, "a thread a point");
    const float u = fabsf(((float)(tid % kAnchTs) + 0.5f) * hs - ah), v = fabsf(((float)(tid / kAnchTs) + 0.5f) * hs - ah), dc = fmaxf(u, v) / ah;
    const uint32_t light = __ballot_sync(0xffffffffu, dc < 0.25f || dc >= 0.6f), in25 = __ballot_sync(0xffffffffu, u / ah < 0.25f),
                   in6 = __ballot_sync(0xffffffffu, u / ah < 0.6f);
    if (lane == 0) s_light[warp] = light;
    if (tid == 0) { s_in[0] = in25 & 0xffffu; s_in[1] = in6 & 0xffffu; }
  }
  __syncthreads();
  const double *lens = use_lens ? s_lens : nullptr;
  const float x0 = (float)a.m0[i], y0 = (float)a.m0[j], X = x0 + ah, Y = y0 + ah;
  const uint8_t *px = a.luma + (int64_t)f * a.fstride;
  // the window
  bool odd = false;
  const LensWindow lw = s_lw;
  for (int t = tid; t < W * W; t += kAnchThreads) {
    const int wx = t % W, wy = t / W;
    float u, v;
    project(s_h, x0 + ((float)(wx - r) + 0.5f) * hs, y0 + ((float)(wy - r) + 0.5f) * hs, &u, &v);
    if (lens) { float dx, dy; lw.at(lens, u, v, &dx, &dy); u += dx; v += dy; }
    const float s = sample(px, a.w, a.h, u, v);
    odd |= !(s >= -0.01f && s <= 1.01f);
    win[wy * W1 + wx] = s;
  }
  // no bound holds about a sample that is not a grey level: every offset is worked out
  const bool all = __syncthreads_or(odd);
  // the pattern's mean (a sum of whole numbers) and its squares' ranges
  int lights = 0;
#pragma unroll
  for (int q = 0; q < kAnchThreads / 32; q++) lights += __popc(s_light[q]);
  const float tm = (float)(2 * lights - kAnchTs * kAnchTs) / (float)(kAnchTs * kAnchTs);
  const int i25 = s_in[0] ? __ffs(s_in[0]) - 1 : kAnchTs, j25 = 31 - __clz(s_in[0]), i6 = s_in[1] ? __ffs(s_in[1]) - 1 : kAnchTs, j6 = 31 - __clz(s_in[1]);
  const double tmd = (double)tm;
  if (!all) {
    // each row's runs of 16, their squares', of the inner squares' widths, at every offset along it, a run of offsets a thread
    float *r16 = run, *q16 = r16 + W * O, *r25 = q16 + W * O, *r6 = r25 + W * O;
    const int parts = max(kAnchThreads / W, (O + kSlide - 1) / kSlide), per = (O + parts - 1) / parts;
    for (int t = tid; t < W * parts; t += kAnchThreads) {
      const int y = t % W, q0 = t / W * per, q1 = min(O, q0 + per);
      const float *w = win + y * W1;
      auto at = [&](int x) { return w[x] - 0.5f; };
      float s = 0, q = 0, s25 = 0, s6 = 0;
      if (q0 < q1) {
#pragma unroll
        for (int x = 0; x < kAnchTs; x++) {
          const float v = at(q0 + x);
          s += v; q += v * v;
          s25 += x >= i25 && x <= j25 ? v : 0.0f;
          s6 += x >= i6 && x <= j6 ? v : 0.0f;
        }
      }
      for (int x = q0; x < q1; x++) {
        r16[y * O + x] = s; q16[y * O + x] = q; r25[y * O + x] = s25; r6[y * O + x] = s6;
        if (x + 1 == q1) break;
        const float out = at(x), in = at(x + kAnchTs);
        s += in - out;
        q += in * in - out * out;
        if (j25 >= i25) s25 += at(x + j25 + 1) - at(x + i25);
        if (j6 >= i6) s6 += at(x + j6 + 1) - at(x + i6);
      }
    }
    __syncthreads();
    // every offset's correlation times the pattern's norm, between two bounds: the upper kept, the largest lower
    float low = -3.0e38f;
    for (int t = tid; t < O * O; t += kAnchThreads) {
      const float *p = run + t;   // row t / O's runs at offset t % O
      float s1 = 0, s2 = 0, s25 = 0, s6 = 0;
#pragma unroll 4
      for (int y = 0; y < kAnchTs; y++) { s1 += p[y * O]; s2 += p[(W + y) * O]; }
      for (int y = i25; y <= j25; y++) s25 += p[(2 * W + y) * O];
      for (int y = i6; y <= j6; y++) s6 += p[(3 * W + y) * O];
      const float var = s2 - s1 * s1 * (1.0f / (kAnchTs * kAnchTs)), ev = kErrVar + kErrVarS * fabsf(s1), st = 2.0f * (s25 - s6) + s1 * (1.0f - tm);
      const float least = var - ev, up = st + kErrSt, down = st - kErrSt;
      // the variance too near none to bound: worked out
      const float h = !(least > kLeastVar) ? 3.0e38f : up > 0 ? up * rsqrtf(least) * 1.0001f : 0.0f;
      hi[t] = h;
      if (least > kLeastVar && down > 0) low = fmaxf(low, down * rsqrtf(var + ev) * 0.9999f);
    }
    for (int q = 16; q > 0; q >>= 1) low = fmaxf(low, __shfl_xor_sync(0xffffffffu, low, q));
    if (lane == 0) s_bv[warp] = low;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kAnchThreads / 32; q++) low = fmaxf(low, s_bv[q]);
    for (int t = tid; t < O * O; t += kAnchThreads)
      if (!(hi[t] < low)) list[atomicAdd(&s_count, 1)] = (uint16_t)t;
    __syncthreads();
  }
  const int count = all ? O * O : s_count;
  for (int t = tid; t < W1; t += kAnchThreads) { I1[t] = 0; I2[t] = 0; I1[t * W1] = 0; I2[t * W1] = 0; }
  __syncthreads();
  // each row's running sums (left to right; a float's square is exact in double, so a fused add rounds as the two steps
  // do), then each column accumulated down the rows; meanwhile the pattern's norm in the reference's order
  if (tid < W) {
    double s = 0, q = 0;
#pragma unroll 4
    for (int wx = 0; wx < W; wx++) {
      const double vv = win[tid * W1 + wx];
      s += vv; q = fma(vv, vv, q);
      I1[(tid + 1) * W1 + wx + 1] = s; I2[(tid + 1) * W1 + wx + 1] = q;
    }
  } else if (tid == kAnchThreads - 1) {
    const float tl = (1.0f - tm) * (1.0f - tm), td = (-1.0f - tm) * (-1.0f - tm);
    float tn = 0;
    for (int q = 0; q < kAnchThreads / 32; q++) {
      const uint32_t bits = s_light[q];
#pragma unroll 8
      for (int x = 0; x < 32; x++) tn += bits >> x & 1 ? tl : td;
    }
    s_tn = sqrtf(tn);
  }
  __syncthreads();
  if (tid < 2 * W) {
    double *I = tid < W ? I1 + tid + 1 : I2 + tid - W + 1, s = 0;
#pragma unroll 4
    for (int wy = 1; wy <= W; wy++) { s += I[wy * W1]; I[wy * W1] = s; }
  }
  __syncthreads();
  const double tnd = (double)s_tn;
  auto corr = [&](int t) {
    const int qx = t % O, qy = t / O;
    const double s1 = abox(I1, W1, qx, qy, kAnchTs), s2 = abox(I2, W1, qx, qy, kAnchTs), var = s2 - s1 * s1 / (double)(kAnchTs * kAnchTs);
    const double s25 = j25 >= i25 ? abox(I1, W1, qx + i25, qy + i25, j25 - i25 + 1) : 0;
    const double s6 = j6 >= i6 ? abox(I1, W1, qx + i6, qy + i6, j6 - i6 + 1) : 0;
    const double st = 2 * (s25 - s6) + s1 * (1 - tmd);
    return var > 1e-12 ? (float)(st / (sqrt(var) * tnd)) : 0.0f;
  };
  // the first largest in scan order
  float bv = -2;
  int bi = O * O;
  for (int e = tid; e < count; e += kAnchThreads) {
    const int t = all ? e : list[e];
    const float c = corr(t);
    if (c > bv || (c == bv && t < bi)) { bv = c; bi = t; }
  }
  for (int s = 16; s > 0; s >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, s);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, s);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  if (lane == 0) { s_bv[warp] = bv; s_bi[warp] = bi; }
  __syncthreads();
  if (tid >= 32) return;
#pragma unroll
  for (int q = 0; q < kAnchThreads / 32; q++)
    if (s_bv[q] > bv || (s_bv[q] == bv && s_bi[q] < bi)) { bv = s_bv[q]; bi = s_bi[q]; }
  const float best = bv;
  const int bx = bi % O - r, by = bi / O - r;
  const bool inx = bx > -r && bx < r, iny = by > -r && by < r;
  if (tid < 4 && (tid < 2 ? inx : iny)) s_nb[tid] = corr(bi + (tid == 0 ? -1 : tid == 1 ? 1 : tid == 2 ? -O : O));
  __syncwarp();
  if (tid != 0) return;
  float sx = 0, sy = 0;
  if (inx) {
    const float l = s_nb[0], c = best, rr = s_nb[1], d = l - 2 * c + rr;
    if (d < 0) sx = 0.5f * (l - rr) / d;
  }
  if (iny) {
    const float l = s_nb[2], c = best, rr = s_nb[3], d = l - 2 * c + rr;
    if (d < 0) sy = 0.5f * (l - rr) / d;
  }
  float u, v, hu, hv;
  anchor_map(s_h, lens, X + ((float)bx + sx) * hs, Y + ((float)by + sy) * hs, &u, &v);
  project(s_h, X, Y, &hu, &hv);
  a.out.peak[o] = best; a.out.dx[o] = u - hu; a.out.dy[o] = v - hv; a.out.u[o] = u; a.out.v[o] = v;
  a.out.ok[o] = best >= kAnchPeak && inx && iny;
}

// Queues the search for a batch of frames (arguments as lizg_anchor_find_dev's, already checked).
cudaError_t anchor_find_launch(int span, const uint8_t *d_luma, int w, int h, int64_t frame_stride, const float *d_H, int h_stride,
                               const double *d_lens, const uint8_t *d_skip, int frames, const lizg_anchor_out &out, cudaStream_t st,
                               const int *d_lens_on, const uint8_t *d_active) {
  AnchArgs a{};
  a.lens_on = d_lens_on; a.active = d_active;
  a.span = span; a.w = w; a.h = h; a.frames = frames; a.hstride = h_stride; a.fstride = frame_stride;
  a.g = anch_geom(span);
  for (int i = 0; i < kAnchK; i++) a.m0[i] = (int)floor(kMarginM + (double)span * (i + 0.5) / kAnchK - a.g.a / 2.0 + 0.5);
  a.luma = d_luma; a.skip = d_skip; a.H = d_H; a.lens = d_lens; a.out = out;
  const int W1 = a.g.W + 1;
  const size_t smem = 2 * sizeof(double) * W1 * W1 + sizeof(float) * (a.g.W * W1 + a.g.O * a.g.O) + sizeof(uint16_t) * a.g.O * a.g.O;
  static SmemOptIn opt;
  cudaError_t e;
  if ((e = opt.set(reinterpret_cast<const void *>(anchor_find_kernel), 120 * 1024)) != cudaSuccess) return e;
  anchor_find_kernel<<<frames * kAnchK * kAnchK, kAnchThreads, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace lizg

extern "C" int lizg_anchor_find_dev(int span, const uint8_t *d_luma, int w, int h, int64_t frame_stride, const float *d_H, int h_stride,
                                    const double *d_lens, const uint8_t *d_skip, int frames, const lizg_anchor_out *out, void *stream) {
  using namespace lizg;
  if (span != 128 && span != 256 && span != 512) return record_error(LIZG_E_ARG, "lizg_anchor_find_dev: span must be 128, 256 or 512");
  if (!d_luma || !d_H || !out || !out->ok || !out->peak || !out->dx || !out->dy || !out->u || !out->v)
    return record_error(LIZG_E_ARG, "lizg_anchor_find_dev: NULL argument");
  if (w < 2 || h < 2 || frames < 1 || frame_stride < (int64_t)w * h || h_stride < 9)
    return record_error(LIZG_E_ARG, "lizg_anchor_find_dev: bad frame geometry, H stride or frame count");
  int sms = 0;
  if (int rc = device_ready(&sms)) return rc;
  const cudaError_t e = anchor_find_launch(span, d_luma, w, h, frame_stride, d_H, h_stride, d_lens, d_skip, frames, *out, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return record_error(LIZG_E_CUDA, (std::string("lizg_anchor_find_dev: ") + cudaGetErrorString(e)).c_str());
  return 0;
}
