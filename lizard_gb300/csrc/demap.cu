// Row (c) of the hot path on sm_103a: the pilots' grid-shift fit, the soft QPSK demap to int8 LLRs, and the
// per-block estimate / pilot reading / decline gate. Compiled with -fmad=false: every float and double operation here
// rounds once, in the reference's order, so from the same spectrum these kernels give the reference's soft values
// bit for bit (liblizard/src/lizard_phy.c:280-329 pilot_align, :1320-1332 sub_scale, :1411-1451 the x86-64 soft4,
// :1775-1818 the block estimate, pilots and decline).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <cooperative_groups.h>
#include "lizg_internal.h"

namespace cg = cooperative_groups;

namespace lizg {

// Coefficient i's value z (spectra are in pos order) turned back by the grid shift (dx, dy): the turn's index in float,
// nearest-even, mod 4096, and the rotation by the table's cos / sin, as liblizard/src/lizard_phy.c:214-218 computes them.
__device__ __forceinline__ float2 turned(const FmtDev &fd, float2 z, int i, float dx, float dy) {
  const float uu = (float)fd.uv[2 * i], vv = (float)fd.uv[2 * i + 1];
  const float t = (uu * dx + vv * dy) * fd.turn_scale;
  const unsigned k = (unsigned)__float2int_rn(t) & (kTurnsDev - 1);
  const float2 cs = fd.rot[k];
  return make_float2(z.x * cs.x + z.y * cs.y, z.y * cs.x - z.x * cs.y);
}

// The pilots' fit, a cluster of kPilotCtas CTAs a frame. The reference adds its six double sums in pilot order
// (liblizard/src/lizard_phy.c:283-317), a chain of as many dependent additions as there are pilots. Only three things of
// the fit are seen: the shift rounded to float after the first pass (the second pass turns the pilots by it), whether
// the shift is worth turning back, and, where it is, the shift rounded to float. So the sums are first added as a
// tree, each quantity's distance from the ordered sums' is bounded (pilot_bound), and where every one of the three
// comes out the same over the whole bound it is the reference's, whatever the order; else the frame is done again
// with the sums in pilot order. A rounding edge falls inside the bound (some 1e-12 of the shift) for about one frame in
// ten thousand; an empty or overflowing spectrum always takes the second way.
// Bound: the double pipe's latency (about 70 cycles an operation). One frame of n = 1536 (984 pilots) decoded: 277 us with
// the ordered sums (95 of them here), 200 with the tree (16 here; 19 for 32 frames).
constexpr int kPilotCtas = 8, kPilotThreads = 128, kPilotWarps = kPilotThreads / 32;
static_assert(kPilotCtas * kPilotWarps == 32, "a lane of one warp a warp of the cluster");
enum { kPilotOn = 0, kPilotGiveUp = 1, kPilotAgain = 2 };

// v[0..5] summed over the warp: value k ends in lane 16 (k >> 2 & 1) + 8 (k >> 1 & 1) + 4 (k & 1) and its three
// neighbours. Each step sends the half of the values that the partner keeps: nine additions in place of thirty.
__device__ __forceinline__ double warp_sum6(double v[8], int lane) {
  v[6] = v[7] = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const double keep = (lane & 16) ? v[j + 4] : v[j], send = (lane & 16) ? v[j] : v[j + 4];
    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const double keep = (lane & 8) ? v[j + 2] : v[j], send = (lane & 8) ? v[j] : v[j + 2];
    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const double keep = (lane & 4) ? v[1] : v[0], send = (lane & 4) ? v[0] : v[1];
  double s = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

// How far the tree's sums (a = S cu cu, b = S cu cv, c = S cv cv, p = S cu zi, q = S cv zi, y = S zi zi over `used` terms)
// and what is worked out from them may be from the ordered sums'. A sum in any order is within used u of the sum of its
// terms' magnitudes (u = 2^-53), itself the sum or, by Cauchy and Schwarz, the root of two; that serves a, b, c and y. p
// and q, whose terms nearly cancel, decide how often the bound cannot tell, so theirs is the ordered chain's own: its
// error is within u times the sum of its partial sums' magnitudes (wp, wq, from a scan in float), the tree's within 20 u
// of the magnitudes' sum. Every figure in float and taken generously; an infinity or a NaN fails the comparisons it is
// used in.
struct PilotBound {
  float ea, eb, ec, ep, eq, ey, det;   // the sums' and a c - b b's
};
constexpr float kU = 1.2e-16f;   // over 2^-53
__device__ __forceinline__ PilotBound pilot_bound(float a, float b, float c, float y, float wp, float wq, int used) {
  PilotBound e;
  const float E = (float)(used + 64) * kU, ra = sqrtf(a), rc = sqrtf(c), ry = sqrtf(y);
  e.ea = E * a; e.ec = E * c; e.ey = E * y;
  e.eb = E * ra * rc;
  e.ep = kU * (1.01f * wp + 24.0f * ra * ry); e.eq = kU * (1.01f * wq + 24.0f * rc * ry);
  e.det = 1.1f * (e.ea * c + a * e.ec + 2.0f * fabsf(b) * e.eb) + 8.0f * kU * (a * c + b * b);
  return e;
}
// The sum over the warp's lanes of |t_0 + ... + t_lane|, with t's inclusive scan.
__device__ __forceinline__ float partials(float t, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, t, o);
    if (lane >= o) t += up;
  }
  float s = fabsf(t);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
// Partial sums' magnitudes over the cluster from each warp's own (w, lane by warp) and its terms' sum (s): a warp's
// partials are its own past what came before it.
__device__ __forceinline__ float partials_all(float w, float s, int lane) {
  float before = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += up;
  }
  float all = w + 32.0f * fabsf(before - s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
  return all;
}

// Frame f's fit by the calling cluster. tm: this CTA's dynamic shared memory (chunk x 6 doubles at least).
__device__ __forceinline__ void pilot_align_frame(const FmtDev &fd, const float2 *spec, int64_t spec_stride, float *align, int f, double *tm) {
  __shared__ double part[kPilotWarps][6], sums[6], dxy[2];
  __shared__ float wander[kPilotWarps][2];
  __shared__ int status;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), used = fd.npilot, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = (used + kPilotCtas - 1) / kPilotCtas, p0 = rank * chunk, p1 = min(used, p0 + chunk);
  const float2 *sp = spec + f * spec_stride;
  const double k = 2.0 * 3.14159265358979323846 / fd.n;
  for (int ordered = 0;; ordered = 1) {
    if (tid == 0) { dxy[0] = dxy[1] = 0; status = used < 8 ? kPilotGiveUp : chunk > kPilotThreads && !ordered ? kPilotAgain : kPilotOn; }
    cl.sync();
    if (status == kPilotGiveUp) break;
    float e_prev = 0;   // rank 0's lanes 0 and 1: the bound on dx's, dy's distance from the ordered one
    for (int it = 0; it < 2 && status == kPilotOn; it++) {
      const float dx = (float)dxy[0], dy = (float)dxy[1];
      double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      float tp = 0, tq = 0;   // the thread's one pilot's p and q terms (the partial sums' bound takes one a thread)
      for (int pi = p0 + tid; pi < p1; pi += kPilotThreads) {
        const int i = fd.pilot_coef[pi], w = fd.pilot_white[pi];
        const float2 y = turned(fd, sp[i], i, dx, dy);
        const double xr = (w & 1) ? -1.0 : 1.0, xi = (w & 2) ? -1.0 : 1.0;
        const double zr = (double)y.x * xr + (double)y.y * xi, zi = (double)y.y * xr - (double)y.x * xi;
        const double cu = k * zr * fd.uv[2 * i], cv = k * zr * fd.uv[2 * i + 1];
        const double t[6] = {cu * cu, cu * cv, cv * cv, cu * zi, cv * zi, zi * zi};
#pragma unroll
        for (int q = 0; q < 6; q++) {
          if (ordered) tm[6 * (pi - p0) + q] = t[q];
          else v[q] += t[q];
        }
        tp = (float)t[3]; tq = (float)t[4];
      }
      if (!ordered) {
        const double s = warp_sum6(v, lane);
        const int q = 4 * (lane >> 4) + 2 * (lane >> 3 & 1) + (lane >> 2 & 1);
        if ((lane & 3) == 0 && q < 6) part[warp][q] = s;
        const float wp = partials(tp, lane), wq = partials(tq, lane);
        if (lane == 0) { wander[warp][0] = wp; wander[warp][1] = wq; }
      }
      cl.sync();
      if (rank == 0 && ordered) {
        if (tid < 6) {
          // in pilot order, CTA by CTA; the loads of eight terms issued ahead of their adds
          double acc = 0;
          for (int r = 0; r < kPilotCtas; r++) {
            const double *rt = cl.map_shared_rank(tm, r) + tid;
            const int cnt = max(0, min(used, (r + 1) * chunk) - r * chunk);
            int q = 0;
            for (; q + 8 <= cnt; q += 8) {
              double x[8];
#pragma unroll
              for (int e = 0; e < 8; e++) x[e] = rt[6 * (q + e)];
#pragma unroll
              for (int e = 0; e < 8; e++) acc += x[e];
            }
            for (; q < cnt; q++) acc += rt[6 * q];
          }
          sums[tid] = acc;
        }
        __syncthreads();
      }
      if (rank == 0 && warp == 0) {
        double a, b, c, p, q, yy;
        float wp = 0, wq = 0;
        if (ordered) {
          a = sums[0]; b = sums[1]; c = sums[2]; p = sums[3]; q = sums[4]; yy = sums[5];
        } else {
          const double *rp = cl.map_shared_rank(&part[0][0], lane / kPilotWarps) + 6 * (lane % kPilotWarps);
#pragma unroll
          for (int j = 0; j < 6; j++) v[j] = rp[j];
          const float *rw = cl.map_shared_rank(&wander[0][0], lane / kPilotWarps) + 2 * (lane % kPilotWarps);
          wp = partials_all(rw[0], (float)v[3], lane); wq = partials_all(rw[1], (float)v[4], lane);
          const double s = warp_sum6(v, lane);
          a = __shfl_sync(0xffffffffu, s, 0); b = __shfl_sync(0xffffffffu, s, 4); c = __shfl_sync(0xffffffffu, s, 8);
          p = __shfl_sync(0xffffffffu, s, 12); q = __shfl_sync(0xffffffffu, s, 16); yy = __shfl_sync(0xffffffffu, s, 20);
        }
        // lane 0 takes x, lane 1 y (the others repeat them): the shift's step (p c - q b) / det, (a q - b p) / det
        const bool ly = lane & 1;
        const double det = a * c - b * b, num = ly ? a * q - b * p : p * c - q * b;
        const double step = num / det, was = ly ? dxy[1] : dxy[0], now = was + step;
        int st = kPilotOn;
        float e_step = 0, e_now = 0;
        const PilotBound e = pilot_bound((float)a, (float)b, (float)c, (float)yy, wp, wq, used);
        if (ordered) {
          if (!(det > 0)) st = kPilotGiveUp;
        } else {
          const float fa = (float)a, fb = fabsf((float)b), fc = (float)c, fp = fabsf((float)p), fq = fabsf((float)q), fdet = (float)det;
          const float m = ly ? fa : fc, em = ly ? e.ea : e.ec, f1 = ly ? fq : fp, e1 = ly ? e.eq : e.ep, f2 = ly ? fp : fq, e2 = ly ? e.ep : e.eq;
          const float e_num = 1.1f * (e1 * m + f1 * em + e2 * fb + f2 * e.eb) + 8.0f * kU * (f1 * m + f2 * fb);
          const float fs = fabsf((float)step);
          e_step = 1.5f * (e_num + fs * e.det) / fdet + 4.0f * kU * fs;   // fdet is over 4 e.det
          e_now = e_prev + e_step + 4.0f * kU * fabsf((float)now);
          // the determinant's sign is not sure, or figures so small that the bound itself could vanish
          if (!(fdet > 4.0f * e.det && fdet > 1e-20f && (yy == 0 || (float)yy > 1e-15f))) st = kPilotAgain;
          // the first pass's shift has to round alike over the bound: the second turns by it
          if (it == 0 && !((float)(now - e_now) == (float)(now + e_now))) st = kPilotAgain;
        }
        st = (int)__reduce_max_sync(0xffffffffu, (unsigned)st);
        if (it == 1 && st == kPilotOn) {
          // worth turning back: chi^2 of the shift over the residual's variance past 13.8
          const double nx = __shfl_sync(0xffffffffu, now, 0), ny = __shfl_sync(0xffffffffu, now, 1);
          const double ex = __shfl_sync(0xffffffffu, step, 0), ey = __shfl_sync(0xffffffffu, step, 1);
          const double s2 = (yy - ex * p - ey * q) / (used - 2);
          const double chi = s2 > 0 ? (nx * nx * a + 2 * nx * ny * b + ny * ny * c) / s2 : 0;
          bool back = chi > 13.8 && nx == nx && ny == ny;
          if (!ordered) {
            const float dsx = __shfl_sync(0xffffffffu, e_step, 0), dsy = __shfl_sync(0xffffffffu, e_step, 1);
            const float dnx = __shfl_sync(0xffffffffu, e_now, 0), dny = __shfl_sync(0xffffffffu, e_now, 1);
            const float fa = (float)a, fb = fabsf((float)b), fc = (float)c, fp = fabsf((float)p), fq = fabsf((float)q), fy = (float)yy;
            const float fx = fabsf((float)ex), fey = fabsf((float)ey), x = fabsf((float)nx), y = fabsf((float)ny), fs2 = (float)s2, fchi = (float)chi;
            const float e_s2 = 2.0f * (e.ey + fx * e.ep + fp * dsx + fey * e.eq + fq * dsy + 8.0f * kU * (fy + fx * fp + fey * fq)) / (float)(used - 2);
            const float e_n = 2.0f * (2.0f * x * dnx * fa + x * x * e.ea + 2.0f * (dnx * y * fb + x * dny * fb + x * y * e.eb) + 2.0f * y * dny * fc +
                                      y * y * e.ec) + 16.0f * kU * (x * x * fa + 2.0f * x * y * fb + y * y * fc);
            const float e_chi = 2.0f * (e_n + fchi * e_s2) / fs2 + 8.0f * kU * fchi;
            bool sure = fs2 > 4.0f * e_s2 && fabs(chi - 13.8) > 4.0 * e_chi;
            if (back && !((float)(nx - dnx) == (float)(nx + dnx) && (float)(ny - dny) == (float)(ny + dny))) sure = false;
            if (!sure) st = kPilotAgain;
          }
          if (lane == 0 && st == kPilotOn) {
            const float d0 = back ? (float)nx : 0.0f, d1 = back ? (float)ny : 0.0f;
            align[3 * f] = d0; align[3 * f + 1] = d1;
            align[3 * f + 2] = d0 != 0 || d1 != 0 ? 1.0f : 0.0f;
          }
        }
        e_prev = e_now;
        // the shift and what to do next, to every CTA of the cluster
        const double nx = __shfl_sync(0xffffffffu, now, 0), ny = __shfl_sync(0xffffffffu, now, 1);
        if (lane < kPilotCtas) {
          double *rd = cl.map_shared_rank(dxy, lane);
          rd[0] = nx; rd[1] = ny;
          *cl.map_shared_rank(&status, lane) = st;
        }
      }
      cl.sync();
    }
    if (status != kPilotAgain) break;
    cl.sync();   // every CTA has read the status before it is set anew
  }
  if (rank == 0 && tid == 0 && status == kPilotGiveUp) align[3 * f] = align[3 * f + 1] = align[3 * f + 2] = 0;
}

__global__ void __cluster_dims__(kPilotCtas, 1, 1) __launch_bounds__(kPilotThreads) pilot_align_kernel(FmtDev fd, const float2 *spec, int64_t spec_stride,
                                                                                           float *align) {
  extern __shared__ double tm[];              // chunk x 6: this CTA's pilots' products
  pilot_align_frame(fd, spec, spec_stride, align, blockIdx.x / kPilotCtas, tm);
}

// ten Brink's J (liblizard/src/lizard_phy.c:73-75)
__device__ __forceinline__ double axis_info(double g) { return g > 0 ? pow(1 - pow(2.0, -0.3073 * pow(2 * sqrt(g), 1.7870)), 1.1064) : 0; }

// 32 sub-channels of a frame a CTA (a frame's last may have 16). Lane q of four sums the moments of a sub-channel's
// coefficients q, q + 4, ... in order (the reference's four float chains, sixteen coefficients' loads in flight) and the
// chains are added (c0 + c1) + (c2 + c3). Warp 0 then works out the scales in double, a sub-channel a lane, while warp 2
// works out what the block stage wants of them (their information, two pows, and their rms), so the double pipe's
// latency, the bound (some 300 dependent operations), is paid beside the soft values and not before them; the soft
// values are each axis times 8 k, NaN to 0, clamped to +-80, rounded half to even, four coefficients a lane, the
// coefficients read again (from L2). One frame at n = 1536, then 32: 31 and 80 us with the scales and the information
// one after the other on the same warps, 18 and 44 so; with the coefficients kept in shared memory 15 and 63 (it leaves
// an SM two CTAs and the pipe idle).
constexpr int kDemapSubs = 32, kDemapThreads = 256, kDemapBatch = 16;
static_assert(kDemapSubs == 32, "a sub-channel a lane of the double warps");
static_assert(kSubDev % (4 * kDemapBatch) == 0, "whole batches");

struct SubMoments {
  double m2, a2, nv;
};
__device__ __forceinline__ SubMoments sub_moments(const float *m) {
  SubMoments r;
  const double M2 = (double)m[0] / kSubDev, M4 = (double)m[1] / kSubDev;
  double a2 = 2 * M2 * M2 - M4;
  a2 = a2 > 0 ? sqrt(a2) : 0;
  double nv = M2 - a2;
  if (nv < 0.02 * M2) nv = 0.02 * M2;
  r.m2 = M2; r.a2 = a2; r.nv = nv;
  return r;
}
// A coefficient's two soft values, in the low bytes.
__device__ __forceinline__ uint32_t soft2(float k8, float x, float y) {
  x = k8 * x; y = k8 * y;
  x = x != x ? 0.0f : fminf(fmaxf(x, -80.0f), 80.0f);
  y = y != y ? 0.0f : fminf(fmaxf(y, -80.0f), 80.0f);
  return (uint32_t)(__float2int_rn(x) & 255) | (uint32_t)(__float2int_rn(y) & 255) << 8;
}

__device__ __forceinline__ void demap_block(const FmtDev &fd, const float2 *spec, int64_t spec_stride, const float *align, int8_t *llrf,
                                            double *sub_est, float *sub_rms, int blk) {
  __shared__ float s_m[kDemapSubs][2], s_k8[kDemapSubs];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per = (fd.subch + kDemapSubs - 1) / kDemapSubs, f = blk / per, j0 = (blk - f * per) * kDemapSubs, subs = min(kDemapSubs, fd.subch - j0);
  const float2 *src = spec + f * spec_stride + j0 * kSubDev;
  const bool turn = align[3 * f + 2] != 0.0f;
  const float dx = align[3 * f], dy = align[3 * f + 1];
  if (tid < 4 * subs) {   // whole warps: subs is 16 or 32
    const int g = tid >> 2, qd = tid & 3;
    float m2 = 0, m4 = 0;
    for (int s0 = qd; s0 < kSubDev; s0 += 4 * kDemapBatch) {
      float2 y[kDemapBatch];
#pragma unroll
      for (int e = 0; e < kDemapBatch; e++) y[e] = src[g * kSubDev + s0 + 4 * e];
      if (turn) {
#pragma unroll
        for (int e = 0; e < kDemapBatch; e++) y[e] = turned(fd, y[e], (j0 + g) * kSubDev + s0 + 4 * e, dx, dy);
      }
#pragma unroll
      for (int e = 0; e < kDemapBatch; e++) {
        const float p = y[e].x * y[e].x + y[e].y * y[e].y;
        m2 = m2 + p; m4 = m4 + p * p;
      }
    }
    // (c0 + c1) + (c2 + c3)
    const float o2 = __shfl_down_sync(0xffffffffu, m2, 1), o4 = __shfl_down_sync(0xffffffffu, m4, 1);
    const float p2 = m2 + o2, p4 = m4 + o4;
    const float r2 = __shfl_down_sync(0xffffffffu, p2, 2), r4 = __shfl_down_sync(0xffffffffu, p4, 2);
    if (qd == 0) { s_m[g][0] = p2 + r2; s_m[g][1] = p4 + r4; }
  }
  __syncthreads();
  if (warp == 2) {   // the block stage's part
    if (lane < subs) {
      const SubMoments m = sub_moments(s_m[lane]);
      sub_rms[f * fd.subch + j0 + lane] = m.m2 > 0 ? (float)sqrt(m.m2 / 2) : 0;
      sub_est[f * fd.subch + j0 + lane] = axis_info(m.a2 / m.nv);
    }
    return;
  }
  if (warp == 0 && lane < subs) {
    const SubMoments m = sub_moments(s_m[lane]);
    const float kk = (float)(0.7 * 2 * sqrt(2 * m.a2) / m.nv);
    s_k8[lane] = 8 * kk;
  }
  asm volatile("bar.sync 1, %0;" ::"n"(kDemapThreads - 32) : "memory");   // every warp but warp 2, which has left
  int8_t *out = llrf + ((int64_t)f * fd.subch + j0) * 2 * kSubDev;
  // four coefficients in, eight soft values out, in the widest accesses the caller's buffers allow
  const bool wide = ((reinterpret_cast<uintptr_t>(src) & 15) | (reinterpret_cast<uintptr_t>(out) & 7)) == 0;
  const int at = warp > 2 ? tid - 32 : tid;   // this thread among the seven warps'
#pragma unroll 4
  for (int c = at; c < subs * kSubDev / 4; c += kDemapThreads - 32) {
    float2 y[4];
    if (wide) {
      const float4 a = reinterpret_cast<const float4 *>(src)[2 * c], b = reinterpret_cast<const float4 *>(src)[2 * c + 1];
      y[0] = make_float2(a.x, a.y); y[1] = make_float2(a.z, a.w); y[2] = make_float2(b.x, b.y); y[3] = make_float2(b.z, b.w);
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++) y[e] = src[4 * c + e];
    }
    if (turn) {
#pragma unroll
      for (int e = 0; e < 4; e++) y[e] = turned(fd, y[e], j0 * kSubDev + 4 * c + e, dx, dy);
    }
    const float k8 = s_k8[c / (kSubDev / 4)];
    const uint32_t lo = soft2(k8, y[0].x, y[0].y) | soft2(k8, y[1].x, y[1].y) << 16, hi = soft2(k8, y[2].x, y[2].y) | soft2(k8, y[3].x, y[3].y) << 16;
    if (wide) {
      *reinterpret_cast<uint2 *>(out + 8 * c) = make_uint2(lo, hi);
    } else {
#pragma unroll
      for (int e = 0; e < 8; e++) out[8 * c + e] = (int8_t)((e < 4 ? lo : hi) >> (8 * (e & 3)));
    }
  }
}

__global__ void __launch_bounds__(kDemapThreads) demap_kernel(FmtDev fd, const float2 *spec, int64_t spec_stride, const float *align,
                                                              int8_t *llrf, double *sub_est, float *sub_rms) {
  demap_block(fd, spec, spec_stride, align, llrf, sub_est, sub_rms, blockIdx.x);
}

// Eight blocks a CTA, a warp a block: its estimate (its sub-channels' information weighted by the slots it holds there, in
// double, in order), its pilot reading (the tail's axis values against the whitening in units of their sub-channel's
// rms, in double, in order; NaN where none was read) and the decline gate (est < 0.2 k / nt in float): decl[f blocks + b]
// = 1. A block's warp works out the terms, a lane each, and the sums run in order a lane a block on one warp, so the
// double pipe does each division and addition once for many blocks. A thread a block took its up to 32 divisions one
// after the other: 24 us a call whatever its size, 8 so for a frame of n = 1536 and 10 for 32.
constexpr int kBlocksPer = 8, kBlocksThreads = 32 * kBlocksPer, kBlocksTerms = 64;
__device__ __forceinline__ void blocks_block(const FmtDev &fd, const float2 *spec, int64_t spec_stride, const float *align,
                                             const double *sub_est, const float *sub_rms, float *est, float *pilot, uint8_t *decl, int blk) {
  __shared__ double s_info[kBlocksPer][kBlocksTerms + 1], s_tail[kBlocksPer][kBlocksTerms + 1];
  __shared__ int s_got[kBlocksPer];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = blk * kBlocksPer + warp;
  if (g < fd.frames * fd.blocks) {
    const int f = g / fd.blocks, b = g - f * fd.blocks;
    const int t = fd.block_tier[b], nb = fd.tier_slots[t], s0 = fd.block_slot[b], nt = fd.tier_nt[t];
    const double *se = sub_est + f * fd.subch;
    const float *sr = sub_rms + f * fd.subch;
    const int ja = s0 / (2 * kSubDev), jn = (s0 + nb + 2 * kSubDev - 1) / (2 * kSubDev) - ja;
    for (int k = lane; k < jn; k += 32) {
      const int j = ja + k, lo = max(s0, 2 * kSubDev * j), hi = min(s0 + nb, 2 * kSubDev * (j + 1));
      s_info[warp][k] = se[j] * (hi - lo);
    }
    const float2 *sp = spec + f * spec_stride;
    const bool turn = align[3 * f + 2] != 0.0f;
    const float dx = align[3 * f], dy = align[3 * f + 1];
    int got = 0;
    for (int i0 = nt; i0 < nb; i0 += 32) {
      const int i = i0 + lane;
      bool read = false;
      if (i < nb) {
        double term = 0;   // where nothing is read: adding 0 leaves the sum as it is
        const int gs = s0 + i, ci = gs / 2;
        const float rms = sr[gs / (2 * kSubDev)];
        if (rms > 0) {
          const float2 z = sp[ci], y = turn ? turned(fd, z, ci, dx, dy) : z;
          const float yv = (i & 1) ? y.y : y.x;
          term = (fd.white[gs] ? -1.0 : 1.0) * yv / rms;
          read = true;
        }
        s_tail[warp][i - nt] = term;
      }
      got += __popc(__ballot_sync(0xffffffffu, read));
    }
    if (lane == 0) s_got[warp] = got;
  }
  __syncthreads();
  const int g2 = blk * kBlocksPer + threadIdx.x;
  if (threadIdx.x >= kBlocksPer || g2 >= fd.frames * fd.blocks) return;
  const int b = g2 % fd.blocks, t = fd.block_tier[b], nb = fd.tier_slots[t], s0 = fd.block_slot[b], nt = fd.tier_nt[t];
  const int jn = (s0 + nb + 2 * kSubDev - 1) / (2 * kSubDev) - s0 / (2 * kSubDev);
  double info = 0, cs = 0;
  for (int k = 0; k < jn; k++) info += s_info[threadIdx.x][k];
  for (int k = 0; k < nb - nt; k++) cs += s_tail[threadIdx.x][k];
  const float e = (float)(info / nb);
  est[g2] = e;
  pilot[g2] = nt < nb && s_got[threadIdx.x] ? (float)(cs / (nb - nt)) : __int_as_float(0x7fc00000);   // NaN: no pilot read
  decl[g2] = e < 0.2f * (float)fd.tier_k[t] / (float)nt;
}

__global__ void __launch_bounds__(kBlocksThreads) blocks_kernel(FmtDev fd, const float2 *spec, int64_t spec_stride, const float *align,
                                                                const double *sub_est, const float *sub_rms, float *est, float *pilot,
                                                                uint8_t *decl) {
  blocks_block(fd, spec, spec_stride, align, sub_est, sub_rms, est, pilot, decl, blockIdx.x);
}

// The three stages over several formats' batches, one launch each: format k's frames (clusters), demap CTAs and block
// CTAs at [pf[k], pf[k + 1]), [df[k], df[k + 1]) and [bf[k], bf[k + 1]).
struct DemapMix {
  DemapSeg seg[kDemapMixSegs];
  int pf[kDemapMixSegs + 1], df[kDemapMixSegs + 1], bf[kDemapMixSegs + 1];
  int nseg;
};
static_assert(sizeof(DemapMix) <= 32000, "the mixed launches' arguments fit a launch");
__device__ __forceinline__ int seg_at(const int *first, int nseg, int b) {
  int k = 0;
  while (k < nseg - 1 && b >= first[k + 1]) k++;
  return k;
}

__global__ void __cluster_dims__(kPilotCtas, 1, 1) __launch_bounds__(kPilotThreads) pilot_align_mixed_kernel(const __grid_constant__ DemapMix m) {
  extern __shared__ double tm[];
  const int c = blockIdx.x / kPilotCtas, k = seg_at(m.pf, m.nseg, c);
  const DemapSeg &g = m.seg[k];
  pilot_align_frame(g.fd, g.spec, g.stride, g.align, c - m.pf[k], tm);
}

__global__ void __launch_bounds__(kDemapThreads) demap_mixed_kernel(const __grid_constant__ DemapMix m) {
  const int k = seg_at(m.df, m.nseg, blockIdx.x);
  const DemapSeg &g = m.seg[k];
  demap_block(g.fd, g.spec, g.stride, g.align, g.llrf, g.sub_est, g.sub_rms, blockIdx.x - m.df[k]);
}

__global__ void __launch_bounds__(kBlocksThreads) blocks_mixed_kernel(const __grid_constant__ DemapMix m) {
  const int k = seg_at(m.bf, m.nseg, blockIdx.x);
  const DemapSeg &g = m.seg[k];
  blocks_block(g.fd, g.spec, g.stride, g.align, g.sub_est, g.sub_rms, g.est, g.pilot, g.decl, blockIdx.x - m.bf[k]);
}

cudaError_t demap_mixed_launch(const DemapSeg *a, int count, cudaStream_t st) {
  if (count < 1 || count > kDemapMixSegs) return cudaErrorInvalidValue;
  DemapMix m{};
  m.nseg = count;
  int psm = 8;
  for (int k = 0; k < count; k++) {
    const FmtDev &fd = a[k].fd;
    m.seg[k] = a[k];
    const int chunk = (fd.npilot + kPilotCtas - 1) / kPilotCtas, bytes = 6 * (chunk > 0 ? chunk : 1) * (int)sizeof(double);
    psm = bytes > psm ? bytes : psm;
    m.pf[k + 1] = m.pf[k] + fd.frames;
    m.df[k + 1] = m.df[k] + fd.frames * ((fd.subch + kDemapSubs - 1) / kDemapSubs);
    m.bf[k + 1] = m.bf[k] + (fd.frames * fd.blocks + kBlocksPer - 1) / kBlocksPer;
  }
  if (psm > 48 * 1024) return cudaErrorInvalidValue;
  pilot_align_mixed_kernel<<<m.pf[count] * kPilotCtas, kPilotThreads, psm, st>>>(m);
  demap_mixed_kernel<<<m.df[count], kDemapThreads, 0, st>>>(m);
  blocks_mixed_kernel<<<m.bf[count], kBlocksThreads, 0, st>>>(m);
  return cudaGetLastError();
}

cudaError_t demap_launch(const FmtDev &fd, const float2 *spec, int64_t spec_stride, float *align, int8_t *llrf,
                         double *sub_est, float *sub_rms, float *est, float *pilot, uint8_t *decl, cudaStream_t st) {
  const int chunk = (fd.npilot + kPilotCtas - 1) / kPilotCtas;
  const int psm = 6 * (chunk > 0 ? chunk : 1) * (int)sizeof(double);
  if (psm > 48 * 1024) return cudaErrorInvalidValue;
  pilot_align_kernel<<<fd.frames * kPilotCtas, kPilotThreads, psm, st>>>(fd, spec, spec_stride, align);
  demap_kernel<<<fd.frames * ((fd.subch + kDemapSubs - 1) / kDemapSubs), kDemapThreads, 0, st>>>(fd, spec, spec_stride, align, llrf, sub_est, sub_rms);
  const int nbk = fd.frames * fd.blocks;
  blocks_kernel<<<(nbk + kBlocksPer - 1) / kBlocksPer, kBlocksThreads, 0, st>>>(fd, spec, spec_stride, align, sub_est, sub_rms, est,
                                                                                       pilot, decl);
  return cudaGetLastError();
}

}  // namespace lizg
