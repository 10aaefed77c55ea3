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

// Coefficient i (spectra are in pos order) turned back by the grid shift (dx, dy): the turn's index in float,
// nearest-even, mod 4096, and the rotation by the table's cos / sin, as liblizard/src/lizard_phy.c:214-218 computes them.
__device__ __forceinline__ float2 turned(const FmtDev &fd, const float2 *spec, int i, float dx, float dy) {
  const float2 z = spec[i];
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
// with the sums in pilot order. A rounding edge falls inside the bound (about 1e-12 of the shift) for about one frame
// in ten thousand; an empty or overflowing spectrum always takes the second way.
// Bound: the double pipe's latency (about 70 cycles an operation). One frame of n = 1536 (984 pilots) decoded: 277 us with
// the ordered sums (95 of them here), 200 with the tree.
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
// and what is worked out from them may be from the ordered sums': a sum in any order is within used u of the sum of its
// terms' magnitudes (u = 2^-53), itself the sum or, by Cauchy and Schwarz, the root of two. Every figure in float and
// taken generously; an infinity or a NaN fails the comparisons it is used in.
struct PilotBound {
  float ea, eb, ec, ep, eq, ey, det;   // the sums' and a c - b b's
};
constexpr float kU = 1.2e-16f;   // over 2^-53
__device__ __forceinline__ PilotBound pilot_bound(float a, float b, float c, float y, int used) {
  PilotBound e;
  const float E = (float)(used + 64) * 2.0f * kU;
  e.ea = E * a; e.ec = E * c; e.ey = E * y;
  e.eb = E * sqrtf(a) * sqrtf(c); e.ep = E * sqrtf(a) * sqrtf(y); e.eq = E * sqrtf(c) * sqrtf(y);
  e.det = 2.0f * (e.ea * c + a * e.ec + 2.0f * fabsf(b) * e.eb) + 8.0f * kU * (a * c + b * b);
  return e;
}

// Frame f's fit by the calling cluster. tm: this CTA's dynamic shared memory (chunk x 6 doubles at least).
__device__ __forceinline__ void pilot_align_frame(const FmtDev &fd, const float2 *spec, int64_t spec_stride, float *align, int f, double *tm) {
  __shared__ double part[kPilotWarps][6], sums[6], dxy[2];
  __shared__ int status;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), used = fd.npilot, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = (used + kPilotCtas - 1) / kPilotCtas, p0 = rank * chunk, p1 = min(used, p0 + chunk);
  const float2 *sp = spec + f * spec_stride;
  const double k = 2.0 * 3.14159265358979323846 / fd.n;
  for (int ordered = 0;; ordered = 1) {
    if (tid == 0) { dxy[0] = dxy[1] = 0; status = used < 8 ? kPilotGiveUp : kPilotOn; }
    cl.sync();
    if (status) break;
    float e_prev = 0;   // rank 0's lanes 0 and 1: the bound on dx's, dy's distance from the ordered one
    for (int it = 0; it < 2; it++) {
      const float dx = (float)dxy[0], dy = (float)dxy[1];
      double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int pi = p0 + tid; pi < p1; pi += kPilotThreads) {
        const int i = fd.pilot_coef[pi], w = fd.pilot_white[pi];
        const float2 y = turned(fd, sp, i, dx, dy);
        const double xr = (w & 1) ? -1.0 : 1.0, xi = (w & 2) ? -1.0 : 1.0;
        const double zr = (double)y.x * xr + (double)y.y * xi, zi = (double)y.y * xr - (double)y.x * xi;
        const double cu = k * zr * fd.uv[2 * i], cv = k * zr * fd.uv[2 * i + 1];
        const double t[6] = {cu * cu, cu * cv, cv * cv, cu * zi, cv * zi, zi * zi};
#pragma unroll
        for (int q = 0; q < 6; q++) {
          if (ordered) tm[6 * (pi - p0) + q] = t[q];
          else v[q] += t[q];
        }
      }
      if (!ordered) {
        const double s = warp_sum6(v, lane);
        const int q = 4 * (lane >> 4) + 2 * (lane >> 3 & 1) + (lane >> 2 & 1);
        if ((lane & 3) == 0 && q < 6) part[warp][q] = s;
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
        if (ordered) {
          a = sums[0]; b = sums[1]; c = sums[2]; p = sums[3]; q = sums[4]; yy = sums[5];
        } else {
          const double *rp = cl.map_shared_rank(&part[0][0], lane / kPilotWarps) + 6 * (lane % kPilotWarps);
#pragma unroll
          for (int j = 0; j < 6; j++) v[j] = rp[j];
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
        const PilotBound e = pilot_bound((float)a, (float)b, (float)c, (float)yy, used);
        if (ordered) {
          if (!(det > 0)) st = kPilotGiveUp;
        } else {
          const float fa = (float)a, fb = fabsf((float)b), fc = (float)c, fp = fabsf((float)p), fq = fabsf((float)q), fdet = (float)det;
          const float m = ly ? fa : fc, em = ly ? e.ea : e.ec, f1 = ly ? fq : fp, e1 = ly ? e.eq : e.ep, f2 = ly ? fp : fq, e2 = ly ? e.ep : e.eq;
          const float e_num = 2.0f * (e1 * m + f1 * em + e2 * fb + f2 * e.eb) + 8.0f * kU * (f1 * m + f2 * fb);
          const float fs = fabsf((float)step);
          e_step = 2.0f * (e_num + fs * e.det) / fdet + 8.0f * kU * fs;
          e_now = e_prev + e_step + 8.0f * kU * fabsf((float)now);
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
      if (status) break;
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

// Four lanes a sub-channel, 64 sub-channels a CTA. Lane q of a group sums the moments of coefficients q, q + 4, ...
// in order (the reference's four float chains) and the chains are added (c0 + c1) + (c2 + c3); one thread a
// sub-channel then works out the scale in double (so a warp's double work serves 32 sub-channels); the soft values
// are each axis times 8 k, NaN to 0, clamped to +-80, rounded half to even.
constexpr int kDemapBatch = 8;   // 320 / 4 = 80 coefficients a lane, 10 batches
static_assert(kSubDev % (4 * kDemapBatch) == 0, "whole batches");

__device__ __forceinline__ void demap_block(const FmtDev &fd, const float2 *spec, int64_t spec_stride, const float *align, int8_t *llrf,
                                            double *sub_est, float *sub_rms, int blk) {
  __shared__ float s_m[64][2], s_k8[64];
  const int grp = threadIdx.x >> 2, qd = threadIdx.x & 3, gid = blk * 64 + grp;
  const int f = gid / fd.subch, j = gid - f * fd.subch;
  const bool live = f < fd.frames;
  const float2 *sp = spec + (live ? f : 0) * spec_stride;
  const bool turn = live && align[3 * f + 2] != 0.0f;
  const float dx = live ? align[3 * f] : 0, dy = live ? align[3 * f + 1] : 0;
  float m2 = 0, m4 = 0;
  if (live) {
    // eight of the lane's coefficients loaded at a time (independent loads in flight), then summed in order
    for (int s0 = qd; s0 < kSubDev; s0 += 4 * kDemapBatch) {
      float2 y[kDemapBatch];
#pragma unroll
      for (int b = 0; b < kDemapBatch; b++) {
        const int i = j * kSubDev + s0 + 4 * b;
        y[b] = turn ? turned(fd, sp, i, dx, dy) : sp[i];
      }
#pragma unroll
      for (int b = 0; b < kDemapBatch; b++) {
        const float e = y[b].x * y[b].x + y[b].y * y[b].y;
        m2 = m2 + e; m4 = m4 + e * e;
      }
    }
  }
  // (c0 + c1) + (c2 + c3)
  const float o2 = __shfl_down_sync(0xffffffffu, m2, 1), o4 = __shfl_down_sync(0xffffffffu, m4, 1);
  const float p2 = m2 + o2, p4 = m4 + o4;
  const float r2 = __shfl_down_sync(0xffffffffu, p2, 2), r4 = __shfl_down_sync(0xffffffffu, p4, 2);
  if (qd == 0) { s_m[grp][0] = p2 + r2; s_m[grp][1] = p4 + r4; }
  __syncthreads();
  if (threadIdx.x < 64) {
    const int g2 = blk * 64 + threadIdx.x, f2 = g2 / fd.subch, j2 = g2 - f2 * fd.subch;
    float k8 = 0;
    if (f2 < fd.frames) {
      const double M2 = (double)s_m[threadIdx.x][0] / kSubDev, M4 = (double)s_m[threadIdx.x][1] / kSubDev;
      sub_rms[f2 * fd.subch + j2] = M2 > 0 ? (float)sqrt(M2 / 2) : 0;
      double a2 = 2 * M2 * M2 - M4;
      a2 = a2 > 0 ? sqrt(a2) : 0;
      double nv = M2 - a2;
      if (nv < 0.02 * M2) nv = 0.02 * M2;
      sub_est[f2 * fd.subch + j2] = axis_info(a2 / nv);
      const float kk = (float)(0.7 * 2 * sqrt(2 * a2) / nv);
      k8 = 8 * kk;
    }
    s_k8[threadIdx.x] = k8;
  }
  __syncthreads();
  if (!live) return;
  const float k8 = s_k8[grp];
  int8_t *out = llrf + (int64_t)f * fd.subch * 2 * kSubDev + 2 * j * kSubDev;
  for (int s0 = qd; s0 < kSubDev; s0 += 4 * kDemapBatch) {
    float2 y[kDemapBatch];
#pragma unroll
    for (int b = 0; b < kDemapBatch; b++) {
      const int i = j * kSubDev + s0 + 4 * b;
      y[b] = turn ? turned(fd, sp, i, dx, dy) : sp[i];
    }
#pragma unroll
    for (int b = 0; b < kDemapBatch; b++) {
      float x = k8 * y[b].x, z = k8 * y[b].y;
      x = x != x ? 0.0f : fminf(fmaxf(x, -80.0f), 80.0f);
      z = z != z ? 0.0f : fminf(fmaxf(z, -80.0f), 80.0f);
      char2 v;
      v.x = (signed char)__float2int_rn(x);
      v.y = (signed char)__float2int_rn(z);
      *reinterpret_cast<char2 *>(out + 2 * (s0 + 4 * b)) = v;
    }
  }
}

__global__ void __launch_bounds__(256) demap_kernel(FmtDev fd, const float2 *spec, int64_t spec_stride, const float *align,
                                                    int8_t *llrf, double *sub_est, float *sub_rms) {
  demap_block(fd, spec, spec_stride, align, llrf, sub_est, sub_rms, blockIdx.x);
}

// One thread a block: its estimate (its sub-channels' information weighted by the slots it holds there, in double, in
// order), its pilot reading (the tail's axis values against the whitening in units of their sub-channel's rms, in
// double, in order; NaN where none was read) and the decline gate (est < 0.2 k / nt in float): decl[f blocks + b] = 1.
constexpr int kBlocksThreads = 128;
__device__ __forceinline__ void blocks_block(const FmtDev &fd, const float2 *spec, int64_t spec_stride, const float *align,
                                             const double *sub_est, const float *sub_rms, float *est, float *pilot, uint8_t *decl, int blk) {
  const int g = blk * kBlocksThreads + threadIdx.x;
  if (g >= fd.frames * fd.blocks) return;
  const int f = g / fd.blocks, b = g - f * fd.blocks;
  const int t = fd.block_tier[b], nb = fd.tier_slots[t], s0 = fd.block_slot[b], nt = fd.tier_nt[t];
  const double *se = sub_est + f * fd.subch;
  const float *sr = sub_rms + f * fd.subch;
  double info = 0;
  for (int j = s0 / (2 * kSubDev); j * 2 * kSubDev < s0 + nb; j++) {
    const int lo = max(s0, 2 * kSubDev * j), hi = min(s0 + nb, 2 * kSubDev * (j + 1));
    info += se[j] * (hi - lo);
  }
  const float e = (float)(info / nb);
  est[g] = e;
  float pv = __int_as_float(0x7fc00000);   // NaN: no pilot read
  if (nt < nb) {
    const float2 *sp = spec + f * spec_stride;
    const bool turn = align[3 * f + 2] != 0.0f;
    const float dx = align[3 * f], dy = align[3 * f + 1];
    double cs = 0;
    int got = 0;
    for (int i = nt; i < nb; i++) {
      const int gs = s0 + i, ci = gs / 2;
      const float rms = sr[gs / (2 * kSubDev)];
      if (!(rms > 0)) continue;
      const float2 y = turn ? turned(fd, sp, ci, dx, dy) : sp[ci];
      const float yv = (i & 1) ? y.y : y.x;
      cs += (fd.white[gs] ? -1.0 : 1.0) * yv / rms;
      got++;
    }
    if (got) pv = (float)(cs / (nb - nt));
  }
  pilot[g] = pv;
  decl[g] = e < 0.2f * (float)fd.tier_k[t] / (float)nt;
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

__global__ void __launch_bounds__(256) demap_mixed_kernel(const __grid_constant__ DemapMix m) {
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
    m.df[k + 1] = m.df[k] + (fd.frames * fd.subch + 63) / 64;
    m.bf[k + 1] = m.bf[k] + (fd.frames * fd.blocks + kBlocksThreads - 1) / kBlocksThreads;
  }
  if (psm > 48 * 1024) return cudaErrorInvalidValue;
  pilot_align_mixed_kernel<<<m.pf[count] * kPilotCtas, kPilotThreads, psm, st>>>(m);
  demap_mixed_kernel<<<m.df[count], 256, 0, st>>>(m);
  blocks_mixed_kernel<<<m.bf[count], kBlocksThreads, 0, st>>>(m);
  return cudaGetLastError();
}

cudaError_t demap_launch(const FmtDev &fd, const float2 *spec, int64_t spec_stride, float *align, int8_t *llrf,
                         double *sub_est, float *sub_rms, float *est, float *pilot, uint8_t *decl, cudaStream_t st) {
  const int chunk = (fd.npilot + kPilotCtas - 1) / kPilotCtas;
  const int psm = 6 * (chunk > 0 ? chunk : 1) * (int)sizeof(double);
  if (psm > 48 * 1024) return cudaErrorInvalidValue;
  pilot_align_kernel<<<fd.frames * kPilotCtas, kPilotThreads, psm, st>>>(fd, spec, spec_stride, align);
  const int groups = fd.frames * fd.subch;
  demap_kernel<<<(groups + 63) / 64, 256, 0, st>>>(fd, spec, spec_stride, align, llrf, sub_est, sub_rms);
  const int nbk = fd.frames * fd.blocks;
  blocks_kernel<<<(nbk + kBlocksThreads - 1) / kBlocksThreads, kBlocksThreads, 0, st>>>(fd, spec, spec_stride, align, sub_est, sub_rms, est,
                                                                                       pilot, decl);
  return cudaGetLastError();
}

}  // namespace lizg
