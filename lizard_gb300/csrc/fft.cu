// Row (b) of the hot path on sm_103a: the anchors' erase, the detrend projections and the 2D mixed-radix FFT of the
// n x n picture grid, restated from the reference's decode (liblizard/src/lizard_phy.c:1596-1716) for the GPU.
//
// Four kernels a batch (five when the samples come straight from captured frames):
//   hole_rhs_kernel   a CTA takes a band of the frame's every-eighth-sample rows: the shading fit's right-hand side
//                     over the samples outside the anchors' squares, one partial sum a band (6 doubles); the frame's
//                     last CTA to finish adds the bands and solves for the shading surface beta;
//   sample16_kernel   (captured frames by the decode's read) the samples, 16 bits each, in a bounded workspace: a batch
//                     past it takes the kernels to here and the column pass in turns;
//   cell_table_kernel (captured frames by the exact walk) each picture row's homography terms and the mesh displacement
//                     line of each mesh cell along it, so the column pass reads them instead of walking the mesh per
//                     sample;
//   fft_cols_kernel   a CTA takes 2L picture columns of a frame (L complex lines: column x0 + l real, x0 + L + l
//                     imaginary), erases the anchors' squares to the shading surface, loads the rest, sums each
//                     column's detrend moments, transforms the L lines along y in shared memory and separates the two
//                     real columns of each, writing Y[v][x] for the kept rows v;
//   fac_kernel        kFacCtas CTAs a frame: the five projections from the columns' moments, then the surface spectrum's
//                     per-column and per-row factors (the double products the reference rounds to float);
//   fft_rows_kernel   a CTA takes L kept rows v of a frame, transforms along x and subtracts the surface's spectrum
//                     (the xy term everywhere, the x terms on v = 0, the y terms on u = 0), writing the used
//                     coefficients in pos order.
// L is the most lines of n points that fit 6144 complex points (so every CTA holds about the same 48 KB of samples).
//
// The transforms are Stockham autosort passes of radix 16, 9, 8, 6, 5, 4, 3 or 2 (every ladder size takes three),
// each pass in place: every thread reads its butterflies' points into registers, the CTA waits, every thread writes
// its outputs. Shared memory holds a line with one spare slot after every 16 points (so the passes' 16-point runs,
// read or written, fall on distinct banks within a half-warp) and lines 16 / L (mod 16) slots apart; the passes'
// twiddles sit beside the lines, per pass [r - 1][k], so a warp reads consecutive entries. FP32 throughout, as the
// reference's; the twiddles and the surface factors are worked out in double.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>
#include "lizg_internal.h"
#include "sample_dev.cuh"

namespace lizg {

constexpr int kThreads = 384;   // threads of a transform CTA
constexpr int kHoleBand = 16;   // every-eighth-sample rows a hole_rhs CTA takes

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// A point's slot in its line: one spare slot after every 16.
__device__ __forceinline__ int pad(int p) { return p + (p >> 4); }

// Forward DFTs (e^{-i}) of R points in place.
template <int R> __device__ __forceinline__ void dft(float2 *v);

template <> __device__ __forceinline__ void dft<2>(float2 *v) { const float2 a = v[0], b = v[1]; v[0] = cadd(a, b); v[1] = csub(a, b); }
template <> __device__ __forceinline__ void dft<4>(float2 *v) {
  const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]), s13 = cadd(v[1], v[3]), d13 = csub(v[1], v[3]);
  v[0] = cadd(s02, s13); v[2] = csub(s02, s13);
  v[1] = make_float2(d02.x + d13.y, d02.y - d13.x);   // d02 - i d13
  v[3] = make_float2(d02.x - d13.y, d02.y + d13.x);   // d02 + i d13
}
template <> __device__ __forceinline__ void dft<3>(float2 *v) {
  const float s3 = 0.86602540378443864676f;
  const float2 a = v[0], t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
  const float2 m = make_float2(a.x - 0.5f * t.x, a.y - 0.5f * t.y);
  v[0] = cadd(a, t);
  v[1] = make_float2(m.x + s3 * d.y, m.y - s3 * d.x);   // m - i s3 d
  v[2] = make_float2(m.x - s3 * d.y, m.y + s3 * d.x);   // m + i s3 d
}
template <> __device__ __forceinline__ void dft<5>(float2 *v) {
  const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;   // cos 2pi/5, cos 4pi/5
  const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;    // sin 2pi/5, sin 4pi/5
  const float2 a = v[0], p1 = cadd(v[1], v[4]), m1 = csub(v[1], v[4]), p2 = cadd(v[2], v[3]), m2 = csub(v[2], v[3]);
  const float2 r1 = make_float2(a.x + c1 * p1.x + c2 * p2.x, a.y + c1 * p1.y + c2 * p2.y);
  const float2 r2 = make_float2(a.x + c2 * p1.x + c1 * p2.x, a.y + c2 * p1.y + c1 * p2.y);
  const float2 q1 = make_float2(s1 * m1.x + s2 * m2.x, s1 * m1.y + s2 * m2.y);   // times -i below
  const float2 q2 = make_float2(s2 * m1.x - s1 * m2.x, s2 * m1.y - s1 * m2.y);
  v[0] = make_float2(a.x + p1.x + p2.x, a.y + p1.y + p2.y);
  v[1] = make_float2(r1.x + q1.y, r1.y - q1.x);
  v[4] = make_float2(r1.x - q1.y, r1.y + q1.x);
  v[2] = make_float2(r2.x + q2.y, r2.y - q2.x);
  v[3] = make_float2(r2.x - q2.y, r2.y + q2.x);
}

// e^{-2 pi i m / R} for the m a composite DFT turns by that are not eighth turns.
template <int R> __device__ __forceinline__ float2 wconst(int m);
template <> __device__ __forceinline__ float2 wconst<16>(int m) {
  return m == 1 ? make_float2(0.92387953251128673848f, -0.38268343236508978178f)
       : m == 3 ? make_float2(0.38268343236508983729f, -0.92387953251128673848f)
                : make_float2(-0.92387953251128684951f, 0.38268343236508967076f);   // m = 9
}
template <> __device__ __forceinline__ float2 wconst<8>(int) { return make_float2(1.0f, 0.0f); }   // every turn of 8 is an eighth
template <> __device__ __forceinline__ float2 wconst<6>(int m) {
  return m == 1 ? make_float2(0.5f, -0.86602540378443864676f) : make_float2(-0.5f, -0.86602540378443864676f);   // m = 2
}
template <> __device__ __forceinline__ float2 wconst<9>(int m) {
  return m == 1 ? make_float2(0.76604444311897801345f, -0.64278760968653925190f)
       : m == 2 ? make_float2(0.17364817766693041445f, -0.98480775301220802032f)
                : make_float2(-0.93969262078590831688f, -0.34202014332566887944f);   // m = 4
}
// a e^{-2 pi i m / R} for a constant m (after unrolling): quarter and eighth turns by adds, the rest by cos/sin.
template <int R> __device__ __forceinline__ float2 twc(float2 a, int m) {
  m %= R;
  const float c = 0.70710678118654757274f;
  if (m == 0) return a;
  if (4 * m == R) return make_float2(a.y, -a.x);
  if (2 * m == R) return make_float2(-a.x, -a.y);
  if (4 * m == 3 * R) return make_float2(-a.y, a.x);
  if (8 * m == R) return make_float2(c * (a.x + a.y), c * (a.y - a.x));
  if (8 * m == 3 * R) return make_float2(c * (a.y - a.x), -c * (a.x + a.y));
  return cmul(a, wconst<R>(m));
}

// R = P Q points by P-point DFTs over the Q interleaved subsequences, twiddles, then Q-point DFTs:
// X[k1 + P k2] = sum_n2 W_Q^{n2 k2} W_R^{n2 k1} sum_n1 x[Q n1 + n2] W_P^{n1 k1}.
template <int P, int Q> __device__ __forceinline__ void dft_pq(float2 *x) {
  constexpr int R = P * Q;
  float2 a[Q][P];
#pragma unroll
  for (int n2 = 0; n2 < Q; n2++) {
#pragma unroll
    for (int n1 = 0; n1 < P; n1++) a[n2][n1] = x[Q * n1 + n2];
    dft<P>(a[n2]);
#pragma unroll
    for (int k1 = 1; k1 < P; k1++) a[n2][k1] = twc<R>(a[n2][k1], n2 * k1);
  }
#pragma unroll
  for (int k1 = 0; k1 < P; k1++) {
    float2 b[Q];
#pragma unroll
    for (int n2 = 0; n2 < Q; n2++) b[n2] = a[n2][k1];
    dft<Q>(b);
#pragma unroll
    for (int k2 = 0; k2 < Q; k2++) x[k1 + P * k2] = b[k2];
  }
}
template <> __device__ __forceinline__ void dft<8>(float2 *v) { dft_pq<4, 2>(v); }
template <> __device__ __forceinline__ void dft<16>(float2 *v) { dft_pq<4, 4>(v); }
template <> __device__ __forceinline__ void dft<6>(float2 *v) { dft_pq<3, 2>(v); }
template <> __device__ __forceinline__ void dft<9>(float2 *v) { dft_pq<3, 3>(v); }

// The transform plan of each ladder size: three passes' radices and the lines a CTA holds (the most lines of n
// points within kFftPoints, n a multiple of twice that). Host and device read the same table.
struct Plan {
  int r0, r1, r2, lines;
};
__host__ __device__ constexpr Plan plan_of(int n) {
  return n == 384    ? Plan{16, 8, 3, 16}
         : n == 512  ? Plan{16, 16, 2, 8}
         : n == 768  ? Plan{16, 16, 3, 8}
         : n == 1024 ? Plan{16, 16, 4, 4}
         : n == 1152 ? Plan{16, 8, 9, 4}
         : n == 1280 ? Plan{16, 16, 5, 4}
         : n == 1536 ? Plan{16, 16, 6, 4}
                     : Plan{0, 0, 0, 0};
}
// Slots from one line to the next: the padded line rounded up to 16 slots, plus 16 / L, so that the L lines x
// 16 / L rows a half-warp stores while loading (and reads while separating) fall on 16 distinct slots.
__host__ __device__ constexpr int lstride_of(int n) { return (n + n / 16 + 15) / 16 * 16 + 16 / plan_of(n).lines; }

// The thread's index, read afresh: the passes' offsets hang on it, so a loop round the passes recomputes them pass by
// pass instead of holding every pass's offsets live across the loop.
__device__ __forceinline__ int tid_fresh() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// pad(a + r S) for a butterfly's points r S apart, S a multiple of 8 (or, from a multiple of 16, 16 points 1 apart): a slot
// worked out once (or once for the even points and once for the odd) and constant steps from it, which the accesses hold
// as offsets. Worked out point by point, slots were most of the integer instructions the passes were bound by (the ALU pipe
// 62 to 65% busy, the FMA pipe 26 to 31%): with them and the outer passes straight from and to memory, 32 pages of n = 1536
// by rows 98 us then 66 and by columns 154 then 127; 24 frames of the refinement's adjoint 74 then 52, 189 then 148.
template <int S> struct Slots {
  static_assert(S == 1 || S % 8 == 0, "the slots' steps");
  int even, odd;
  __device__ __forceinline__ explicit Slots(int a) : even(pad(a)), odd(S % 16 == 8 ? pad(a + S) : 0) {}
  __device__ __forceinline__ int operator()(int r) const {
    return S == 1 ? even + r : S % 16 == 0 ? even + r * (S + S / 16) : (r & 1 ? odd : even) + (r >> 1) * (2 * S + S / 8);
  }
};

// One Stockham pass of radix R over the CTA's lines (Lr <= L of them) in place, n = N points a line. Butterfly j of
// a line (j < NR = N / R, k = j mod NS) reads points j + r NR, turns point r by e^{-2 pi i r k / (NS R)}
// (tw[NS + (r - 1) NS + k]) and writes its DFT's output r to point (j / NS) NS R + k + r NS. A thread takes butterflies
// tid, tid + kThreads, ... (at most B = ceil(L NR / kThreads) of them), a line's one after another, or with LFAST the
// lines' j-th ones together (Lr = L). `in(l, j)` gives a butterfly's points and `out(l, point)` takes its outputs, as
// callables of r; LinesIn and LinesOut are the lines themselves. An output elsewhere is the last pass's: nothing waits
// for its reads, and the CTA is not synchronised after it.
template <int N, int NR> struct LinesIn {
  const float2 *buf;
  struct At {
    const float2 *line;
    Slots<NR> at;
    __device__ __forceinline__ float2 operator()(int r) const { return line[at(r)]; }
  };
  __device__ __forceinline__ At operator()(int l, int j) const { return At{buf + l * lstride_of(N), Slots<NR>(j)}; }
};
template <int N, int NS> struct LinesOut {
  float2 *buf;
  struct At {
    float2 *line;
    Slots<NS> at;
    __device__ __forceinline__ void operator()(int r, float2 v) const { line[at(r)] = v; }
  };
  __device__ __forceinline__ At operator()(int l, int p) const { return At{buf + l * lstride_of(N), Slots<NS>(p)}; }
};
template <int N, int R, int NS, int L, bool LFAST, bool ELSEWHERE, class In, class Out>
__device__ __forceinline__ void pass_via(const float2 *tw, int Lr, const In &in, const Out &out) {
  constexpr int NR = N / R, B = (L * NR + kThreads - 1) / kThreads;
  static_assert(NS != 1 || R == 16, "a first pass's outputs start on a multiple of 16");
  const int total = Lr * NR, tid = tid_fresh();
  float2 v[ELSEWHERE ? 1 : B][R];
#pragma unroll
  for (int b = 0; b < B; b++) {
    const int t = tid + b * kThreads;
    float2 *x = v[ELSEWHERE ? 0 : b];
    if (t < total) {
      const int l = LFAST ? t % L : t / NR, j = LFAST ? t / L : t - l * NR, k = j % NS;
      const auto from = in(l, j);
#pragma unroll
      for (int r = 0; r < R; r++) x[r] = from(r);
      if (NS > 1) {
#pragma unroll
        for (int r = 1; r < R; r++) x[r] = cmul(x[r], tw[NS + (r - 1) * NS + k]);
      }
      dft<R>(x);
      if (ELSEWHERE) {
        const auto to = out(l, (j / NS) * NS * R + k);
#pragma unroll
        for (int r = 0; r < R; r++) to(r, x[r]);
      }
    }
  }
  if (ELSEWHERE) return;
  __syncthreads();
#pragma unroll
  for (int b = 0; b < B; b++) {
    const int t = tid + b * kThreads;
    if (t < total) {
      const int l = LFAST ? t % L : t / NR, j = LFAST ? t / L : t - l * NR, jq = j / NS, k = j - jq * NS;
      const auto to = out(l, jq * NS * R + k);
#pragma unroll
      for (int r = 0; r < R; r++) to(r, v[ELSEWHERE ? 0 : b][r]);
    }
  }
  __syncthreads();
}
template <int N, int R, int NS, int L>
__device__ __forceinline__ void pass(float2 *buf, const float2 *tw, int Lr) {
  pass_via<N, R, NS, L, false, false>(tw, Lr, LinesIn<N, N / R>{buf}, LinesOut<N, NS>{buf});
}

// The Lr lines at buf (line l at buf + l lstride_of(N), point p at slot pad(p)) transformed along their N points by the
// size's three passes. tw: the passes' twiddles, pass s's at NS (a multiple of 16 past the first pass, so a
// half-warp's 16 twiddles are one aligned 128-byte row). Every thread of the CTA takes part. In place (later_passes);
// or with the first pass's points from elsewhere (first_pass_from, in(l, j) at points r N / r0 apart from j) and the last
// pass's outputs elsewhere (last_pass_to, out(l, p) at points r N / r2 apart from p).
template <int N, bool LFAST = false, class In>
__device__ __forceinline__ void first_pass_from(float2 *buf, const float2 *tw, int Lr, const In &in) {
  constexpr Plan P = plan_of(N);
  pass_via<N, P.r0, 1, P.lines, LFAST, false>(tw, Lr, in, LinesOut<N, 1>{buf});
}
template <int N>
__device__ __forceinline__ void middle_pass(float2 *buf, const float2 *tw, int Lr) {
  constexpr Plan P = plan_of(N);
  pass<N, P.r1, P.r0, P.lines>(buf, tw, Lr);
}
template <int N, bool LFAST = false, class Out>
__device__ __forceinline__ void last_pass_to(const float2 *buf, const float2 *tw, int Lr, const Out &out) {
  constexpr Plan P = plan_of(N);
  pass_via<N, P.r2, P.r0 * P.r1, P.lines, LFAST, true>(tw, Lr, LinesIn<N, N / P.r2>{buf}, out);
}
template <int N>
__device__ __forceinline__ void later_passes(float2 *buf, const float2 *tw, int Lr) {
  constexpr Plan P = plan_of(N);
  middle_pass<N>(buf, tw, Lr);
  pass<N, P.r2, P.r0 * P.r1, P.lines>(buf, tw, Lr);
}

// A frame's shading-fit sample (x, y) = (8 kx, 8 ky) from a supplied grid or by the exact walk of the captured frame
// (the decode's read walks the row: hole_rhs_band).
__device__ __forceinline__ float shade_at(const SrcDev &s, int f, int x, int y) {
  if (!s.luma) return s.grid[f * s.gstride + (int64_t)y * s.sd.n + x];
  const float *H = s.reg + (int64_t)f * s.regstride;
  return sample_xy_exact(s.sd, s.luma + f * s.fstride, s.w, s.h, s.pitch, H, H + 9, s.sd.colt[x], s.sd.rowt[y]);
}

__device__ __forceinline__ bool in_square(const FftDev &xd, int t) {
  bool in = false;
#pragma unroll
  for (int i = 0; i < 7; i++) in |= t >= xd.elo[i] && t <= xd.ehi[i];
  return in;
}

// The shading fit's right-hand side (liblizard/src/lizard_phy.c:1609-1623) over kHoleBand of the frame's every-eighth
// rows, hole[f][band][0..5], then, by the frame's last CTA to finish (its ticket), the surface beta[f][0..5] from the
// bands in order. A warp takes a row: its samples outside the squares summed in float as z, z c(x), z q(x) (the basis is
// separable: 1, c(x), q(x), c(y), q(y), c(x) c(y)), then the row's six terms added in double, rows w and w + 8, then w
// in order. The decode's read is the reference's one call over every eighth column (liblizard/src/lizard_phy.c:1611):
// lane l takes columns l, l + 32, ..., so its homography lane is walked on eight steps from one to the next, and its G
// samples' loads (hole_cols: 2 at n = 384, 6 at 1536) are in flight together. Bound: latency. A frame of n = 1536: 26 us
// with two rows a warp, each sample walked from the first column, 15 so; and the column pass no longer adds the bands in
// every CTA (39 us, 35).
constexpr int kHoleThreads = 32 * kHoleBand;
static_assert(kHoleBand == 16, "rows w and w + 8 of a band share a sum");
__host__ __device__ constexpr int hole_cols(int n) { return (n / 8 + 31) / 32; }   // a lane's columns
struct HoleShared {
  double red[8][6], rhs[6];
  float row[kHoleBand][3];
  bool last;
};
template <int G>
__device__ __forceinline__ void hole_rhs_band(const FftDev &xd, const SrcDev &src, int bands, double *hole, double *beta, int *ticket, int f,
                                              int band, HoleShared &sh) {
  const int n = xd.n, c = n / 8, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ky = band * kHoleBand + warp, y = 8 * ky;
  if (ky < c) {
    const bool ysq = in_square(xd, y);
    float v[G];
    if (src.luma && src.sd.read == LIZG_READ_DECODE) {
      const float *H = src.reg + (int64_t)f * src.regstride;
      const uint8_t *px = src.luma + f * src.fstride;
      const RowTerms r = row_terms(H, src.sd.rowt[y]);
      const LinCol lc = lin_col_shade(src.sd, H, lane);
      LinNum s = lin_start(lc, r.kw, r.ku, r.kv);
      lin_steps(lc, s, lc.g);
#pragma unroll
      for (int m = 0; m < G; m++) {
        const int x = 8 * min(lane + 32 * m, c - 1);
        v[m] = lin_point(px, src.w, src.h, src.pitch, s, lin_cell(src.sd, H + 9, src.sd.colt[x], r.j), r.v);
#pragma unroll
        for (int q = 0; q < 8; q++) lin_steps(lc, s, 1);
      }
    } else {
#pragma unroll
      for (int m = 0; m < G; m++) v[m] = shade_at(src, f, 8 * min(lane + 32 * m, c - 1), y);
    }
    float s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
    for (int m = 0; m < G; m++) {
      const int kx = lane + 32 * m, x = 8 * kx;
      if (kx < c && !(ysq && in_square(xd, x))) { s0 += v[m]; s1 += __ldg(xd.cx + x) * v[m]; s2 += __ldg(xd.qx + x) * v[m]; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) { sh.row[warp][0] = s0; sh.row[warp][1] = s1; sh.row[warp][2] = s2; }
  }
  __syncthreads();
  if (tid < 48) {
    const int w = tid / 6, r = tid % 6, k = r < 3 ? r : r == 5 ? 1 : 0;   // terms s0, s1, s2, c(y) s0, q(y) s0, c(y) s1
    double acc = 0;
    for (int row = w; row < kHoleBand; row += 8) {
      const int kr = band * kHoleBand + row;
      if (kr >= c) break;
      const double sv = sh.row[row][k], b = r < 3 ? 1.0 : r == 4 ? xd.qx[8 * kr] : xd.cx[8 * kr];
      acc = fma(b, sv, acc);
    }
    sh.red[w][r] = acc;
  }
  __syncthreads();
  if (tid < 6) {
    double acc = 0;
    for (int w = 0; w < 8; w++) acc += sh.red[w][tid];
    __stcg(hole + ((int64_t)f * bands + band) * 6 + tid, acc);
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) {
    sh.last = atomicAdd(ticket + f, 1) == bands - 1;
    __threadfence();
  }
  __syncthreads();
  if (!sh.last || tid >= 32) return;
  if (tid < 6) {
    double acc = 0;
    for (int b0 = 0; b0 < bands; b0 += 12) {   // the bands' loads in flight, then added in order
      double v[12];
#pragma unroll
      for (int k = 0; k < 12; k++) v[k] = b0 + k < bands ? __ldcg(hole + ((int64_t)f * bands + b0 + k) * 6 + tid) : 0.0;
#pragma unroll
      for (int k = 0; k < 12; k++) if (b0 + k < bands) acc += v[k];
    }
    sh.rhs[tid] = acc;
  }
  __syncwarp();
  if (tid < 6) {
    double acc = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) acc += xd.hole_inv[tid * 6 + k] * sh.rhs[k];
    beta[6 * f + tid] = acc;
  }
  if (tid == 0) ticket[f] = 0;   // as the next call finds it
}
template <int G>
__global__ void __launch_bounds__(kHoleThreads) hole_rhs_kernel(FftDev xd, SrcDev src, int bands, double *hole, double *beta, int *ticket) {
  __shared__ HoleShared sh;
  hole_rhs_band<G>(xd, src, bands, hole, beta, ticket, blockIdx.x / bands, blockIdx.x % bands, sh);
}

// The transform CTA's dynamic shared memory: the lines, the twiddles.
struct SmemMap {
  float2 *buf, *tw;
};
__host__ __device__ constexpr int smem_bytes_of(int n) { return (plan_of(n).lines * lstride_of(n) + n) * (int)sizeof(float2); }
template <int N>
__device__ __forceinline__ SmemMap smem_map(unsigned char *raw) {
  float2 *buf = reinterpret_cast<float2 *>(raw);
  return SmemMap{buf, buf + plan_of(N).lines * lstride_of(N)};
}

__host__ __device__ constexpr int cmax_i(int x, int y) { return x > y ? x : y; }

// The mixed-size grids' kernel arguments: each format's tables and buffers, and its first CTA (first[nseg] CTAs in all).
struct FftColsSeg {
  FftDev xd;
  SrcDev src;
  const float4 *ctab;
  const int16_t *g16;
  const double *beta;
  double *part;
  float2 *Y;
};
struct FftColsMix {
  FftColsSeg seg[kFftMixSegs];
  int first[kFftMixSegs + 1];
  int nseg;
};
struct FftRowsSeg {
  CUtensorMap ymap;
  FftDev xd;
  const float2 *fac;
  const int32_t *tpos;
  float2 *C;
  int *err;
  int need;
};
struct FftRowsMix {
  FftRowsSeg seg[kFftMixSegs];
  int first[kFftMixSegs + 1];
  int nseg;
};
static_assert(sizeof(FftColsMix) <= 32000 && sizeof(FftRowsMix) <= 32000, "the mixed grids' arguments fit a launch");

// The exact walk's per-row quantities of a batch, worked out once a frame before the column pass reads them, with the
// same functions and inputs as the per-sample walk (the cell's 1 / width as the column table computes it), so the
// column pass reads the walk's own values. A thread an entry, entries in table order: for picture row y and mesh cell
// i < nx - 1 the displacement line cell_terms gives, and at i = nx - 1 the homography's row terms (kw, ku, kv).
__device__ __forceinline__ void cell_table_entry(const SrcDev &src, int per_frame, float4 *ctab, int f, int t) {
  if (t >= per_frame) return;
  const SampleDev &sd = src.sd;
  const float *H = src.reg + (int64_t)f * src.regstride;
  const int nn = sd.nx, y = t / nn, i = t - y * nn;
  const RowTerms r = row_terms(H, sd.rowt[y]);
  float4 o;
  if (i == nn - 1) {
    o = make_float4(r.kw, r.ku, r.kv, 0.0f);
  } else {
    const float inv = __fdiv_rn(1.0f, __fsub_rn(sd.node_x[i + 1], sd.node_x[i]));
    const CellTerms c = cell_terms(sd, H + 9, i, inv, r);
    o = make_float4(c.ex, c.cx, c.ey, c.cy);
  }
  ctab[(int64_t)f * per_frame + t] = o;
}

// Two floats in a 64-bit register, added in one instruction on sm_103a, each rounded as its scalar sum is. (Not multiplied
// so: the assembler fuses a packed product with the sum it goes into, rounding modifier or not.)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 addx2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// The place of picture sample (x, y) in a frame of 16-bit samples: a column tile's samples together, row by row, a line's
// two columns side by side, so that a warp of the column pass loads one run of bytes (row by row of the picture they
// were 16 bytes a line, 279 us a pass over 32 frames of n = 1536 against 210).
__device__ __forceinline__ int g16_at(int n, int lines, int x, int y) { return pic_at(n, lines, x) + y * 2 * lines; }

// The decode's read of a strip of 64 columns of a frame's rows, the blend's whole numbers (16 bits a sample,
// exact) into g16 for the column pass. A warp takes `rows` rows, two at a time, lane l columns l and l + 32 of the
// strip: a load reads neighbouring pixels of one row of the picture, the homography's lanes are stepped two rows
// to an instruction (on to the lane's column, then eight steps to the second), and a column's displacement terms are
// worked out once a mesh row.
// Bound: instruction issue (77%; 103 instructions a sample) and the luma's latency. Fused into the column pass instead,
// the samples waited on a third of the warps between the transform's barriers: 32 frames of n = 1536 decoded in 906 us
// against 883, one of n = 384 in 135 against 123.
constexpr int kSampleThreads = kHoleThreads, kSampleWarps = kSampleThreads / 32;
template <class Off>
__device__ __forceinline__ void sample_strip(const SrcDev &src, int16_t *g16, int f, int strip, int y0, int y1) {
  const SampleDev &sd = src.sd;
  const int n = sd.n, lane = threadIdx.x & 31, x = strip * 64 + lane, w2 = src.w - 2, h2 = src.h - 2;
  const float *reg = src.reg + (int64_t)f * src.regstride;
  float H[8];
#pragma unroll
  for (int k = 0; k < 8; k++) H[k] = __ldg(reg + k);
  const uint8_t *px = src.luma + f * src.fstride;
  const LinCol lc = lin_col_grid(sd, H, x);
  const f32x2 cw = pack2(lc.cw, lc.cw), cu = pack2(lc.cu, lc.cu), cv = pack2(lc.cv, lc.cv);
  const float4 c0 = sd.colt[x], c1 = sd.colt[x + 32];
  const int lines = plan_of(n).lines, row = 2 * lines;   // a row of a tile
  int16_t *out = g16 + (int64_t)f * n * n + g16_at(n, lines, x, y0);
  const int to32 = g16_at(n, lines, x + 32, 0) - g16_at(n, lines, x, 0);
  float4 T0{}, T1{};
  int j = -1;
  for (int y = y0; y < y1;) {
    const float4 ta = __ldg(sd.rowt + y), tb = __ldg(sd.rowt + min(y + 1, y1 - 1));
    const RowTerms ra = row_terms(H, ta), rb = row_terms(H, tb);
    const bool two = y + 1 < y1 && rb.j == ra.j;   // else the row alone (its pair's work goes nowhere)
    if (ra.j != j) {
      j = ra.j;
      T0 = lin_cell(sd, reg + 9, c0, j); T1 = lin_cell(sd, reg + 9, c1, j);
    }
    f32x2 W = pack2(__fadd_rn(lc.bw, __fadd_rn(lc.w0, ra.kw)), __fadd_rn(lc.bw, __fadd_rn(lc.w0, rb.kw)));
    f32x2 U = pack2(__fadd_rn(lc.bu, __fadd_rn(lc.u0, ra.ku)), __fadd_rn(lc.bu, __fadd_rn(lc.u0, rb.ku)));
    f32x2 V = pack2(__fadd_rn(lc.bv, __fadd_rn(lc.v0, ra.kv)), __fadd_rn(lc.bv, __fadd_rn(lc.v0, rb.kv)));
#pragma unroll
    for (int s = 0; s < 7; s++)
      if (s < lc.g) { W = addx2(W, cw); U = addx2(U, cu); V = addx2(V, cv); }
    int o[2][2];
#pragma unroll
    for (int half = 0; half < 2; half++) {
      const float4 T = half ? T1 : T0;
      float wa, wb, ua, ub, va, vb;
      unpack2(W, wa, wb); unpack2(U, ua, ub); unpack2(V, va, vb);
      const float rwa = __frcp_rn(wa), rwb = __frcp_rn(wb);
      const float xa = __fadd_rn(__fadd_rn(T.x, __fmul_rn(T.y, ra.v)), __fmul_rn(ua, rwa));
      const float xb = __fadd_rn(__fadd_rn(T.x, __fmul_rn(T.y, rb.v)), __fmul_rn(ub, rwb));
      const float ya = __fadd_rn(__fadd_rn(T.z, __fmul_rn(T.w, ra.v)), __fmul_rn(va, rwa));
      const float yb = __fadd_rn(__fadd_rn(T.z, __fmul_rn(T.w, rb.v)), __fmul_rn(vb, rwb));
      o[half][0] = lin_read_whole<Off>(px, w2, h2, src.pitch, lin_hold(xa), lin_hold(ya));
      o[half][1] = lin_read_whole<Off>(px, w2, h2, src.pitch, lin_hold(xb), lin_hold(yb));
      if (half == 0) {
#pragma unroll
        for (int s = 0; s < 8; s++) { W = addx2(W, cw); U = addx2(U, cu); V = addx2(V, cv); }
      }
    }
    out[0] = (int16_t)o[0][0]; out[to32] = (int16_t)o[1][0];
    if (two) { out[row] = (int16_t)o[0][1]; out[row + to32] = (int16_t)o[1][1]; }
    const int step = two ? 2 : 1;
    y += step; out += step * row;
  }
}
// The sampler's CTAs a frame at `rows` rows a warp.
__host__ __device__ constexpr int sample_ctas(int n, int rows) { return (n / 64) * ((n + kSampleWarps * rows - 1) / (kSampleWarps * rows)); }
// Rows a warp: 16 spread a column's set-up over 32 samples; where they would leave SMs idle (two CTAs each), 4, for a
// shorter chain of rows.
static int sample_rows(int n, int frames, int sms) { return frames * sample_ctas(n, 16) >= 2 * sms ? 16 : 4; }
__device__ __forceinline__ void sample_cta(const SrcDev &src, int16_t *g16, int rows, int f, int b) {
  const int strips = src.sd.n / 64, y0 = (b / strips * kSampleWarps + (threadIdx.x >> 5)) * rows, y1 = min(src.sd.n, y0 + rows);
  if (y0 >= y1) return;
  if ((int64_t)src.pitch * src.h <= UINT32_MAX) sample_strip<uint32_t>(src, g16, f, b % strips, y0, y1);
  else sample_strip<int64_t>(src, g16, f, b % strips, y0, y1);
}
__global__ void __launch_bounds__(kSampleThreads, 2) sample16_kernel(SrcDev src, int16_t *g16, int rows) {
  const int per = sample_ctas(src.sd.n, rows);
  sample_cta(src, g16, rows, blockIdx.x / per, blockIdx.x % per);
}
__global__ void __launch_bounds__(256) cell_table_kernel(SrcDev src, int per_frame, float4 *ctab) {
  cell_table_entry(src, per_frame, ctab, blockIdx.y, blockIdx.x * blockDim.x + threadIdx.x);
}

// A column tile's samples. Line l holds column xa = x0 + l as its real part and xb = x0 + L + l as its imaginary part; inside
// the anchors' squares the value is the one erase_tile laid into the line. The five detrend projections' raw sums, z c(x),
// z c(y), z c(x) c(y), z q(x), z q(y) (liblizard/src/lizard_phy.c:1584-1591, 1657-1667), run over a thread's rows t / L,
// + kThreads / L, ... of line t mod L in order, whatever the samples come from.
struct TileSums {
  float cxa, qxa, cxb, qxb;
  float p[5] = {0, 0, 0, 0, 0};
  __device__ __forceinline__ TileSums(const FftDev &xd, int xa, int xb)
      : cxa(__ldg(xd.cx + xa)), qxa(__ldg(xd.qx + xa)), cxb(__ldg(xd.cx + xb)), qxb(__ldg(xd.qx + xb)) {}
  __device__ __forceinline__ void add(float cy, float qy, float va, float vb) {
    const float t0 = va + vb, t1 = cxa * va + cxb * vb, t2 = qxa * va + qxb * vb;
    p[0] += t1; p[1] += cy * t0; p[2] += cy * t1; p[3] += t2; p[4] += qy * t0;
  }
};

// By the exact walk of the captured frame, into the lines: thread t takes column x0 + t mod 2L at rows t / 2L, +
// kThreads / 2L, ... (a warp's 8 columns by 4 rows of the largest sizes touch half the cache lines of 4 by 8).
template <int N>
__device__ __forceinline__ void load_exact(const FftDev &xd, const SrcDev &src, const float4 *ctab, int f, int x0, float2 *buf) {
  constexpr int L = plan_of(N).lines, C = 2 * L, G = kThreads / C;
  const int q = threadIdx.x % C, x = x0 + q;
  const bool in = in_square(xd, x);
  float *col = reinterpret_cast<float *>(buf + (q % L) * lstride_of(N)) + q / L;   // the column's row y at col[2 pad(y)]
  const float *H = src.reg + (int64_t)f * src.regstride;
  const int nn = src.sd.nx;
  const float4 *T = ctab + (int64_t)f * N * nn;   // the frame's row and cell table
  const uint8_t *px = src.luma + f * src.fstride;
  const float4 cx = src.sd.colt[x];
  const float mx = cx.x, h6 = __fmul_rn(H[6], mx), h0 = __fmul_rn(H[0], mx), h3 = __fmul_rn(H[3], mx);
  const int i = __float_as_int(cx.y);
#pragma unroll 4
  for (int y = threadIdx.x / C; y < N; y += G) {
    if (in && __float_as_int(__ldg(xd.rowc + y).x)) continue;   // erased
    const float4 *Ty = T + y * nn;
    const float4 rt = Ty[nn - 1], tc = Ty[i];
    RowTerms rr;
    rr.kw = rt.x; rr.ku = rt.y; rr.kv = rt.z;
    col[2 * pad(y)] = sample_at(px, src.w, src.h, src.pitch, mx, h6, h0, h3, rr, CellTerms{tc.x, tc.y, tc.z, tc.w});
  }
  __syncthreads();
}

// The samples with the transform's first pass: from a supplied grid of floats (kSrcGrid), from the decode's read as the
// sampler left it (kSrcSampled), or from the lines (kSrcExact: load_exact before). Where a first-pass butterfly reads the
// rows a thread sums over (N / r0 = kThreads / L: n = 384, 768, 1536) the thread transforms what it loads, all of its
// loads in flight together and nothing passing through shared memory on the way; at the other sizes the rows go to the
// lines first. Called by every thread; ends with the first pass's outputs in the lines, the CTA synchronised.
constexpr int kSrcGrid = 0, kSrcExact = 1, kSrcSampled = 2;
template <int N, int SRC>
__device__ __forceinline__ void load_first_pass(const FftDev &xd, const SrcDev &src, const int16_t *g16, int f, int x0, float2 *buf,
                                                const float2 *tw, float p[5]) {
  constexpr int L = plan_of(N).lines, R = plan_of(N).r0, G = kThreads / L;
  constexpr bool kFused = N / R == G;
  const int l = threadIdx.x % L, j = threadIdx.x / L, xa = x0 + l, xb = x0 + L + l;
  const bool ina = in_square(xd, xa), inb = in_square(xd, xb);
  float2 *line = buf + l * lstride_of(N);
  const short2 *gs = reinterpret_cast<const short2 *>(g16 + (int64_t)f * N * N + (int64_t)x0 * N) + l;
  const float *gf = src.grid + f * src.gstride;
  TileSums sum(xd, xa, xb);
  // row y's samples, erased where a square holds them, into the sums
  auto take = [&](int y, float2 v) {
    const float4 rc = __ldg(xd.rowc + y);
    if (SRC != kSrcExact && (ina || inb) && __float_as_int(rc.x)) {
      const float2 e = line[pad(y)];
      if (ina) v.x = e.x;
      if (inb) v.y = e.y;
    }
    sum.add(rc.z, rc.w, v.x, v.y);
    return v;
  };
  // B rows y0, y0 + G, ... loaded together (past the last row, the last again)
  auto load = [&](int y0, float2 *v, auto count) {
    constexpr int B = decltype(count)::value;
    if (SRC == kSrcSampled) {
      short2 w[B];
#pragma unroll
      for (int k = 0; k < B; k++) w[k] = __ldg(gs + (kFused ? y0 + k * G : min(y0 + k * G, N - 1)) * L);
#pragma unroll
      for (int k = 0; k < B; k++) v[k] = make_float2(lin_sample(w[k].x), lin_sample(w[k].y));
    } else {
#pragma unroll
      for (int k = 0; k < B; k++) {
        const int y = kFused ? y0 + k * G : min(y0 + k * G, N - 1);
        if (SRC == kSrcExact) v[k] = line[pad(y)];
        else v[k] = make_float2(__ldg(gf + (int64_t)y * N + xa), __ldg(gf + (int64_t)y * N + xb));
      }
    }
  };
  if constexpr (kFused) {
    float2 v[R];
    load(j, v, std::integral_constant<int, R>{});
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = take(j + r * G, v[r]);
    dft<R>(v);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; r++) line[pad(j * R) + r] = v[r];   // R = 16
    __syncthreads();
  } else {
    constexpr int B = 8;
    for (int y0 = j; y0 < N; y0 += B * G) {
      float2 v[B];
      load(y0, v, std::integral_constant<int, B>{});
#pragma unroll
      for (int k = 0; k < B; k++)
        if (y0 + k * G < N) line[pad(y0 + k * G)] = take(y0 + k * G, v[k]);
    }
    __syncthreads();
    pass<N, R, 1, L>(buf, tw, L);
  }
#pragma unroll
  for (int q = 0; q < 5; q++) p[q] = sum.p[q];
}

// The column pass's per-CTA scalars in shared memory.
struct ColsShared {
  double beta[6];
  double h2[32], cx[32];   // a column's part of the surface and its c(x), the tile's columns inside a square
  float part[kThreads / 32][5];
};

// The anchors' squares of one tile laid into its lines before the samples are read: at (x, y) the shading surface
// beta . (1, c(x), q(x), c(y), q(y), c(x) c(y)) in double, rounded to float (liblizard/src/lizard_phy.c:336-346). A tile
// meets at most one square's columns (a tile is at most 32 wide, the squares' gaps are wider); a thread takes a row
// inside a square over those columns, the columns' terms (the first three, the same for every row) worked out once.
// The double pipe is the reason: worked out where each sample is read, in warps with a few lanes inside a square, it was
// 86% busy and most of the pass on grids (the transform of 64 grids of n = 768: 572 us, 253 with the values laid in
// first; 32 captured frames of n = 1536 decoded: 1093 us, 1071).
template <int N>
__device__ __forceinline__ void erase_tile(const FftDev &xd, int x0, float2 *buf, ColsShared &s) {
  constexpr int L = plan_of(N).lines, LSTR = lstride_of(N);
  static_assert(2 * L <= 32, "a tile's columns");
  int lo = 0, cols = 0, rows = 0;
#pragma unroll
  for (int i = 0; i < 7; i++) {
    const int a = max(xd.elo[i], x0), b = min(xd.ehi[i], x0 + 2 * L - 1);
    if (a <= b) { lo = a; cols = b - a + 1; }
    rows += xd.ehi[i] - xd.elo[i] + 1;
  }
  if (cols == 0) return;
  const int tid = threadIdx.x;
  if (tid < cols) {
    const double cx = xd.cx[lo + tid], qx = xd.qx[lo + tid];
    s.h2[tid] = fma(s.beta[2], qx, fma(s.beta[1], cx, s.beta[0]));
    s.cx[tid] = cx;
  }
  __syncthreads();
  for (int k = tid; k < rows; k += kThreads) {
    int y = k;   // the k-th row inside a square
#pragma unroll
    for (int i = 0; i < 7; i++) {
      const int w = xd.ehi[i] - xd.elo[i] + 1;
      if (y < w) { y += xd.elo[i]; break; }
      y -= w;
    }
    const double cy = xd.cx[y], qy = xd.qx[y];
    for (int c = 0; c < cols; c++) {
      const double h = fma(s.beta[5], s.cx[c] * cy, fma(s.beta[4], qy, fma(s.beta[3], cy, s.h2[c])));
      const int q = lo - x0 + c;
      reinterpret_cast<float *>(buf + (q % L) * LSTR + pad(y))[q / L] = (float)h;
    }
  }
  __syncthreads();
}

// The column pass on one tile (frame f, columns x0 = 2 L tile .. x0 + 2L - 1): the tile's samples (erased, projections
// summed: part[f][tile][0..4]), the L lines' transforms along y, and the two real columns of each line separated: A(v) =
// (Z(v) + conj Z(n - v)) / 2, B(v) = -i (Z(v) - conj Z(n - v)) / 2, written to Y[f][v][x] for the kept rows v. Every
// thread of the CTA takes part.
template <int N>
__device__ __forceinline__ void cols_tile(const FftDev &xd, const SrcDev &src, const float4 *ctab, const int16_t *g16, const double *beta,
                                          double *part, float2 *Y, int f, int tile, unsigned char *smraw, ColsShared &s) {
  constexpr int n = N, L = plan_of(N).lines, LSTR = lstride_of(N), tiles = n / (2 * L), ystep = kThreads / L;
  const SmemMap sm = smem_map<N>(smraw);
  const int tid = threadIdx.x, l = tid % L, warp = tid >> 5, lane = tid & 31, x0 = tile * 2 * L;
  for (int i = tid; i < n; i += kThreads) sm.tw[i] = xd.tws[i];
  float2 *line = sm.buf + l * LSTR;
  if (tid < 6) s.beta[tid] = beta[6 * f + tid];
  __syncthreads();
  erase_tile<N>(xd, x0, sm.buf, s);
  float p[5];
  if (src.grid) {
    load_first_pass<N, kSrcGrid>(xd, src, g16, f, x0, sm.buf, sm.tw, p);
  } else if (src.sd.read == LIZG_READ_DECODE) {
    load_first_pass<N, kSrcSampled>(xd, src, g16, f, x0, sm.buf, sm.tw, p);
  } else {
    load_exact<N>(xd, src, ctab, f, x0, sm.buf);
    load_first_pass<N, kSrcExact>(xd, src, g16, f, x0, sm.buf, sm.tw, p);
  }
#pragma unroll
  for (int q = 0; q < 5; q++)
    for (int o = 16; o > 0; o >>= 1) p[q] += __shfl_xor_sync(0xffffffffu, p[q], o);
  if (lane == 0)
    for (int q = 0; q < 5; q++) s.part[warp][q] = p[q];
  __syncthreads();
  if (tid < 5) {
    double acc = 0;
    for (int w = 0; w < kThreads / 32; w++) acc += s.part[w][tid];
    part[((int64_t)f * tiles + tile) * 5 + tid] = acc;
  }
  later_passes<N>(sm.buf, sm.tw, L);
  float2 *Yf = Y + (int64_t)f * xd.vrows * n;
  const int xa = x0 + l, xb = x0 + L + l;
  for (int v = tid / L; v < xd.vrows; v += ystep) {
    const float2 zv = line[pad(v)], zm = line[pad(v ? n - v : 0)];
    Yf[(int64_t)v * n + xa] = make_float2(0.5f * (zv.x + zm.x), 0.5f * (zv.y - zm.y));
    Yf[(int64_t)v * n + xb] = make_float2(0.5f * (zv.y + zm.y), -0.5f * (zv.x - zm.x));
  }
}

// The column pass of one picture size: CTA b takes tile b mod tiles of frame b / tiles.
template <int N>
__global__ void __launch_bounds__(kThreads, 3) fft_cols_kernel(FftDev xd, SrcDev src, const float4 *ctab, const int16_t *g16, const double *beta, double *part,
                                                                float2 *Y) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ ColsShared s;
  constexpr int tiles = N / (2 * plan_of(N).lines);
  cols_tile<N>(xd, src, ctab, g16, beta, part, Y, blockIdx.x / tiles, blockIdx.x % tiles, smraw, s);
}

// The column pass over several picture sizes in one grid: a queue of (format, frame, tile) items, format k's at CTAs
// [first[k], first[k + 1]), each taken by its size's body (every size's tile holds about the same 48 KB of samples,
// so one CTA shape serves them all; the dynamic shared memory is the largest size's).
__global__ void __launch_bounds__(kThreads, 3) fft_cols_mixed_kernel(const __grid_constant__ FftColsMix m) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ ColsShared s;
  int k = 0;
  while (k < m.nseg - 1 && (int)blockIdx.x >= m.first[k + 1]) k++;
  const FftColsSeg &g = m.seg[k];
  const int b = (int)blockIdx.x - m.first[k], tiles = g.xd.n / (2 * plan_of(g.xd.n).lines), f = b / tiles, tile = b - f * tiles;
  switch (g.xd.n) {
    case 384: cols_tile<384>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
    case 512: cols_tile<512>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
    case 768: cols_tile<768>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
    case 1024: cols_tile<1024>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
    case 1152: cols_tile<1152>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
    case 1280: cols_tile<1280>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
    default: cols_tile<1536>(g.xd, g.src, g.ctab, g.g16, g.beta, g.part, g.Y, f, tile, smraw, s); break;
  }
}

// The five projections of each frame from its column tiles' sums, normalised (liblizard/src/lizard_phy.c:1697), then the
// surface spectrum's factors (liblizard/src/lizard_phy.c:1702-1716), rounded to float as there: fac[f] = xy[u] (pxy
// X1[u]) for u < n, x0[u] (n (px X1[u] + pxx X2[u])) for u < n, y0[v] (n (py X1[v] + pyy X2[v])) for v < vrows. Each of
// a frame's kFacCtas CTAs adds the tiles itself (a warp a projection, as a tree) and takes its share of the factors: one
// CTA a frame adding the tiles in a chain held one SM's double pipe 27 us at n = 1536; 6 so (9 for 32 frames). The tiles
// are this pass's own, so no order of the reference's is at stake; the tree's sums (at most 6 in a lane, then 5 steps)
// are nearer the exact ones than the chain's of up to 192, and both have rounded to the same factors wherever compared.
constexpr int kFacCtas = 8;
__device__ __forceinline__ void fac_frame(const FftDev &xd, int tiles, const double *part, float2 *fac, int f, int piece) {
  const int n = xd.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ double s_p[5];
  if (warp < 5) {
    double acc = 0;
#pragma unroll 6
    for (int t = lane; t < tiles; t += 32) acc += part[((int64_t)f * tiles + t) * 5 + warp];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    // z c(x), z c(y): n sx2; z c(x) c(y): sx2 sx2; z q(x), z q(y): n sq2
    if (lane == 0) s_p[warp] = acc / (warp < 2 ? n * xd.sx2 : warp == 2 ? xd.sx2 * xd.sx2 : n * xd.sq2);
  }
  __syncthreads();
  const double px = s_p[0], py = s_p[1], pxy = s_p[2], pxx = s_p[3], pyy = s_p[4];
  float2 *o = fac + (int64_t)f * (2 * n + xd.vrows);
  for (int i = piece * blockDim.x + threadIdx.x; i < 2 * n + xd.vrows; i += kFacCtas * blockDim.x) {
    const int k = i < n ? i : i < 2 * n ? i - n : i - 2 * n;
    const float2 x1 = xd.x1[k];
    if (i < n) {
      o[i] = make_float2((float)(pxy * x1.x), (float)(pxy * x1.y));
    } else {
      const float2 x2 = xd.x2[k];
      const double a = i < 2 * n ? px : py, b = i < 2 * n ? pxx : pyy;
      o[i] = make_float2((float)(n * (a * x1.x + b * x2.x)), (float)(n * (a * x1.y + b * x2.y)));
    }
  }
}
__global__ void __launch_bounds__(256) fac_kernel(FftDev xd, int tiles, const double *part, float2 *fac) {
  fac_frame(xd, tiles, part, fac, blockIdx.x / kFacCtas, blockIdx.x % kFacCtas);
}

// The shading sums, the sampler or the exact walk's tables and the surface factors over several formats' batches, one
// launch a stage:
// format k's shading-band CTAs at [hf[k], hf[k + 1]), then its table CTAs at [tf[k], tf[k + 1]) (one launch takes
// both), its frames' factor CTAs at [ff[k], ff[k + 1]).
struct FftLightSeg {
  FftDev xd;
  SrcDev src;
  double *hole, *beta, *part;
  int *ticket;
  float4 *ctab;
  int16_t *g16;
  float2 *fac;
  int bands, per_frame, tblocks, tiles;
};
struct FftLightMix {
  FftLightSeg seg[kFftMixSegs];
  int hf[kFftMixSegs + 1], tf[kFftMixSegs + 1], ff[kFftMixSegs + 1];
  int nseg;
};
static_assert(sizeof(FftLightMix) <= 32000, "the light stages' arguments fit a launch");
__device__ __forceinline__ int seg_at(const int *first, int nseg, int b) {
  int k = 0;
  while (k < nseg - 1 && b >= first[k + 1]) k++;
  return k;
}
__global__ void __launch_bounds__(kHoleThreads, 2) fft_pre_mixed_kernel(const __grid_constant__ FftLightMix m) {
  __shared__ HoleShared sh;
  const int b = blockIdx.x;
  if (b < m.hf[m.nseg]) {
    const int k = seg_at(m.hf, m.nseg, b);
    const FftLightSeg &g = m.seg[k];
    const int lb = b - m.hf[k];
    switch (hole_cols(g.xd.n)) {
      case 2: hole_rhs_band<2>(g.xd, g.src, g.bands, g.hole, g.beta, g.ticket, lb / g.bands, lb % g.bands, sh); break;
      case 3: hole_rhs_band<3>(g.xd, g.src, g.bands, g.hole, g.beta, g.ticket, lb / g.bands, lb % g.bands, sh); break;
      case 4: hole_rhs_band<4>(g.xd, g.src, g.bands, g.hole, g.beta, g.ticket, lb / g.bands, lb % g.bands, sh); break;
      case 5: hole_rhs_band<5>(g.xd, g.src, g.bands, g.hole, g.beta, g.ticket, lb / g.bands, lb % g.bands, sh); break;
      default: hole_rhs_band<6>(g.xd, g.src, g.bands, g.hole, g.beta, g.ticket, lb / g.bands, lb % g.bands, sh); break;
    }
  } else {
    const int k = seg_at(m.tf, m.nseg, b);
    const FftLightSeg &g = m.seg[k];
    const int lb = b - m.tf[k], f = lb / g.tblocks;
    if (g.src.sd.read == LIZG_READ_DECODE) sample_cta(g.src, g.g16, 16, f, lb - f * g.tblocks);
    else cell_table_entry(g.src, g.per_frame, g.ctab, f, (lb - f * g.tblocks) * kHoleThreads + threadIdx.x);
  }
}
__global__ void __launch_bounds__(256) fac_mixed_kernel(const __grid_constant__ FftLightMix m) {
  const int k = seg_at(m.ff, m.nseg, blockIdx.x);
  const FftLightSeg &g = m.seg[k];
  const int b = blockIdx.x - m.ff[k];
  fac_frame(g.xd, g.tiles, g.part, g.fac, b / kFacCtas, b % kFacCtas);
}

// A bounded wait on an mbarrier's phase (try_wait blocks a while in hardware before it answers): false when the
// limit ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit) {
  for (int i = 0; i < limit; i++) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}

// The row pass on one tile (frame f, rows v0 = L rtile .. v0 + L - 1): transforms them along x and takes the surface's
// spectrum off: the xy term pxy X1[u] X1[v] everywhere, the x terms on v = 0, the y terms on u = 0. The used
// coefficients go straight to their place in pos order: C[f][tpos[v][u]] (tpos -1 where (u, v) is not used).
// The tile's rows come in by the tensor memory accelerator: bulk tensor copies of 128 complex points of a row each,
// issued by one thread, landing densely at the start of each line's slots (at a 128-byte boundary) and counted on an
// mbarrier; the first transform pass reads its points from the dense rows and writes the padded lines (all read, then all
// written), and the last one's outputs go to their coefficients from registers. 32 frames of n = 1536: 120 us with a copy
// from dense to padded before the passes and the lines read again after them, 97 so.
template <int N>
__device__ __forceinline__ void rows_tile(const FftDev &xd, const float2 *fac, const CUtensorMap *ymap, const int32_t *tpos, int need, float2 *C,
                                          int *err, int f, int rtile, unsigned char *smraw, uint64_t *s_bar) {
  constexpr int n = N, L = plan_of(N).lines, LSTR = lstride_of(N), SEGS = N / 128;
  static_assert(LSTR >= N + 16, "a line's slots hold its dense row at a 128-byte boundary");
  const SmemMap sm = smem_map<N>(smraw);
  const int tid = threadIdx.x;
  const int v0 = rtile * L, Lr = min(L, xd.vrows - v0);
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(s_bar);
  // line l's dense row: at the first 128-byte boundary of its slots (room: a line's slots exceed n by 16 or more)
  auto dense = [&](int l) { return (uint32_t)(((uint32_t)__cvta_generic_to_shared(sm.buf + l * LSTR) + 127u) & ~127u); };
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (tid == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((uint32_t)(Lr * N * 8)) : "memory");
    const int y0 = f * xd.vrows + v0;
    for (int l = 0; l < Lr; l++)
      for (int s = 0; s < SEGS; s++)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                     ::"r"(dense(l) + 1024u * s), "l"(ymap), "r"(256 * s), "r"(y0 + l), "r"(bar) : "memory");
  }
  for (int i = tid; i < n; i += kThreads) sm.tw[i] = xd.tws[i];
  if (!mbar_wait(bar, 0, 1 << 22)) {   // never expected: record it, wait for the copies once more, leave the tile
    atomicOr(err, 1);
    mbar_wait(bar, 0, 1 << 22);
    return;
  }
  __syncthreads();   // the twiddles
  first_pass_from<N>(sm.buf, sm.tw, Lr, [&](int l, int j) {
    const uint32_t row = dense(l) + 8u * j;
    return [=](int r) {
      float2 p;
      asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(p.x), "=f"(p.y) : "r"(row + 8u * (N / plan_of(N).r0) * r));
      return p;
    };
  });
  middle_pass<N>(sm.buf, sm.tw, Lr);
  float2 *Cf = C + (int64_t)f * need;
  const int32_t *tp = tpos + (int64_t)v0 * n;
  const float2 *fx = fac + (int64_t)f * (2 * n + xd.vrows), *fx0 = fx + n, *fy0 = fx + 2 * n;
  last_pass_to<N>(sm.buf, sm.tw, Lr, [&](int l, int p) {
    const int v = v0 + l;
    const float2 x1v = xd.x1[v];
    const int32_t *at = tp + l * n + p;
    const float2 *a0 = fx + p;
    return [=](int r, float2 o) {
      const int u = p + r * (N / plan_of(N).r2), i = __ldg(at + r * (N / plan_of(N).r2));
      if (i < 0) return;
      const float2 a = a0[r * (N / plan_of(N).r2)];
      o.x -= __fmaf_rn(a.x, x1v.x, -__fmul_rn(a.y, x1v.y));   // the contraction named: the compiler's hangs on the code round it
      o.y -= __fmaf_rn(a.y, x1v.x, __fmul_rn(a.x, x1v.y));
      if (v == 0) { const float2 c = fx0[u]; o.x -= c.x; o.y -= c.y; }
      if (u == 0) { const float2 c = fy0[v]; o.x -= c.x; o.y -= c.y; }
      Cf[i] = o;
    };
  });
}

// The row pass of one picture size: CTA b takes row tile b mod tiles of frame b / tiles.
template <int N>
__global__ void __launch_bounds__(kThreads, 3) fft_rows_kernel(FftDev xd, const float2 *fac, const __grid_constant__ CUtensorMap ymap,
                                                               const int32_t *tpos, int need, float2 *C, int *err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(8) uint64_t s_bar;
  const int tiles = (xd.vrows + plan_of(N).lines - 1) / plan_of(N).lines;
  rows_tile<N>(xd, fac, &ymap, tpos, need, C, err, blockIdx.x / tiles, blockIdx.x % tiles, smraw, &s_bar);
}

// The row pass over several picture sizes in one grid: format k's (frame, row tile) items at CTAs
// [first[k], first[k + 1]), each with its own tensor map over its Y.
__global__ void __launch_bounds__(kThreads, 3) fft_rows_mixed_kernel(const __grid_constant__ FftRowsMix m) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(8) uint64_t s_bar;
  int k = 0;
  while (k < m.nseg - 1 && (int)blockIdx.x >= m.first[k + 1]) k++;
  const FftRowsSeg &g = m.seg[k];
  const int L = plan_of(g.xd.n).lines, tiles = (g.xd.vrows + L - 1) / L, b = (int)blockIdx.x - m.first[k], f = b / tiles, rt = b - f * tiles;
  switch (g.xd.n) {
    case 384: rows_tile<384>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
    case 512: rows_tile<512>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
    case 768: rows_tile<768>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
    case 1024: rows_tile<1024>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
    case 1152: rows_tile<1152>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
    case 1280: rows_tile<1280>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
    default: rows_tile<1536>(g.xd, g.fac, &g.ymap, g.tpos, g.need, g.C, g.err, f, rt, smraw, &s_bar); break;
  }
}

// The column pass's row entries: 256 where row y is inside an anchor's square, c(y), q(y).
__global__ void row_table_kernel(FftDev xd, float4 *rowc) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  if (y < xd.n) rowc[y] = make_float4(__int_as_float(in_square(xd, y) ? 256 : 0), 0.0f, xd.cx[y], xd.qx[y]);
}
cudaError_t fft_row_table_launch(const FftDev &xd, float4 *rowc, cudaStream_t st) {
  row_table_kernel<<<(xd.n + 255) / 256, 256, 0, st>>>(xd, rowc);
  return cudaGetLastError();
}

int fft_plan(int n, int radix[3], int *lines) {
  const Plan p = plan_of(n);
  if (!p.lines) return -1;
  radix[0] = p.r0; radix[1] = p.r1; radix[2] = p.r2;
  *lines = p.lines;
  return 0;
}

int fft_hole_bands(int n) { return (n / 8 + kHoleBand - 1) / kHoleBand; }

int fft_y_map(CUtensorMap *map, float2 *Y, int n, int64_t rows) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess || !fn) return -1;
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  const cuuint64_t dims[2] = {(cuuint64_t)2 * n, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)2 * n * sizeof(float)};
  const cuuint32_t box[2] = {256, 1}, estr[2] = {1, 1};
  return (int)encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, Y, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

int fft_turn(const FftSegArgs &a) {
  if (a.src.grid || a.src.sd.read != LIZG_READ_DECODE) return a.frames;
  if (a.b.g16_frames < 1) return 0;
  const int turns = (a.frames + a.b.g16_frames - 1) / a.b.g16_frames;
  return (a.frames + turns - 1) / turns;   // alike: 128 frames of n = 1536 as 56, 56 and 16 had a short last grid
}

FftSegArgs fft_frames_of(const FftSegArgs &a, int f0, int count) {
  FftSegArgs s = a;
  s.frames = count;
  if (f0 == 0) return s;
  const int n = a.xd.n;
  if (s.src.grid) s.src.grid += f0 * s.src.gstride;
  if (s.src.luma) { s.src.luma += f0 * s.src.fstride; s.src.reg += (int64_t)f0 * s.src.regstride; }
  s.b.hole += (int64_t)f0 * fft_hole_bands(n) * 6; s.b.beta += 6 * (int64_t)f0; s.b.ticket += f0;
  s.b.part += (int64_t)f0 * (n / (2 * plan_of(n).lines)) * 5;
  s.b.Y += (int64_t)f0 * a.xd.vrows * n;
  return s;
}

// What the column pass reads of captured frames: the decode's samples or the exact walk's table.
static cudaError_t fft_read_launch(const FftSegArgs &a, int sms, cudaStream_t st) {
  if (a.src.grid) return cudaSuccess;
  if (a.src.sd.read == LIZG_READ_DECODE) {
    if (!a.b.g16 || a.frames > a.b.g16_frames) return cudaErrorInvalidValue;
    const int rows = sample_rows(a.xd.n, a.frames, sms);
    sample16_kernel<<<a.frames * sample_ctas(a.xd.n, rows), kSampleThreads, 0, st>>>(a.src, a.b.g16, rows);
  } else {
    if (!a.b.ctab || a.src.sd.nx != a.src.sd.ny) return cudaErrorInvalidValue;
    const int per_frame = a.xd.n * a.src.sd.nx;
    cell_table_kernel<<<dim3((per_frame + 255) / 256, a.frames), 256, 0, st>>>(a.src, per_frame, a.b.ctab);
  }
  return cudaGetLastError();
}

static cudaError_t fft_fac_launch(const FftSegArgs &a, cudaStream_t st) {
  fac_kernel<<<a.frames * kFacCtas, 256, 0, st>>>(a.xd, a.xd.n / (2 * plan_of(a.xd.n).lines), a.b.part, a.b.fac);
  return cudaGetLastError();
}

template <int N>
static cudaError_t fft_launch_n(const FftDev &xd, int frames, const SrcDev &src, const FftBufs &b, int sms, cudaStream_t st) {
  constexpr int L = plan_of(N).lines, smem = smem_bytes_of(N), tiles = N / (2 * L);
  static_assert(smem <= kFftSmemMax, "transform CTA's shared memory");
  static_assert(hole_cols(N) >= 2 && hole_cols(N) <= 6, "the shading fit's columns a lane");
  static_assert(N % (2 * L) == 0 && L * N <= kFftPoints && kThreads % L == 0 && L <= 32, "transform plan");
  static SmemOptIn opt_cols, opt_rows;
  cudaError_t e;
  if ((e = opt_cols.set(reinterpret_cast<const void *>(fft_cols_kernel<N>), smem)) != cudaSuccess ||
      (e = opt_rows.set(reinterpret_cast<const void *>(fft_rows_kernel<N>), smem)) != cudaSuccess)
    return e;
  const FftSegArgs all{xd, src, b, frames};
  const int turn = fft_turn(all);
  if (turn < 1) return cudaErrorInvalidValue;
  const int bands = fft_hole_bands(N);
  hole_rhs_kernel<hole_cols(N)><<<frames * bands, kHoleThreads, 0, st>>>(xd, src, bands, b.hole, b.beta, b.ticket);
  for (int f0 = 0; f0 < frames; f0 += turn) {
    const FftSegArgs a = fft_frames_of(all, f0, frames - f0 < turn ? frames - f0 : turn);
    if ((e = fft_read_launch(a, sms, st)) != cudaSuccess) return e;
    fft_cols_kernel<N><<<a.frames * tiles, kThreads, smem, st>>>(xd, a.src, a.b.ctab, a.b.g16, a.b.beta, a.b.part, a.b.Y);
  }
  if ((e = fft_fac_launch(all, st)) != cudaSuccess) return e;
  if (!b.ymap || !b.err) return cudaErrorInvalidValue;
  fft_rows_kernel<N><<<frames * ((xd.vrows + L - 1) / L), kThreads, smem, st>>>(xd, b.fac, *b.ymap, b.tpos, b.need, b.C, b.err);
  return cudaGetLastError();
}

// The largest transform CTA's shared memory over the ladder: the mixed grids' dynamic size.
constexpr int kFftSmemLadder = cmax_i(cmax_i(cmax_i(smem_bytes_of(384), smem_bytes_of(512)), cmax_i(smem_bytes_of(768), smem_bytes_of(1024))),
                                      cmax_i(cmax_i(smem_bytes_of(1152), smem_bytes_of(1280)), smem_bytes_of(1536)));
static_assert(kFftSmemLadder <= kFftSmemMax, "transform CTA's shared memory");

static int ladder_size(int n) { return plan_of(n).lines != 0; }

static cudaError_t light_mix(const FftSegArgs *a, int count, FftLightMix &m) {
  if (count < 1 || count > kFftMixSegs) return cudaErrorInvalidValue;
  m = FftLightMix{};
  m.nseg = count;
  for (int k = 0; k < count; k++) {
    const FftSegArgs &s = a[k];
    const bool sampled = s.src.sd.read == LIZG_READ_DECODE;
    if (!ladder_size(s.xd.n) || s.frames < 1 || s.src.grid || s.src.sd.nx != s.src.sd.ny || !(sampled ? (void *)s.b.g16 : s.b.ctab))
      return cudaErrorInvalidValue;
    FftLightSeg &g = m.seg[k];
    g.xd = s.xd; g.src = s.src; g.hole = s.b.hole; g.beta = s.b.beta; g.ticket = s.b.ticket; g.g16 = s.b.g16; g.part = s.b.part; g.ctab = s.b.ctab; g.fac = s.b.fac;
    g.bands = fft_hole_bands(s.xd.n); g.per_frame = s.xd.n * s.src.sd.nx; g.tblocks = sampled ? sample_ctas(s.xd.n, 16) : (g.per_frame + kHoleThreads - 1) / kHoleThreads;
    g.tiles = s.xd.n / (2 * plan_of(s.xd.n).lines);
    m.hf[k + 1] = m.hf[k] + s.frames * g.bands;
    m.ff[k + 1] = m.ff[k] + s.frames * kFacCtas;
  }
  m.tf[0] = m.hf[count];
  for (int k = 0; k < count; k++) m.tf[k + 1] = m.tf[k] + a[k].frames * m.seg[k].tblocks;
  return cudaSuccess;
}

cudaError_t fft_pre_mixed_launch(const FftSegArgs *a, int count, cudaStream_t st) {
  FftLightMix m;
  if (cudaError_t e = light_mix(a, count, m)) return e;
  for (int k = 0; k < count; k++)
    if (a[k].frames > fft_turn(a[k])) return cudaErrorInvalidValue;
  fft_pre_mixed_kernel<<<m.tf[count], kHoleThreads, 0, st>>>(m);
  return cudaGetLastError();
}

cudaError_t fft_fac_mixed_launch(const FftSegArgs *a, int count, cudaStream_t st) {
  FftLightMix m;
  if (cudaError_t e = light_mix(a, count, m)) return e;
  fac_mixed_kernel<<<m.ff[count], 256, 0, st>>>(m);
  return cudaGetLastError();
}

cudaError_t fft_cols_mixed_launch(const FftSegArgs *a, int count, cudaStream_t st) {
  if (count < 1 || count > kFftMixSegs) return cudaErrorInvalidValue;
  static SmemOptIn opt;
  cudaError_t e;
  if ((e = opt.set(reinterpret_cast<const void *>(fft_cols_mixed_kernel), kFftSmemLadder)) != cudaSuccess) return e;
  FftColsMix m{};
  m.nseg = count;
  int smem = 0;
  for (int k = 0; k < count; k++) {
    const FftSegArgs &s = a[k];
    if (!ladder_size(s.xd.n) || s.frames < 1) return cudaErrorInvalidValue;
    FftColsSeg &g = m.seg[k];
    g.xd = s.xd; g.src = s.src; g.ctab = s.b.ctab; g.g16 = s.b.g16; g.beta = s.b.beta; g.part = s.b.part; g.Y = s.b.Y;
    m.first[k + 1] = m.first[k] + s.frames * (s.xd.n / (2 * plan_of(s.xd.n).lines));
    smem = cmax_i(smem, smem_bytes_of(s.xd.n));
  }
  fft_cols_mixed_kernel<<<m.first[count], kThreads, smem, st>>>(m);
  return cudaGetLastError();
}

cudaError_t fft_rows_mixed_launch(const FftSegArgs *a, int count, cudaStream_t st) {
  if (count < 1 || count > kFftMixSegs) return cudaErrorInvalidValue;
  static SmemOptIn opt;
  cudaError_t e;
  if ((e = opt.set(reinterpret_cast<const void *>(fft_rows_mixed_kernel), kFftSmemLadder)) != cudaSuccess) return e;
  FftRowsMix m{};
  m.nseg = count;
  int smem = 0;
  for (int k = 0; k < count; k++) {
    const FftSegArgs &s = a[k];
    if (!ladder_size(s.xd.n) || s.frames < 1 || !s.b.ymap || !s.b.err) return cudaErrorInvalidValue;
    FftRowsSeg &g = m.seg[k];
    const int L = plan_of(s.xd.n).lines;
    g.xd = s.xd; g.ymap = *s.b.ymap; g.fac = s.b.fac; g.tpos = s.b.tpos; g.C = s.b.C; g.err = s.b.err; g.need = s.b.need;
    m.first[k + 1] = m.first[k] + s.frames * ((s.xd.vrows + L - 1) / L);
    smem = cmax_i(smem, smem_bytes_of(s.xd.n));
  }
  fft_rows_mixed_kernel<<<m.first[count], kThreads, smem, st>>>(m);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- the sender's inverse (liblizard/src/lizard_phy.c:1134-1199)
//
// The half-plane spectrum's rows (v < vrows, each along u), then the picture's columns, in one of two forms. Over rows
// (the refinement's adjoint): the spectrum complex, transformed in place, the picture row-major. PAGE (the sender): the
// spectrum a byte a point and frame (its two signs), and both results by column tiles, a line's two columns side by
// side, so that the column pass reads and writes runs of bytes (row by row they are 16 to 32 bytes a cache line, and the
// pass is bound by the lines it touches: 250 us over 32 pages of n = 1536, 145 so).

// The half-plane spectrum's rows inverse-transformed: S[v][x] = sum_u S[v][u] e^{+2 pi i u x / n}, as the conjugate of the
// forward transform of the conjugate. L rows a CTA.
template <int N, bool PAGE>
__global__ void __launch_bounds__(kThreads, 3) enc_cols_kernel(EncFft e, const uint32_t *signs, float2 *S) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int L = plan_of(N).lines, LSTR = lstride_of(N), C = 2 * L;
  float2 *buf = reinterpret_cast<float2 *>(smraw), *tw = buf + L * LSTR;
  const int tiles = (e.vrows + L - 1) / L, f = blockIdx.x / tiles, v0 = (blockIdx.x % tiles) * L, Lr = min(L, e.vrows - v0);
  for (int i = threadIdx.x; i < N; i += kThreads) tw[i] = e.tws[i];
  __syncthreads();
  constexpr int from = N / plan_of(N).r0, to = N / plan_of(N).r2;   // a butterfly's points, its outputs
  if (PAGE) {
    const uint32_t *rows = signs + ((int64_t)(f / kFrameGroup) * e.vrows + v0) * N;
    const int shift = 8 * (f % kFrameGroup);
    first_pass_from<N>(buf, tw, Lr, [&](int l, int j) {
      const uint32_t *at = rows + l * N + j;
      return [=](int r) {
        const uint32_t s = __ldg(at + r * from) >> shift;
        const float a = s & 1 ? kEncQpsk : 0.0f;
        return make_float2(s & 2 ? -a : a, s & 4 ? a : -a);
      };
    });
  } else {
    const float2 *rows = S + ((int64_t)f * e.vrows + v0) * N;
    first_pass_from<N>(buf, tw, Lr, [&](int l, int j) {
      const float2 *at = rows + l * N + j;
      return [=](int r) { const float2 z = at[r * from]; return make_float2(z.x, -z.y); };
    });
  }
  middle_pass<N>(buf, tw, Lr);
  float2 *out = S + (int64_t)f * e.vrows * N;
  last_pass_to<N>(buf, tw, Lr, [&](int l, int p) {
    // by column tiles: outputs `to` columns apart are as far into their tiles where that is whole tiles
    const int c = p % C;
    float2 *at = PAGE ? out + (p - c) * e.vrows + (v0 + l) * C + (c < L ? 2 * c : 2 * (c - L) + 1) : out + (v0 + l) * N + p;
    const int step = PAGE ? to * e.vrows : to;
    return [=](int r, float2 z) { at[r * step] = make_float2(z.x, -z.y); };
  });
  static_assert(!PAGE || to % C == 0, "a butterfly's outputs in like places of their tiles");
}

// The picture's columns: 2L of them a CTA, columns xa = x0 + l and xb = x0 + L + l sharing line l as H_a + i H_b, each H
// the column's Hermitian completion over v (H(0) = 2 Re T(0), H(v) = T(v), H(n - v) = conj T(v) for 0 < v < vrows, zero
// between), inverse-transformed along v: the real part column xa, the imaginary part column xb
// (liblizard/src/lizard_phy.c:733-773 turn_pack). Then clipped at +-lim and mapped to 0.5 + v sc (clip_row, :775-782),
// into pic[y][x], or by column tiles (pic_at), as they are or (GREY) as the page's grey levels.
template <int N, bool PAGE, bool GREY>
__global__ void __launch_bounds__(kThreads, 3) enc_rows_kernel(EncFft e, const float2 *T, void *pic) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int L = plan_of(N).lines, LSTR = lstride_of(N), C = 2 * L, tiles = N / C;
  float2 *buf = reinterpret_cast<float2 *>(smraw), *tw = buf + L * LSTR;
  const int f = blockIdx.x / tiles, x0 = (blockIdx.x % tiles) * C;
  for (int i = threadIdx.x; i < N; i += kThreads) tw[i] = e.tws[i];
  const float2 *Tf = T + (int64_t)f * e.vrows * N;
  const float4 *Tt = reinterpret_cast<const float4 *>(Tf + (int64_t)x0 * e.vrows);   // the tile's (a, b) pairs, row by row
  // l fastest: a row's 2L columns read together, each row v < vrows once for the rows v and n - v that it fills
#pragma unroll 4
  for (int t = threadIdx.x; t < L * e.vrows; t += kThreads) {
    const int v = t / L, l = t - v * L;
    float2 a, b;
    if (PAGE) {
      const float4 ab = __ldg(Tt + t);
      a = make_float2(ab.x, ab.y); b = make_float2(ab.z, ab.w);
    } else {
      a = Tf[(int64_t)v * N + x0 + l]; b = Tf[(int64_t)v * N + x0 + L + l];
    }
    float2 *line = buf + l * LSTR;
    if (v == 0) {
      line[0] = make_float2(2.0f * a.x, -(2.0f * b.x));
    } else {
      line[pad(v)] = make_float2(a.x - b.y, -(a.y + b.x));
      line[pad(N - v)] = make_float2(a.x + b.y, -(b.x - a.y));
    }
  }
  for (int t = threadIdx.x; t < L * (N - 2 * e.vrows + 1); t += kThreads) {
    const int v = e.vrows + t / L, l = t % L;
    buf[l * LSTR + pad(v)] = make_float2(0.0f, -0.0f);
  }
  __syncthreads();
  pass<N, plan_of(N).r0, 1, L>(buf, tw, L);
  middle_pass<N>(buf, tw, L);
  float *pf = static_cast<float *>(pic) + (int64_t)f * N * N;
  uint8_t *gf = static_cast<uint8_t *>(pic) + (int64_t)f * N * N;
  constexpr int to = N / plan_of(N).r2;
  last_pass_to<N, true>(buf, tw, L, [&](int l, int y) {
    return [=](int r, float2 z) {
      float a = z.x, b = -z.y;
      if (PAGE) {   // finite: the signs' transform (two operations a clip for four: 117 us for 32 pages of n = 1536, 127 before)
        a = fmaxf(fminf(a, e.lim), -e.lim); b = fmaxf(fminf(b, e.lim), -e.lim);
      } else {
        a = a > e.lim ? e.lim : a;
        a = a < -e.lim ? -e.lim : a;
        b = b > e.lim ? e.lim : b;
        b = b < -e.lim ? -e.lim : b;
      }
      a = __fadd_rn(0.5f, __fmul_rn(a, e.sc)); b = __fadd_rn(0.5f, __fmul_rn(b, e.sc));   // rounded as clip_row rounds, unfused
      const int yr = y + r * to;
      if (GREY) {   // held to 0..1 and rounded as the page's paint does
        reinterpret_cast<uchar2 *>(gf + (int64_t)x0 * N)[yr * L + l] = make_uchar2(grey_level(__saturatef(a)), grey_level(__saturatef(b)));
      } else if (PAGE) {
        reinterpret_cast<float2 *>(pf + (int64_t)x0 * N)[yr * L + l] = make_float2(a, b);
      } else {
        pf[(int64_t)yr * N + x0 + l] = a;
        pf[(int64_t)yr * N + x0 + L + l] = b;
      }
    };
  });
}

template <int N, bool PAGE, bool GREY>
static cudaError_t enc_fft_launch_n(const EncFft &e, int frames, const uint32_t *signs, float2 *S, void *pic, cudaStream_t st) {
  constexpr int L = plan_of(N).lines, smem = smem_bytes_of(N);
  static SmemOptIn opt_cols, opt_rows;
  cudaError_t err;
  if ((err = opt_cols.set(reinterpret_cast<const void *>(enc_cols_kernel<N, PAGE>), smem)) != cudaSuccess ||
      (err = opt_rows.set(reinterpret_cast<const void *>(enc_rows_kernel<N, PAGE, GREY>), smem)) != cudaSuccess)
    return err;
  enc_cols_kernel<N, PAGE><<<frames * ((e.vrows + L - 1) / L), kThreads, smem, st>>>(e, signs, S);
  enc_rows_kernel<N, PAGE, GREY><<<frames * (N / (2 * L)), kThreads, smem, st>>>(e, S, pic);
  return cudaGetLastError();
}
template <bool PAGE, bool GREY>
static cudaError_t enc_fft_launch_of(const EncFft &e, int frames, const uint32_t *signs, float2 *S, void *pic, cudaStream_t st) {
  if (e.vrows < 1 || 2 * e.vrows > e.n + 1) return cudaErrorInvalidValue;
  switch (e.n) {
    case 384: return enc_fft_launch_n<384, PAGE, GREY>(e, frames, signs, S, pic, st);
    case 512: return enc_fft_launch_n<512, PAGE, GREY>(e, frames, signs, S, pic, st);
    case 768: return enc_fft_launch_n<768, PAGE, GREY>(e, frames, signs, S, pic, st);
    case 1024: return enc_fft_launch_n<1024, PAGE, GREY>(e, frames, signs, S, pic, st);
    case 1152: return enc_fft_launch_n<1152, PAGE, GREY>(e, frames, signs, S, pic, st);
    case 1280: return enc_fft_launch_n<1280, PAGE, GREY>(e, frames, signs, S, pic, st);
    case 1536: return enc_fft_launch_n<1536, PAGE, GREY>(e, frames, signs, S, pic, st);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t enc_fft_launch(const EncFft &e, int frames, float2 *S, float *pic, cudaStream_t st) {
  return enc_fft_launch_of<false, false>(e, frames, nullptr, S, pic, st);
}
cudaError_t enc_page_launch(const EncFft &e, int frames, const uint32_t *signs, float2 *T, void *pic, bool grey, cudaStream_t st) {
  return grey ? enc_fft_launch_of<true, true>(e, frames, signs, T, pic, st) : enc_fft_launch_of<true, false>(e, frames, signs, T, pic, st);
}

cudaError_t fft_launch(const FftDev &xd, int frames, const SrcDev &src, const FftBufs &b, int sms, cudaStream_t st) {
  switch (xd.n) {
    case 384: return fft_launch_n<384>(xd, frames, src, b, sms, st);
    case 512: return fft_launch_n<512>(xd, frames, src, b, sms, st);
    case 768: return fft_launch_n<768>(xd, frames, src, b, sms, st);
    case 1024: return fft_launch_n<1024>(xd, frames, src, b, sms, st);
    case 1152: return fft_launch_n<1152>(xd, frames, src, b, sms, st);
    case 1280: return fft_launch_n<1280>(xd, frames, src, b, sms, st);
    case 1536: return fft_launch_n<1536>(xd, frames, src, b, sms, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace lizg
