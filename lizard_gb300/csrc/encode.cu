// The sender on sm_103a (the GPU encoder): a batch of frames' blocks to the ring's drive and its grey page, as the
// reference's lizard_encode and lizard_paint_grey make them (liblizard/src/lizard_phy.c:1087-1236, 700-716):
//   - each block's data bits and CRC-32C, the LDPC code's parity as the running XOR of the checks' data bits
//     (liblizard/src/ldpc.c:117-126), its slots through the tier's bit map and the whitening, the pilots' count bit
//     past the codeword (map_out, :121-159), Gray QPSK of unit magnitude at each coefficient (:1134-1141); the
//     padding past the last block the whitening alone (:1146-1152);
//   - the half-plane's Hermitian inverse, clipped at 2 sqrt(640 subch) and mapped to 0..1 (fft.cu enc_*);
//   - the picture onto the ring's pixels by the Lanczos-3 resampler over the picture and its guard interval, the
//     picture periodic (:962-1075), six weights a pass in order; the border's cells 0 or 1 at pxm pixels a module
//     (:1153-1165), the format word among them; the anchors' squares over the picture (:1218-1234);
//   - the page: round(drive 255) inside a white margin of 2 modules (lizard_paint_grey).
// The transform's floats are this library's (a different order from the reference's), so a drive pixel may differ in
// its last bits and a grey level by one at a rounding tie; every other step is the reference's float order
// (-fmad=false). A receiver reads the same blocks.
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>
#include "format.h"
#include "lizard_codes.h"
#include "lizard_gb300.h"
#include "lizg_internal.h"

namespace lizg {

constexpr int kEncThreads = 256, kCp = 3, kQuiet = 2, kMaxCheckRows = 30;

struct EncTier {
  // per coefficient that carries codeword bits: its two bits' places, 16 bits each (data bits in order, parity bit
  // k + i mb + r at k + 128 r + i)
  const uint32_t *bit;
  const uint8_t *rowptr;
  const uint16_t *circ;
  int nt, k, m, slots, mb;
};

struct EncDev {
  int n, subch, blocks, used, vrows;
  const uint32_t *tixw;   // per coefficient, its place in the half-plane << 3 | 1 | its whitening's real bit << 1 | imaginary bit << 2
  const int32_t *block_tier, *block_slot;
  const uint32_t *crc;   // x^(8 (476 - 4 j)) mod P for word j of a block, then the all-ones init's term
  EncTier tier[kMaxTiers];
  int lines;   // the picture's column tiles are 2 lines wide
  int pxm, px, W, q, o, side, aside, a0[kAnchK];   // drive geometry (pixels), the anchors' first pixels
  int copy;   // every tap is the one sample's (the ring's pixels an exact copy of the picture's samples)
  const int32_t *rs_i0;
  const float *rs_w;
  const uint8_t *kind;
  // per ring pixel p < q: the exact copy's picture index (rs_i0 + 2) mod n and the first tap's rs_i0 mod n (both in
  // [0, n)); per drive pixel d < px: its border cell d / pxm
  const int32_t *rs_cp, *rs_c0, *cellx;
};

// ---------------------------------------------------------------- blocks to coefficients

// a * b mod the CRC's polynomial in the reflected representation (bit 31 is x^0).
__device__ __forceinline__ uint32_t crc_mul(uint32_t a, uint32_t b) {
  uint32_t p = 0;
#pragma unroll
  for (int i = 0; i < 32; i++) {
    p ^= b & (0u - ((a >> (31 - i)) & 1u));
    b = (b >> 1) ^ (0x82f63b78u & (0u - (b & 1u)));
  }
  return p;
}

// A block of kFrameGroup frames, one CTA: their bits, their codewords, their slots, their coefficients' signs into the
// half-plane, a byte a frame of a word a point (the frames of a group share the place, and the scattered stores, a
// sector each, are what a byte a store is bound by). Everything is words: a column of 128 data bits is four, a check
// row's data bits the XOR of its circulants' columns rotated (check c = i mb + r holds data bit col z + (i - shift) mod
// z of row r's circulants), CRC-32C (Castagnoli, reflected 0x82F63B78, liblizard/src/layout.c:44-54) a word a thread
// times its place, the parity's running XOR over the checks (i, then r) a prefix over the rows and one over the 128 bits
// of their sum. 3,968 blocks (32 pages of n = 1536): 140 us a bit a byte with the CRC on one thread, 92 in words a frame
// at a time (the stores), 27 four frames at a time.
constexpr int kBlockThreads = 128 * kFrameGroup, kBlockWords = 244;
__global__ void __launch_bounds__(kBlockThreads) enc_blocks_kernel(EncDev e, const uint8_t *blocks, int frames, int pilots, uint32_t *signs) {
  // frame g's word w at [w][g]: bit t of the codeword at bit t & 31 of word t >> 5, the parity rows of 128 past the data
  __shared__ __align__(16) uint32_t bits[kBlockWords][kFrameGroup];
  __shared__ uint32_t syn[kFrameGroup][4 * kMaxCheckRows], before[kFrameGroup][4], s_crc[kFrameGroup][4];
  const int group = blockIdx.x / e.blocks, b = blockIdx.x % e.blocks, g = threadIdx.x >> 7, tid = threadIdx.x & 127, lane = tid & 31;
  const int held = min(kFrameGroup, frames - group * kFrameGroup);
  const bool mine = g < held;
  const EncTier &t = e.tier[e.block_tier[b]];
  const uint8_t *src = blocks + ((int64_t)(group * kFrameGroup + g) * e.blocks + b) * LIZG_BLOCK_BYTES;
  constexpr int kWords = LIZG_BLOCK_BYTES / 4;
  uint32_t c = 0;
  if (tid < kWords) {
    uint32_t w = 0;
    if (!mine) w = 0;
    else if ((reinterpret_cast<uintptr_t>(src) & 3) == 0) w = __ldg(reinterpret_cast<const uint32_t *>(src) + tid);
    else w = src[4 * tid] | src[4 * tid + 1] << 8 | src[4 * tid + 2] << 16 | (uint32_t)src[4 * tid + 3] << 24;
    bits[tid][g] = __brev(__byte_perm(w, 0u, 0x0123u));   // bytes MSB first
    c = crc_mul(w, __ldg(e.crc + tid));
  }
  c = __reduce_xor_sync(0xffffffffu, c);
  if (lane == 0) s_crc[g][tid >> 5] = c;
  for (int w = kWords + 1 + tid; w < t.k / 32; w += 128) bits[w][g] = 0;
  __syncthreads();
  if (tid == 0) bits[kWords][g] = __brev(~(s_crc[g][0] ^ s_crc[g][1] ^ s_crc[g][2] ^ s_crc[g][3] ^ __ldg(e.crc + kWords)));   // MSB first
  __syncthreads();
  if (tid < 4 * t.mb) {
    const int r = tid >> 2, w = tid & 3;
    uint32_t acc = 0;
    for (int k = t.rowptr[r]; k < t.rowptr[r + 1]; k++) {
      const int cs = t.circ[k], sh = cs & 255, at = w - (sh >> 5), col = 4 * (cs >> 8);
      acc ^= __funnelshift_l(bits[col + ((at - 1) & 3)][g], bits[col + (at & 3)][g], sh & 31);
    }
    syn[g][tid] = acc;
  }
  __syncthreads();
  if (tid < 4) {
    uint32_t q = 0;
    for (int r = 0; r < t.mb; r++) { q ^= syn[g][4 * r + tid]; syn[g][4 * r + tid] = q; }
    // over the bits: each word's inclusive prefix, what the words before hold, one bit on
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) q ^= q << o;
    uint32_t carry = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const uint32_t up = __shfl_sync(0xfu, q, k) >> 31;
      if (tid > k) carry ^= up;
    }
    q ^= 0u - carry;
    const uint32_t last = __shfl_up_sync(0xfu, q, 1) >> 31;
    before[g][tid] = q << 1 | (tid ? last : 0u);
  }
  __syncthreads();
  if (tid < 4 * t.mb) bits[t.k / 32 + tid][g] = syn[g][tid] ^ before[g][tid & 3];
  __syncthreads();
  // the coefficients: two codeword bits or the pilots' count bit twice, whitened
  const int first = e.block_slot[b] / 2;
  const uint32_t present = 0x01010101u >> 8 * (kFrameGroup - held), q = present * (((uint32_t)(pilots >> (b & 1)) & 1) * 6);
  uint32_t *out = signs + (int64_t)group * e.vrows * e.n;
#pragma unroll 2
  for (int s = threadIdx.x; s < t.slots / 2; s += kBlockThreads) {
    const uint32_t at = __ldg(e.tixw + first + s);
    uint32_t v = q;
    if (2 * s < t.nt) {
      const uint32_t p = __ldg(t.bit + s), p0 = p & 31, p1 = p >> 16 & 31;
      const uint4 a = *reinterpret_cast<const uint4 *>(bits[(p & 0xffffu) >> 5]), d = *reinterpret_cast<const uint4 *>(bits[p >> 21]);
      v = (a.x >> p0 & 1) << 1 | (d.x >> p1 & 1) << 2 | (a.y >> p0 & 1) << 9 | (d.y >> p1 & 1) << 10 | (a.z >> p0 & 1) << 17 |
          (d.z >> p1 & 1) << 18 | (a.w >> p0 & 1) << 25 | (d.w >> p1 & 1) << 26;
    }
    out[at >> 3] = (v ^ (at & 7) * 0x01010101u) & present * 7;
  }
}

// The coefficients past the last block: the whitening alone.
__global__ void __launch_bounds__(kEncThreads) enc_pad_kernel(EncDev e, int frames, int per, uint32_t *signs) {
  const int group = blockIdx.x / per, s = e.used / 2 + (blockIdx.x % per) * blockDim.x + threadIdx.x;
  if (s >= e.subch * kSub) return;
  const uint32_t at = e.tixw[s], present = 0x01010101u >> 8 * (kFrameGroup - min(kFrameGroup, frames - group * kFrameGroup));
  signs[(int64_t)group * e.vrows * e.n + (at >> 3)] = (at & 7) * present;
}

// ---------------------------------------------------------------- resample and paint

// Down the picture: row y of the q x n intermediate from the six picture rows its taps read (the picture periodic).
__global__ void __launch_bounds__(kEncThreads) enc_vert_kernel(EncDev e, const float *pic, float *tmp) {
  const int f = blockIdx.x / e.q, y = blockIdx.x % e.q;
  const float *wt = e.rs_w + 6 * y;
  const float *pf = pic + (int64_t)f * e.n * e.n;
  int r[6];
#pragma unroll
  for (int t = 0; t < 6; t++) {
    int i = (e.rs_i0[y] + t) % e.n;
    if (i < 0) i += e.n;
    r[t] = i * 2 * e.lines;
  }
  float *out = tmp + ((int64_t)f * e.q + y) * e.n;
  for (int k = threadIdx.x; k < e.n; k += blockDim.x) {
    const float *col = pf + pic_at(e.n, e.lines, k);
    out[k] = wt[0] * col[r[0]] + wt[1] * col[r[1]] + wt[2] * col[r[2]] + wt[3] * col[r[3]] + wt[4] * col[r[4]] + wt[5] * col[r[5]];
  }
}

__device__ __forceinline__ float held01(float v) { return v < 0 ? 0.0f : v > 1 ? 1.0f : v; }

// A row of modules of the page, one CTA: the white margin, the border's cells, the picture resampled across, the anchors
// over it, put together in shared memory and written out in words. Margin, cells, picture and anchors all start and end
// on whole modules, so what the border shows is worked out once for the pxm rows. PIC_GREY: an exact copy for the grey page,
// of the picture in grey levels already, read tile by tile (a tile's pxm rows are one run of bytes); PIC_COPY: an exact
// copy of the picture (both passes' six terms are 0 x, 1 x the sample, 0 x ..., whose sums are the sample itself);
// PIC_TAPS: the taps across over the intermediate. 32 pages of 1944 x 1944: 290 us a page row a CTA with a pixel's place
// worked out at the pixel, 373 a thread a column, 155 with the grey levels read a byte a pixel, 74 so (issue, 73%).
enum { PIC_TAPS, PIC_COPY, PIC_GREY };
template <int SRC>
__global__ void __launch_bounds__(kEncThreads) enc_paint_kernel(EncDev e, int pitch, const void *src, float *drive, uint8_t *grey) {
  extern __shared__ __align__(16) uint8_t page[];   // the rows, `pitch` bytes apart, or where they are alike one of them
  const int strips = e.W / e.pxm, f = blockIdx.x / strips, cy = blockIdx.x % strips - kQuiet, m = kQuiet * e.pxm;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, dy0 = cy * e.pxm;
  const bool cells = cy >= 0 && cy < e.side, pic = dy0 >= e.o && dy0 < e.o + e.q;
  float *dr = drive && cells ? drive + ((int64_t)f * e.px + dy0) * e.px : nullptr;
  // the margin and the border's cells, beside the picture where the strip has one
  const int rows = pic ? e.pxm : 1, left = pic ? m + e.o : e.W;
  for (int i = tid; i < (pic ? e.W - e.q : e.W); i += kEncThreads) {
    const int X = i < left ? i : i + e.q, dx = X - m;
    uint8_t level = 255;
    if (cells && dx >= 0 && dx < e.px) {
      const float d = (e.kind[cy * e.side + e.cellx[dx]] & 3) == 2 ? 0.0f : 1.0f;
      level = grey_level(d);
      if (dr) for (int r = 0; r < e.pxm; r++) dr[(int64_t)r * e.px + dx] = d;
    }
    for (int r = 0; r < rows; r++) page[r * pitch + X] = level;
  }
  if (pic) {
    const int y0 = dy0 - e.o;
    uint8_t *to = page + m + e.o;
    if (SRC == PIC_GREY) {
      // two of a tile's bytes a thread, columns l and L + l of row r; the tiles in the order the page shows them
      const int L = e.lines, C = 2 * L, per = e.pxm * L, groups = max(1, kEncThreads / per), cp0 = e.rs_cp[0], tiles = e.n / C;
      const int skip = cp0 % C, units = (e.q + skip + C - 1) / C;
      const uint8_t *lev = static_cast<const uint8_t *>(src) + (int64_t)f * e.n * e.n;
      for (int i = tid; i < groups * per; i += kEncThreads) {
        const int g = i / per, r = (i - g * per) / L, l = i - g * per - r * L;
        const uint8_t *at = lev + e.rs_cp[y0 + r] * C + 2 * l;
        uint8_t *row = to + r * pitch;
        int tile = (cp0 / C + g) % tiles, x = g * C - skip + l;
        const int hop = groups % tiles;
#pragma unroll 4
        for (int u = g; u < units; u += groups, x += groups * C) {
          const uint32_t ab = __ldg(reinterpret_cast<const uint16_t *>(at + tile * C * e.n));
          if (x >= 0 && x < e.q) row[x] = (uint8_t)ab;
          if (x + L >= 0 && x + L < e.q) row[x + L] = (uint8_t)(ab >> 8);
          tile += hop;
          tile = tile >= tiles ? tile - tiles : tile;
        }
      }
    } else {
      for (int x = tid; x < e.q; x += kEncThreads) {
        float *d = dr ? dr + e.o + x : nullptr;
        if (SRC == PIC_COPY) {
          const float *col = static_cast<const float *>(src) + (int64_t)f * e.n * e.n + pic_at(e.n, e.lines, e.rs_cp[x]);
#pragma unroll 4
          for (int r = 0; r < e.pxm; r++) {
            const float v = held01(__ldg(col + e.rs_cp[y0 + r] * 2 * e.lines));
            to[r * pitch + x] = grey_level(v);
            if (d) d[(int64_t)r * e.px] = v;
          }
        } else {
          const float *row = static_cast<const float *>(src) + ((int64_t)f * e.q + y0) * e.n;
          int c[6];
          float wt[6];
          c[0] = e.rs_c0[x];
#pragma unroll
          for (int t = 0; t < 6; t++) {
            wt[t] = e.rs_w[6 * x + t];
            if (t) c[t] = c[t - 1] + 1 == e.n ? 0 : c[t - 1] + 1;
          }
#pragma unroll 2
          for (int r = 0; r < e.pxm; r++, row += e.n) {
            float v = wt[0] * __ldg(row + c[0]);
#pragma unroll
            for (int t = 1; t < 6; t++) v = v + wt[t] * __ldg(row + c[t]);
            v = held01(v);
            to[r * pitch + x] = grey_level(v);
            if (d) d[(int64_t)r * e.px] = v;
          }
        }
      }
    }
    // the anchors' pattern over it: light middle and rim, a dark ring (Chebyshev distance from its middle)
    int aj = -1;
#pragma unroll
    for (int j = 0; j < kAnchK; j++) if (dy0 >= e.a0[j] && dy0 < e.a0[j] + e.aside) aj = dy0 - e.a0[j];
    if (aj >= 0) {
      __syncthreads();
      const float half = 0.5f * (float)e.aside;
      for (int i = tid; i < kAnchK * e.aside; i += kEncThreads) {
        const int k = i / e.aside, ax = i - k * e.aside, dx = e.a0[k] + ax;
        const float ddx = fabsf((float)ax + 0.5f - half);
        for (int r = 0; r < e.pxm; r++) {
          const float rr = fmaxf(ddx, fabsf((float)(aj + r) + 0.5f - half)) / half, d = rr < 0.25f || rr >= 0.6f ? 1.0f : 0.0f;
          page[r * pitch + m + dx] = grey_level(d);
          if (dr) dr[(int64_t)r * e.px + dx] = d;
        }
      }
    }
  }
  if (!grey) return;
  __syncthreads();
  for (int r = warp; r < e.pxm; r += kEncThreads / 32) {   // a row a warp: bytes up to a word's edge, words, bytes
    uint8_t *out = grey + ((int64_t)f * e.W + (cy + kQuiet) * e.pxm + r) * e.W;
    const uint8_t *row = page + (pic ? r * pitch : 0);
    const int head = (int)(-reinterpret_cast<uintptr_t>(out) & 3), words = (e.W - head) / 4, tail = e.W - head - 4 * words;
    const uint32_t *from = reinterpret_cast<const uint32_t *>(row);   // pitch is whole words
    if (lane < head) out[lane] = row[lane];
    if (lane < tail) out[head + 4 * words + lane] = row[head + 4 * words + lane];
    for (int i = lane; i < words; i += 32)
      reinterpret_cast<uint32_t *>(out + head)[i] = __funnelshift_r(from[i], from[i + 1], 8 * head);
  }
}

// ---------------------------------------------------------------- host: the layout, the word, the resampler's taps

// Reed-Solomon parity of the format word over GF(256), polynomial 0x11d, roots alpha^0 .. (liblizard/src/rs.c:19-35).
static void word_encode(uint8_t *cw, int k, int nroots) {
  uint8_t ex[512], lg[256];
  int x = 1;
  for (int i = 0; i < 255; i++) { ex[i] = (uint8_t)x; lg[x] = (uint8_t)i; x <<= 1; if (x & 256) x ^= 0x11d; }
  for (int i = 255; i < 512; i++) ex[i] = ex[i - 255];
  auto mul = [&](int a, int b) -> uint8_t { return a && b ? ex[lg[a] + lg[b]] : 0; };
  uint8_t gen[256] = {1};
  for (int i = 0; i < nroots; i++) {
    gen[i + 1] = 0;
    for (int j = i + 1; j > 0; j--) gen[j] ^= mul(gen[j - 1], ex[i]);
  }
  uint8_t *par = cw + k;
  std::memset(par, 0, (size_t)nroots);
  for (int i = 0; i < k; i++) {
    const uint8_t fb = cw[i] ^ par[0];
    std::memmove(par, par + 1, (size_t)nroots - 1);
    par[nroots - 1] = 0;
    if (fb) for (int j = 0; j < nroots; j++) par[j] ^= mul(fb, gen[j + 1]);
  }
}

static int track_bit(int side, int j) {   // liblizard/src/layout.c:57-61
  uint32_t v = (uint32_t)(side * 4099 + (j >> 1)) * 2654435761u + 40503u;
  v ^= v >> 15;
  v *= 2246822519u;
  v ^= v >> 13;
  return (int)((v ^ (uint32_t)j) & 1);
}

// The border's cell kinds, side x side modules: the corner marks, the line, the timing track, the format word's
// cells (liblizard/src/layout.c:69-141 thin_init, thin_corner, ob_layout_set_fmt). 2 dark, 1 light, 0 the picture's;
// | 8 on the word's cells (CELL_WORD: the registration's templates skip them).
void layout_kind(int span, int version, int fps, std::vector<uint8_t> &kind) {
  const int side = span + 2 * kMargin, S = 12, reserve = 15, margin = kMargin;
  kind.assign((size_t)side * side, 1);
  for (int y = 0; y < side; y++)
    for (int x = 0; x < side; x++) {
      const int dx = std::min(x, side - 1 - x), dy = std::min(y, side - 1 - y), d = std::min(dx, dy);
      uint8_t k;
      if (dx < S && dy < S) {   // a corner mark
        const bool in = dx >= 1 && dx <= S - 2 && dy >= 1 && dy <= S - 2;
        const int cd = std::min(dx, dy);
        k = in && !(cd >= 3 && cd < 5) ? 2 : 1;
      } else {
        bool dark = d >= 1 && d <= 2;
        if (d >= 5 && d < 7) {
          const int along = dy <= dx ? x : y, len = side;
          const int sd = dy <= dx ? (y < side / 2 ? 0 : 2) : (x < side / 2 ? 3 : 1);
          const int cell = (along - reserve) / 2, run = cell / 4;
          if (along >= reserve && along < len - reserve && !(run & 1)) dark = track_bit(sd, run / 2 * 4 + cell % 4);
        }
        k = d >= margin - kCp ? 0 : dark ? 2 : 1;
      }
      kind[(size_t)y * side + x] = k;
    }
  // the word: RS(bytes, 3) of magic, version, fps over the word cells; blank (light) where the version is no format's
  const int thin = (side - 2 * reserve) / 2, wc = thin / 8 * 4, cells = wc >= 32 ? wc : 0, bytes = std::min(64, 4 * (cells / 8));
  uint8_t cw[64] = {0};
  if (bytes >= 16 && version >= 4 && version <= 64 && fps >= 0 && fps <= 255) {
    cw[0] = 0x4c; cw[1] = (uint8_t)version; cw[2] = (uint8_t)fps;
    word_encode(cw, 3, bytes - 3);
  }
  for (int sd = 0; sd < 4; sd++)
    for (int i = 0; i < cells; i++) {
      const int kb = 4 * (i >> 3) + sd;
      const int bit = kb < bytes ? (cw[kb] >> (7 - (i & 7))) & 1 : 0;
      const int off = ((i / 4) * 8 + i % 4 + 4) * 2;
      for (int j = 0; j < 2; j++)
        for (int ee = 0; ee < 2; ee++) {
          const int t = reserve + off + j, dd = 5 + ee;
          const int x = sd == 0 || sd == 2 ? t : sd == 3 ? dd : side - 1 - dd;
          const int y = sd == 0 ? dd : sd == 2 ? side - 1 - dd : t;
          kind[(size_t)y * side + x] = (bit ? 2 : 1) | 8;
        }
    }
}

static double lanczos3(double x) {   // liblizard/src/lizard_phy.c:970-975
  x = std::fabs(x);
  if (x >= 3) return 0;
  const double px = 3.14159265358979323846 * x;
  return 3 * std::sin(px) * std::sin(px / 3) / (px * px);
}

}  // namespace lizg

struct lizg_encoder {
  lizg::Format f;
  lizg::EncDev e{};
  lizg::EncFft xf{};
  int max_frames = 0, fps = 0;
  std::vector<void *> owned;
  float2 *S = nullptr;      // the row transforms, by column tiles
  float *pic = nullptr, *tmp = nullptr;   // the picture; the resampler's intermediate
  uint32_t *signs = nullptr;   // the half-plane's signs, in tmp's place: read by the row transforms, before tmp is written
  uint8_t *kind = nullptr;
};

namespace {
template <class T>
bool upload(lizg_encoder *x, const T **dst, const T *src, size_t count) {
  void *p = nullptr;
  if (cudaMalloc(&p, std::max<size_t>(1, count) * sizeof(T)) != cudaSuccess) return false;
  x->owned.push_back(p);
  if (count && cudaMemcpy(p, src, count * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) return false;
  *dst = static_cast<const T *>(p);
  return true;
}
bool alloc(lizg_encoder *x, void **dst, size_t bytes) {
  if (cudaMalloc(dst, std::max<size_t>(1, bytes)) != cudaSuccess) return false;
  x->owned.push_back(*dst);
  return true;
}
bool paint_kind(lizg_encoder *x) {
  std::vector<uint8_t> kind;
  lizg::layout_kind(x->f.span, x->f.subch % 16 == 0 ? x->f.subch / 16 : 0, x->fps, kind);
  return cudaMemcpy(x->kind, kind.data(), kind.size(), cudaMemcpyHostToDevice) == cudaSuccess;
}
}  // namespace

extern "C" {

lizg_encoder *lizg_encoder_new(int n, int subch, int span, int max_frames) {
  using namespace lizg;
  if (max_frames < 1 || max_frames > 4096) { record_error(LIZG_E_ARG, "lizg_encoder_new: max_frames must be 1..4096"); return nullptr; }
  int sms = 0;
  if (device_ready(&sms)) return nullptr;
  lizg_encoder *x = new (std::nothrow) lizg_encoder();
  if (!x) { record_error(LIZG_E_NOMEM, "lizg_encoder_new: out of host memory"); return nullptr; }
  Format &f = x->f;
  int rad[3], lines = 0;
  if (format_build(n, subch, span, f) || fft_plan(n, rad, &lines) || 2 * (f.vmax + 1) > n) {
    delete x;
    record_error(LIZG_E_ARG, "lizg_encoder_new: no such format");
    return nullptr;
  }
  x->max_frames = max_frames;
  EncDev &e = x->e;
  e.n = n; e.subch = subch; e.blocks = f.blocks; e.used = f.used; e.vrows = f.vmax + 1;
  e.pxm = (int)std::ceil((float)n / span - 1e-4f);
  e.side = span + 2 * kMargin;
  e.px = e.side * e.pxm;
  e.W = e.px + 2 * kQuiet * e.pxm;
  e.q = (span + 2 * kCp) * e.pxm;
  e.o = (kMargin - kCp) * e.pxm;
  const int a = span / 64;
  e.aside = a * e.pxm;
  for (int i = 0; i < kAnchK; i++) e.a0[i] = (int)std::floor(kMargin + (double)span * (i + 0.5) / kAnchK - a / 2.0 + 0.5) * e.pxm;
  std::vector<uint32_t> tixw(f.tix.size());
  for (size_t i = 0; i < tixw.size(); i++) tixw[i] = (uint32_t)f.tix[i] << 3 | 1u | (f.white[2 * i] ? 2u : 0u) | (f.white[2 * i + 1] ? 4u : 0u);
  bool ok = upload(x, &e.tixw, tixw.data(), tixw.size()) &&
            upload(x, &e.block_tier, f.block_tier.data(), f.block_tier.size()) && upload(x, &e.block_slot, f.block_slot.data(), f.block_slot.size());
  for (int t = 0; ok && t < f.tiers; t++) {
    const lizg_code_def_t &d = LIZG_CODES[f.tier[t].code];
    EncTier &et = e.tier[t];
    et.nt = f.tier[t].nt; et.k = f.tier[t].k; et.mb = d.mb; et.m = d.mb * LIZG_Z; et.slots = f.tier[t].slots;
    std::vector<uint32_t> bit((size_t)et.nt / 2);
    for (int i = 0; i < et.nt / 2 * 2; i++) {
      const int v = f.perm[t][i], at = v < et.k ? v : et.k + (v - et.k) % d.mb * LIZG_Z + (v - et.k) / d.mb;
      bit[i / 2] |= (uint32_t)at << 16 * (i & 1);
    }
    ok = upload(x, &et.bit, bit.data(), bit.size()) && upload(x, &et.rowptr, d.rowptr, (size_t)d.mb + 1) &&
         upload(x, &et.circ, d.circ, (size_t)d.rowptr[d.mb]) && et.m <= kMaxCheckRows * LIZG_Z && et.k + et.m <= 32 * kBlockWords && et.nt % 2 == 0;
  }
  {
    // CRC-32C as a sum of word products: x^(8 (476 - 4 j)) mod P, and the all-ones init's x^(8 476) times itself
    auto step = [](uint32_t r, int bits) { while (bits-- > 0) r = (r >> 1) ^ (0x82f63b78u & (0u - (r & 1u))); return r; };
    std::vector<uint32_t> crc;
    for (int j = 0; j < LIZG_BLOCK_BYTES / 4; j++) crc.push_back(step(0x80000000u, 8 * (LIZG_BLOCK_BYTES - 4 * j)));
    crc.push_back(step(0xffffffffu, 8 * LIZG_BLOCK_BYTES));
    ok = ok && upload(x, &e.crc, crc.data(), crc.size());
  }
  e.lines = lines;
  // the resampler's taps (liblizard/src/lizard_phy.c:980-1000)
  std::vector<int32_t> i0(e.q);
  std::vector<float> w(6 * (size_t)e.q);
  const double sc = (double)n / span;
  for (int p = 0; p < e.q; p++) {
    const double u = (p + 0.5) * sc / e.pxm - kCp * sc - 0.5, r = std::floor(u + 0.5);
    if (std::fabs(u - r) < 1e-6) {
      i0[p] = (int)r - 2;
      for (int t = 0; t < 6; t++) w[6 * p + t] = t == 2 ? 1.0f : 0.0f;
      continue;
    }
    const int a0 = (int)std::floor(u) - 2;
    double tw[6], sum = 0;
    for (int t = 0; t < 6; t++) { tw[t] = lanczos3(u - (a0 + t)); sum += tw[t]; }
    i0[p] = a0;
    for (int t = 0; t < 6; t++) w[6 * p + t] = (float)(tw[t] / sum);
  }
  ok = ok && upload(x, &e.rs_i0, i0.data(), i0.size()) && upload(x, &e.rs_w, w.data(), w.size());
  {
    std::vector<int32_t> cp(e.q), c0(e.q), cell(e.px);
    for (int p = 0; p < e.q; p++) {
      int a = (i0[p] + 2) % n, b = i0[p] % n;
      cp[p] = a < 0 ? a + n : a;
      c0[p] = b < 0 ? b + n : b;
    }
    for (int d = 0; d < e.px; d++) cell[d] = d / e.pxm;
    ok = ok && upload(x, &e.rs_cp, cp.data(), cp.size()) && upload(x, &e.rs_c0, c0.data(), c0.size()) && upload(x, &e.cellx, cell.data(), cell.size());
  }
  e.copy = 1;
  for (int p = 0; p < e.q && e.copy; p++)
    for (int t = 0; t < 6; t++) e.copy &= w[6 * p + t] == (t == 2 ? 1.0f : 0.0f);
  // the transform's twiddles
  std::vector<float2> tws(n);
  for (int st = 0, ns = 1; st < 3; ns *= rad[st], st++)
    for (int qq = 1; qq < rad[st]; qq++)
      for (int k = 0; k < ns; k++) {
        const double th = -2.0 * 3.14159265358979323846 * qq * k / ((double)ns * rad[st]);
        tws[ns + (qq - 1) * ns + k] = make_float2((float)std::cos(th), (float)std::sin(th));
      }
  const float2 *dtw = nullptr;
  ok = ok && upload(x, &dtw, tws.data(), tws.size());
  x->xf.n = n; x->xf.vrows = e.vrows; x->xf.tws = dtw;
  x->xf.lim = 2.0f * 2.0f * std::sqrt(0.5f * (float)(subch * kSub));   // LIZARD_CLIP 2, twice the half-plane's rms
  x->xf.sc = 0.5f / x->xf.lim;
  ok = ok && alloc(x, reinterpret_cast<void **>(&x->S), sizeof(float2) * (size_t)max_frames * e.vrows * n) &&
       alloc(x, reinterpret_cast<void **>(&x->pic), sizeof(float) * (size_t)max_frames * n * n) &&
       alloc(x, reinterpret_cast<void **>(&x->tmp), sizeof(float) * (size_t)max_frames * e.q * n) &&
       alloc(x, reinterpret_cast<void **>(&x->kind), (size_t)e.side * e.side);
  e.kind = x->kind;
  // signs: vrows n words for every kFrameGroup frames; tmp: q n floats a frame, q >= n >= 2 vrows
  x->signs = reinterpret_cast<uint32_t *>(x->tmp);
  ok = ok && e.q >= e.vrows && paint_kind(x);
  if (!ok) {
    lizg_encoder_free(x);
    record_error(LIZG_E_NOMEM, "lizg_encoder_new: device allocation or copy failed");
    return nullptr;
  }
  return x;
}

void lizg_encoder_free(lizg_encoder *x) {
  if (!x) return;
  for (void *p : x->owned) cudaFree(p);
  delete x;
}

int lizg_encoder_fps(lizg_encoder *x, int fps) {
  if (!x || fps < 0 || fps > 255) return lizg::record_error(LIZG_E_ARG, "lizg_encoder_fps: NULL handle or fps outside 0..255");
  x->fps = fps;
  return paint_kind(x) ? 0 : lizg::record_error(LIZG_E_CUDA, "lizg_encoder_fps: copy failed");
}

int lizg_layout_kind(int span, int version, int fps, uint8_t *kind) {
  if ((span != 128 && span != 256 && span != 512) || !kind) return lizg::record_error(LIZG_E_ARG, "lizg_layout_kind: span must be 128, 256 or 512");
  std::vector<uint8_t> k;
  lizg::layout_kind(span, version, fps, k);
  std::memcpy(kind, k.data(), k.size());
  return span + 2 * lizg::kMargin;
}

int lizg_encoder_info(const lizg_encoder *x, int32_t *out) {
  if (!x || !out) return lizg::record_error(LIZG_E_ARG, "lizg_encoder_info: NULL argument");
  out[0] = x->e.blocks; out[1] = x->e.pxm; out[2] = x->e.px; out[3] = x->e.W; out[4] = x->max_frames;
  return 0;
}

int lizg_encode_dev(lizg_encoder *x, const uint8_t *d_blocks, int frames, int pilots, float *d_drive, uint8_t *d_grey, void *stream) {
  using namespace lizg;
  if (!x || !d_blocks || (!d_drive && !d_grey) || frames < 1 || frames > x->max_frames || pilots < 0 || pilots > 3)
    return record_error(LIZG_E_ARG, "lizg_encode_dev: NULL argument, frames outside 1..max_frames or pilots outside 0..3");
  const EncDev &e = x->e;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int groups = (frames + kFrameGroup - 1) / kFrameGroup;
  cudaError_t err = cudaMemsetAsync(x->signs, 0, sizeof(uint32_t) * (size_t)groups * e.vrows * e.n, st);
  if (err == cudaSuccess) {
    enc_blocks_kernel<<<groups * e.blocks, kBlockThreads, 0, st>>>(e, d_blocks, frames, pilots, x->signs);
    const int pad = e.subch * kSub - e.used / 2, per = (pad + kEncThreads - 1) / kEncThreads;
    if (per > 0) enc_pad_kernel<<<groups * per, kEncThreads, 0, st>>>(e, frames, per, x->signs);
    err = cudaGetLastError();
  }
  // a copy for the grey page alone has its grey levels taken by the transform, a byte a sample written and read instead of
  // four: the column pass 154 us against 145 (117 now), the paint's 302 MB of samples 75
  const bool bytes = e.copy && !d_drive;
  if (err == cudaSuccess) err = enc_page_launch(x->xf, frames, x->signs, x->S, x->pic, bytes, st);
  if (err == cudaSuccess) {
    // rows an odd number of words apart, with one to read past the last
    const int pitch = ((e.W + 4) / 4 | 1) * 4, smem = pitch * e.pxm, grid = frames * (e.W / e.pxm);
    if (bytes) {
      enc_paint_kernel<PIC_GREY><<<grid, kEncThreads, smem, st>>>(e, pitch, x->pic, d_drive, d_grey);
    } else if (e.copy) {
      enc_paint_kernel<PIC_COPY><<<grid, kEncThreads, smem, st>>>(e, pitch, x->pic, d_drive, d_grey);
    } else {
      enc_vert_kernel<<<frames * e.q, kEncThreads, 0, st>>>(e, x->pic, x->tmp);
      enc_paint_kernel<PIC_TAPS><<<grid, kEncThreads, smem, st>>>(e, pitch, x->tmp, d_drive, d_grey);
    }
    err = cudaGetLastError();
  }
  return err == cudaSuccess ? 0 : record_error(LIZG_E_CUDA, (std::string("lizg_encode_dev: ") + cudaGetErrorString(err)).c_str());
}

}  // extern "C"
