// Problem policies that turn the persistent tcgen05 kernel (tc_kernel.cuh) into implicit-GEMM
// convolutions over a channels-last (NHWC) copy of the activations.
//
// Why channels-last: a filter tap shifts the window by whole pixels.  In NCHW the shifted
// pixel is the contiguous index, which breaks TMA's 16-byte start rule; in NHWC the shift
// lands on the w / h coordinates of the tensor map (any value, negative = zero padding for
// free) and the contiguous coordinate is the channel, always a multiple of 32 here.
//
//  PatchConvProblem  (forward, and backward-data with transposed taps)
//     rows  m = output pixels of a rectangular patch  NB images x PH rows x QW columns = 128
//     cols  n = output channels
//     k     = taps x 32-channel chunks:  A = one TMA box [32 c][QW][PH][NB] of the source at
//             the tap's offset (element strides implement the convolution stride),
//             B = packed filter [tap][n][c] (K-major)
//     out   = NCHW, optionally strided (the parity classes of a strided backward-data);
//             lanes of a warp hold consecutive pixels of a row, so each column is stored
//             as one coalesced run per patch row
//
//  PatchWgradProblem (backward-filter), one GEMM per group of taps:
//     rows  m = output channels (A = dy in NHWC, MN-major boxes [32 co][32 pixels])
//     cols  n = (tap of the group, input channel)  (B = x in NHWC at each tap's offset,
//             MN-major); layers with few input channels put several taps side by side so
//             that the dy tile is loaded once for all of them
//     k     = 32-pixel patches (QW x PH) of every image; split over CTAs, partial sums are
//             reduced in a fixed order by a second kernel.
#pragma once
#include "tc_pair.cuh"

namespace flb200 {
namespace tc {

// The taps a launch walks form a grid: tap (i, j) reads the source at offset
// (dh0 + i*dh_step, dw0 + j*dw_step) and uses filter element (r0 + i*r_step, s0 + j*s_step).
// Forward: every (r, s).  A parity class of a strided backward-data: the arithmetic
// progressions of r and s whose offsets divide by the stride.
struct TapGrid {
  int ni, nj;
  int dh0, dh_step, dw0, dw_step;
  int r0, r_step, s0, s_step, kW;
};

// One parity class of a launch (a forward pass has a single class): its taps and where its
// pixels land in the output.
struct PatchClass {
  TapGrid taps;
  int ntaps, oh_add, ow_add;
};
constexpr int kMaxPatchClasses = 4;

template <int BN>
struct PatchConvProblem {
  static constexpr bool kTwoProducers = false;
  static constexpr int kMinBlocks = 1;
  int a_mn_major, b_mn_major;  // 0, 0
  int operand;
  int kel;                     // channels per stage: 32 fp32, 64 16-bit
  // patch geometry (all powers of two, NB * PH * QW == 128)
  int QW, PH, NB, qw_shift, ph_shift;
  int tiles_q, tiles_p, tiles_b, tiles_n;
  int pix_w, pix_h, images;  // extent of the pixel grid the rows walk over
  int n_out;                 // number of output channels (columns)
  // K loop
  int cchunks;
  int a_w_mul, a_h_mul;      // A box origin = (q0 * a_w_mul + dw, p0 * a_h_mul + dh)
  // Parity classes served by this launch (strided backward-data with equal class extents: the
  // classes of one pixel patch are consecutive tiles, so that the interleaved stores of the
  // classes meet in L2 instead of reaching DRAM as half-written sectors of separate launches).
  int ncls;
  PatchClass cls[kMaxPatchClasses];
  // output: out[img][co][oh][ow], oh = p * oh_mul + oh_add, ow = q * ow_mul + ow_add
  float* out;                // 16-bit elements where operand says so (channels-last only)
  const float* bias;
  int out_H, out_W, out_C;
  int oh_mul, ow_mul;
  int fill_cell;  // see store()
  int out_cl;     // output stored channels-last: out[img][oh][ow][co]
  float* stats;   // EpiStats matrix [pixel tiles * 4][2 * n_out] (tc_kernel.cuh), or null

  struct Tile { int q0, p0, b0, n0, c; };
  struct LoadState { int i, j, cc, aw, ah, wtap, c, n0; };

  __device__ __forceinline__ int num_tiles() const {
    return tiles_q * tiles_p * tiles_b * tiles_n * ncls;
  }
  __device__ __forceinline__ void decode(int tile, Tile& t) const {
    int r = tile;
    t.c = r % ncls; r /= ncls;
    t.n0 = (r % tiles_n) * BN; r /= tiles_n;
    t.q0 = (r % tiles_q) * QW; r /= tiles_q;
    t.p0 = (r % tiles_p) * PH; r /= tiles_p;
    t.b0 = r * NB;
  }
  // CTA pairs: the two halves of a pair tile are consecutive pixel patches that share the
  // column block n0 (hence the whole B tile and the K loop).  Patches are enumerated fastest,
  // column blocks slowest; an odd patch count leaves the last pair a phantom half whose image
  // index is out of range (its loads are zero-filled, its stores masked).
  __device__ __forceinline__ int num_pair_tiles() const {
    return ((tiles_q * tiles_p * tiles_b + 1) >> 1) * tiles_n * ncls;
  }
  __device__ __forceinline__ void decode_pair(int tile, int rank, Tile& t) const {
    const int pairs_m = (tiles_q * tiles_p * tiles_b + 1) >> 1;
    t.c = tile % ncls;
    tile /= ncls;
    const int nt = tile / pairs_m;
    int r = 2 * (tile - nt * pairs_m) + rank;
    t.n0 = nt * BN;
    t.q0 = (r % tiles_q) * QW; r /= tiles_q;
    t.p0 = (r % tiles_p) * PH; r /= tiles_p;
    t.b0 = r * NB;
  }
  template <int>
  __device__ __forceinline__ void load_begin_pair(const Tile& t, LoadState& ls, int rank) const {
    load_begin<kBoth>(t, ls);
    ls.n0 = t.n0 + rank * (BN / 2);  // this CTA's half of B
  }
  template <int>
  __device__ __forceinline__ void load_pair(const CUtensorMap* ma, const CUtensorMap* mb,
                                            const Tile& t, LoadState& ls, uint32_t full_bar,
                                            char* a_dst, char* b_dst) const {
    int ca[4] = {ls.cc * kel, ls.aw, ls.ah, t.b0};
    tma_load_pair(ma, full_bar, a_dst, 4, ca);
    int cb[4] = {ls.cc * kel, ls.n0, ls.wtap, 0};
    tma_load_pair(mb, full_bar, b_dst, 3, cb);
    advance(ls);
  }
  __device__ __forceinline__ void advance(LoadState& ls) const {
    if (++ls.cc == cchunks) {  // next tap: j fastest
      const TapGrid& taps = cls[ls.c].taps;
      ls.cc = 0;
      ls.aw += taps.dw_step;
      ls.wtap += taps.s_step;
      if (++ls.j == taps.nj) {
        ls.j = 0;
        ++ls.i;
        ls.aw -= taps.nj * taps.dw_step;
        ls.ah += taps.dh_step;
        ls.wtap += taps.r_step * taps.kW - taps.nj * taps.s_step;
      }
    }
  }
  __device__ __forceinline__ int k_begin(const Tile&) const { return 0; }
  __device__ __forceinline__ int k_end(const Tile& t) const { return cls[t.c].ntaps * cchunks; }
  template <int>
  __device__ __forceinline__ void load_begin(const Tile& t, LoadState& ls) const {
    ls.n0 = t.n0;
    ls.i = 0;
    ls.j = 0;
    ls.cc = 0;
    const TapGrid& taps = cls[t.c].taps;
    ls.c = t.c;
    ls.aw = t.q0 * a_w_mul + taps.dw0;
    ls.ah = t.p0 * a_h_mul + taps.dh0;
    ls.wtap = taps.r0 * taps.kW + taps.s0;
  }
  __device__ __forceinline__ uint32_t stage_bytes(const Tile&) const {
    return (kBM + BN) * kBK * 4;  // NB * PH * QW == 128 rows of 128 bytes + B tile
  }
  template <int>
  __device__ __forceinline__ void load(const CUtensorMap* ma, const CUtensorMap* mb,
                                       const Tile& t, LoadState& ls, uint64_t* bar, char* a_dst,
                                       char* b_dst) const {
    int ca[4] = {ls.cc * kel, ls.aw, ls.ah, t.b0};
    tma_load(ma, bar, a_dst, 4, ca);
    int cb[4] = {ls.cc * kel, ls.n0, ls.wtap, 0};
    tma_load(mb, bar, b_dst, 3, cb);
    advance(ls);
  }
  __device__ __forceinline__ bool chunk_live(const Tile& t, int c0) const {
    return t.n0 + c0 < n_out;
  }
  // pixel index (in the whole output) of row `r` of the tile, class offsets applied, or -1 for a
  // row outside the image
  __device__ __forceinline__ long long cl_pixel(const Tile& t, int r) const {
    const int q = t.q0 + (r & (QW - 1));
    const int p = t.p0 + ((r >> qw_shift) & (PH - 1));
    const int img = t.b0 + (r >> (qw_shift + ph_shift));
    if (q >= pix_w || p >= pix_h || img >= images) return -1;
    const int oh_add = fill_cell ? 0 : cls[t.c].oh_add, ow_add = fill_cell ? 0 : cls[t.c].ow_add;
    return ((long long)img * out_H + p * oh_mul + oh_add) * out_W + q * ow_mul + ow_add;
  }
  // Pixel rows 4k + lane / 8 (k = 0..7) of the warp's staged chunk, 4 channels per lane, bias
  // added; STATS (uniform across the grid, so a copy of the loop each): per-channel sums of the
  // stored values into the statistics matrix.  FILL: the strided backward-data whose only
  // class with taps is (0, 0) — every pixel also writes the zeros of its cell, whole
  // rows like its own values, so the tensor needs no clearing pass.
  template <typename T, bool STATS, bool FILL>
  __device__ __forceinline__ void staged_pixels(const Tile& t, int row, int nb, float* stage,
                                                int lane) const {
    float4 bq = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias) bq = *reinterpret_cast<const float4*>(bias + nb + 4 * (lane & 7));
    const int r_first = row - lane;
    // every lane works out the address of its own row; the rows it stores come by shuffle
    const long long own = cl_pixel(t, row);
    float4 val[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) val[k] = epi_stage_read(stage, lane, k);
    EpiStats acc;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const long long pix = __shfl_sync(0xffffffffu, own, 4 * k + (lane >> 3));
      float4 v = val[k];
      v.x += bq.x; v.y += bq.y; v.z += bq.z; v.w += bq.w;
      if (pix >= 0) {
        T* dst = reinterpret_cast<T*>(out) + pix * out_C + nb + 4 * (lane & 7);
        if (STATS) {
          v = epi_round<T>(v);
          acc.add(v);
        }
        epi_store4(dst, v);
        if (FILL) {
          // this pixel owns its whole oh_mul x ow_mul cell: the other pixels receive zeros
          const int r = r_first + 4 * k + (lane >> 3);
          const int ow0 = (t.q0 + (r & (QW - 1))) * ow_mul;
          const int oh0 = (t.p0 + ((r >> qw_shift) & (PH - 1))) * oh_mul;
          for (int a = 0; a < oh_mul && oh0 + a < out_H; ++a)
            for (int b = a == 0 ? 1 : 0; b < ow_mul && ow0 + b < out_W; ++b)
              epi_store4(dst + ((long long)a * out_W + b) * out_C, make_float4(0.f, 0.f, 0.f, 0.f));
        }
      }
    }
    if (STATS) {
      const long long tile_m = ((long long)(t.b0 >> (7 - qw_shift - ph_shift)) * tiles_p +
                                (t.p0 >> ph_shift)) * tiles_q + (t.q0 >> qw_shift);
      acc.flush(stats, tile_m * 4 + (row >> 5), n_out, nb, lane, stage);
    }
  }
  template <typename T>
  __device__ __forceinline__ void store_cl(const Tile& t, int row, int nb, const float* v,
                                           float* stage, int lane) const {
    if (nb + 32 <= n_out && (out_C & 3) == 0) {
      // through the warp's staging tile, 4 whole pixel rows per store instruction (tc_kernel.cuh)
      epi_stage_write(stage, lane, v);
      if (fill_cell) staged_pixels<T, false, true>(t, row, nb, stage, lane);
      else if (stats) staged_pixels<T, true, false>(t, row, nb, stage, lane);
      else staged_pixels<T, false, false>(t, row, nb, stage, lane);
      __syncwarp();
      return;
    }
    // the channel tail, one pixel per lane; the other pixels of a cell receive zeros
    const long long pix = cl_pixel(t, row);
    if (pix < 0) return;
    const int q = t.q0 + (row & (QW - 1)), p = t.p0 + ((row >> qw_shift) & (PH - 1));
    const int cell_h = fill_cell ? min(oh_mul, out_H - p * oh_mul) : 1;
    const int cell_w = fill_cell ? min(ow_mul, out_W - q * ow_mul) : 1;
    for (int a = 0; a < cell_h; ++a)
      for (int b = 0; b < cell_w; ++b) {
        T* dst = reinterpret_cast<T*>(out) + (pix + (long long)a * out_W + b) * out_C + nb;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (nb + j < n_out)
            dst[j] = Num<T>::from_f(a == 0 && b == 0 ? v[j] + (bias ? bias[nb + j] : 0.f) : 0.f);
      }
  }
  __device__ __forceinline__ void store(const Tile& t, int row, int c0, const float* v,
                                        float* stage, int lane) const {
    const int nb = t.n0 + c0;
    if (out_cl) {
      if (operand == kOperandTf32) store_cl<float>(t, row, nb, v, stage, lane);
      else if (operand == kOperandBf16) store_cl<__nv_bfloat16>(t, row, nb, v, stage, lane);
      else store_cl<__half>(t, row, nb, v, stage, lane);
      return;
    }
    // row -> (image, p, q) inside the patch
    const int q = t.q0 + (row & (QW - 1));
    const int p = t.p0 + ((row >> qw_shift) & (PH - 1));
    const int img = t.b0 + (row >> (qw_shift + ph_shift));
    if (q >= pix_w || p >= pix_h || img >= images) return;
    const long long plane = (long long)out_H * out_W;
    if (fill_cell) {
      // Strided backward-data whose only class with taps is (0, 0): this pixel owns the whole
      // oh_mul x ow_mul cell and writes its zeros too, so the tensor needs no separate
      // clearing pass and every 32-byte sector is written whole.
      float* cell = out + ((long long)img * out_C + nb) * plane +
                    (long long)(p * oh_mul) * out_W + q * ow_mul;
      const bool pair = ow_mul == 2 && (out_W & 1) == 0;
      for (int a = 0; a < oh_mul; ++a) {
        if (p * oh_mul + a >= out_H) break;
        float* rowp = cell + (long long)a * out_W;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (nb + j >= n_out) break;
          const float val = a == 0 ? v[j] : 0.f;
          if (pair) {
            *reinterpret_cast<float2*>(rowp + j * plane) = make_float2(val, 0.f);
          } else {
            for (int b = 0; b < ow_mul; ++b)
              if (q * ow_mul + b < out_W) rowp[j * plane + b] = b == 0 ? val : 0.f;
          }
        }
      }
      return;
    }
    float* dst = out + ((long long)img * out_C + nb) * plane +
                 (long long)(p * oh_mul + cls[t.c].oh_add) * out_W + (q * ow_mul + cls[t.c].ow_add);
    if (nb + 32 <= n_out) {
      if (bias) {
        const float* bn = bias + nb;
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[j * plane] = v[j] + bn[j];
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[j * plane] = v[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (nb + j < n_out) dst[j * plane] = v[j] + (bias ? bias[nb + j] : 0.f);
    }
  }
};

template <int BN>
struct PatchWgradProblem {
  static constexpr bool kTwoProducers = true;
  static constexpr int kMinBlocks = 1;
  int a_mn_major, b_mn_major;  // 1, 1
  int operand;
  int QW, PH;                  // pixel patch of one stage: QW * PH == 32 (16-bit operands: 64)
  int cb_shift;                // log2 of the channels of one box: 5 (16-bit operands: 6)
  int tiles_q, tiles_p, images;
  int tiles_m, tiles_n, M, N;  // M = output channels, N = input channels
  // The BN columns of a tile are tg taps x (1 << cn_shift) boxes of 32 input channels, so a
  // narrow layer shares one load of dy between several taps.
  int ntaps, tap_groups, tg, cn_shift;
  int a_nbox;                  // 32-channel boxes of dy per stage: min(4, ceil(M / 32))
  int a_each, b_each;          // 1: a copy per box (nhwc_operand), else one copy of all of them
  int splits, iters_per_split, k_iters;  // k_iters = images * tiles_p * tiles_q
  int b_w_mul, b_h_mul;        // B box origin = (q0 * b_w_mul + dw, p0 * b_h_mul + dh)
  int kW, dil_x, dil_y, pad_x, pad_y;  // tap t = (r, s) = (t / kW, t % kW): dw = s*dil_x - pad_x
  float* partial;              // [split][tap][M][N]

  struct Tile { int m0, n0, tap0, ntap, cn_live, split, k0, k1; };
  // (tr, ts): the first of the taps [tap, tap_end) that this producer loads
  struct LoadState { int qi, pi, img, tr, ts, tap, tap_end; };

  __device__ __forceinline__ int num_tiles() const {
    return tiles_m * tiles_n * tap_groups * splits;
  }
  __device__ __forceinline__ void decode(int tile, Tile& t) const {
    int r = tile;
    t.split = r % splits; r /= splits;
    t.n0 = (r % tiles_n) * BN; r /= tiles_n;
    t.m0 = (r % tiles_m) * kBM; r /= tiles_m;
    t.tap0 = r * tg;
    t.ntap = min(tg, ntaps - t.tap0);
    t.cn_live = min(1 << cn_shift, (N - t.n0 + (1 << cb_shift) - 1) >> cb_shift);
    t.k0 = t.split * iters_per_split;
    t.k1 = min(t.k0 + iters_per_split, k_iters);
  }
  __device__ __forceinline__ int k_begin(const Tile& t) const { return t.k0; }
  __device__ __forceinline__ int k_end(const Tile& t) const { return t.k1; }
  template <int kWhich>
  __device__ __forceinline__ void load_begin(const Tile& t, LoadState& ls) const {
    int r = t.k0;
    ls.qi = r % tiles_q; r /= tiles_q;
    ls.pi = r % tiles_p; r /= tiles_p;
    ls.img = r;
    // of two producers A's takes the last taps of a tile of several
    const int moved = kWhich == kBoth ? 0 : (t.ntap - 1) >> 1;
    ls.tap = kWhich == kA ? t.ntap - moved : 0;
    ls.tap_end = kWhich == kB ? t.ntap - moved : t.ntap;
    ls.tr = (t.tap0 + ls.tap) / kW;
    ls.ts = t.tap0 + ls.tap - ls.tr * kW;
  }
  // 32 pixels x 32 fp32 or 64 pixels x 64 16-bit channels
  __device__ __forceinline__ int box_bytes() const { return 128 << cb_shift; }
  __device__ __forceinline__ uint32_t stage_bytes(const Tile& t) const {
    return (a_nbox + (t.ntap << cn_shift)) * box_bytes();
  }
  // With the channel index of a map split into (32 contiguous channels, group of 32) one copy
  // brings every 32 x 32 box of an operand: a_nbox boxes of dy, and per tap 1 << cn_shift boxes
  // of x.  Boxes past the last channel are zero-filled or hold a neighbouring pixel's channels;
  // they only reach accumulator rows / columns that the epilogue never stores.  Over whole
  // channels each box is a copy of its own, zero-filled past the last channel.
  template <int kWhich>
  __device__ __forceinline__ void load(const CUtensorMap* ma, const CUtensorMap* mb,
                                       const Tile& t, LoadState& ls, uint64_t* bar, char* a_dst,
                                       char* b_dst) const {
    const int q0 = ls.qi * QW, p0 = ls.pi * PH;
    if constexpr (kWhich != kB) {
      if (a_each) {
        for (int i = 0; i < a_nbox; ++i) {
          int ca[5] = {t.m0 + (i << cb_shift), q0, p0, ls.img, 0};
          tma_load(ma, bar, a_dst + i * box_bytes(), 4, ca);
        }
      } else {
        int ca[5] = {0, q0, p0, ls.img, t.m0 >> cb_shift};
        tma_load(ma, bar, a_dst, 5, ca);
      }
    }
    if (ls.tap < ls.tap_end) {
      const int w0 = q0 * b_w_mul - pad_x, h0 = p0 * b_h_mul - pad_y;
      int w = w0 + ls.ts * dil_x, h = h0 + ls.tr * dil_y, ts = ls.ts;
      for (int tap = ls.tap;;) {
        char* dst = b_dst + (tap << cn_shift) * box_bytes();
        if (b_each) {
          for (int i = 0; i < 1 << cn_shift; ++i) {
            int cb[5] = {t.n0 + (i << cb_shift), w, h, ls.img, 0};
            tma_load(mb, bar, dst + i * box_bytes(), 4, cb);
          }
        } else {
          int cb[5] = {0, w, h, ls.img, t.n0 >> cb_shift};
          tma_load(mb, bar, dst, 5, cb);
        }
        if (++tap >= ls.tap_end) break;
        w += dil_x;
        if (++ts == kW) { ts = 0; w = w0; h += dil_y; }
      }
    }
    if (++ls.qi == tiles_q) {
      ls.qi = 0;
      if (++ls.pi == tiles_p) { ls.pi = 0; ++ls.img; }
    }
  }
  __device__ __forceinline__ bool chunk_live(const Tile& t, int c0) const {
    const int j = c0 >> cb_shift;
    return (j >> cn_shift) < t.ntap && (j & ((1 << cn_shift) - 1)) < t.cn_live;
  }
  __device__ __forceinline__ void store(const Tile& t, int row, int c0, const float* v,
                                        float* stage, int lane) const {
    const int m = t.m0 + row, m_first = m - lane;
    const int j = c0 >> cb_shift;
    const int tap = t.tap0 + (j >> cn_shift);
    const int nb = t.n0 + ((j & ((1 << cn_shift) - 1)) << cb_shift) + (c0 & ((1 << cb_shift) - 1));
    if (nb >= N || m_first >= M) return;
    float* base = partial + (((long long)t.split * ntaps + tap) * M + m_first) * N + nb;
    if (nb + 32 <= N && (N & 3) == 0) {
      // whole 128-byte rows per store instruction (tc_kernel.cuh)
      epi_stage_write(stage, lane, v);
      float4 val[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) val[k] = epi_stage_read(stage, lane, k);
      float* dst = base + (long long)(lane >> 3) * N + 4 * (lane & 7);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (m_first + 4 * k + (lane >> 3) < M)
          *reinterpret_cast<float4*>(dst + 4LL * k * N) = val[k];
      __syncwarp();
      return;
    }
    if (m >= M) return;
    float* dst = base + (long long)lane * N;
#pragma unroll
    for (int jj = 0; jj < 32; ++jj)
      if (nb + jj < N) dst[jj] = v[jj];
  }
};

}  // namespace tc
}  // namespace flb200
