// conv2d forward, backward-data and backward-filter(+bias) as implicit GEMMs
// over fl's native layout: x [N][C][H][W], w [Cout][C/groups][kH][kW],
// y [N][Cout][Ho][Wo] (row-major views of fl's column-major tensors; the byte
// buffers are identical, cf. flashlight/fl/autograd/tensor/backend/onednn/Conv2D.cpp:171-178).
// Stands behind fl::AutogradExtension::conv2d / ::conv2dBackwardData /
// ::conv2dBackwardFilterBias (flashlight/fl/autograd/tensor/AutogradExtension.h:58-69,
// 110-138).  Cross-correlation, stride (sx,sy), symmetric zero padding (px,py),
// dilation (dx,dy), groups.
//
// GEMM views (per group):
//   forward   M = batch*Ho*Wo, N = Cout/g,        K = (C/g)*kH*kW
//   bwd data  M = batch*H*W,   N = C/g,           K = (Cout/g)*kH*kW
//   bwd filt  M = Cout/g,      N = (C/g)*kH*kW,   K = batch*Ho*Wo   (split-K)
// STRICT mode: the fp32-FMA kernel of simt_gemm.cuh with the loaders below.  Channels-last images
// of a multiple of 4 channels are read in 16-byte runs of channels, K ordered (tap, channel),
// against a filter repacked to that order; anything else element by element with the lanes along
// the pixels, K in the filter's own order (channel, tap).
// TF32 mode: shapes covered by the tensor-core kernels go to tc_conv, the rest
// fall through to the fp32 kernel.
#include "filter_permute.cuh"
#include "simt_gemm.cuh"
#include "tc_conv.cuh"
#include "tc_gemm.cuh"

namespace flb200 {

int make_conv_geo(const char* name, const flb200_conv2d_desc* d, ConvGeo* g) {
  FLB200_REQUIRE(d, "%s: null descriptor", name);
  FLB200_REQUIRE(d->W >= 1 && d->H >= 1 && d->C >= 1 && d->N >= 1, "%s: empty input", name);
  FLB200_REQUIRE(d->kW >= 1 && d->kH >= 1 && d->Cout >= 1, "%s: empty filter", name);
  FLB200_REQUIRE(d->sx >= 1 && d->sy >= 1 && d->dx >= 1 && d->dy >= 1 && d->px >= 0 && d->py >= 0,
                 "%s: bad stride/dilation/padding", name);
  FLB200_REQUIRE(d->groups >= 1 && d->C % d->groups == 0 && d->Cout % d->groups == 0,
                 "%s: channels (%d in, %d out) not divisible by groups (%d)", name, d->C, d->Cout,
                 d->groups);
  FLB200_REQUIRE(d->dtype == FLB200_F32 || d->dtype == FLB200_F16 || d->dtype == FLB200_BF16,
                 "%s: unknown dtype %d", name, d->dtype);
  FLB200_REQUIRE(d->math_mode >= FLB200_MATH_STRICT_F32 && d->math_mode <= FLB200_MATH_F32X3,
                 "%s: unknown math mode %d", name, d->math_mode);
  const int ekw = 1 + (d->kW - 1) * d->dx, ekh = 1 + (d->kH - 1) * d->dy;
  FLB200_REQUIRE(d->W + 2 * d->px >= ekw && d->H + 2 * d->py >= ekh,
                 "%s: filter larger than padded input", name);
  g->W = d->W; g->H = d->H; g->C = d->C; g->N = d->N;
  g->kW = d->kW; g->kH = d->kH; g->Cout = d->Cout;
  g->sx = d->sx; g->sy = d->sy; g->px = d->px; g->py = d->py; g->dx = d->dx; g->dy = d->dy;
  g->groups = d->groups;
  g->Wo = 1 + (d->W + 2 * d->px - ekw) / d->sx;
  g->Ho = 1 + (d->H + 2 * d->py - ekh) / d->sy;
  g->Cg = d->C / d->groups;
  g->Coutg = d->Cout / d->groups;
  g->HW = d->H * d->W;
  g->HoWo = g->Ho * g->Wo;
  g->RS = d->kH * d->kW;
  FLB200_REQUIRE(d->layout == FLB200_LAYOUT_NCHW || d->layout == FLB200_LAYOUT_NHWC ||
                     d->layout == FLB200_LAYOUT_NCHW_IN_NHWC_OUT,
                 "%s: unknown layout %d", name, d->layout);
  g->x_cl = d->layout == FLB200_LAYOUT_NHWC;
  g->y_cl = d->layout != FLB200_LAYOUT_NCHW;
  g->x_cs = g->x_cl ? 1 : g->HW;
  g->x_ps = g->x_cl ? d->C : 1;
  g->y_cs = g->y_cl ? 1 : g->HoWo;
  g->y_ps = g->y_cl ? d->Cout : 1;
  g->operand = tc::kOperandTf32;
  return FLB200_OK;
}

namespace {

// Pixel index and filter tap of the two image views: the forward pass reads x at
// (p*sy - py + r*dy, q*sx - px + s*dx), backward-data reads dy where h + py - r*dy and
// w + px - s*dx divide by the stride.
struct PixelRow { long long base; int h0, w0; };

// ---- images read channel-run-wise (channels-last, a multiple of 4 channels per group)
template <bool DGRAD>
struct ImageVec {
  static constexpr int kKind = kVecK;
  const float* p;
  ConvGeo g;
  int n_total, c4;  // pixels, 4-channel runs per tap
  typedef PixelRow Row;
  struct Iter { int cq, r, s; };
  __device__ const float* base() const { return p; }
  __device__ Row row(int n, int z) const {
    if (n >= n_total) return Row{-1, 0, 0};
    if (DGRAD) {
      const int img = n / g.HW, hw = n - img * g.HW, h = hw / g.W, w = hw - h * g.W;
      return Row{(long long)img * g.Cout * g.HoWo + (long long)z * g.Coutg, h + g.py, w + g.px};
    }
    const int img = n / g.HoWo, pq = n - img * g.HoWo, y = pq / g.Wo, q = pq - y * g.Wo;
    return Row{(long long)img * g.C * g.HW + (long long)z * g.Cg, y * g.sy - g.py, q * g.sx - g.px};
  }
  __device__ Iter iter(int k, int) const {
    const int run = k >> 2, tap = run / c4, r = tap / g.kW;
    return Iter{run - tap * c4, r, tap - r * g.kW};
  }
  __device__ void advance(Iter& it) const {
    it.cq += kBKf / 4;
    while (it.cq >= c4) {
      it.cq -= c4;
      if (++it.s == g.kW) { it.s = 0; ++it.r; }
    }
  }
  __device__ const float* at(const Row& row, const Iter& it) const {
    if (row.base < 0) return nullptr;
    if (DGRAD) {
      const int th = row.h0 - it.r * g.dy, tw = row.w0 - it.s * g.dx;
      if (th < 0 || tw < 0) return nullptr;
      int y = th, q = tw;
      if (g.sy != 1) { y = th / g.sy; if (y * g.sy != th) return nullptr; }
      if (g.sx != 1) { q = tw / g.sx; if (q * g.sx != tw) return nullptr; }
      if (y >= g.Ho || q >= g.Wo) return nullptr;
      return p + row.base + (long long)(y * g.Wo + q) * g.Cout + 4 * it.cq;
    }
    const int h = row.h0 + it.r * g.dy, w = row.w0 + it.s * g.dx;
    if (h < 0 || h >= g.H || w < 0 || w >= g.W) return nullptr;
    return p + row.base + (long long)(h * g.W + w) * g.C + 4 * it.cq;
  }
};

// ---- images read element by element, K = (channel, tap).  Row and k carry their part of the offset
// whether or not they meet inside the image, so that an element costs two additions, the test of its
// position and one address; only backward-data with a stride has to divide.
constexpr int kNowhere = -(1 << 30);  // a position that no tap brings inside
template <bool DGRAD>
struct ImageElem {
  static constexpr int kKind = kElemRows;
  const float* p;
  ConvGeo g;
  int n_total;
  struct Row { long long off; int h0, w0; };
  struct Kk { long long off; int dh, dw; };
  __device__ const float* base() const { return p; }
  __device__ bool divides() const { return DGRAD && (g.sx != 1 || g.sy != 1); }
  __device__ Row row(int n, int z) const {
    if (n >= n_total) return Row{0, kNowhere, kNowhere};
    Row r;
    if (DGRAD) {
      const int img = n / g.HW, hw = n - img * g.HW, h = hw / g.W, w = hw - h * g.W;
      r.off = (long long)img * g.Cout * g.HoWo + (long long)z * g.Coutg * g.y_cs;
      r.h0 = h + g.py;
      r.w0 = w + g.px;
      if (!divides()) r.off += ((long long)r.h0 * g.Wo + r.w0) * g.y_ps;
    } else {
      const int img = n / g.HoWo, pq = n - img * g.HoWo, y = pq / g.Wo, q = pq - y * g.Wo;
      r.h0 = y * g.sy - g.py;
      r.w0 = q * g.sx - g.px;
      r.off = (long long)img * g.C * g.HW + (long long)z * g.Cg * g.x_cs +
              ((long long)r.h0 * g.W + r.w0) * g.x_ps;
    }
    return r;
  }
  __device__ Kk kk(int k, int) const {
    const int c = k / g.RS, rs = k - c * g.RS, r = rs / g.kW, s = rs - r * g.kW;
    Kk v{(long long)c * (DGRAD ? g.y_cs : g.x_cs), r * g.dy, s * g.dx};
    if (DGRAD) {
      v.dh = -v.dh;
      v.dw = -v.dw;
    }
    if (!divides()) v.off += ((long long)v.dh * (DGRAD ? g.Wo : g.W) + v.dw) * (DGRAD ? g.y_ps : g.x_ps);
    return v;
  }
  __device__ const float* at(const Row& row, const Kk& k) const {
    int h = row.h0 + k.dh, w = row.w0 + k.dw;
    long long off = row.off + k.off;
    if (divides()) {
      if (h < 0 || w < 0) return nullptr;
      const int y = h / g.sy, q = w / g.sx;
      if (y * g.sy != h || q * g.sx != w) return nullptr;
      h = y;
      w = q;
      off += ((long long)y * g.Wo + q) * g.y_ps;
    }
    const bool inside = (unsigned)h < (unsigned)(DGRAD ? g.Ho : g.H) && (unsigned)w < (unsigned)(DGRAD ? g.Wo : g.W);
    return inside ? p + off : nullptr;
  }
};

// ---- filters.  The filter in the K order of the image view: row = co (forward) or ci
// (backward-data), tap_major: k = (tap, channel) else (channel, tap).
struct FilterElem {
  static constexpr int kKind = kElemK;
  const float* w;
  ConvGeo g;
  int dgrad, tap_major, rows;
  struct Row { long long off; };
  struct Kk { long long off; };
  __device__ const float* base() const { return w; }
  __device__ Row row(int r, int z) const {
    if (r >= rows) return Row{-1};
    const long long group = (long long)z * g.Coutg * g.Cg * g.RS;
    return Row{group + (long long)r * g.RS * (dgrad ? 1 : g.Cg)};
  }
  __device__ Kk kk(int k, int) const {
    const int ch = dgrad ? g.Coutg : g.Cg;
    const int c = tap_major ? k % ch : k / g.RS, tap = tap_major ? k / ch : k - c * g.RS;
    return Kk{(long long)c * g.RS * (dgrad ? g.Cg : 1) + tap};
  }
  __device__ const float* at(const Row& r, const Kk& k) const {
    return r.off >= 0 ? w + r.off + k.off : nullptr;
  }
};
// ---- image-shaped results: rows are pixels, columns channels
struct PixelOut {
  float* out;
  const float* bias;
  float alpha, beta;
  int along_m, vec;
  long long image, chan, pix;  // element strides
  int pixels, per_group;       // pixels per image, columns per group
  __device__ long long row(int m, int) const {
    const int img = m / pixels;
    return img * image + (m - img * pixels) * pix;
  }
  __device__ long long col(int n, int z) const { return (long long)(z * per_group + n) * chan; }
  __device__ int bias_at(int n, int z) const { return z * per_group + n; }
};
PixelOut pixel_out(float* out, const float* bias, const ConvGeo& g, bool dgrad) {
  PixelOut o{out, bias, 1.f, 0.f, 0, 0, 0, 0, 0, 0, 0};
  o.image = dgrad ? (long long)g.C * g.HW : (long long)g.Cout * g.HoWo;
  o.chan = dgrad ? g.x_cs : g.y_cs;
  o.pix = dgrad ? g.x_ps : g.y_ps;
  o.pixels = dgrad ? g.HW : g.HoWo;
  o.per_group = dgrad ? g.Cg : g.Coutg;
  o.along_m = o.pix == 1;
  o.vec = (o.along_m ? o.pixels % 4 == 0 && o.chan % 4 == 0
                     : o.chan == 1 && o.per_group % 4 == 0 && o.pix % 4 == 0) && aligned16(out);
  return o;
}

// ---- backward filter: K = pixels of the output
// x around output pixel k, 16-byte runs of channels, n = (tap, channel)
struct WindowVec {
  static constexpr int kKind = kVecRow;
  const float* x;
  ConvGeo g;
  int n_total;
  struct Row { int off, dh, dw; };
  struct Iter { long long img; int y, q; };
  __device__ const float* base() const { return x; }
  __device__ Row row(int n, int z) const {
    if (n >= n_total) return Row{-1, 0, 0};
    const int tap = n / g.Cg, c = n - tap * g.Cg, r = tap / g.kW, s = tap - r * g.kW;
    return Row{z * g.Cg + c, r * g.dy - g.py, s * g.dx - g.px};
  }
  __device__ Iter iter(int k, int) const {
    const int img = k / g.HoWo, pq = k - img * g.HoWo, y = pq / g.Wo;
    return Iter{(long long)img * g.C * g.HW, y, pq - y * g.Wo};
  }
  __device__ void advance(Iter& it) const {
    it.q += kBKf;
    while (it.q >= g.Wo) {
      it.q -= g.Wo;
      if (++it.y == g.Ho) { it.y = 0; it.img += (long long)g.C * g.HW; }
    }
  }
  __device__ const float* at(const Row& r, const Iter& it) const {
    const int h = it.y * g.sy + r.dh, w = it.q * g.sx + r.dw;
    if (r.off < 0 || h < 0 || h >= g.H || w < 0 || w >= g.W) return nullptr;
    return x + it.img + (long long)(h * g.W + w) * g.C + r.off;
  }
};
// element by element, n = (channel, tap); offsets split as in ImageElem
struct WindowElem {
  static constexpr int kKind = kElemK;
  const float* x;
  ConvGeo g;
  int n_total;
  struct Row { long long off; int dh, dw; };
  struct Kk { long long off; int h0, w0; };
  __device__ const float* base() const { return x; }
  __device__ Row row(int n, int z) const {
    if (n >= n_total) return Row{0, kNowhere, kNowhere};
    const int c = n / g.RS, rs = n - c * g.RS, r = rs / g.kW, s = rs - r * g.kW;
    const int dh = r * g.dy - g.py, dw = s * g.dx - g.px;
    return Row{((long long)z * g.Cg + c) * g.x_cs + ((long long)dh * g.W + dw) * g.x_ps, dh, dw};
  }
  __device__ Kk kk(int k, int) const {
    const int img = k / g.HoWo, pq = k - img * g.HoWo, y = pq / g.Wo, q = pq - y * g.Wo;
    const int h0 = y * g.sy, w0 = q * g.sx;
    return Kk{(long long)img * g.C * g.HW + ((long long)h0 * g.W + w0) * g.x_ps, h0, w0};
  }
  __device__ const float* at(const Row& r, const Kk& k) const {
    const int h = k.h0 + r.dh, w = k.w0 + r.dw;
    const bool inside = (unsigned)h < (unsigned)g.H && (unsigned)w < (unsigned)g.W;
    return inside ? x + k.off + r.off : nullptr;
  }
};
// dy element by element, lanes along the pixels
struct GradElem {
  static constexpr int kKind = kElemK;
  const float* gy;
  ConvGeo g;
  struct Row { long long off; };
  struct Kk { long long off; };
  __device__ const float* base() const { return gy; }
  __device__ Row row(int m, int z) const {
    return Row{m < g.Coutg ? ((long long)z * g.Coutg + m) * g.y_cs : -1};
  }
  __device__ Kk kk(int k, int) const {
    const int img = k / g.HoWo;
    return Kk{(long long)img * g.Cout * g.HoWo + (long long)(k - img * g.HoWo) * g.y_ps};
  }
  __device__ const float* at(const Row& r, const Kk& k) const {
    return r.off >= 0 ? gy + r.off + k.off : nullptr;
  }
};
struct FilterOut {
  float* out;
  const float* bias;
  float alpha, beta;
  int along_m, vec;
  ConvGeo g;
  int tap_major;
  __device__ long long row(int m, int z) const {
    return ((long long)z * g.Coutg + m) * ((long long)g.Cg * g.RS);
  }
  __device__ long long col(int n, int) const {
    return tap_major ? (long long)(n % g.Cg) * g.RS + n / g.Cg : n;
  }
  __device__ int bias_at(int n, int) const { return n; }
};

// ---- the three passes on the fp32 kernel
inline size_t up256c(size_t v) { return (v + 255) / 256 * 256; }

// Products of some size first bring their operands into the order that the 16-byte loaders read:
// the filter with its rows contiguous, an image in fl's order as a channels-last copy.  Below this
// many multiply-adds a copy and its launch cost more than the element-wise loads they replace.
constexpr double kStrictCopyWork = 3.2e7;
struct StrictScratch { size_t filter, x, gy; };
StrictScratch strict_scratch(const ConvGeo& g, int which) {
  StrictScratch s{0, 0, 0};
  if ((double)g.N * (which == 1 ? g.HW : g.HoWo) * g.Cout * g.Cg * g.RS < kStrictCopyWork) return s;
  const size_t x = up256c((size_t)g.N * g.C * g.HW * 4), gy = up256c((size_t)g.N * g.Cout * g.HoWo * 4);
  const bool images = g.N <= 65535;  // the copying kernels put them in the grid's third extent
  const bool x_copy = !g.x_cl && g.Cg % 4 == 0 && g.C >= 8 && images;
  const bool gy_copy = !g.y_cl && g.Coutg % 4 == 0 && g.Cout >= 8 && images;
  if (which != 2 && g.RS <= kPermuteMaxTaps) s.filter = up256c((size_t)g.Cout * g.Cg * g.RS * 4);
  if (which == 0 && x_copy) s.x = x;
  if (which == 1 && gy_copy) s.gy = gy;
  if (which == 2 && (g.x_cl || x_copy) && (g.y_cl || gy_copy)) {
    if (!g.x_cl) s.x = x;
    if (!g.y_cl) s.gy = gy;
  }
  return s;
}
size_t strict_scratch_bytes(const ConvGeo& g, int which) {
  const StrictScratch s = strict_scratch(g, which);
  return s.filter + s.x + s.gy;
}

// forward (DGRAD = false) and backward-data: an image against the filter
template <bool DGRAD>
int strict_image_pass(const char* name, const ConvGeo& g0, const float* src, const float* w,
                      const float* bias, float* dst, void* ws, size_t ws_bytes, cudaStream_t st) {
  ConvGeo g = g0;
  const long long M = (long long)g.N * (DGRAD ? g.HW : g.HoWo);
  FLB200_REQUIRE(M < 0x7fffffffLL, "%s: too many pixels", name);
  const int ch = DGRAD ? g.Coutg : g.Cg, N = DGRAD ? g.Cg : g.Coutg;
  const long long K = (long long)ch * g.RS;
  FLB200_REQUIRE(K < 0x7fffff00LL, "%s: filter too large", name);
  const PixelOut ep = pixel_out(dst, bias, g, DGRAD);
  const StrictScratch need = strict_scratch(g, DGRAD ? 1 : 0);
  const bool scratch = ws && aligned16(ws) && ws_bytes >= need.filter + need.x + need.gy;
  char* at = static_cast<char*>(ws);
  if (scratch && need.x + need.gy) {
    float* copy = reinterpret_cast<float*>(at);
    const int C = DGRAD ? g.Cout : g.C, pixels = DGRAD ? g.HoWo : g.HW;
    if (int rc = to_channels_last(src, copy, g.N, C, pixels, st)) return rc;
    at += need.x + need.gy;
    src = copy;
    if (DGRAD) { g.y_cl = 1; g.y_cs = 1; g.y_ps = g.Cout; }
    else { g.x_cl = 1; g.x_cs = 1; g.x_ps = g.C; }
  }
  const bool vec = (DGRAD ? g.y_cl : g.x_cl) && ch % 4 == 0 && aligned16(src);
  const FilterElem f{w, g, DGRAD ? 1 : 0, vec ? 1 : 0, N};
  const float* packed = nullptr;
  if (scratch && need.filter && N % 4 == 0) {
    // out[z][k][row], k = (tap, channel) for channel runs, else (channel, tap)
    float* out = reinterpret_cast<float*>(at);
    const long long s_tap = (long long)N * (vec ? ch : 1), s_ch = (long long)N * (vec ? 1 : g.RS);
    if (int rc = filter_permute(w, out, g.Coutg, g.Cg, g.RS, s_tap, DGRAD ? s_ch : 1, DGRAD ? 1 : s_ch, st,
                                g.groups))
      return rc;
    packed = out;
    at += need.filter;
  }
  ws_bytes -= at - static_cast<char*>(ws);
  const StridedLoader<kVecRow> fv{packed, 1, N, (long long)N * K, N};
  if (vec) {
    const ImageVec<DGRAD> iv{src, g, (int)M, ch / 4};
    if (packed) return launch_simt_gemm(name, iv, fv, ep, M, N, K, g.groups, at, ws_bytes, st);
    return launch_simt_gemm(name, iv, f, ep, M, N, K, g.groups, at, ws_bytes, st);
  }
  const ImageElem<DGRAD> ie{src, g, (int)M};
  if (packed) return launch_simt_gemm(name, ie, fv, ep, M, N, K, g.groups, at, ws_bytes, st);
  return launch_simt_gemm(name, ie, f, ep, M, N, K, g.groups, at, ws_bytes, st);
}

// (beta: what of gw's own values stays)
int strict_filter_pass(const char* name, const ConvGeo& g0, const float* gy, const float* x, float* gw,
                       void* ws, size_t ws_bytes, cudaStream_t st, float beta = 0.f) {
  ConvGeo g = g0;
  const long long N = (long long)g.Cg * g.RS, K = (long long)g.N * g.HoWo;
  FLB200_REQUIRE(N < 0x7fffffffLL, "%s: extent out of range", name);
  constexpr long long kMostK = 1LL << 30;  // the kernel counts k in 32 bits: more pixels in pieces
  if (K > kMostK && g.N > 1) {
    const int most = (int)std::max(1LL, kMostK / g.HoWo);
    for (int n = 0; n < g0.N; n += most) {
      g.N = std::min(most, g0.N - n);
      if (int rc = strict_filter_pass(name, g, gy + (long long)n * g.Cout * g.HoWo, x + (long long)n * g.C * g.HW,
                                      gw, ws, ws_bytes, st, n ? 1.f : 0.f))
        return rc;
    }
    return FLB200_OK;
  }
  FLB200_REQUIRE(K < 0x7fffff00LL, "%s: extent out of range", name);
  const StrictScratch need = strict_scratch(g, 2);
  char* at = static_cast<char*>(ws);
  if (ws && aligned16(ws) && ws_bytes >= need.x + need.gy) {
    if (need.x) {
      if (int rc = to_channels_last(x, reinterpret_cast<float*>(at), g.N, g.C, g.HW, st)) return rc;
      x = reinterpret_cast<const float*>(at);
      at += need.x;
      g.x_cl = 1; g.x_cs = 1; g.x_ps = g.C;
    }
    if (need.gy) {
      if (int rc = to_channels_last(gy, reinterpret_cast<float*>(at), g.N, g.Cout, g.HoWo, st)) return rc;
      gy = reinterpret_cast<const float*>(at);
      at += need.gy;
      g.y_cl = 1; g.y_cs = 1; g.y_ps = g.Cout;
    }
    ws_bytes -= need.x + need.gy;
  }
  FilterOut ep{gw, nullptr, 1.f, beta, 0, 0, g, 0};
  if (g.x_cl && g.y_cl && g.Cg % 4 == 0 && g.Coutg % 4 == 0 && aligned16(x) && aligned16(gy)) {
    const StridedLoader<kVecRow> gl{gy, 1, g.Cout, g.Coutg, g.Coutg};
    ep.tap_major = 1;
    ep.vec = g.RS == 1 && aligned16(gw);
    return launch_simt_gemm(name, gl, WindowVec{x, g, (int)N}, ep, g.Coutg, N, K, g.groups, at, ws_bytes,
                            st);
  }
  ep.vec = N % 4 == 0 && aligned16(gw);
  return launch_simt_gemm(name, GradElem{gy, g}, WindowElem{x, g, (int)N}, ep, g.Coutg, N, K, g.groups, at,
                          ws_bytes, st);
}

inline size_t max_sz(size_t a, size_t b) { return a > b ? a : b; }

// The tensor-core routes hand the tensors to TMA (16-byte aligned base addresses) and carve
// 256-byte-aligned sub-buffers out of the workspace that the kernels access with 16-byte
// vectors: an offset view or an odd workspace must not reach them (a misaligned vector access
// is a sticky device fault).  Such calls run on the fp32 kernels, which take any alignment.
inline bool tc_operands_aligned(const void* a, const void* b, const void* c, const void* d,
                                const void* ws) {
  return aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && aligned16(ws);
}


// ---- 16-bit tensors ---------------------------------------------------------------------------
// Casts between fp32 and 16-bit tensors, and f16 / bf16 convolutions (the reference accepts f16,
// backend/cudnn/Conv2D.cpp:231,266,321) that the tensor cores do not read as they are: widen the
// operands into fp32 copies at the front of the workspace, run the fp32 operator in the call's math
// mode (TF32 tensor cores keep 10 mantissa bits, as many as f16 has and more than bf16), round the
// result once to the 16-bit type.  Accumulation is fp32 throughout.
// Eight elements of 16-byte aligned tensors, or what is left of them, one by one elsewhere.
template <typename T>
__device__ __forceinline__ void widen8(const T* in, float* out) {
  float v[8];
  unpack16(load16(in), v);
#pragma unroll
  for (int j = 0; j < 8; j += 4)
    *reinterpret_cast<float4*>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
}
// Both kernels are bound by memory, on a weight matrix by their launch: 16-byte accesses, two groups
// of a thread in flight.  (51 bf16 copies of 134 M weights: 387 us with 4-byte loads, 348 so; 131 M
// scores to fp32: 165 and 152.)
template <typename T>
__global__ void widen_kernel(const T* __restrict__ in, float* __restrict__ out, long long n) {
  chain_begin();
  const long long stride = (long long)gridDim.x * blockDim.x * 8;
  long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
    for (; i + stride + 8 <= n; i += 2 * stride) {
      widen8(in + i, out + i);
      widen8(in + i + stride, out + i + stride);
    }
    for (; i + 8 <= n; i += stride) widen8(in + i, out + i);
  }
  for (; i < n; i += stride)
    for (long long j = i; j < n && j < i + 8; ++j) out[j] = Num<T>::to_f(in[j]);
}
template <typename T>
__global__ void narrow_kernel(const float* __restrict__ in, T* __restrict__ out, long long n) {
  chain_begin();
  const long long stride = (long long)gridDim.x * blockDim.x * 8;
  long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
    const auto group = [&](const float4& lo, const float4& hi) {
      const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      return pack16<T>(v);
    };
    const auto at = [&](long long k) { return *reinterpret_cast<const float4*>(in + k); };
    for (; i + stride + 8 <= n; i += 2 * stride) {
      const float4 a = at(i), b = at(i + 4), c = at(i + stride), d = at(i + stride + 4);
      store16(out + i, group(a, b));
      store16(out + i + stride, group(c, d));
    }
    for (; i + 8 <= n; i += stride) store16(out + i, group(at(i), at(i + 4)));
  }
  for (; i < n; i += stride)
    for (long long j = i; j < n && j < i + 8; ++j) out[j] = Num<T>::from_f(in[j]);
}
int widen(const void* in, float* out, long long n, int dtype, cudaStream_t st) {
  if (n == 0 || !in) return FLB200_OK;
  const unsigned grid = (unsigned)std::min<long long>(n / 8 / 256 + 1, 16LL * device_info().sm_count);
  if (dtype == FLB200_F16)
    launch_chained(widen_kernel<__half>, grid, 256, 0, st, static_cast<const __half*>(in), out, n);
  else
    launch_chained(widen_kernel<__nv_bfloat16>, grid, 256, 0, st, static_cast<const __nv_bfloat16*>(in), out,
                   n);
  FLB200_AFTER_LAUNCH("conv_widen");
  return FLB200_OK;
}
int narrow(const float* in, void* out, long long n, int dtype, cudaStream_t st) {
  if (n == 0 || !out) return FLB200_OK;
  const unsigned grid = (unsigned)std::min<long long>(n / 8 / 256 + 1, 16LL * device_info().sm_count);
  if (dtype == FLB200_F16)
    launch_chained(narrow_kernel<__half>, grid, 256, 0, st, in, static_cast<__half*>(out), n);
  else
    launch_chained(narrow_kernel<__nv_bfloat16>, grid, 256, 0, st, in, static_cast<__nv_bfloat16*>(out), n);
  FLB200_AFTER_LAUNCH("conv_narrow");
  return FLB200_OK;
}
// Channels-last 16-bit convolutions of a multiple of 8 channels need none of this in the tensor-core
// modes: their operands go to the tensor cores as they are (products of 16-bit values are exact
// in either case, the sums are fp32 in tensor memory, the result is rounded once).  The copies of a
// residual block of 64 x 56 x 56 x 256 f16 alone took 0.84 of its 2.8 ms.
bool native16(const flb200_conv2d_desc* d, ConvGeo* g, int which) {
  if (d->dtype == FLB200_F32 || d->math_mode == FLB200_MATH_STRICT_F32) return false;
  g->operand = tc::operand_of(d->dtype);
  if (tc_conv_native16(*g, which)) return true;
  g->operand = tc::kOperandTf32;
  return false;
}

// byte offsets of the fp32 copies pass `which` needs, in the order of its tensors:
// 0: x, w, bias, y | 1: grad_y, w, grad_x | 2: grad_y, x, grad_w, grad_bias
struct WideCopies {
  long long n[4];
  size_t off[4], total;
};
WideCopies wide_copies(const ConvGeo& g, int which) {
  const long long x = (long long)g.N * g.C * g.HW, w = (long long)g.Cout * g.Cg * g.RS,
                  y = (long long)g.N * g.Cout * g.HoWo, b = g.Cout;
  const long long n[3][4] = {{x, w, b, y}, {y, w, x, 0}, {y, x, w, b}};
  WideCopies c{};
  size_t off = 0;
  for (int i = 0; i < 4; ++i) {
    c.n[i] = n[which][i];
    c.off[i] = off;
    off += up256c((size_t)c.n[i] * 4);
  }
  c.total = off;
  return c;
}

}  // namespace
}  // namespace flb200

using namespace flb200;

extern "C" {

int flb200_conv2d_output_dims(const flb200_conv2d_desc* d, int32_t* Wo, int32_t* Ho) {
  ConvGeo g;
  if (int st = make_conv_geo("conv2d_output_dims", d, &g)) return st;
  if (Wo) *Wo = g.Wo;
  if (Ho) *Ho = g.Ho;
  return FLB200_OK;
}

// Key of the three queries below.  (A call with a descriptor that they refuse is not kept: it sets the
// error text again.)
struct ConvQuery { flb200_conv2d_desc d; int which, sm, cc, outer_x3; };
static ConvQuery conv_query(const flb200_conv2d_desc* d, int which) {
  ConvQuery q;
  memset(&q, 0, sizeof(q));
  q.d = *d;
  const DeviceInfo& di = device_info();
  q.which = which; q.sm = di.sm_count; q.cc = di.cc_major; q.outer_x3 = tc::x3_enabled() ? 1 : 0;
  return q;
}

static size_t conv2d_workspace_bytes(const flb200_conv2d_desc* d, int which, ConvGeo g) {
  size_t need = 0;
  if (which == 0) {
    need = strict_scratch_bytes(g, 0) +
           plan_simt((long long)g.N * g.HoWo, g.Coutg, (long long)g.Cg * g.RS, g.groups).workspace_bytes;
  } else if (which == 1) {
    need = strict_scratch_bytes(g, 1) +
           plan_simt((long long)g.N * g.HW, g.Cg, (long long)g.Coutg * g.RS, g.groups).workspace_bytes;
  } else {
    need = strict_scratch_bytes(g, 2) +
           plan_simt(g.Coutg, (long long)g.Cg * g.RS, (long long)g.N * g.HoWo, g.groups).workspace_bytes;
    need = max_sz(need, g.y_cl ? flb200_channel_sum_workspace_bytes((int64_t)g.N * g.HoWo, g.Cout, 1)
                               : flb200_channel_sum_workspace_bytes(g.N, g.Cout, g.HoWo));
  }
  if (native16(d, &g, which))  // + the fp32 bias or its gradient
    return up256c(max_sz(need, tc_conv_workspace_bytes(g, which))) + up256c((size_t)g.Cout * 4) +
           wide_copies(g, which).total;
  tc::X3Scope x3(d->math_mode == FLB200_MATH_F32X3);  // plans differ by mode
  if (d->math_mode != FLB200_MATH_STRICT_F32) need = max_sz(need, tc_conv_workspace_bytes(g, which));
  if (d->dtype != FLB200_F32 && which >= 0 && which <= 2)
    need = up256c(need) + wide_copies(g, which).total;  // fp32 copies of the 16-bit tensors
  return need;
}

size_t flb200_conv2d_workspace_bytes(const flb200_conv2d_desc* d, int which) {
  static thread_local Memo<ConvQuery, size_t> memo;
  ConvQuery q;
  if (d) {
    q = conv_query(d, which);
    if (const size_t* known = memo.find(q)) return *known;
  }
  ConvGeo g;
  if (make_conv_geo("conv2d_workspace_bytes", d, &g)) return 0;
  return memo.put(q, conv2d_workspace_bytes(d, which, g));
}

int flb200_conv2d_forward(const flb200_conv2d_desc* d, const void* x, const void* w,
                          const void* bias, void* y, void* workspace, size_t workspace_bytes,
                          void* stream) {
  return flb200_conv2d_forward_cached(d, x, w, bias, y, workspace, workspace_bytes, nullptr,
                                      stream);
}

size_t flb200_conv2d_cache_bytes(const flb200_conv2d_desc* d, int which) {
  static thread_local Memo<ConvQuery, size_t> memo;
  ConvQuery q;
  if (d) {
    q = conv_query(d, which);
    if (const size_t* known = memo.find(q)) return *known;
  }
  ConvGeo g;
  if (make_conv_geo("conv2d_cache_bytes", d, &g)) return 0;
  if (d->math_mode == FLB200_MATH_STRICT_F32 || which < 0 || which > 1) return 0;
  return memo.put(q, tc_conv_cache_bytes(g, which));
}

int flb200_conv2d_forward_cached(const flb200_conv2d_desc* d, const void* x, const void* w,
                                 const void* bias, void* y, void* workspace,
                                 size_t workspace_bytes, flb200_conv2d_cache* cache,
                                 void* stream) {
  ConvGeo g;
  if (int st = make_conv_geo("conv2d_forward", d, &g)) return st;
  FLB200_REQUIRE(x && w && y, "conv2d_forward: null tensor");
  cudaStream_t st = as_stream(stream);
  if (native16(d, &g, 0)) {
    const size_t bias_bytes = bias ? up256c((size_t)g.Cout * 4) : 0;
    if (tc_operands_aligned(x, w, y, nullptr, workspace) && workspace_bytes >= bias_bytes &&
        tc_conv_supported(g, 0, workspace_bytes - bias_bytes)) {
      float* b32 = bias ? static_cast<float*>(workspace) : nullptr;
      if (int rc = widen(bias, b32, g.Cout, d->dtype, st)) return rc;
      return tc_conv_forward(g, static_cast<const float*>(x), static_cast<const float*>(w), b32,
                             static_cast<float*>(y), static_cast<char*>(workspace) + bias_bytes,
                             workspace_bytes - bias_bytes, st, nullptr);
    }
    g.operand = tc::kOperandTf32;
  }
  if (d->dtype != FLB200_F32) {
    const WideCopies c = wide_copies(g, 0);
    if (!workspace || workspace_bytes < c.total)
      return fail(FLB200_WORKSPACE_TOO_SMALL, "conv2d_forward: workspace %zu < %zu",
                  workspace_bytes, c.total);
    char* ws = static_cast<char*>(workspace);
    float* x32 = reinterpret_cast<float*>(ws + c.off[0]);
    float* w32 = reinterpret_cast<float*>(ws + c.off[1]);
    float* b32 = bias ? reinterpret_cast<float*>(ws + c.off[2]) : nullptr;
    float* y32 = reinterpret_cast<float*>(ws + c.off[3]);
    if (int rc = widen(x, x32, c.n[0], d->dtype, st)) return rc;
    if (int rc = widen(w, w32, c.n[1], d->dtype, st)) return rc;
    if (int rc = widen(bias, b32, c.n[2], d->dtype, st)) return rc;
    flb200_conv2d_desc d32 = *d;
    d32.dtype = FLB200_F32;
    if (int rc = flb200_conv2d_forward_cached(&d32, x32, w32, b32, y32, ws + c.total,
                                              workspace_bytes - c.total, nullptr, stream))
      return rc;
    return narrow(y32, y, c.n[3], d->dtype, st);
  }
  const float* xf = static_cast<const float*>(x);
  const float* wf = static_cast<const float*>(w);
  const float* bf = static_cast<const float*>(bias);
  float* yf = static_cast<float*>(y);
  tc::X3Scope x3(d->math_mode == FLB200_MATH_F32X3);
  if (d->math_mode != FLB200_MATH_STRICT_F32 && tc_operands_aligned(x, w, y, bias, workspace) &&
      tc_conv_supported(g, 0, workspace_bytes))
    return tc_conv_forward(g, xf, wf, bf, yf, workspace, workspace_bytes, st, cache);
  return strict_image_pass<false>("conv2d_forward", g, xf, wf, bf, yf, workspace, workspace_bytes, st);
}

static long long conv2d_stats_groups(const flb200_conv2d_desc* d, ConvGeo g) {
  if (d->math_mode == FLB200_MATH_STRICT_F32 || (d->dtype != FLB200_F32 && !native16(d, &g, 0))) return 0;
  tc::X3Scope x3(g.operand == tc::kOperandTf32 && d->math_mode == FLB200_MATH_F32X3);
  const long long n = tc_conv_stats_groups(g);
  return n == 0 || !tc_conv_supported(g, 0, tc_conv_workspace_bytes(g, 0)) ? 0 : n;
}
size_t flb200_conv2d_stats_bytes(const flb200_conv2d_desc* d, int64_t* groups) {
  static thread_local Memo<ConvQuery, long long> memo;
  if (groups) *groups = 0;
  ConvQuery q;
  const long long* n = nullptr;
  if (d) {
    q = conv_query(d, 0);
    n = memo.find(q);
  }
  if (!n) {
    ConvGeo g;
    if (make_conv_geo("conv2d_stats_bytes", d, &g)) return 0;
    n = &memo.put(q, conv2d_stats_groups(d, g));
  }
  if (*n == 0) return 0;
  if (groups) *groups = *n;
  // CTA pairs may write one phantom tile (four all-zero rows) past the last real one
  return (size_t)(*n + 4) * 2 * d->Cout * sizeof(float);
}

int flb200_conv2d_forward_stats(const flb200_conv2d_desc* d, const void* x, const void* w,
                                const void* bias, void* y, float* stats, size_t stats_bytes,
                                void* workspace, size_t workspace_bytes,
                                flb200_conv2d_cache* cache, void* stream) {
  ConvGeo g;
  if (int st = make_conv_geo("conv2d_forward_stats", d, &g)) return st;
  FLB200_REQUIRE(x && w && y && stats, "conv2d_forward_stats: null tensor");
  const size_t need = flb200_conv2d_stats_bytes(d, nullptr);
  const bool half = native16(d, &g, 0);
  const size_t bias_bytes = half && bias ? up256c((size_t)g.Cout * 4) : 0;
  if (need == 0 || workspace_bytes < bias_bytes || !tc_operands_aligned(x, w, y, bias, workspace) || !aligned16(stats) ||
      !tc_conv_supported(g, 0, workspace_bytes - bias_bytes))
    return fail(FLB200_UNSUPPORTED,
                "conv2d_forward_stats: needs a tensor-core route with a channels-last output "
                "of a multiple of 32 channels, 16-byte aligned tensors and the forward workspace");
  if (stats_bytes < need)
    return fail(FLB200_WORKSPACE_TOO_SMALL, "conv2d_forward_stats: statistics buffer %zu < %zu",
                stats_bytes, need);
  ConvStats cs{stats};
  tc::X3Scope x3(!half && d->math_mode == FLB200_MATH_F32X3);
  const float* b32 = static_cast<const float*>(bias);
  if (bias_bytes) {
    if (int rc = widen(bias, static_cast<float*>(workspace), g.Cout, d->dtype, as_stream(stream))) return rc;
    b32 = static_cast<const float*>(workspace);
  }
  return tc_conv_forward(g, static_cast<const float*>(x), static_cast<const float*>(w), b32,
                         static_cast<float*>(y), workspace ? static_cast<char*>(workspace) + bias_bytes : nullptr,
                         workspace_bytes - bias_bytes, as_stream(stream), cache, &cs);
}

int flb200_conv2d_backward_data(const flb200_conv2d_desc* d, const void* grad_y, const void* w,
                                void* grad_x, void* workspace, size_t workspace_bytes,
                                void* stream) {
  return flb200_conv2d_backward_data_cached(d, grad_y, w, grad_x, workspace, workspace_bytes,
                                            nullptr, stream);
}

int flb200_conv2d_backward_data_cached(const flb200_conv2d_desc* d, const void* grad_y,
                                       const void* w, void* grad_x, void* workspace,
                                       size_t workspace_bytes, flb200_conv2d_cache* cache,
                                       void* stream) {
  ConvGeo g;
  if (int st = make_conv_geo("conv2d_backward_data", d, &g)) return st;
  FLB200_REQUIRE(grad_y && w && grad_x, "conv2d_backward_data: null tensor");
  cudaStream_t st = as_stream(stream);
  if (native16(d, &g, 1)) {
    if (tc_operands_aligned(grad_y, w, grad_x, nullptr, workspace) &&
        tc_conv_supported(g, 1, workspace_bytes))
      return tc_conv_backward_data(g, static_cast<const float*>(grad_y), static_cast<const float*>(w),
                                   static_cast<float*>(grad_x), workspace, workspace_bytes, st, nullptr);
    g.operand = tc::kOperandTf32;
  }
  if (d->dtype != FLB200_F32) {
    const WideCopies c = wide_copies(g, 1);
    if (!workspace || workspace_bytes < c.total)
      return fail(FLB200_WORKSPACE_TOO_SMALL, "conv2d_backward_data: workspace %zu < %zu",
                  workspace_bytes, c.total);
    char* ws = static_cast<char*>(workspace);
    float* gy32 = reinterpret_cast<float*>(ws + c.off[0]);
    float* w32 = reinterpret_cast<float*>(ws + c.off[1]);
    float* gx32 = reinterpret_cast<float*>(ws + c.off[2]);
    if (int rc = widen(grad_y, gy32, c.n[0], d->dtype, st)) return rc;
    if (int rc = widen(w, w32, c.n[1], d->dtype, st)) return rc;
    flb200_conv2d_desc d32 = *d;
    d32.dtype = FLB200_F32;
    if (int rc = flb200_conv2d_backward_data_cached(&d32, gy32, w32, gx32, ws + c.total,
                                                    workspace_bytes - c.total, nullptr, stream))
      return rc;
    return narrow(gx32, grad_x, c.n[2], d->dtype, st);
  }
  const float* gyf = static_cast<const float*>(grad_y);
  const float* wf = static_cast<const float*>(w);
  float* gxf = static_cast<float*>(grad_x);
  tc::X3Scope x3(d->math_mode == FLB200_MATH_F32X3);
  if (d->math_mode != FLB200_MATH_STRICT_F32 &&
      tc_operands_aligned(grad_y, w, grad_x, nullptr, workspace) &&
      tc_conv_supported(g, 1, workspace_bytes))
    return tc_conv_backward_data(g, gyf, wf, gxf, workspace, workspace_bytes, st, cache);
  return strict_image_pass<true>("conv2d_backward_data", g, gyf, wf, nullptr, gxf, workspace,
                                 workspace_bytes, st);
}

int flb200_conv2d_backward_filter_bias(const flb200_conv2d_desc* d, const void* grad_y,
                                       const void* x, void* grad_w, void* grad_bias,
                                       void* workspace, size_t workspace_bytes, void* stream) {
  return flb200_conv2d_backward_filter_bias_cached(d, grad_y, x, grad_w, grad_bias, workspace,
                                                   workspace_bytes, nullptr, stream);
}

int flb200_conv2d_backward_filter_bias_cached(const flb200_conv2d_desc* d, const void* grad_y,
                                              const void* x, void* grad_w, void* grad_bias,
                                              void* workspace, size_t workspace_bytes,
                                              flb200_conv2d_cache* cache, void* stream) {
  ConvGeo g;
  if (int st = make_conv_geo("conv2d_backward_filter_bias", d, &g)) return st;
  FLB200_REQUIRE(grad_y && x && grad_w, "conv2d_backward_filter_bias: null tensor");
  cudaStream_t st = as_stream(stream);
  if (native16(d, &g, 2)) {
    if (tc_operands_aligned(grad_y, x, grad_w, nullptr, workspace) &&
        tc_conv_supported(g, 2, workspace_bytes)) {
      if (int rc = tc_conv_backward_filter(g, static_cast<const float*>(grad_y),
                                           static_cast<const float*>(x), static_cast<float*>(grad_w),
                                           workspace, workspace_bytes, st, nullptr))
        return rc;
      if (!grad_bias) return FLB200_OK;
      float* gb32 = static_cast<float*>(workspace);
      const size_t gb_bytes = up256c((size_t)g.Cout * 4);
      if (int rc = flb200_channel_sum(grad_y, gb32, (int64_t)g.N * g.HoWo, g.Cout, 1, d->dtype,
                                      static_cast<char*>(workspace) + gb_bytes,
                                      workspace_bytes - gb_bytes, stream))
        return rc;
      return narrow(gb32, grad_bias, g.Cout, d->dtype, st);
    }
    g.operand = tc::kOperandTf32;
  }
  if (d->dtype != FLB200_F32) {
    const WideCopies c = wide_copies(g, 2);
    if (!workspace || workspace_bytes < c.total)
      return fail(FLB200_WORKSPACE_TOO_SMALL, "conv2d_backward_filter_bias: workspace %zu < %zu",
                  workspace_bytes, c.total);
    char* ws = static_cast<char*>(workspace);
    float* gy32 = reinterpret_cast<float*>(ws + c.off[0]);
    float* x32 = reinterpret_cast<float*>(ws + c.off[1]);
    float* gw32 = reinterpret_cast<float*>(ws + c.off[2]);
    float* gb32 = grad_bias ? reinterpret_cast<float*>(ws + c.off[3]) : nullptr;
    if (int rc = widen(grad_y, gy32, c.n[0], d->dtype, st)) return rc;
    if (int rc = widen(x, x32, c.n[1], d->dtype, st)) return rc;
    flb200_conv2d_desc d32 = *d;
    d32.dtype = FLB200_F32;
    if (int rc = flb200_conv2d_backward_filter_bias_cached(&d32, gy32, x32, gw32, gb32,
                                                           ws + c.total, workspace_bytes - c.total,
                                                           nullptr, stream))
      return rc;
    if (int rc = narrow(gw32, grad_w, c.n[2], d->dtype, st)) return rc;
    return narrow(gb32, grad_bias, c.n[3], d->dtype, st);
  }
  const float* gyf = static_cast<const float*>(grad_y);
  const float* xf = static_cast<const float*>(x);
  float* gwf = static_cast<float*>(grad_w);
  int rc;
  tc::X3Scope x3(d->math_mode == FLB200_MATH_F32X3);
  if (d->math_mode != FLB200_MATH_STRICT_F32 &&
      tc_operands_aligned(grad_y, x, grad_w, nullptr, workspace) &&
      tc_conv_supported(g, 2, workspace_bytes)) {
    rc = tc_conv_backward_filter(g, gyf, xf, gwf, workspace, workspace_bytes, st, cache);
  } else {
    rc = strict_filter_pass("conv2d_backward_filter", g, gyf, xf, gwf, workspace, workspace_bytes, st);
  }
  if (rc) return rc;
  if (grad_bias) {
    // db[co] = sum over batch and output pixels of dy — one pass over dy
    // (flashlight/fl/autograd/tensor/backend/cudnn/Conv2D.cpp:737).
    if (g.y_cl)  // [pixels][Cout]: column sums
      return flb200_channel_sum(grad_y, static_cast<float*>(grad_bias), (int64_t)g.N * g.HoWo,
                                g.Cout, 1, FLB200_F32, workspace, workspace_bytes, stream);
    return flb200_channel_sum(grad_y, static_cast<float*>(grad_bias), g.N, g.Cout, g.HoWo,
                              FLB200_F32, workspace, workspace_bytes, stream);
  }
  return FLB200_OK;
}


int flb200_astype(const void* in, int in_dtype, void* out, int out_dtype, int64_t n,
                  void* stream) {
  FLB200_REQUIRE(n >= 0, "astype: negative length");
  if (n == 0) return FLB200_OK;
  FLB200_REQUIRE(in && out, "astype: null tensor");
  cudaStream_t st = as_stream(stream);
  const bool in16 = in_dtype == FLB200_F16 || in_dtype == FLB200_BF16;
  const bool out16 = out_dtype == FLB200_F16 || out_dtype == FLB200_BF16;
  if (in_dtype == out_dtype) {
    const size_t es = in_dtype == FLB200_F32 ? 4 : 2;
    FLB200_REQUIRE(in_dtype == FLB200_F32 || in16, "astype: unknown dtype %d", in_dtype);
    FLB200_CUDA_CHECK(cudaMemcpyAsync(out, in, (size_t)n * es, cudaMemcpyDeviceToDevice, st));
    return FLB200_OK;
  }
  if (in_dtype == FLB200_F32 && out16) return narrow(static_cast<const float*>(in), out, n, out_dtype, st);
  if (in16 && out_dtype == FLB200_F32) return widen(in, static_cast<float*>(out), n, in_dtype, st);
  return fail(FLB200_UNSUPPORTED, "astype: %d -> %d is not built (f32 <-> f16 / bf16 only)",
              in_dtype, out_dtype);
}

}  // extern "C"
