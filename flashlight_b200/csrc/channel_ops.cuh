// Per-channel reductions and per-channel affine passes over a tensor viewed as
// [outer][channels][inner] (row-major).  This is the one access pattern behind
// batchnorm / LayerNorm forward and backward, the convolution bias gradient and
// sumAs / tile of a bias, so they share these templates.
//
// Work split: grid = (channels, splits).  A CTA owns one channel and a
// contiguous range of that channel's outer*inner elements, walks it with
// 128-bit accesses when inner is a multiple of the vector width, and leaves two
// partial sums per (channel, split) in a small scratch array that a one-thread-
// per-channel kernel finishes in double precision.  The channel is constant per
// CTA, so the per-channel constants live in registers.
#pragma once
#include <algorithm>

#include "common.cuh"

namespace flb200 {

constexpr int kChanThreads = 256;

struct ChannelGeo {
  long long outer, channels, inner;
  long long per_channel;  // outer * inner
  int splits;             // gridDim.y
  long long chunk;        // elements of one channel per split (multiple of 16)
};

// Picks the number of splits so that the grid fills the device a few times but
// a CTA still has at least 8K elements to amortise its reduction.
inline ChannelGeo make_channel_geo(long long outer, long long channels, long long inner) {
  ChannelGeo g;
  g.outer = outer;
  g.channels = channels;
  g.inner = inner;
  g.per_channel = outer * inner;
  const long long target_ctas = 4LL * 8 * device_info().sm_count;
  long long splits = (target_ctas + channels - 1) / channels;
  const long long max_by_work = (g.per_channel + 8191) / 8192;
  if (splits > max_by_work) splits = max_by_work;
  if (splits < 1) splits = 1;
  if (splits > 4096) splits = 4096;
  long long chunk = (g.per_channel + splits - 1) / splits;
  chunk = (chunk + 15) / 16 * 16;
  splits = (g.per_channel + chunk - 1) / chunk;
  if (splits < 1) splits = 1;
  g.splits = static_cast<int>(splits);
  g.chunk = chunk;
  return g;
}

// Address of element e (0 <= e < outer*inner) of channel c.
__device__ __forceinline__ long long channel_elem_offset(const ChannelGeo& g, long long c,
                                                         long long e) {
  // 32-bit division when it fits: it does for every shape of the five workloads.
  long long o, i;
  if (g.per_channel < 0x7fffffffLL) {
    const unsigned eo = static_cast<unsigned>(e) / static_cast<unsigned>(g.inner);
    o = eo;
    i = static_cast<unsigned>(e) - eo * static_cast<unsigned>(g.inner);
  } else {
    o = e / g.inner;
    i = e - o * g.inner;
  }
  return (o * g.channels + c) * g.inner + i;
}

// F: struct with
//   struct K {...};  __device__ K channel(long long c) const;
//   __device__ void accumulate(const K&, float a, float b, float& s0, float& s1) const;
// NIN = number of input tensors (1 or 2).  partial[(c*splits + s)] = (s0, s1).
template <typename T, int NIN, bool VEC, typename F>
__global__ void __launch_bounds__(kChanThreads)
channel_reduce_kernel(const T* __restrict__ a, const T* __restrict__ b,
                      float2* __restrict__ partial, ChannelGeo g, F f) {
  chain_begin();
  __shared__ float scratch[32];
  const long long c = blockIdx.x;
  const int s = blockIdx.y;
  const typename F::K k = f.channel(c);
  long long begin = (long long)s * g.chunk;
  long long end = begin + g.chunk;
  if (end > g.per_channel) end = g.per_channel;
  float s0 = 0.f, s1 = 0.f;
  if (VEC) {
    constexpr int V = Vec16<T>::N;
    // chunk is a multiple of 16 and inner a multiple of V, so vectors never straddle rows.
    for (long long e = begin + (long long)threadIdx.x * V; e < end;
         e += (long long)kChanThreads * V * 2) {
      const long long e2 = e + (long long)kChanThreads * V;
      const bool two = e2 < end;
      const long long off = channel_elem_offset(g, c, e);
      const long long off2 = two ? channel_elem_offset(g, c, e2) : off;
      Vec16<T> va = load16(a + off), vb, va2, vb2;
      if (NIN == 2) vb = load16(b + off);
      if (two) {
        va2 = load16(a + off2);
        if (NIN == 2) vb2 = load16(b + off2);
      }
#pragma unroll
      for (int j = 0; j < V; ++j)
        f.accumulate(k, Num<T>::to_f(va.v[j]), NIN == 2 ? Num<T>::to_f(vb.v[j]) : 0.f, s0, s1);
      if (two) {
#pragma unroll
        for (int j = 0; j < V; ++j)
          f.accumulate(k, Num<T>::to_f(va2.v[j]), NIN == 2 ? Num<T>::to_f(vb2.v[j]) : 0.f, s0,
                       s1);
      }
    }
  } else {
    for (long long e = begin + threadIdx.x; e < end; e += kChanThreads) {
      const long long off = channel_elem_offset(g, c, e);
      f.accumulate(k, Num<T>::to_f(a[off]), NIN == 2 ? Num<T>::to_f(b[off]) : 0.f, s0, s1);
    }
  }
  s0 = block_sum(s0, scratch);
  s1 = block_sum(s1, scratch);
  if (threadIdx.x == 0) partial[c * g.splits + s] = make_float2(s0, s1);
}

// F: struct with K / channel(c) as above and
//   __device__ float apply(const K&, float a, float b) const;
template <typename T, int NIN, bool VEC, typename F>
__global__ void __launch_bounds__(kChanThreads)
channel_apply_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ out,
                     ChannelGeo g, F f) {
  chain_begin();
  const long long c = blockIdx.x;
  const int s = blockIdx.y;
  const typename F::K k = f.channel(c);
  long long begin = (long long)s * g.chunk;
  long long end = begin + g.chunk;
  if (end > g.per_channel) end = g.per_channel;
  if (VEC) {
    constexpr int V = Vec16<T>::N;
    for (long long e = begin + (long long)threadIdx.x * V; e < end;
         e += (long long)kChanThreads * V * 2) {
      const long long e2 = e + (long long)kChanThreads * V;
      const bool two = e2 < end;
      const long long off = channel_elem_offset(g, c, e);
      const long long off2 = two ? channel_elem_offset(g, c, e2) : off;
      Vec16<T> va = load16(a + off), vb, va2, vb2, vo;
      if (NIN == 2) vb = load16(b + off);
      if (two) {
        va2 = load16(a + off2);
        if (NIN == 2) vb2 = load16(b + off2);
      }
#pragma unroll
      for (int j = 0; j < V; ++j)
        vo.v[j] = Num<T>::from_f(
            f.apply(k, Num<T>::to_f(va.v[j]), NIN == 2 ? Num<T>::to_f(vb.v[j]) : 0.f));
      store16(out + off, vo);
      if (two) {
#pragma unroll
        for (int j = 0; j < V; ++j)
          vo.v[j] = Num<T>::from_f(
              f.apply(k, Num<T>::to_f(va2.v[j]), NIN == 2 ? Num<T>::to_f(vb2.v[j]) : 0.f));
        store16(out + off2, vo);
      }
    }
  } else {
    for (long long e = begin + threadIdx.x; e < end; e += kChanThreads) {
      const long long off = channel_elem_offset(g, c, e);
      out[off] = Num<T>::from_f(
          f.apply(k, Num<T>::to_f(a[off]), NIN == 2 ? Num<T>::to_f(b[off]) : 0.f));
    }
  }
}

// inner == 1 ([rows][channels], channel fastest): a CTA of 32 x 8 threads owns
// 32 adjacent channels and a range of rows; lanes read 128 contiguous bytes.
template <typename T, int NIN, typename F>
__global__ void __launch_bounds__(256)
column_reduce_kernel(const T* __restrict__ a, const T* __restrict__ b,
                     float2* __restrict__ partial, long long rows, long long channels,
                     int splits, long long rows_per_split, F f) {
  chain_begin();
  __shared__ float sh0[8][33];
  __shared__ float sh1[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long c = (long long)blockIdx.x * 32 + tx;
  const int s = blockIdx.y;
  float s0 = 0.f, s1 = 0.f;
  if (c < channels) {
    const typename F::K k = f.channel(c);
    long long r0 = (long long)s * rows_per_split;
    long long r1 = r0 + rows_per_split;
    if (r1 > rows) r1 = rows;
    for (long long r = r0 + ty; r < r1; r += 8) {
      const long long off = r * channels + c;
      f.accumulate(k, Num<T>::to_f(a[off]), NIN == 2 ? Num<T>::to_f(b[off]) : 0.f, s0, s1);
    }
  }
  sh0[ty][tx] = s0;
  sh1[ty][tx] = s1;
  __syncthreads();
  if (ty == 0 && c < channels) {
#pragma unroll
    for (int j = 1; j < 8; ++j) {
      s0 += sh0[j][tx];
      s1 += sh1[j][tx];
    }
    partial[c * splits + s] = make_float2(s0, s1);
  }
}

// Element by element.  The threads walk in steps of a multiple of the channels, so that each stays on
// one channel and makes its constants once, the batch-norm scale in fp64 among them (64 x 30 x 112 x 112
// f16 in evaluation mode: 95 us with a scale per element, 61 with scales from a kernel before, 37 so).
// Only where the channels outnumber the threads does a thread change them.
template <typename T, int NIN, typename F>
__global__ void __launch_bounds__(256)
column_apply_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ out,
                    long long rows, long long channels, F f) {
  chain_begin();
  const long long total = rows * channels;
  const long long threads = (long long)gridDim.x * blockDim.x;
  const bool fixed = threads >= channels;
  const long long stride = fixed ? threads - threads % channels : threads;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= stride || t >= total) return;
  typename F::K k = f.channel(t % channels);
  while (true) {
    out[t] = Num<T>::from_f(f.apply(k, Num<T>::to_f(a[t]), NIN == 2 ? Num<T>::to_f(b[t]) : 0.f));
    t += stride;
    if (t >= total) return;
    if (!fixed) k = f.channel(t % channels);
  }
}

// ------------------------------------------------------------------------------------------
// inner == 1 with channels a multiple of the 16-byte vector (4 fp32, 8 16-bit values) and 16-byte
// aligned tensors (channels-last image tensors [pixels][channels], rows of features): the same
// column reduction and per-channel pass with 16-byte accesses.  A CTA of 256 threads is CQ column
// vectors (CQ a power of two <= 64) x 256 / CQ row lanes; a thread keeps the constants of its
// channels in registers and walks the rows of its split with several independent loads in flight.
// (Element by element, 16-bit tensors ran at a quarter to half of the bandwidth of fp32 ones: the
// three reductions for relu(batch-norm) gradients in a block of 64 x 56 x 56 x 256 f16 took 166 us,
// with vectors 76; its statistics passes 40 us each, now 23.)
struct ColumnTiling {
  int cq_shift;    // log2(CQ)
  int col_blocks;  // ceil(channels / (V * CQ))
};
inline ColumnTiling column_tiling(long long channels, int v = 4) {
  const long long vecs = (channels + v - 1) / v;
  int shift = 0;
  while ((2LL << shift) <= vecs && shift < 6) ++shift;
  ColumnTiling t;
  t.cq_shift = shift;
  t.col_blocks = (int)((vecs + (1LL << shift) - 1) >> shift);
  return t;
}

// NIN = 3: the second input is b + b2, rounded to T as the sum of two tensors is, and written to `sum` unless
// that is null (a gradient that reaches an operator from two consumers, added where it is read: on 256 x 56 x
// 56 x 256 f32 the addition, 369 us, and the reduction of two tensors, 255, become one pass of 380; of 64
// f16 images 49 and 34 become 68, where the registers bound the loads in flight).
template <typename T, int NIN, typename F>
__global__ void __launch_bounds__(256, 3)
column_reduce_vec_kernel(const T* __restrict__ a, const T* __restrict__ b,
                         float2* __restrict__ partial, long long rows, long long channels,
                         int splits, long long rows_per_split, int cq_shift, F f,
                         const T* __restrict__ b2, T* __restrict__ sum) {
  chain_begin();
  constexpr int V = Vec16<T>::N;
  __shared__ float sh0[256 * V];
  __shared__ float sh1[256 * V];
  const int cq = 1 << cq_shift, rl = 256 >> cq_shift;
  const int tq = threadIdx.x & (cq - 1), tr = threadIdx.x >> cq_shift;
  const long long c = ((long long)blockIdx.x * cq + tq) * V;
  const int s = blockIdx.y;
  float s0[V], s1[V];
#pragma unroll
  for (int j = 0; j < V; ++j) s0[j] = s1[j] = 0.f;
  if (c < channels) {
    typename F::K k[V];
#pragma unroll
    for (int j = 0; j < V; ++j) k[j] = f.channel(c + j);
    const long long r0 = (long long)s * rows_per_split;
    long long r1 = r0 + rows_per_split;
    if (r1 > rows) r1 = rows;
    long long r = r0 + tr;
    auto take = [&](const Vec16<T>& ra, const Vec16<T>& rb, float* t0, float* t1) {
      float va[V], vb[V];
      unpack16(ra, va);
      if (NIN >= 2) unpack16(rb, vb);
#pragma unroll
      for (int j = 0; j < V; ++j) f.accumulate(k[j], va[j], NIN >= 2 ? vb[j] : 0.f, t0[j], t1[j]);
    };
    auto add = [&](const Vec16<T>& rb, const Vec16<T>& rb2, long long off) {
      float x[V], y[V];
      unpack16(rb, x);
      unpack16(rb2, y);
#pragma unroll
      for (int j = 0; j < V; ++j) x[j] += y[j];
      const Vec16<T> s = pack16<T>(x);
      if (sum) store16(sum + off, s);
      return s;
    };
    // eight 16-byte loads in flight per thread: 8 rows of one tensor or 4 rows of two; six of 2 rows
    // of three, added up in the groups of the two
    constexpr int U = NIN == 1 ? 8 : (NIN == 2 ? 4 : 2), G = NIN == 3 ? 2 : 1;
    for (; r + (long long)(G * U - 1) * rl < r1; r += (long long)G * U * rl) {
      // the rows in flight are summed by themselves first: a long chain of positive fp32 terms is
      // biased (variance of 104000 bf16 rows, 117 to a thread: 1.4e-6 off, in groups of 8 4e-8)
      float g0[V], g1[V];
#pragma unroll
      for (int j = 0; j < V; ++j) g0[j] = g1[j] = 0.f;
#pragma unroll
      for (int h = 0; h < G; ++h) {
        Vec16<T> va[U], vb[U], vb2[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const long long off = (r + (long long)(h * U + u) * rl) * channels + c;
          va[u] = load16(a + off);
          if (NIN >= 2) vb[u] = load16(b + off);
          if (NIN == 3) vb2[u] = load16(b2 + off);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          take(va[u], NIN == 3 ? add(vb[u], vb2[u], (r + (long long)(h * U + u) * rl) * channels + c) : vb[u], g0, g1);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) {
        s0[j] += g0[j];
        s1[j] += g1[j];
      }
    }
    for (; r < r1; r += rl) {
      const long long off = r * channels + c;
      const Vec16<T> va = load16(a + off);
      Vec16<T> vb;
      if (NIN >= 2) vb = load16(b + off);
      take(va, NIN == 3 ? add(vb, load16(b2 + off), off) : vb, s0, s1);
    }
  }
  // sh[tr][tq * V + j]: 256 threads x V values
#pragma unroll
  for (int j = 0; j < V; ++j) {
    sh0[(tr * cq + tq) * V + j] = s0[j];
    sh1[(tr * cq + tq) * V + j] = s1[j];
  }
  __syncthreads();
  // the block's V * CQ columns, each finished by one thread
  for (int t = threadIdx.x; t < V * cq; t += 256) {
    const long long cc = (long long)blockIdx.x * cq * V + t;
    if (cc < channels) {
      float t0 = 0.f, t1 = 0.f;
      for (int i0 = 0; i0 < rl; i0 += 4) {  // (rl is 4 or a multiple of it; short chains as above)
        float g0 = 0.f, g1 = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          g0 += sh0[(i0 + i) * cq * V + t];
          g1 += sh1[(i0 + i) * cq * V + t];
        }
        t0 += g0;
        t1 += g1;
      }
      partial[cc * splits + s] = make_float2(t0, t1);
    }
  }
}

template <typename T, int NIN, typename F>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : NIN == 2 ? 2 : 3)
column_apply_vec_kernel(const T* __restrict__ a, const T* __restrict__ b,
                        T* __restrict__ out, long long rows, long long channels,
                        long long rows_per_split, int cq_shift, F f) {
  chain_begin();
  constexpr int V = Vec16<T>::N;
  const int cq = 1 << cq_shift, rl = 256 >> cq_shift;
  const int tq = threadIdx.x & (cq - 1), tr = threadIdx.x >> cq_shift;
  const long long c = ((long long)blockIdx.x * cq + tq) * V;
  if (c >= channels) return;
  typename F::K k[V];
#pragma unroll
  for (int j = 0; j < V; ++j) k[j] = f.channel(c + j);
  const long long r0 = (long long)blockIdx.y * rows_per_split;
  long long r1 = r0 + rows_per_split;
  if (r1 > rows) r1 = rows;
  long long r = r0 + tr;
  auto apply = [&](const Vec16<T>& ra, const Vec16<T>& rb) {
    float va[V], vb[V], o[V];
    unpack16(ra, va);
    if (NIN == 2) unpack16(rb, vb);
#pragma unroll
    for (int j = 0; j < V; ++j) o[j] = f.apply(k[j], va[j], NIN == 2 ? vb[j] : 0.f);
    return pack16<T>(o);
  };
  for (; r + 3LL * rl < r1; r += 4LL * rl) {
    Vec16<T> va[4], vb[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long off = (r + (long long)u * rl) * channels + c;
      va[u] = load16(a + off);
      if (NIN == 2) vb[u] = load16(b + off);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      store16(out + (r + (long long)u * rl) * channels + c, apply(va[u], vb[u]));
  }
  for (; r < r1; r += rl) {
    const long long off = r * channels + c;
    const Vec16<T> va = load16(a + off);
    Vec16<T> vb;
    if (NIN == 2) vb = load16(b + off);
    store16(out + off, apply(va, vb));
  }
}

// Splits of the column path (rows handled per CTA), at most 512.  The vector kernel: one wave of three
// CTAs per SM (its registers allow that many with 16-bit data) over its column blocks, at least 32 rows
// each; where that would round to a few splits, two waves of them.  The element kernel has fewer loads
// in flight per thread: two waves, at least 64 rows each (the gradient sums of 64 x 33 x 56 x 56 f32:
// 57 us with the vector kernel's splits, 43 so, and shorter chains of additions).
inline int column_splits(long long rows, long long channels, bool vec) {
  const long long sm = device_info().sm_count, col_blocks = column_tiling(channels).col_blocks;
  const long long two_waves = (6 * sm + col_blocks - 1) / col_blocks;
  long long splits = vec ? 3 * sm / col_blocks : two_waves;
  if (splits < 8) splits = two_waves;
  const long long least = vec ? 32 : 64, max_by_work = (rows + least - 1) / least;
  if (splits > max_by_work) splits = max_by_work;
  if (splits > 512) splits = 512;
  if (splits < 1) splits = 1;
  return static_cast<int>(splits);
}

// Rows of one CTA of a per-channel pass with `per_sm` CTAs per SM that walk `lanes` rows at once, a
// multiple of the four rows that a thread has in flight.  Every thread first loads the constants of
// its channels: with eight 16-bit channels per thread those cost as much as a few rows, so 16-bit
// passes are six CTAs per SM (two waves of three, or three of two; the three relu(batch-norm)
// gradient passes of a 64 x 56 x 56 x 256 f16 block took 155 us at 16 per SM, 97 so); fp32 ones keep
// 16, which measured 4 to 8 % faster than one wave.
inline long long apply_rows_per_split(long long rows, long long col_blocks, long long lanes,
                                      long long per_sm) {
  const long long ctas = per_sm * device_info().sm_count;
  const long long splits = std::max(1LL, std::min(65535LL, ctas / col_blocks));
  const long long unit = 4 * lanes;
  return ((rows + splits - 1) / splits + unit - 1) / unit * unit;
}

// Scratch bytes for the (channel, split) partial sums of any op built on these, whichever kernel
// the alignment of its tensors leads to.
inline size_t channel_partial_bytes(long long outer, long long channels, long long inner) {
  long long splits;
  if (inner == 1) {
    splits = std::max(column_splits(outer, channels, true), column_splits(outer, channels, false));
  } else {
    splits = make_channel_geo(outer, channels, inner).splits;
  }
  return static_cast<size_t>(channels) * static_cast<size_t>(splits) * sizeof(float2);
}

}  // namespace flb200
