// Repacking of convolution filters: w[co][ci][tap] to out[tap * s_tap + co * s_co + ci * s_ci],
// where one of s_co, s_ci is 1; the grid's z walks groups of Cout * C * RS words on both sides; `pad`
// (at most 3) zeros follow each contiguous run of the target.  A
// CTA brings 32 output channels x a short run of input channels x all taps into shared memory along
// the filter's own contiguous order and writes it out along the contiguous index of the target, so
// both sides move whole sectors; the runs are short (8 input channels) because most filters are
// small and a few CTAs would be bound by their own latency.  (A thread per target element read the
// filter kH * kW elements apart: 57 us for a 13-tap 1024 x 1024 filter, 54 MB; now 37.  With a
// launch per group, 256 groups of 4 x 4 channels took 1 ms.)
#pragma once
#include "common.cuh"

namespace flb200 {

constexpr int kPermuteCo = 32;
// The most taps of a filter whose tile fits in shared memory at one input channel per CTA (32 rows of
// up to 1816 words: 227 KB); longer filters are left as they are.
constexpr int kPermuteMaxTaps = 1815;
// log2 of the input channels per CTA
inline int permute_ci_shift(int RS) { return RS == 1 ? 5 : (RS <= 40 ? 3 : (RS <= 80 ? 2 : 0)); }

template <typename T>
__global__ void __launch_bounds__(256)
filter_permute_kernel(const T* __restrict__ w, T* __restrict__ out, int Cout, int C, int RS,
                      unsigned rs_magic, int ci_shift, long long s_tap, long long s_co, long long s_ci, int pad) {
  chain_begin();
  extern __shared__ char permute_smem[];
  T* tile = reinterpret_cast<T*>(permute_smem);
  const int ci_run = 1 << ci_shift;
  const int co0 = blockIdx.y * kPermuteCo, ci0 = blockIdx.x * ci_run;
  const int nco = min(kPermuteCo, Cout - co0), nci = min(ci_run, C - ci0);
  const int run = nci * RS, pitch = (ci_run * RS) | 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long group = (long long)blockIdx.z * Cout * C * RS;
  w += group;
  out += group;
  // i / RS for the small i of a tile (rs_magic = ceil(2^32 / RS), 0 for RS == 1)
  auto over_rs = [&](int i) { return rs_magic ? (int)__umulhi((unsigned)i, rs_magic) : i; };
#pragma unroll
  for (int r4 = 0; r4 < kPermuteCo / 8; ++r4) {
    const int r = warp + 8 * r4;
    if (r >= nco) break;
    const T* src = w + ((long long)(co0 + r) * C + ci0) * RS;
#pragma unroll 4
    for (int i = lane; i < run; i += 32) tile[r * pitch + i] = src[i];
  }
  __syncthreads();
  out += (long long)co0 * s_co + (long long)ci0 * s_ci;
  if (s_co == 1) {
#pragma unroll 4
    for (int i = warp; i < run; i += 8) {  // one (ci, tap) per warp, lanes along co
      const int ci = over_rs(i), tap = i - ci * RS;
      if (lane < nco) out[tap * s_tap + lane + ci * s_ci] = tile[lane * pitch + i];
      if (lane < pad && co0 + nco == Cout) out[tap * s_tap + nco + lane + ci * s_ci] = T(0);
    }
  } else {
    const int total = nco * RS << ci_shift;  // (co, tap, ci), ci fastest
#pragma unroll 4
    for (int e = threadIdx.x; e < total; e += 256) {
      const int ci = e & (ci_run - 1), i = e >> ci_shift, r = over_rs(i), tap = i - r * RS;
      if (ci < nci) out[tap * s_tap + r * s_co + ci] = tile[r * pitch + ci * RS + tap];
      if (ci < pad && ci0 + nci == C) out[tap * s_tap + r * s_co + nci + ci] = T(0);
    }
  }
}

template <typename T>
int filter_permute(const T* w, T* out, int Cout, int C, int RS, long long s_tap, long long s_co,
                   long long s_ci, cudaStream_t st, int groups = 1, int pad = 0) {
  FLB200_REQUIRE(RS <= kPermuteMaxTaps, "filter_permute: %d taps do not fit", RS);
  int shift = permute_ci_shift(RS);
  // few CTAs: shorter runs (64 x 64 filters of 31 taps: 8.6 us in 16 CTAs, 2.6 in 128), as long as the
  // stores stay together, and `pad` threads are there for the zeros
  const long long over_co = (Cout + kPermuteCo - 1) / kPermuteCo;
  while (shift > (s_co == 1 ? 0 : 2) && over_co * ((C + (1 << shift) - 1) >> shift) * groups < 148) --shift;
  const int run = 1 << shift;
  const size_t smem = (size_t)kPermuteCo * ((run * RS) | 1) * sizeof(T);
  if (smem > 48 * 1024)  // more than 380 taps
    FLB200_CUDA_CHECK(cudaFuncSetAttribute(filter_permute_kernel<T>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((unsigned)((C + run - 1) / run), (unsigned)((Cout + kPermuteCo - 1) / kPermuteCo),
            (unsigned)groups);
  FLB200_REQUIRE(grid.y <= 65535 && groups <= 65535, "filter_permute: too many channels");
  const unsigned magic = RS == 1 ? 0u : (unsigned)(((1ull << 32) + RS - 1) / RS);
  launch_chained(filter_permute_kernel<T>, grid, 256, smem, st, w, out, Cout, C, RS, magic, shift, s_tap, s_co,
                 s_ci, pad);
  FLB200_AFTER_LAUNCH("filter_permute");
  return FLB200_OK;
}

}  // namespace flb200
