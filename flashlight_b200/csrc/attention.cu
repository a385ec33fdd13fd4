// Fused attention, forward and backward (flash style):  o = softmax(scale * q k^T [+ causal mask]) v
// and dq, dk, dv, without materialising the T x T score tensors in device memory.  The reference
// builds the chain out of whole-tensor operators and keeps the probabilities for the gradient
// (flashlight/fl/autograd/Functions.cpp:1828-1891, 1021-1042); here the forward pass keeps only
// the row-wise log-sum-exp of the scaled scores, and the backward kernel recomputes the
// probabilities of one 128 x 128 block at a time in tensor memory.
//
// bf16 tensors of head dimension 64 and any length T, read and written in place through strides:
// [batch * heads][T][64], or the packed projection [batch][T][3][heads][64] as its contraction left
// it, which saves a reordering copy on each side.  Rows past T arrive as zeros from TMA, are masked
// and never stored.
// Backward: one CTA per (batch-head, block of 128 keys): K_j and V_j stay in shared memory, the CTA
// walks the query blocks i (i >= j with the causal mask) and per block issues five tcgen05
// contractions with fp32 accumulators in tensor memory:
//     S  = Q_i K_j^T                    (128 x 128, K = 64)   columns   0..127
//     dP = dO_i V_j^T                   (128 x 128, K = 64)   columns 128..255
//     dV_j += P^T dO_i                  (128 x  64, K = 128)  columns 256..319   (kept over i)
//     dK_j += dS^T Q_i                  (128 x  64, K = 128)  columns 320..383   (kept over i)
//     dQ_i  = dS K_j                    (128 x  64, K = 128)  columns 384..447
// with P = exp(scale * S - lse), dS = scale * P * (dP - D) and D = rowsum(dO * O) from a small
// pre-pass, computed by the row threads (two per query row, half of the columns each) between
// the two groups of contractions and written to shared memory as bf16
// operand tiles.  One storage order serves every role a tile plays: row r of a tile is 128
// bytes (64 bf16) at r * 128 with its 16-byte chunks XOR-swizzled by r & 7 — read as a K-major
// operand (rows = m or n, 64 k per row) or as an MN-major operand (rows = k, 64 m or n per
// row), so Q_i, dO_i and K_j are used as TMA delivered them, and P / dS (two 64-key halves,
// 16 KB apart) feed both the transposed products and dS K_j.  dQ blocks of different CTAs are
// summed in fp32 into scratch, a bulk reduction each, and rounded to bf16 by a second small kernel.
// The chain from contraction to softmax to contraction bounds it, with one CTA per SM (its tiles and
// accumulators fill both memories): so Q_i+2 and dO_i+2 are fetched behind block i, S and dP of block i + 1
// run behind its gradients, and dQ comes first of these, its sums leaving while dV and dK are made.
// Every mbarrier wait is bounded (tc_core.cuh): a wait that runs out raises the library's status
// flag and the CTA finishes its loop without waiting again.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <mutex>
#include <set>
#include <utility>

#include "common.cuh"
#include "flb200.h"
#include "tc_core.cuh"
#include "tc_gemm.cuh"

namespace flb200 {
namespace {

using namespace tc;

constexpr int kAttnThreads = 288;      // warps 0..7: two threads per query row (each half of the
                                       // columns); warp 8: TMA + MMA
constexpr int kTile = 128 * 128;       // bytes of a [128 rows][64 bf16] tile
// K V, two buffers of Q dO, P dS, dQ (fp32), align, bars
constexpr int kAttnSmem = 2 * kTile + 4 * kTile + 2 * 2 * kTile + 2 * kTile + 1024 + 256;

// element (batch b, head h, position t, d) of a tensor is at b * batch + h * head + t * row + d
struct HeadStrides { long long batch, head, row; };

struct AttnArgs {
  HeadStrides gs;     // of dq, dk and dv
  int heads;
  const float* dsum;  // rowsum(dO * O), from attention_dsum_kernel, [batch * heads][T]
  const float* lse;
  float* dq_acc;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int T, causal;
  float scale;
  int* status;
};

// byte offset of the 16-byte chunk holding keys key0 .. key0 + 7 of query row r in a P / dS tile
__device__ __forceinline__ uint32_t score_chunk(int r, int key0) {
  return (uint32_t)(key0 >> 6) * kTile + (uint32_t)r * 128 +
         ((((uint32_t)(key0 & 63) >> 3) ^ ((uint32_t)r & 7)) << 4);
}

// Row r of a dQ block is 64 floats in 16 chunks; chunk q is kept at q ^ (r & 15), in shared memory for the sake
// of the banks and so in the fp32 sums too (narrow_dq_kernel reads it back).
__device__ __forceinline__ int dq_chunk(int r, int q) { return q ^ (r & 15); }
// adds `bytes` of fp32 in shared memory to device memory, asynchronously
__device__ __forceinline__ void bulk_add(float* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

// two 32-column loads of this thread's tensor-memory lane in flight together
__device__ __forceinline__ void tmem_ld32_pair(uint32_t ta, float* a, uint32_t tb, float* b) {
  uint32_t x[32], y[32];
#define FLB200_LD32(addr, r)                                                                     \
  asm volatile(                                                                                  \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                                  \
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "                  \
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"  \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),      \
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),  \
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),            \
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),            \
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])             \
      : "r"(addr)                                                                                \
      : "memory")
  FLB200_LD32(ta, x);
  FLB200_LD32(tb, y);
#undef FLB200_LD32
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    a[i] = __uint_as_float(x[i]);
    b[i] = __uint_as_float(y[i]);
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// e^x as 2^(x log2 e), results below 2^-126 as zero.  x is what is left of a score once the row's maximum or lse
// has been subtracted: the base is converted behind the subtraction, so that the conversion's rounding is one of
// that difference.  (With the score and the lse converted first the error grows with the score itself: of P
// 4.6e-6 -> 8.2e-6 for scores of spread 100.  For 8 x 12 heads of 512 positions that takes 22.6 us forward and
// 45.8 backward, this 24.5 and 47.8.)
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float exp_of(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * kLog2e));
  return y;
}

__global__ void __launch_bounds__(kAttnThreads)
attention_backward_kernel(const __grid_constant__ CUtensorMap map_q,
                          const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_v,
                          const __grid_constant__ CUtensorMap map_do, const AttnArgs a) {
  chain_begin();
  extern __shared__ __align__(1024) char smem_raw[];
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                       ~static_cast<uintptr_t>(1023));
  char* sK = base;
  char* sV = base + kTile;
  char* sQ = base + 2 * kTile;   // the second buffer of both 2 tiles further
  char* sDO = base + 3 * kTile;
  char* sP = base + 6 * kTile;   // two 64-key halves
  char* sDS = base + 8 * kTile;  // two 64-key halves
  char* sDQ = base + 10 * kTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + 12 * kTile);
  uint64_t* bar_kv = bars;      // K_j, V_j landed
  uint64_t* bar_q = bars + 1;   // [2] Q_i, dO_i landed
  uint64_t* bar_s = bars + 3;   // S and dP complete
  uint64_t* bar_dq = bars + 4;  // dQ contraction complete
  uint64_t* bar_o = bars + 5;   // dV and dK contractions complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);
  volatile int* failed = reinterpret_cast<volatile int*>(bars + 7);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int nblk = (a.T + 127) / 128;
  const int j = blockIdx.x % nblk;        // key block
  const int bh = blockIdx.x / nblk;       // batch * heads index
  const int batch = bh / a.heads, head = bh - batch * a.heads;
  const long long row0 = (long long)bh * a.T;  // first row of this head in lse, dsum and dq_acc

  if (threadIdx.x == 0) {
    for (int k = 0; k < 6; ++k) mbar_init(bars + k, 1);
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 8) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool row_thread = warp < 8;
  const int r = (warp & 3) * 32 + lane;  // query row inside the block (row threads)
  const int half = warp >> 2;            // which half of the columns this row thread handles

  // operand descriptors (see the file comment): K-major tiles step 32 bytes per 16 k,
  // MN-major tiles step 16 rows = 2048 bytes per 16 k
  const uint64_t dK_k = umma_desc(smem_u32(sK), 16, 1024, 2);
  const uint64_t dV_k = umma_desc(smem_u32(sV), 16, 1024, 2);
  const uint64_t dQ_k = umma_desc(smem_u32(sQ), 16, 1024, 2);
  const uint64_t dDO_k = umma_desc(smem_u32(sDO), 16, 1024, 2);
  const uint64_t dP_mn = umma_desc(smem_u32(sP), kTile, 1024, 2);    // 64-key boxes 16 KB apart
  const uint64_t dDS_mn = umma_desc(smem_u32(sDS), kTile, 1024, 2);
  const uint64_t dDS_k = umma_desc(smem_u32(sDS), 16, 1024, 2);
  const uint64_t dDO_mn = umma_desc(smem_u32(sDO), 8192, 1024, 2);   // one box of 64 d
  const uint64_t dQ_mn = umma_desc(smem_u32(sQ), 8192, 1024, 2);
  const uint64_t dK_mn = umma_desc(smem_u32(sK), 8192, 1024, 2);
  const uint32_t id_s = umma_idesc_f16(kOperandBf16, 128, 0, 0);   // S, dP
  const uint32_t id_t = umma_idesc_f16(kOperandBf16, 64, 1, 1);    // dV, dK: both operands MN-major
  const uint32_t id_q = umma_idesc_f16(kOperandBf16, 64, 0, 1);    // dQ: dS K-major, K_j MN-major

  auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
    if (*failed == 0 && !mbar_wait(bar, phase)) *failed = code;
    tc_fence_after();
  };
  auto load_q = [&](int i, uint32_t buf) {
    mbar_expect_tx(&bar_q[buf], 2 * kTile);
    int c[4] = {0, i * 128, head, batch};
    tma_load(&map_q, &bar_q[buf], sQ + buf * 2 * kTile, 4, c);
    tma_load(&map_do, &bar_q[buf], sDO + buf * 2 * kTile, 4, c);
  };
  auto scores = [&](uint32_t buf, uint32_t phase) {
    wait(&bar_q[buf], phase, 2);
    const uint32_t off = buf * 2 * kTile;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)  // K = 64 d in steps of 16
      umma_f16(tmem, umma_desc_advance(dQ_k, off + kk * 32), umma_desc_advance(dK_k, kk * 32), id_s, kk > 0);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      umma_f16(tmem + 128, umma_desc_advance(dDO_k, off + kk * 32), umma_desc_advance(dV_k, kk * 32), id_s, kk > 0);
    umma_commit(bar_s);
  };
  const int i_first = a.causal ? j : 0, blocks = nblk - i_first;
  if (warp == 8 && elect_one()) {
    mbar_expect_tx(bar_kv, 2 * kTile);
    int c[4] = {0, j * 128, head, batch};
    tma_load(&map_k, bar_kv, sK, 4, c);
    load_q(i_first, 0);
    tma_load(&map_v, bar_kv, sV, 4, c);
    if (blocks > 1) load_q(i_first + 1, 1);
    wait(bar_kv, 0, 1);
    scores(0, 0);
  }
  float lse = 0.f, dsum = 0.f;
  auto fetch_row = [&](int i) {
    lse = dsum = 0.f;
    if (row_thread && i * 128 + r < a.T) {
      dsum = a.dsum[row0 + (long long)i * 128 + r];
      lse = a.lse[row0 + (long long)i * 128 + r];
    }
  };
  fetch_row(i_first);

#ifdef FLB200_ATTN_PROFILE
  long long pc[6] = {0, 0, 0, 0, 0, 0};
#define ATTN_MARK(k, t) pc[k] += clock64() - t; t = clock64()
  long long tp = clock64();
#else
#define ATTN_MARK(k, t)
#endif
  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  for (int it = 0; it < blocks; ++it) {
    const int i = i_first + it;
    const uint32_t ph = it & 1;
    if (row_thread) {
      wait(bar_s, ph, 3);
      ATTN_MARK(1, tp);
      const int q_pos = i * 128 + r;
      // Keys in front of `live` count; blocks off the diagonal and the ends have no others, and the test
      // per element is most of what such a block costs (4900 clocks, without it 1750).
      const bool whole = !(a.causal && i == j) && (i + 1) * 128 <= a.T && (j + 1) * 128 <= a.T;
      const int live = q_pos >= a.T ? 0 : min(a.T, a.causal ? q_pos + 1 : a.T) - j * 128;
#pragma unroll 1
      for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 32) {
        float s[32], dp[32];
        tmem_ld32_pair(lane_addr + (uint32_t)c0, s, lane_addr + 128u + (uint32_t)c0, dp);
        if (whole) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            s[e] = exp_of(fmaf(a.scale, s[e], -lse));
            dp[e] = a.scale * s[e] * (dp[e] - dsum);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            s[e] = c0 + e < live ? exp_of(fmaf(a.scale, s[e], -lse)) : 0.f;
            dp[e] = a.scale * s[e] * (dp[e] - dsum);
          }
        }
        // the last block's dV and dK have read P and dS
        if (it > 0 && c0 == 64 * half) wait(bar_o, ph ^ 1, 4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t off = score_chunk(r, c0 + 8 * u);
          *reinterpret_cast<uint4*>(sP + off) =
              make_uint4(pack_bf16(s[8 * u], s[8 * u + 1]), pack_bf16(s[8 * u + 2], s[8 * u + 3]),
                         pack_bf16(s[8 * u + 4], s[8 * u + 5]), pack_bf16(s[8 * u + 6], s[8 * u + 7]));
          *reinterpret_cast<uint4*>(sDS + off) = make_uint4(
              pack_bf16(dp[8 * u], dp[8 * u + 1]), pack_bf16(dp[8 * u + 2], dp[8 * u + 3]),
              pack_bf16(dp[8 * u + 4], dp[8 * u + 5]), pack_bf16(dp[8 * u + 6], dp[8 * u + 7]));
        }
      }
      fence_proxy_async();  // the tensor core reads these generic-proxy writes next
      if (threadIdx.x == 0) bulk_wait_read<0>();  // the last dQ has left its tile
      ATTN_MARK(2, tp);
    }
    tc_fence_before();
    __syncthreads();  // P and dS are complete; S, dP and the last dQ have been read
    if (warp == 8) {
      if (elect_one()) {
        const uint32_t off = ph * 2 * kTile;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // K = 128 keys: two 64-key halves of dS, 16 key rows of K_j
          umma_f16(tmem + 384, umma_desc_advance(dDS_k, (kk >> 2) * kTile + (kk & 3) * 32),
                   umma_desc_advance(dK_mn, kk * 2048), id_q, kk > 0);
        umma_commit(bar_dq);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {  // K = 128 query rows in steps of 16
          umma_f16(tmem + 256, umma_desc_advance(dP_mn, kk * 2048),
                   umma_desc_advance(dDO_mn, off + kk * 2048), id_t, (it > 0 || kk > 0) ? 1u : 0u);
          umma_f16(tmem + 320, umma_desc_advance(dDS_mn, kk * 2048),
                   umma_desc_advance(dQ_mn, off + kk * 2048), id_t, (it > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(bar_o);
        if (it + 1 < blocks) scores(ph ^ 1, ((it + 1) >> 1) & 1);
        if (it + 2 < blocks) {
          wait(bar_o, ph, 4);
          load_q(i + 2, ph);
        }
      }
      __syncwarp();
    } else {
      if (it + 1 < blocks) fetch_row(i + 1);
      wait(bar_dq, ph, 5);
      ATTN_MARK(3, tp);
      float v[32];
      tmem_ld32(lane_addr + 384u + 32u * half, v);
      float4* to = reinterpret_cast<float4*>(sDQ) + r * 16;
#pragma unroll
      for (int e = 0; e < 32; e += 4)
        to[dq_chunk(r, 8 * half + e / 4)] = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      fence_proxy_async();
      asm volatile("bar.sync 1, 256;" ::: "memory");  // the row threads
      if (threadIdx.x == 0) {
        bulk_add(a.dq_acc + (row0 + (long long)i * 128) * 64, sDQ, (uint32_t)min(128, a.T - i * 128) * 256u);
        bulk_commit();
      }
      ATTN_MARK(4, tp);
    }
  }
  if (*failed)  // copies and contractions under way when a wait ran out have ended after this
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {
    }
  if (row_thread) wait(bar_o, (blocks - 1) & 1, 4);
  if (threadIdx.x == 0) bulk_wait<0>();
#ifdef FLB200_ATTN_PROFILE
  if (blockIdx.x == 0 && threadIdx.x == 0)
    printf("attention profile (CTA 0, %d blocks): wait S,dP %lld | softmax %lld | wait dQ %lld | dQ %lld\n",
           blocks, pc[1], pc[2], pc[3], pc[4]);
#endif

  if (row_thread) {
    // the first half of the row threads stores dV_j, the second dK_j
    const int key = j * 128 + r;
    const uint32_t from = lane_addr + 256u + 64u * half;
    __nv_bfloat16* out = (half == 0 ? a.dv : a.dk) + batch * a.gs.batch + head * a.gs.head +
                         (long long)key * a.gs.row;
#pragma unroll 1
    for (int c0 = 0; c0 < 64; c0 += 32) {
      float v[32];
      __syncwarp();  // the lanes past the end store nothing, and are back for the next load
      tmem_ld32(from + (uint32_t)c0, v);
      if (key < a.T) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<uint4*>(out + c0 + 8 * u) =
              make_uint4(pack_bf16(v[8 * u], v[8 * u + 1]), pack_bf16(v[8 * u + 2], v[8 * u + 3]),
                         pack_bf16(v[8 * u + 4], v[8 * u + 5]), pack_bf16(v[8 * u + 6], v[8 * u + 7]));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *failed != 0 && a.status) atomicExch(a.status, *failed);
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// D[row] = sum_d dO[row][d] * O[row][d]: eight lanes per row, one 16-byte load each.  Rows in the
// order [batch][T][heads] of o, results in [batch][heads][T].
__global__ void attention_dsum_kernel(const __nv_bfloat16* __restrict__ o,
                                      const __nv_bfloat16* __restrict__ d_o,
                                      float* __restrict__ dsum, long long rows, int T,
                                      int heads) {
  chain_begin();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long row = t >> 3;
  float acc = 0.f;
  if (row < rows) {
    const uint4 vo = reinterpret_cast<const uint4*>(o)[t];
    const uint4 vg = reinterpret_cast<const uint4*>(d_o)[t];
    const __nv_bfloat162* ho = reinterpret_cast<const __nv_bfloat162*>(&vo);
    const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&vg);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 fo = __bfloat1622float2(ho[e]), fg = __bfloat1622float2(hg[e]);
      acc += fo.x * fg.x + fo.y * fg.y;
    }
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  if (row < rows && (threadIdx.x & 7) == 0) {
    const long long bt = row / heads, b = bt / T;
    dsum[(b * heads + row - bt * heads) * T + bt - b * T] = acc;
  }
}

__global__ void narrow_dq_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                 long long n8, int T, int heads, HeadStrides gs) {
  chain_begin();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8;
       i += (long long)gridDim.x * blockDim.x) {
    const long long row = i >> 3, bh = row / T, b = bh / heads;
    const int in_block = (int)(row - bh * T) & 127, q = 2 * ((int)i & 7);
    const float4 lo = reinterpret_cast<const float4*>(acc)[row * 16 + dq_chunk(in_block, q)];
    const float4 hi = reinterpret_cast<const float4*>(acc)[row * 16 + dq_chunk(in_block, q + 1)];
    __nv_bfloat16* to = dq + b * gs.batch + (bh - b * heads) * gs.head + (row - bh * T) * gs.row + 8 * (i & 7);
    *reinterpret_cast<uint4*>(to) = make_uint4(pack_bf16(lo.x, lo.y), pack_bf16(lo.z, lo.w),
                                                 pack_bf16(hi.x, hi.y), pack_bf16(hi.z, hi.w));
  }
}

// ---------------------------------------------------------------------------------- forward
// One CTA per (batch-head, block of 128 queries), largest blocks of a causal head first; it walks the
// key blocks j with two contractions each:
//     S  = Q_i K_j^T   (128 x 128, K = 64)    columns   0..127
//     O  = P V_j       (128 x  64, K = 128)   columns 128..191
// Two threads per query row (half of the columns each) read S, agree on the new row maximum m through
// shared memory, write P = exp(scale * S - m) as a bf16 operand tile, and keep the row's sum and its
// output in fp32 registers, rescaled by exp(m_old - m) per block.  K_{j+1} is fetched while the
// probabilities of block j are computed, S_{j+1} runs behind O_j.  What bounds it is that chain from
// contraction to contraction, not the tensor pipe: two CTAs share an SM and fill each other's waits.
// 8 x 12 heads of 512 positions: 24.5 us (39 with a mask test per element); scores, softmax and context
// as three operators with a reordering copy before and after were five launches, three T x T passes and
// about 90 us.  A pass of 12 layers over 128 positions went from 2.1 to 1.4 ms with the 48 launches that
// are gone.
constexpr int kFwdSmem = 5 * kTile + 1024 + 1024 + 256;  // Q K V P(2), row exchange, align, bars
struct AttnFwdArgs {
  __nv_bfloat16* out;
  HeadStrides os;
  float* lse;  // [batch * heads][T], or null
  int T, heads, causal;
  float scale;
  int* status;
};

__global__ void __launch_bounds__(kAttnThreads, 2)
attention_forward_kernel(const __grid_constant__ CUtensorMap map_q,
                         const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const AttnFwdArgs a) {
  chain_begin();
  extern __shared__ __align__(1024) char smem_raw[];
  char* base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  char* sQ = base;
  char* sK = base + kTile;
  char* sV = base + 2 * kTile;
  char* sP = base + 3 * kTile;  // two 64-key halves
  float* row_x = reinterpret_cast<float*>(base + 5 * kTile);  // [2 halves][128 rows]
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_x + 256);
  uint64_t* bar_q = bars;
  uint64_t* bar_k = bars + 1;
  uint64_t* bar_v = bars + 2;
  uint64_t* bar_s = bars + 3;
  uint64_t* bar_o = bars + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
  volatile int* failed = reinterpret_cast<volatile int*>(bars + 6);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int nblk = (a.T + 127) / 128;
  const int i = nblk - 1 - (int)blockIdx.x % nblk;  // query block
  const int bh = blockIdx.x / nblk;
  const int batch = bh / a.heads, head = bh - batch * a.heads;

  if (threadIdx.x == 0) {
    for (int k = 0; k < 5; ++k) mbar_init(bars + k, 1);
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 8) tmem_alloc(tmem_slot, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int r = (warp & 3) * 32 + lane, half = warp >> 2;
  const int q_pos = i * 128 + r;
  const int blocks = a.causal ? i + 1 : nblk;

  const uint64_t dQ = umma_desc(smem_u32(sQ), 16, 1024, 2);
  const uint64_t dK = umma_desc(smem_u32(sK), 16, 1024, 2);
  const uint64_t dP = umma_desc(smem_u32(sP), 16, 1024, 2);
  const uint64_t dV = umma_desc(smem_u32(sV), 8192, 1024, 2);  // one box of 64 d, rows = keys
  const uint32_t id_s = umma_idesc_f16(kOperandBf16, 128, 0, 0);
  const uint32_t id_o = umma_idesc_f16(kOperandBf16, 64, 0, 1);
  auto load = [&](const CUtensorMap* m, uint64_t* bar, char* to, int block) {
    mbar_expect_tx(bar, kTile);
    int c[4] = {0, block * 128, head, batch};
    tma_load(m, bar, to, 4, c);
  };
  auto wait = [&](uint64_t* bar, uint32_t phase, int code) {
    if (*failed == 0 && !mbar_wait(bar, phase)) *failed = code;
    tc_fence_after();
  };
  auto scores = [&](uint32_t phase) {
    wait(bar_k, phase, 2);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)  // K = 64 d in steps of 16
      umma_f16(tmem, umma_desc_advance(dQ, kk * 32), umma_desc_advance(dK, kk * 32), id_s, kk > 0);
    umma_commit(bar_s);
  };
  if (warp == 8 && elect_one()) {
    load(&map_q, bar_q, sQ, i);
    load(&map_k, bar_k, sK, 0);
    load(&map_v, bar_v, sV, 0);
    wait(bar_q, 0, 1);
    scores(0);
  }
  // the running maximum starts at the lowest finite value: keys whose scores are all -inf then count
  // as zeros, where -inf - (-inf) would leave NaN to every later block of the row
  float m = -FLT_MAX, sum = 0.f, o[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) o[e] = 0.f;
  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);

  for (int j = 0; j < blocks; ++j) {
    const uint32_t ph = j & 1;
    float alpha = 1.f;
    if (warp < 8) {
      wait(bar_s, ph, 3);
      // this thread's 64 keys; those in front of `live` count
      const int k0 = j * 128 + 64 * half;
      const int live = min(a.T, a.causal ? q_pos + 1 : a.T) - k0;
      // (blocks off the diagonal and the end need no test per element: 39 us for 8 x 12 heads of 512
      // positions with it, 28 without)
      const bool whole = !(a.causal && i == j) && (j + 1) * 128 <= a.T;
      float mx = -INFINITY;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float s[32];
        tmem_ld32(lane_addr + 64u * half + c0, s);
        if (whole) {
#pragma unroll
          for (int e = 0; e < 32; ++e) mx = fmaxf(mx, a.scale * s[e]);
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) mx = fmaxf(mx, c0 + e < live ? a.scale * s[e] : -INFINITY);
        }
      }
      row_x[half * 128 + r] = mx;
      // the two warps that share these rows
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
      mx = fmaxf(mx, row_x[(half ^ 1) * 128 + r]);
      const float m_new = fmaxf(m, mx);
      alpha = exp_of(m - m_new);
      m = m_new;
      sum *= alpha;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float s[32];
        tmem_ld32(lane_addr + 64u * half + c0, s);
        if (whole) {
#pragma unroll
          for (int e = 0; e < 32; ++e) s[e] = exp_of(fmaf(a.scale, s[e], -m));
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) s[e] = c0 + e < live ? exp_of(fmaf(a.scale, s[e], -m)) : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) sum += s[e];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<uint4*>(sP + score_chunk(r, 64 * half + c0 + 8 * u)) =
              make_uint4(pack_bf16(s[8 * u], s[8 * u + 1]), pack_bf16(s[8 * u + 2], s[8 * u + 3]),
                         pack_bf16(s[8 * u + 4], s[8 * u + 5]), pack_bf16(s[8 * u + 6], s[8 * u + 7]));
      }
      fence_proxy_async();
    } else if (elect_one()) {
      wait(bar_s, ph, 3);
      if (j + 1 < blocks) load(&map_k, bar_k, sK, j + 1);
    }
    tc_fence_before();
    __syncthreads();  // P is complete, S and the last block's O have been read
    if (warp == 8 && elect_one()) {
      wait(bar_v, ph, 4);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)  // K = 128 keys: two 64-key halves of P, 16 key rows of V_j
        umma_f16(tmem + 128, umma_desc_advance(dP, (kk >> 2) * kTile + (kk & 3) * 32),
                 umma_desc_advance(dV, kk * 2048), id_o, kk > 0);
      umma_commit(bar_o);
      if (j + 1 < blocks) scores(ph ^ 1);
      wait(bar_o, ph, 5);
      if (j + 1 < blocks) load(&map_v, bar_v, sV, j + 1);
    } else if (warp < 8) {
      wait(bar_o, ph, 5);
      float v[32];
      tmem_ld32(lane_addr + 128u + 32u * half, v);
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] = o[e] * alpha + v[e];
    }
    __syncwarp();
  }
  if (warp < 8) {
    asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");  // row_x has been read
    row_x[half * 128 + r] = sum;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
    sum = half == 0 ? sum + row_x[128 + r] : row_x[r] + sum;
    if (q_pos < a.T) {
      const float inv = 1.f / sum;
      __nv_bfloat16* to = a.out + batch * a.os.batch + head * a.os.head + (long long)q_pos * a.os.row + 32 * half;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        *reinterpret_cast<uint4*>(to + 8 * u) = make_uint4(
            pack_bf16(o[8 * u] * inv, o[8 * u + 1] * inv), pack_bf16(o[8 * u + 2] * inv, o[8 * u + 3] * inv),
            pack_bf16(o[8 * u + 4] * inv, o[8 * u + 5] * inv), pack_bf16(o[8 * u + 6] * inv, o[8 * u + 7] * inv));
      if (half == 0 && a.lse) a.lse[(long long)bh * a.T + q_pos] = m + logf(sum);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *failed != 0 && a.status) atomicExch(a.status, *failed);
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// Blocks of 128 positions of one head of a strided tensor; positions past T are zeros.
int head_map(CUtensorMap* m, const void* base, const HeadStrides& s, long long batch, long long heads,
             long long T) {
  const uint64_t dims[4] = {64, (uint64_t)T, (uint64_t)heads, (uint64_t)batch};
  const uint64_t strides[3] = {(uint64_t)s.row * 2, (uint64_t)s.head * 2, (uint64_t)s.batch * 2};
  const uint32_t box[4] = {64, 128, 1, 1};
  return tc::make_tensor_map(m, base, 4, dims, strides, box, tc::kMapKMajor, nullptr, tc::kOperandBf16);
}
int configure(const void* kernel, int smem) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> done;
  int dev = 0;
  FLB200_CUDA_CHECK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({dev, kernel})) return FLB200_OK;
  FLB200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  done.insert({dev, kernel});
  return FLB200_OK;
}
bool head_shape_ok(long long T, long long head_dim, int dtype) {
  return flb200_has_tensor_core_path() && dtype == FLB200_BF16 && head_dim == 64 && T > 0 && T < (1 << 24);
}

// is: strides of q, k, v; os: of o and grad_o; gs: of the gradients
int run_attention_backward(const void* q, const void* k, const void* v, const HeadStrides& is, const void* o,
                           const void* grad_o, const HeadStrides& os, const float* lse, void* grad_q,
                           void* grad_k, void* grad_v, const HeadStrides& gs, long long batch,
                           long long heads, long long T, float scale, int causal, void* workspace,
                           cudaStream_t st) {
  const long long rows = batch * heads * T;
  CUtensorMap mq, mk, mv, mg;
  if (int rc = head_map(&mq, q, is, batch, heads, T)) return rc;
  if (int rc = head_map(&mk, k, is, batch, heads, T)) return rc;
  if (int rc = head_map(&mv, v, is, batch, heads, T)) return rc;
  if (int rc = head_map(&mg, grad_o, os, batch, heads, T)) return rc;
  if (int rc = configure(reinterpret_cast<const void*>(attention_backward_kernel), kAttnSmem)) return rc;
  const size_t acc_bytes = (size_t)rows * 64 * sizeof(float);
  FLB200_CUDA_CHECK(cudaMemsetAsync(workspace, 0, acc_bytes, st));
  float* dsum = reinterpret_cast<float*>(static_cast<char*>(workspace) + acc_bytes);
  launch_chained(attention_dsum_kernel, (unsigned)((rows * 8 + 255) / 256), 256, 0, st,
                 static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(grad_o), dsum, rows,
                 (int)T, (int)heads);
  FLB200_AFTER_LAUNCH("attention_dsum");
  AttnArgs a{};
  a.gs = gs;
  a.heads = (int)heads;
  a.dsum = dsum;
  a.lse = lse;
  a.dq_acc = static_cast<float*>(workspace);
  a.dk = static_cast<__nv_bfloat16*>(grad_k);
  a.dv = static_cast<__nv_bfloat16*>(grad_v);
  a.T = (int)T;
  a.causal = causal ? 1 : 0;
  a.scale = scale;
  a.status = tc::status_ptr();
  const unsigned grid = (unsigned)(batch * heads * ((T + 127) / 128));
  launch_chained(attention_backward_kernel, grid, kAttnThreads, kAttnSmem, st, mq, mk, mv, mg, a);
  FLB200_AFTER_LAUNCH("attention_backward");
  tc::count_tc_launch();
  const long long n8 = rows * 64 / 8;
  launch_chained(narrow_dq_kernel, (unsigned)std::min<long long>((n8 + 255) / 256, 148 * 8), 256, 0, st,
                 a.dq_acc, static_cast<__nv_bfloat16*>(grad_q), n8, (int)T, (int)heads, gs);
  FLB200_AFTER_LAUNCH("attention_narrow_dq");
  return FLB200_OK;
}

}  // namespace
}  // namespace flb200

using namespace flb200;

extern "C" {

size_t flb200_attention_backward_workspace_bytes(int64_t batch_heads, int64_t seq_len,
                                                 int64_t head_dim) {
  if (batch_heads <= 0 || seq_len <= 0 || head_dim <= 0) return 0;
  // fp32 sums of dq, then rowsum(dO * O)
  return (size_t)batch_heads * seq_len * head_dim * sizeof(float) +
         (size_t)batch_heads * seq_len * sizeof(float);
}

int flb200_attention_backward_supported(int64_t seq_len, int64_t head_dim, int dtype) {
  return flb200_has_tensor_core_path() && dtype == FLB200_BF16 && head_dim == 64 && seq_len > 0 &&
                 seq_len % 128 == 0
             ? 1
             : 0;
}

int flb200_attention_backward(const void* q, const void* k, const void* v, const void* o,
                              const void* grad_o, const float* lse, void* grad_q, void* grad_k,
                              void* grad_v, int64_t batch_heads, int64_t seq_len,
                              int64_t head_dim, float scale, int causal, int dtype,
                              void* workspace, size_t workspace_bytes, void* stream) {
  FLB200_REQUIRE(q && k && v && o && grad_o && lse && grad_q && grad_k && grad_v,
                 "attention_backward: null tensor");
  FLB200_REQUIRE(batch_heads > 0, "attention_backward: empty batch");
  if (!flb200_attention_backward_supported(seq_len, head_dim, dtype))
    return fail(FLB200_UNSUPPORTED,
                "attention_backward: built for bf16, head dimension 64 and a sequence length that "
                "is a multiple of 128 (got dtype %d, head %lld, length %lld)",
                dtype, (long long)head_dim, (long long)seq_len);
  const long long rows = (long long)batch_heads * seq_len;
  FLB200_REQUIRE(rows < 0x7fffffffLL, "attention_backward: too many rows");
  const size_t need = flb200_attention_backward_workspace_bytes(batch_heads, seq_len, head_dim);
  if (!workspace || workspace_bytes < need)
    return fail(FLB200_WORKSPACE_TOO_SMALL, "attention_backward: workspace %zu < %zu",
                workspace_bytes, need);
  const void* ptrs[] = {q, k, v, o, grad_o, grad_q, grad_k, grad_v, workspace};
  for (const void* p : ptrs)
    FLB200_REQUIRE(aligned16(p), "attention_backward: tensors must be 16-byte aligned");
  const HeadStrides dense{seq_len * 64, seq_len * 64, 64};
  return run_attention_backward(q, k, v, dense, o, grad_o, dense, lse, grad_q, grad_k, grad_v, dense,
                                batch_heads, 1, seq_len, scale, causal, workspace, as_stream(stream));
}

int flb200_attention_packed_supported(int64_t seq_len, int64_t head_dim, int dtype) {
  return head_shape_ok(seq_len, head_dim, dtype) ? 1 : 0;
}

int flb200_attention_packed_forward(const void* qkv, void* out, float* lse, int64_t batch, int64_t heads,
                                    int64_t seq_len, int64_t head_dim, float scale, int causal, int dtype,
                                    void* stream) {
  FLB200_REQUIRE(qkv && out, "attention_packed_forward: null tensor");
  FLB200_REQUIRE(batch > 0 && heads > 0 && batch * heads * seq_len < 0x7fffffffLL,
                 "attention_packed_forward: bad extents");
  if (!head_shape_ok(seq_len, head_dim, dtype) || !aligned16(qkv) || !aligned16(out))
    return fail(FLB200_UNSUPPORTED,
                "attention_packed_forward: built for 16-byte aligned bf16 tensors of head dimension 64");
  const long long width = heads * 64;
  const HeadStrides is{seq_len * 3 * width, 64, 3 * width}, os{seq_len * width, 64, width};
  const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(qkv);
  CUtensorMap mq, mk, mv;
  if (int rc = head_map(&mq, q, is, batch, heads, seq_len)) return rc;
  if (int rc = head_map(&mk, q + width, is, batch, heads, seq_len)) return rc;
  if (int rc = head_map(&mv, q + 2 * width, is, batch, heads, seq_len)) return rc;
  if (int rc = configure(reinterpret_cast<const void*>(attention_forward_kernel), kFwdSmem)) return rc;
  AttnFwdArgs a{};
  a.out = static_cast<__nv_bfloat16*>(out);
  a.os = os;
  a.lse = lse;
  a.T = (int)seq_len;
  a.heads = (int)heads;
  a.causal = causal ? 1 : 0;
  a.scale = scale;
  a.status = tc::status_ptr();
  const unsigned grid = (unsigned)(batch * heads * ((seq_len + 127) / 128));
  launch_chained(attention_forward_kernel, grid, kAttnThreads, kFwdSmem, as_stream(stream), mq, mk, mv, a);
  FLB200_AFTER_LAUNCH("attention_forward");
  tc::count_tc_launch();
  return FLB200_OK;
}

int flb200_attention_packed_backward(const void* qkv, const void* out, const void* grad_out, const float* lse,
                                     void* grad_qkv, int64_t batch, int64_t heads, int64_t seq_len,
                                     int64_t head_dim, float scale, int causal, int dtype, void* workspace,
                                     size_t workspace_bytes, void* stream) {
  FLB200_REQUIRE(qkv && out && grad_out && lse && grad_qkv, "attention_packed_backward: null tensor");
  FLB200_REQUIRE(batch > 0 && heads > 0 && batch * heads * seq_len < 0x7fffffffLL,
                 "attention_packed_backward: bad extents");
  const void* ptrs[] = {qkv, out, grad_out, grad_qkv, workspace};
  bool aligned = true;
  for (const void* p : ptrs) aligned = aligned && aligned16(p);
  if (!head_shape_ok(seq_len, head_dim, dtype) || !aligned)
    return fail(FLB200_UNSUPPORTED,
                "attention_packed_backward: built for 16-byte aligned bf16 tensors of head dimension 64");
  const size_t need = flb200_attention_backward_workspace_bytes(batch * heads, seq_len, head_dim);
  if (!workspace || workspace_bytes < need)
    return fail(FLB200_WORKSPACE_TOO_SMALL, "attention_packed_backward: workspace %zu < %zu",
                workspace_bytes, need);
  const long long width = heads * 64;
  const HeadStrides is{seq_len * 3 * width, 64, 3 * width}, os{seq_len * width, 64, width};
  const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(qkv);
  __nv_bfloat16* g = static_cast<__nv_bfloat16*>(grad_qkv);
  return run_attention_backward(q, q + width, q + 2 * width, is, out, grad_out, os, lse, g, g + width,
                                g + 2 * width, is, batch, heads, seq_len, scale, causal, workspace,
                                as_stream(stream));
}

}  // extern "C"
