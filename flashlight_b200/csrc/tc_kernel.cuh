// Persistent tcgen05 contraction kernel for sm_100a and the "problem" policies that feed it.
//
//   D = sum_k A(m,k) * B(k,n),  fp32 operands read as TF32, fp32 accumulation in TMEM.
//
// One CTA per SM walks a static list of 128 x BN output tiles:
//   warp 0   : TMA producer — issues cp.async.bulk.tensor loads (never multicast) into a
//              STAGES-deep ring of 128-byte-swizzled shared-memory tiles and runs ahead into
//              the next output tile while the current one drains.  One elected lane owns the
//              barriers and issues the copies; per stage it adds to the coordinates and no more,
//              since a stage's MMAs take only 160 to 512 clocks.  (A lane per copy, coordinates
//              by multiplication: 470 clocks per stage of two copies, 730 of four.)
//   warp 1   : allocates TMEM (2 accumulators of BN columns); one lane issues tcgen05.mma
//              for each ready stage and tcgen05.commit to free the stage / publish the tile
//   warps 6-9: only in the 3xTF32 instantiation (fp32-grade products): split every landed
//              operand element into a TF32-exact high part and the remainder, so that the MMA
//              warp can issue a_lo*b_hi + a_hi*b_lo + a_hi*b_hi
//   warps 2-5 (and four more behind the producers for tiles of 128+ columns, each group
//              taking every other 32-column chunk):
//              epilogue — tcgen05.ld the finished accumulator (32 lanes each) and store it
//              from registers (coalesced 128-byte rows when the row index is contiguous in
//              memory, 16-byte vectors when the column index is) while the MMA warp already
//              fills the other accumulator
// Hand-offs: full/empty mbarriers per stage, full/empty mbarriers per accumulator.
// Every wait is bounded by a clock budget; a wait that runs out raises a flag, all roles
// drain and the CTA frees its TMEM and returns (the host then reports FLB200_TIMEOUT).
//
// A problem policy P tells the skeleton what a tile is:
//   int  a_mn_major, b_mn_major, operand;   // operand: kOperandTf32 / kOperandBf16 / kOperandF16
//   static constexpr bool kTwoProducers;  // a producer warp per operand, else one for both
//   static constexpr int kMinBlocks;      // second argument of tc_persistent_kernel's launch
//                                         // bounds: 1 = the register allocator may use the whole
//                                         // file for the one resident CTA, 0 = its own choice
//   struct Tile;  struct LoadState;
//   __device__ int  num_tiles() const;
//   __device__ void decode(int tile, Tile&) const;
//   __device__ int  k_begin(const Tile&) const;  __device__ int k_end(const Tile&) const;
//   template <int kWhich> __device__ void load_begin(const Tile&, LoadState&) const;   // once per tile
//   __device__ uint32_t stage_bytes(const Tile&) const;   // that the copies of a stage bring
//   template <int kWhich>
//   __device__ void load(const CUtensorMap* a, const CUtensorMap* b, const Tile&, LoadState&,
//                        uint64_t* bar, char* a_dst, char* b_dst) const;
//                        // one stage: issues the copies and advances the LoadState
//   __device__ bool chunk_live(const Tile&, int c0) const;                // warp-uniform
//   __device__ void store(const Tile&, int row, int c0, const float* v, float* stage,
//                         int lane) const;   // 32 columns of row `row`; called by all 32 lanes
//                         // of an epilogue warp (rows row - lane .. + 31), `stage` is the
//                         // warp's 4 KB staging tile for policies that store through it
#pragma once
#include <cuda_bf16.h>

#include <type_traits>

#include "tc_core.cuh"

namespace flb200 {
namespace tc {

// Staging tile of one epilogue warp and the transposing store through it.  The accumulator
// arrives with one row per lane (32 consecutive columns in registers).  Written to a row-major
// output as it is, every store instruction touches 32 rows at 16 bytes each (32 memory sectors,
// half filled); staged through shared memory, an instruction stores 4 whole 128-byte rows.
// Layout: row r, 16-byte chunk q at chunk (q ^ (r & 7)) of row r: conflict-free both ways.
constexpr int kEpiStageBytes = 32 * 128;
__device__ __forceinline__ void epi_stage_write(float* stage, int lane, const float* v) {
  float4* rowp = reinterpret_cast<float4*>(stage) + lane * 8;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    rowp[q ^ (lane & 7)] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  __syncwarp();
}
// The float4 that lane `lane` stores in step k (0..7): row 4 * k + lane / 8, columns
// 4 * (lane % 8) .. + 3 of the chunk.
__device__ __forceinline__ float4 epi_stage_read(const float* stage, int lane, int k) {
  const int r = 4 * k + (lane >> 3), q = lane & 7;
  return reinterpret_cast<const float4*>(stage)[r * 8 + (q ^ (r & 7))];
}

// Batch-norm statistics of a convolution's output taken from its accumulators: while a warp
// stores its 32 x 32 chunk through the staging tile, every lane adds up the values (and their
// squares) it holds — 4 channels of 8 rows — and the four row groups are added through the
// staging tile; lanes 0..7 then write them, 128 contiguous bytes each for sums and squares,
// into row `group` of a [groups][2 * channels] matrix (sums first, then squares).  Its column
// sums are the per-channel totals; no atomics, so the result does not depend on timing.
struct EpiStats {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
  __device__ __forceinline__ void add(float4 v) {
    s0 += v.x; s1 += v.y; s2 += v.z; s3 += v.w;
    q0 = fmaf(v.x, v.x, q0); q1 = fmaf(v.y, v.y, q1);
    q2 = fmaf(v.z, v.z, q2); q3 = fmaf(v.w, v.w, q3);
  }
  // `stage`: the warp's staging tile, free again once every lane has read its values out of
  // it (the caller's loop is done); the four row groups of a chunk (lane / 8) meet through it.
  __device__ __forceinline__ void flush(float* stats, long long group, int channels, int c0,
                                        int lane, float* stage) {
    __syncwarp();
    float4* slot = reinterpret_cast<float4*>(stage);
    slot[2 * lane] = make_float4(s0, s1, s2, s3);
    slot[2 * lane + 1] = make_float4(q0, q1, q2, q3);
    __syncwarp();
    if (lane < 8) {
#pragma unroll
      for (int g = 1; g < 4; ++g) {
        const float4 a = slot[2 * (lane + 8 * g)], b = slot[2 * (lane + 8 * g) + 1];
        s0 += a.x; s1 += a.y; s2 += a.z; s3 += a.w;
        q0 += b.x; q1 += b.y; q2 += b.z; q3 += b.w;
      }
      float* row = stats + group * (2LL * channels) + c0 + 4 * lane;
      *reinterpret_cast<float4*>(row) = make_float4(s0, s1, s2, s3);
      *reinterpret_cast<float4*>(row + channels) = make_float4(q0, q1, q2, q3);
    }
  }
};

// Four consecutive elements of a row-major output, rounded to its type.
__device__ __forceinline__ void epi_store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <typename T>
__device__ __forceinline__ void epi_store4(T* p, float4 v) {
  T h[4] = {Num<T>::from_f(v.x), Num<T>::from_f(v.y), Num<T>::from_f(v.z), Num<T>::from_f(v.w)};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
}
template <typename T>
__device__ __forceinline__ float4 epi_round(float4 v) {
  return make_float4(Num<T>::to_f(Num<T>::from_f(v.x)), Num<T>::to_f(Num<T>::from_f(v.y)),
                     Num<T>::to_f(Num<T>::from_f(v.z)), Num<T>::to_f(Num<T>::from_f(v.w)));
}

// gelu in the tanh form of flashlight/fl/autograd/Functions.cpp:1791-1796 (the constants of
// flb200_gelu_forward)
// tanh(u) = 1 - 2 / (1 + exp(2u)) from the fast exponential: branch-free (no library call inside
// the store loop of the contraction kernels), absolute error below 1e-6
__device__ __forceinline__ float epi_gelu(float x) {
  const float u = 0.7978845608f * (x + 0.044715f * x * x * x);
  const float t = 1.f - __fdividef(2.f, 1.f + __expf(2.f * u));
  return 0.5f * x * (1.f + t);
}

// X3 = 1: every stage also holds the low-order tiles of the 3xTF32 split (see the kernel).
template <int BN, int STAGES, int X3 = 0>
struct SmemLayout {
  static constexpr int kABytes = kBM * kBK * 4;  // 16 KB
  static constexpr int kBBytes = BN * kBK * 4;
  static constexpr int kLoOffset = kABytes + kBBytes;  // low-order A tile, then low-order B tile
  static constexpr int kStageBytes = (X3 ? 2 : 1) * (kABytes + kBBytes);
  static constexpr int kTileBytes = STAGES * kStageBytes;
  static constexpr int kBarBytes = 512;
  // 4 KB per epilogue warp: a 32 x 32 accumulator chunk is turned from "one row per lane" into
  // "128 contiguous bytes per 8 lanes" through it before it is stored to a row-major output
  static constexpr int kStagingBytes = ((X3 == 0 && BN >= 128) ? 8 : 4) * kEpiStageBytes;
  static constexpr int kTotal = kTileBytes + kBarBytes + kStagingBytes + 1024;  // + slack to align
};

// ~200 KB of tiles per CTA
constexpr int stages_for(int bn) { return bn >= 256 ? 4 : (bn >= 128 ? 6 : (bn >= 64 ? 8 : 10)); }
constexpr int stages_for_x3(int bn) { return bn >= 256 ? 2 : (bn >= 128 ? 3 : (bn >= 64 ? 4 : 5)); }
constexpr int kThreadsX3 = kThreads + 128;  // four more warps split the operands
// The copies of a stage: of one operand or of both.  Policies whose operands may be several boxes per
// stage have a producer warp for each (warps 0 and 6).
enum { kA = 0, kB = 1, kBoth = 2 };
// Tiles of 128 or more columns get a second group of four epilogue warps (each group drains
// every other 32-column chunk of the accumulator): with one group, shapes with a short K loop
// and a large output (1x1 layers on 56x56 planes: 2 K blocks per 128 KB tile) were bound by the
// time four warps need to store a tile.
template <int X3, int BN>
constexpr int epilogue_groups() { return (X3 == 0 && BN >= 128) ? 2 : 1; }
template <class P, int X3>
constexpr int second_epilogue_first_warp() { return P::kTwoProducers && X3 == 0 ? 7 : 6; }
template <class P, int X3, int BN>
constexpr int threads_for() {
  if (X3) return kThreadsX3;
  if (epilogue_groups<X3, BN>() == 2) return (second_epilogue_first_warp<P, X3>() + 4) * 32;
  return P::kTwoProducers ? kThreads + 32 : kThreads;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Stall accounting, compiled in with -DFLB200_TC_PROFILE only (FLB200_NVCC_EXTRA of the build
// script): every role of every CTA sums the clocks it spends in each of its waits, and the
// host prints the means after each launch.  Slots: producer {wait empty, total}, MMA issuer
// {wait full, wait accumulator free, total}, epilogue warp 2 {wait accumulator full, store, total}.
#ifdef FLB200_TC_PROFILE
static __device__ long long g_tc_profile[256 * 8];
#define TC_PROF_VAR(x) long long x = 0
#define TC_PROF_NOW(t) const long long t = clock64()
#define TC_PROF_ADD(x, t) x += clock64() - t
#define TC_PROF_PUT(slot, v) g_tc_profile[(blockIdx.x & 255) * 8 + (slot)] = (v)
#else
#define TC_PROF_VAR(x)
#define TC_PROF_NOW(t)
#define TC_PROF_ADD(x, t)
#define TC_PROF_PUT(slot, v)
#endif

template <class P, int BN, int STAGES, int X3 = 0, int KSUB = 1>
__global__ void __launch_bounds__(threads_for<P, X3, BN>(), P::kMinBlocks)
tc_persistent_kernel(const __grid_constant__ CUtensorMap map_a,
                     const __grid_constant__ CUtensorMap map_b, const P prob, int* status) {
  chain_begin();
  using SL = SmemLayout<BN, STAGES, X3>;
  // The ring's STAGES sub-stages (one 128-byte-wide K block of both operands each) are handed
  // over in groups of KSUB: one pair of barriers, one wait and one commit per group.  A
  // hand-off costs each side a chain of dependent barrier instructions (measured: ~270 clocks
  // for wait + arrive alone, ~400 with one copy issued), which a narrow tile's four MMAs do
  // not cover; a group amortises it over 4 * KSUB MMAs.
  static_assert(STAGES % KSUB == 0 && (X3 == 0 || KSUB == 1), "ring must be whole groups");
  constexpr int NG = STAGES / KSUB;
  extern __shared__ char smem_raw[];
  // (an offset rather than a rounded address: the compiler keeps knowing that the tiles are
  // shared memory, and may move the epilogue's reads of them ahead of its stores)
  char* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + SL::kTileBytes);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;   // [2] accumulator ready for the epilogue
  uint64_t* tempty_bar = tfull_bar + 2;       // [2] accumulator drained, MMA may overwrite
  uint64_t* split_bar = tempty_bar + 2;       // [STAGES] X3: low-order tiles of the stage written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(split_bar + STAGES);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // (uniform to the compiler too, and one lane elected: see elect_one)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  constexpr uint32_t kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;
  const int n_tiles = prob.num_tiles();

  if (threadIdx.x == 0) {
    for (int s = 0; s < NG; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
      mbar_init(&split_bar[s], 4);  // one arrival per splitting warp
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 4 * epilogue_groups<X3, BN>());  // one arrival per epilogue warp
    }
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  constexpr bool kTwo = P::kTwoProducers && X3 == 0;
  if (warp == 0 || (kTwo && warp == 6)) {
    // One elected lane waits for a group of stages to be free, posts its byte count (not kB) and issues
    // the copies: of both operands, or of one where the policy has two producers.
    auto produce = [&](auto which) {
      constexpr int kWhich = decltype(which)::value;
      uint32_t s = 0, round = 0;
      typename P::Tile t;
      typename P::LoadState ls;
      TC_PROF_VAR(p_wait);
      TC_PROF_NOW(p_t0);
      for (int tile = blockIdx.x; tile < n_tiles && *failed == 0; tile += gridDim.x) {
        prob.decode(tile, t);
        prob.template load_begin<kWhich>(t, ls);
        const int k1 = prob.k_end(t);
        for (int k = prob.k_begin(t); k < k1; k += KSUB) {
          TC_PROF_NOW(w0);
          if (round > 0 && !mbar_wait(&empty_bar[s], (round - 1) & 1)) {
            *failed = 1;
            break;
          }
          TC_PROF_ADD(p_wait, w0);
          const int kn = min(KSUB, k1 - k);
#pragma unroll
          for (int sub = 0; sub < KSUB; ++sub) {
            if (sub >= kn) break;
            char* a_dst = tiles + (s * KSUB + sub) * SL::kStageBytes;
            if constexpr (kWhich != kB) mbar_post_tx(&full_bar[s], prob.stage_bytes(t), sub == kn - 1);
            prob.template load<kWhich>(&map_a, &map_b, t, ls, &full_bar[s], a_dst, a_dst + SL::kABytes);
          }
          if (++s == NG) { s = 0; ++round; }
        }
      }
#ifdef FLB200_TC_PROFILE
      if (kWhich != kB) { TC_PROF_PUT(0, p_wait); TC_PROF_PUT(1, clock64() - p_t0); }
#endif
    };
    if (elect_one()) {
      if constexpr (kTwo) {
        if (warp == 0) produce(std::integral_constant<int, kA>{});
        else produce(std::integral_constant<int, kB>{});
      } else {
        produce(std::integral_constant<int, kBoth>{});
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const bool half = prob.operand != kOperandTf32;
      const uint32_t idesc =
          half ? umma_idesc_f16(prob.operand, BN, prob.a_mn_major, prob.b_mn_major)
               : umma_idesc_tf32(BN, prob.a_mn_major, prob.b_mn_major);
      // MN-major tiles: fp32 in 32 x 32 boxes with the 32-byte-chunk swizzle (4 KB apart, k
      // atoms 512 B apart, 8 k-rows = 1 KB per MMA); 16-bit in 64 x 64 boxes with the plain
      // 128-byte swizzle (8 KB apart, k atoms 1 KB apart, 16 k-rows = 2 KB per MMA)
      const uint32_t mn_lbo = half ? 8192 : kBK * 128, mn_sbo = half ? 1024 : 512;
      const uint32_t mn_step = half ? 2048 : 1024, mn_layout = half ? 2 : 1;
      // descriptors of the ring's first sub-stage; every MMA offsets them (umma_desc_advance)
      const uint32_t ring = smem_u32(tiles);
      const uint64_t a_desc0 = prob.a_mn_major ? umma_desc(ring, mn_lbo, mn_sbo, mn_layout)
                                               : umma_desc(ring, 16, 1024, 2);
      const uint64_t b_desc0 = prob.b_mn_major
                                   ? umma_desc(ring + SL::kABytes, mn_lbo, mn_sbo, mn_layout)
                                   : umma_desc(ring + SL::kABytes, 16, 1024, 2);
      // K-major: step 8 elements = 32 bytes inside the swizzled row;
      // MN-major: step 8 (bf16: 16) k-rows = 1024 (2048) bytes inside each box.
      const uint32_t a_jstep = prob.a_mn_major ? mn_step : 32;
      const uint32_t b_jstep = prob.b_mn_major ? mn_step : 32;
      TC_PROF_VAR(m_full);
      TC_PROF_VAR(m_acc);
      TC_PROF_NOW(m_t0);
      // One copy of the loop per operand kind: with the kind tested between two MMAs the chains
      // that feed their descriptors to the tensor core no longer overlap, and every MMA took
      // 200 clocks to issue whatever its shape (bf16 4096 x 3072 x 768: 27.7 us, now 17.5).
      auto mma_tiles = [&](auto half_kind) {
        constexpr bool kHalf = decltype(half_kind)::value;
        uint32_t s = 0, round = 0, nt = 0;
        typename P::Tile t;
        for (int tile = blockIdx.x; tile < n_tiles && *failed == 0; tile += gridDim.x, ++nt) {
          prob.decode(tile, t);
          const uint32_t acc = nt & 1, around = nt >> 1;
          TC_PROF_NOW(w0);
          if (around > 0 && !mbar_wait(&tempty_bar[acc], (around - 1) & 1)) {
            *failed = 4;
            break;
          }
          TC_PROF_ADD(m_acc, w0);
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN;
          const int k0 = prob.k_begin(t), k1 = prob.k_end(t);
          for (int k = k0; k < k1; k += KSUB) {
            TC_PROF_NOW(w1);
            if (!mbar_wait(X3 ? &split_bar[s] : &full_bar[s], round & 1)) {
              *failed = 2;
              break;
            }
            TC_PROF_ADD(m_full, w1);
            tc_fence_after();
            if constexpr (X3 != 0) {
              // a * b ~ a_hi * b_hi + a_lo * b_hi + a_hi * b_lo with x = x_hi + x_lo, x_hi exact
              // in TF32: fp32-grade products out of three tensor-core passes
              const uint32_t off = s * SL::kStageBytes;
#pragma unroll
              for (int j = 0; j < kBK / kUmmaK; ++j) {
                const uint64_t ah = umma_desc_advance(a_desc0, off + j * a_jstep);
                const uint64_t bh = umma_desc_advance(b_desc0, off + j * b_jstep);
                const uint64_t al = umma_desc_advance(a_desc0, off + SL::kLoOffset + j * a_jstep);
                const uint64_t bl = umma_desc_advance(b_desc0, off + SL::kLoOffset + j * b_jstep);
                umma_tf32(d_tmem, al, bh, idesc, (k > k0 || j > 0) ? 1u : 0u);
                umma_tf32(d_tmem, ah, bl, idesc, 1u);
                umma_tf32(d_tmem, ah, bh, idesc, 1u);
              }
              umma_commit(&empty_bar[s]);
              if (++s == NG) { s = 0; ++round; }
              continue;
            }
            const int kn = min(KSUB, k1 - k);
#pragma unroll
            for (int sub = 0; sub < KSUB; ++sub) {
              if (sub >= kn) break;
              const uint32_t off = (s * KSUB + sub) * SL::kStageBytes;
#pragma unroll
              for (int j = 0; j < kBK / kUmmaK; ++j) {
                const uint64_t ad = umma_desc_advance(a_desc0, off + j * a_jstep);
                const uint64_t bd = umma_desc_advance(b_desc0, off + j * b_jstep);
                const uint32_t accumulate = (k > k0 || sub > 0 || j > 0) ? 1u : 0u;
                if constexpr (kHalf) umma_f16(d_tmem, ad, bd, idesc, accumulate);
                else umma_tf32(d_tmem, ad, bd, idesc, accumulate);
              }
            }
            umma_commit(&empty_bar[s]);  // frees the group once these MMAs have read it
            if (++s == NG) { s = 0; ++round; }
          }
          umma_commit(&tfull_bar[acc]);  // accumulator complete
        }
      };
      if (half) mma_tiles(std::true_type{});
      else mma_tiles(std::false_type{});
#ifdef FLB200_TC_PROFILE
      TC_PROF_PUT(2, m_full); TC_PROF_PUT(3, m_acc); TC_PROF_PUT(4, clock64() - m_t0);
#endif
    }
  } else if (X3 != 0 && warp >= 6) {
    // splitting warps (X3 only): once a stage has landed, rewrite every operand element x in
    // place as x_hi (low 13 mantissa bits cleared: exact in TF32 however the tensor core
    // converts) and write x_lo = x - x_hi at the same offset of the stage's low-order tiles;
    // elementwise at equal offsets, so the swizzled layout carries over unchanged.
    const int t128 = threadIdx.x - 6 * 32;
    uint32_t s = 0, round = 0;
    typename P::Tile t;
    bool live = true;
    for (int tile = blockIdx.x; live && tile < n_tiles; tile += gridDim.x) {
      prob.decode(tile, t);
      const int k0 = prob.k_begin(t), k1 = prob.k_end(t);
      for (int k = k0; k < k1; ++k) {
        if (*failed != 0 || !mbar_wait(&full_bar[s], round & 1)) {
          if (*failed == 0) *failed = 5;
          live = false;
          break;
        }
        float4* hi = reinterpret_cast<float4*>(tiles + s * SL::kStageBytes);
        float4* lo = reinterpret_cast<float4*>(tiles + s * SL::kStageBytes + SL::kLoOffset);
        constexpr int kVec = SL::kLoOffset / 16;
#pragma unroll 4
        for (int i = t128; i < kVec; i += 128) {
          const float4 v = hi[i];
          float4 h;
          h.x = __uint_as_float(__float_as_uint(v.x) & 0xffffe000u);
          h.y = __uint_as_float(__float_as_uint(v.y) & 0xffffe000u);
          h.z = __uint_as_float(__float_as_uint(v.z) & 0xffffe000u);
          h.w = __uint_as_float(__float_as_uint(v.w) & 0xffffe000u);
          hi[i] = h;
          lo[i] = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
        }
        fence_proxy_async();  // these generic-proxy writes are read by the tensor core next
        __syncwarp();
        if (lane == 0) mbar_arrive(&split_bar[s]);
        if (++s == NG) { s = 0; ++round; }
      }
    }
  } else if ((warp >= 2 && warp < 6) ||
             (epilogue_groups<X3, BN>() == 2 && warp >= second_epilogue_first_warp<P, X3>() &&
              warp < second_epilogue_first_warp<P, X3>() + 4)) {
    // an epilogue warp owns TMEM lanes 32*(warp % 4) .. +31; group 0 = warps 2..5 drains the
    // even 32-column chunks (all of them when there is one group), group 1 the odd ones
    constexpr int kGroups = epilogue_groups<X3, BN>();
    const int group = warp < 6 ? 0 : 1;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    float* stage = reinterpret_cast<float*>(tiles + SL::kTileBytes + SL::kBarBytes +
                                            (group * 4 + (warp < 6 ? warp - 2
                                                                   : warp - second_epilogue_first_warp<P, X3>())) *
                                                kEpiStageBytes);
    uint32_t nt = 0;
    typename P::Tile t;
    TC_PROF_VAR(e_wait);
    TC_PROF_VAR(e_store);
    TC_PROF_NOW(e_t0);
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++nt) {
      prob.decode(tile, t);
      const uint32_t acc = nt & 1, around = nt >> 1;
      if (*failed != 0) break;
      TC_PROF_NOW(w0);
      if (!mbar_wait(&tfull_bar[acc], around & 1)) {
        *failed = 3;
        break;
      }
      TC_PROF_ADD(e_wait, w0);
      TC_PROF_NOW(w1);
      tc_fence_after();
      if (*failed != 0) break;
#pragma unroll 1
      for (int c0 = 32 * group; c0 < BN; c0 += 32 * kGroups) {
        if (!prob.chunk_live(t, c0)) continue;  // uniform across the warp; need not be a prefix
        float v[32];
        tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN + (uint32_t)c0, v);
        prob.store(t, row, c0, v, stage, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      TC_PROF_ADD(e_store, w1);
    }
#ifdef FLB200_TC_PROFILE
    if (threadIdx.x == 64) { TC_PROF_PUT(5, e_wait); TC_PROF_PUT(6, e_store); TC_PROF_PUT(7, clock64() - e_t0); }
#endif
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *failed != 0 && status) atomicExch(status, *failed);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------ plain GEMM
// Tiles ordered split-fastest, then n, then m, then batch, so that CTAs running
// together share the (large) A tile through L2.
template <int BN>
struct GemmProblem {
  static constexpr bool kTwoProducers = true;
  static constexpr int kMinBlocks = 1;
  int operand;  // kOperandTf32, or 16-bit (64 elements per stage)
  OperandCoords a, b;
  EpiloguePlan ep;
  int a_mn_major, b_mn_major;
  int M, N, k_iters, splits, iters_per_split;
  int tiles_m, tiles_n, Z;
  int pair_n_fast;  // order of the pair tiles: column tiles of one row pair next to each other
  float* partial;  // split-K scratch [z*splits + s][M][N]

  struct Tile { int m0, n0, z, split, k0, k1; };
  struct Walk { int c[4], lo; };  // coordinates of an operand's first box, stage of the inner k level
  struct LoadState { Walk a, b; };

  __device__ __forceinline__ int num_tiles() const { return tiles_m * tiles_n * Z * splits; }
  __device__ __forceinline__ void decode(int tile, Tile& t) const {
    int r = tile;
    t.split = r % splits; r /= splits;
    t.n0 = (r % tiles_n) * BN; r /= tiles_n;
    t.m0 = (r % tiles_m) * kBM; r /= tiles_m;
    t.z = r;
    t.k0 = t.split * iters_per_split;
    t.k1 = min(t.k0 + iters_per_split, k_iters);
  }
  __device__ __forceinline__ int k_begin(const Tile& t) const { return t.k0; }
  __device__ __forceinline__ int k_end(const Tile& t) const { return t.k1; }
  static __device__ __forceinline__ void walk_begin(const OperandCoords& o, Walk& w, int mn, const Tile& t) {
    const int hi = o.k_inner > 0 ? t.k0 / o.k_inner : 0;
    w.lo = t.k0 - hi * o.k_inner;
    operand_coords(o, mn, w.lo, hi, t.z, w.c);
  }
  // Boxes [first, first + count) of an operand's stage.  A K-major operand is one box, an MN-major one a
  // box per 32 (16-bit: 64) rows, or one copy of them all where the map is grouped.
  template <bool kPair, int kRank, class Bar>
  __device__ __forceinline__ void copy_boxes(const OperandCoords& o, const CUtensorMap* map, Bar bar, char* dst,
                                             const Walk& w, int first, int count) const {
    const int box_mn = operand ? 64 : 32, box_bytes = operand ? 8192 : kBK * 128;
    int c[4];
#pragma unroll
    for (int d = 0; d < kRank; ++d) c[d] = w.c[d] + first * box_mn * o.mn_mul[d];
    dst += first * box_bytes;
    for (int i = 0;;) {
      if constexpr (kPair) tma_load_pair(map, bar, dst, kRank, c);
      else tma_load(map, bar, dst, kRank, c);
      if (++i >= count) break;
      dst += box_bytes;
#pragma unroll
      for (int d = 0; d < kRank; ++d) c[d] += box_mn * o.mn_mul[d];
    }
  }
  template <bool kPair, class Bar>
  __device__ __forceinline__ void walk_load(const OperandCoords& o, const CUtensorMap* map, Bar bar, char* dst,
                                            Walk& w, int first, int count) const {
    if (o.rank == 2) copy_boxes<kPair, 2>(o, map, bar, dst, w, first, count);
    else if (o.rank == 3) copy_boxes<kPair, 3>(o, map, bar, dst, w, first, count);
    else copy_boxes<kPair, 4>(o, map, bar, dst, w, first, count);
#pragma unroll
    for (int d = 0; d < 4; ++d) w.c[d] += o.k_mul[d];
    if (++w.lo == o.k_inner) {
      w.lo = 0;
#pragma unroll
      for (int d = 0; d < 4; ++d) w.c[d] += o.k2_mul[d] - o.k_inner * o.k_mul[d];
    }
  }
  __device__ __forceinline__ int boxes_of(const OperandCoords& o, int rows) const {
    return o.mn_major && !o.mn_shift ? rows / (operand ? 64 : 32) : 1;
  }
  // Of two producers A's takes the last boxes of B where B has more than A.
  template <int kWhich, bool kPair, class Bar>
  __device__ __forceinline__ void load_stage(const CUtensorMap* ma, const CUtensorMap* mb, LoadState& ls, Bar bar,
                                             char* a_dst, char* b_dst, int b_rows) const {
    const int na = boxes_of(a, kBM), nb = boxes_of(b, b_rows);
    const int moved = kWhich == kBoth ? 0 : max(0, (nb - na) >> 1);
    if constexpr (kWhich != kB) walk_load<kPair>(a, ma, bar, a_dst, ls.a, 0, na);
    if (kWhich != kA) walk_load<kPair>(b, mb, bar, b_dst, ls.b, 0, nb - moved);
    else if (moved > 0) walk_load<kPair>(b, mb, bar, b_dst, ls.b, nb - moved, moved);
  }
  template <int kWhich>
  __device__ __forceinline__ void load_begin(const Tile& t, LoadState& ls) const {
    if constexpr (kWhich != kB) walk_begin(a, ls.a, t.m0, t);
    walk_begin(b, ls.b, t.n0, t);
  }
  __device__ __forceinline__ uint32_t stage_bytes(const Tile&) const { return (kBM + BN) * kBK * 4; }
  template <int kWhich>
  __device__ __forceinline__ void load(const CUtensorMap* ma, const CUtensorMap* mb, const Tile&,
                                       LoadState& ls, uint64_t* bar, char* a_dst, char* b_dst) const {
    load_stage<kWhich, false>(ma, mb, ls, bar, a_dst, b_dst, BN);
  }
  // CTA pairs (tc_pair.cuh): the halves of a pair tile are two consecutive 128-row blocks of
  // the same column block, batch and K slice; row blocks run fastest, then splits, columns,
  // batches.  With an odd number of row blocks the last pair has a phantom half past M
  // (zero-filled loads, masked stores).
  __device__ __forceinline__ int num_pair_tiles() const {
    return ((tiles_m + 1) >> 1) * splits * tiles_n * Z;
  }
  __device__ __forceinline__ void decode_pair(int tile, int rank, Tile& t) const {
    const int pairs_m = (tiles_m + 1) >> 1;
    int r = tile;
    if (pair_n_fast) {
      t.n0 = (r % tiles_n) * BN; r /= tiles_n;
      t.split = r % splits; r /= splits;
      t.m0 = (2 * (r % pairs_m) + rank) * kBM; r /= pairs_m;
    } else {
      t.m0 = (2 * (r % pairs_m) + rank) * kBM; r /= pairs_m;
      t.split = r % splits; r /= splits;
      t.n0 = (r % tiles_n) * BN; r /= tiles_n;
    }
    t.z = r;
    t.k0 = t.split * iters_per_split;
    t.k1 = min(t.k0 + iters_per_split, k_iters);
  }
  // this CTA's 128 rows of A and its BN / 2 columns of B
  template <int kWhich>
  __device__ __forceinline__ void load_begin_pair(const Tile& t, LoadState& ls, int rank) const {
    if constexpr (kWhich != kB) walk_begin(a, ls.a, t.m0, t);
    walk_begin(b, ls.b, t.n0 + rank * (BN / 2), t);
  }
  template <int kWhich>
  __device__ __forceinline__ void load_pair(const CUtensorMap* ma, const CUtensorMap* mb, const Tile&,
                                            LoadState& ls, uint32_t full_bar, char* a_dst,
                                            char* b_dst) const {
    load_stage<kWhich, true>(ma, mb, ls, full_bar, a_dst, b_dst, BN / 2);
  }
  __device__ __forceinline__ bool chunk_live(const Tile& t, int c0) const {
    return t.n0 + c0 < N;
  }

  // How store() writes a chunk of 32 whole columns; decided once on the host (see set_store_mode),
  // so that a chunk costs one test and not the chain of them.
  enum {
    kStoreGeneral = 0,  // element offsets of any kind, one row per lane
    kStorePartial,      // split-K partial sums, row-major fp32
    kStoreF32,          // row-major result: + 1 bias_n, + 2 bias_n and gelu, + 3 statistics too
    kStoreF32Bias,
    kStoreF32Gelu,
    kStoreF32Stats,
    kStoreBf16,
    kStoreBf16Bias,
    kStoreBf16Gelu,
    kStoreBf16Stats,
    kStoreF16,
    kStoreF16Bias,
    kStoreF16Gelu,
    kStoreF16Stats,
  };
  int store_mode;

  void set_store_mode() {
    store_mode = kStoreGeneral;
    if (splits > 1) {
      if ((N & 3) == 0) store_mode = kStorePartial;
      return;
    }
    if (ep.beta != 0.f || ep.n_div != 0 || ep.m_div != 0 || ep.n_stride != 1 ||
        ep.bias_m != nullptr || (ep.m_stride & 3) != 0 || (ep.z_stride & 3) != 0 ||
        (reinterpret_cast<uintptr_t>(ep.out) & 15) != 0)
      return;
    const int base = ep.out16 == 0 ? kStoreF32 : (ep.out16 == kOperandBf16 ? kStoreBf16 : kStoreF16);
    store_mode = base + (ep.stats ? 3 : (ep.act ? 2 : (ep.bias_n ? 1 : 0)));
  }

  // The warp's staged 32 x 32 chunk to a row-major output of type T: lane i stores columns
  // 4 (i % 8) .. + 3 of rows 4 k + i / 8, k = 0..7 (whole 128-byte rows of fp32, 64-byte rows of
  // 16-bit values).  All eight reads are issued before the first store; `rows` < 32 only at the
  // ragged end.  MODE 0: the values times alpha; 1: + bias_n; 2: + bias_n, then gelu, the
  // pre-activation kept in ep.pre when that is set; 3: + bias_n, and per-channel sums of the
  // stored values into row `group` of ep.stats.
  template <typename T, int MODE>
  __device__ __forceinline__ void staged_rows(float* stage, int lane, int rows, T* dst, T* pre,
                                              long long ld, int nb, long long group) const {
    float4 bq = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE != 0 && ep.bias_n)
      bq = *reinterpret_cast<const float4*>(ep.bias_n + nb + 4 * (lane & 7));
    float4 val[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) val[k] = epi_stage_read(stage, lane, k);
    EpiStats acc;
    const long long step = 4 * ld;
    const int r0 = lane >> 3;
    if (MODE == 0) {
      if (rows >= 32) {
#pragma unroll
        for (int k = 0; k < 8; ++k, dst += step) epi_store4(dst, val[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k, dst += step)
          if (4 * k + r0 < rows) epi_store4(dst, val[k]);
      }
      return;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k, dst += step) {
      float4 v = val[k];
      v.x += bq.x; v.y += bq.y; v.z += bq.z; v.w += bq.w;
      const bool live = 4 * k + r0 < rows;
      if (MODE == 2) {
        // the activation sees the value that the pre-activation tensor holds (rounded to T)
        v = epi_round<T>(v);
        if (pre) {
          if (live) epi_store4(pre, v);
          pre += step;
        }
        v = make_float4(epi_gelu(v.x), epi_gelu(v.y), epi_gelu(v.z), epi_gelu(v.w));
      }
      if (MODE == 3) {
        v = epi_round<T>(v);
        if (live) acc.add(v);
      }
      if (live) epi_store4(dst, v);
    }
    if (MODE == 3) acc.flush(ep.stats, group, N, nb, lane, stage);
  }
  template <typename T, int MODE>
  __device__ __forceinline__ void staged_result(float* stage, int lane, int m_first, int nb,
                                                const Tile& t) const {
    const long long off = (long long)(m_first + (lane >> 3)) * ep.m_stride +
                          (long long)t.z * ep.z_stride + nb + 4 * (lane & 7);
    T* pre = MODE == 2 && ep.pre ? static_cast<T*>(ep.pre) + off : nullptr;
    staged_rows<T, MODE>(stage, lane, M - m_first, reinterpret_cast<T*>(ep.out) + off, pre,
                         ep.m_stride, nb, m_first >> 5);
  }

  // a row's 32 columns one by one: column tails, strided and accumulating 16-bit results
  template <typename T>
  __device__ __forceinline__ void store_16(long long m_off, int nb, float bm, const float* v) const {
    T* out16 = reinterpret_cast<T*>(ep.out);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int n = nb + j;
      if (n < N) {
        T* dst = out16 + m_off + epi_off(n, ep.n_div, ep.n_stride, ep.n_outer);
        float r = ep.alpha * v[j] + bm + (ep.bias_n ? ep.bias_n[n] : 0.f);
        if (ep.beta != 0.f) r += ep.beta * Num<T>::to_f(*dst);
        *dst = Num<T>::from_f(r);
      }
    }
  }

  __device__ __forceinline__ void store(const Tile& t, int row, int c0, const float* v,
                                        float* stage, int lane) const {
    const int m = t.m0 + row;
    const int nb = t.n0 + c0;
    if (store_mode != kStoreGeneral && nb + 32 <= N) {
      // through the staging tile, whole row segments per store instruction
      const int m_first = m - lane;  // first row of this warp
      if (m_first >= M && store_mode != kStoreF32Stats && store_mode != kStoreBf16Stats &&
          store_mode != kStoreF16Stats)
        return;  // (statistics of a phantom tile are zeros that somebody adds up)
      if (store_mode == kStorePartial || ep.alpha == 1.f) {
        epi_stage_write(stage, lane, v);
      } else {
        float w[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) w[j] = ep.alpha * v[j];
        epi_stage_write(stage, lane, w);
      }
      switch (store_mode) {
        case kStorePartial: {
          float* dst = partial + ((long long)(t.z * splits + t.split) * M + m_first + (lane >> 3)) * N +
                       nb + 4 * (lane & 7);
          staged_rows<float, 0>(stage, lane, M - m_first, dst, nullptr, N, nb, 0);
          break;
        }
        case kStoreF32: staged_result<float, 0>(stage, lane, m_first, nb, t); break;
        case kStoreF32Bias: staged_result<float, 1>(stage, lane, m_first, nb, t); break;
        case kStoreF32Gelu: staged_result<float, 2>(stage, lane, m_first, nb, t); break;
        case kStoreF32Stats: staged_result<float, 3>(stage, lane, m_first, nb, t); break;
        case kStoreBf16: staged_result<__nv_bfloat16, 0>(stage, lane, m_first, nb, t); break;
        case kStoreBf16Bias: staged_result<__nv_bfloat16, 1>(stage, lane, m_first, nb, t); break;
        case kStoreBf16Gelu: staged_result<__nv_bfloat16, 2>(stage, lane, m_first, nb, t); break;
        case kStoreBf16Stats: staged_result<__nv_bfloat16, 3>(stage, lane, m_first, nb, t); break;
        case kStoreF16: staged_result<__half, 0>(stage, lane, m_first, nb, t); break;
        case kStoreF16Bias: staged_result<__half, 1>(stage, lane, m_first, nb, t); break;
        case kStoreF16Gelu: staged_result<__half, 2>(stage, lane, m_first, nb, t); break;
        default: staged_result<__half, 3>(stage, lane, m_first, nb, t); break;
      }
      __syncwarp();  // the tile is rewritten by the next chunk
      return;
    }
    if (m >= M) return;
    if (splits > 1) {
      float* dst = partial + ((long long)(t.z * splits + t.split) * M + m) * N + nb;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (nb + j < N) dst[j] = v[j];
      return;
    }
    if (ep.m_valid != 0 && ep.m_div != 0 && (m % ep.m_div) >= ep.m_valid) return;
    const long long m_off =
        epi_off(m, ep.m_div, ep.m_stride, ep.m_outer) + (long long)t.z * ep.z_stride;
    const float bm = ep.bias_m ? ep.bias_m[m] : 0.f;
    if (ep.out16) {
      if (ep.out16 == kOperandBf16) store_16<__nv_bfloat16>(m_off, nb, bm, v);
      else store_16<__half>(m_off, nb, bm, v);
      return;
    }
    const bool simple = ep.beta == 0.f && ep.n_div == 0;
    if (simple && nb + 32 <= N) {
      // strided columns (convolution output planes): the rows of a warp are contiguous
      float* dst = ep.out + m_off + (long long)nb * ep.n_stride;
      const long long ns = ep.n_stride;
      if (ep.bias_n != nullptr) {
        const float* bn = ep.bias_n + nb;
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[j * ns] = ep.alpha * v[j] + bm + bn[j];
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[j * ns] = ep.alpha * v[j] + bm;
      }
      return;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int n = nb + j;
      if (n < N) {
        float* dst = ep.out + m_off + epi_off(n, ep.n_div, ep.n_stride, ep.n_outer);
        float r = ep.alpha * v[j] + bm + (ep.bias_n ? ep.bias_n[n] : 0.f);
        if (ep.beta != 0.f) r += ep.beta * *dst;
        *dst = r;
      }
    }
  }
};

// ------------------------------------------------------------- host launch
// Launches the persistent kernel for problem P: one CTA per SM (fewer when there are fewer tiles).
template <class P, int BN, int STAGES, int X3, int KSUB = 1>
int launch_problem_as(const char* name, const CUtensorMap& ma, const CUtensorMap& mb, const P& prob,
                      long long tiles, cudaStream_t st) {
  using SL = SmemLayout<BN, STAGES, X3>;
  static bool configured[64] = {false};
  int dev = 0;
  FLB200_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    FLB200_CUDA_CHECK(cudaFuncSetAttribute(tc_persistent_kernel<P, BN, STAGES, X3, KSUB>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           SL::kTotal));
    configured[dev] = true;
  }
  const long long sms = device_info().sm_count;
  const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
  launch_chained(tc_persistent_kernel<P, BN, STAGES, X3, KSUB>, grid, threads_for<P, X3, BN>(), SL::kTotal, st,
                 ma, mb, prob, status_ptr());
  FLB200_AFTER_LAUNCH(name);
  count_tc_launch();
#ifdef FLB200_TC_PROFILE
  {
    cudaStreamSynchronize(st);
    static long long h[256 * 8];
    cudaMemcpyFromSymbol(h, g_tc_profile, sizeof(h));
    double a[8] = {0};
    for (unsigned c = 0; c < grid && c < 256; ++c)
      for (int i = 0; i < 8; ++i) a[i] += (double)h[c * 8 + i] / (grid < 256 ? grid : 256);
    fprintf(stderr,
            "tc profile %s BN=%d stages=%d ksub=%d tiles=%lld grid=%u | producer wait %.0f of %.0f | "
            "mma wait full %.0f, accumulator %.0f of %.0f | epilogue wait %.0f, store %.0f of %.0f "
            "(mean clocks per CTA)\n",
            name, BN, STAGES, KSUB, tiles, grid, a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
  }
#endif
  return FLB200_OK;
}

template <class P, int BN>
int launch_problem(const char* name, const CUtensorMap& ma, const CUtensorMap& mb, const P& prob,
                   long long tiles, cudaStream_t st) {
  if (tiles <= 0) return FLB200_OK;
  if (x3_enabled())
    return launch_problem_as<P, BN, stages_for_x3(BN), 1>(name, ma, mb, prob, tiles, st);
  // Narrow tiles hand the ring over in groups of two sub-stages (measured 5-10 % faster than
  // single sub-stages, no further gain from four); 256-column tiles keep four single stages.
  constexpr int kS = stages_for(BN);
  if constexpr (BN <= 128)
    return launch_problem_as<P, BN, kS, 0, 2>(name, ma, mb, prob, tiles, st);
  else
    return launch_problem_as<P, BN, kS, 0, 1>(name, ma, mb, prob, tiles, st);
}

}  // namespace tc
}  // namespace flb200
