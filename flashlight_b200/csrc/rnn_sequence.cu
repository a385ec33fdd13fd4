// The recurrence of a layer as one persistent kernel: all T steps, with the recurrent weights
// resident in tensor memory and shared memory, and both directions (or several parts of a large batch) side by side
// as jobs of one launch where the device holds them.
//
// What bounds a step is latency: between two steps every unit's new state has to reach all CTAs.
// The states travel without barriers, fences or counters: each one is a 4-byte word of an exchange
// buffer whose low 13 bits, which a TF32 operand does not use, carry the step's number, and a reader
// looks at the words themselves.  A word is complete the moment it is visible, so a step costs one
// write to L2 and one read back.  Two slots, used in turn, are enough: a CTA can only be asked to write
// step s + 2 once everybody has consumed step s, which the data dependence itself ensures (each state
// needs all states of the step before).
//
// Both directions of a 1024-unit LSTM are 32 MB of weights, as much as the shared memory of all SMs; of a CTA's
// 16 k tiles 8 (forward) or 12 (backward) lie in tensor memory instead, beside the accumulators, as the A
// operand of the MMAs, which is also the faster place to read them from.  So they run side by side: 32 rows of the batch take 4.4 us per step forward and 5.1 backward,
// where one direction after the other took 2 x 3.9 and 2 x 6.6 (weights in shared memory only, words
// fetched by the threads that polled them, the backward pass with a second exchange through L2 for its
// partial sums).  Of a backward step of 9600 clocks about 1000 are the cell gradient, 1700 until its words
// are seen by others (a round trip to L2 takes 900), 3000 the copy of 128 KB per SM, 1500 what the MMAs
// lag behind, 1400 the sums' way through the cluster, 700 memory the passes before and after need.
//
// All CTAs of a launch must be resident at once; the host asks the occupancy calculator and launches
// fewer jobs at a time, or a kernel per step, where they are not.  Every wait is bounded by a clock
// budget: on expiry (or once the device status flag is seen raised by anybody) a CTA leaves its loop
// over the steps, and the host reports FLB200_TIMEOUT.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "rnn_sequence.cuh"
#include "rnn_step.cuh"
#include "tc_core.cuh"
#include "tc_gemm.cuh"

namespace flb200 {
namespace {

using namespace tc;

constexpr int kMaxJobs = 4;                 // jobs of one launch
constexpr int kABytes = kBM * kBK * 4;      // 16 KB: one 32-wide k tile of the weights
constexpr int kWorkers = 8;                 // warps that bring tiles, move sums and update states
constexpr int kWorkThreads = 32 * kWorkers;
constexpr int kMaxTiles = 2 * kWorkers;     // k tiles a CTA keeps at most
constexpr int kIssuers = 2;                 // warps that only issue MMAs, of every other k tile
constexpr int kSeqThreads = kWorkThreads + 32 * kIssuers;
constexpr int kTmemColumns = 512;
constexpr uint32_t kTagMask = 0x1fff;       // bits of an fp32 word that a TF32 operand ignores
constexpr int kUnits = 32;                  // hidden units of a forward cluster

__device__ __forceinline__ float sigmoid_(float v) { return 1.f / (1.f + expf(-v)); }
__device__ __forceinline__ uint4 ld_relaxed_v4(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_volatile_i32(const int* p) {
  int v;
  asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// four floats into the shared memory of a CTA of the cluster, counted by its barrier
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, float a, float b, float c,
                                            float d) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
          addr),
      "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool is_tagged(const uint4& v, uint32_t tag) {
  return (((v.x ^ tag) | (v.y ^ tag) | (v.z ^ tag) | (v.w ^ tag)) & kTagMask) == 0;
}

struct Waits {
  volatile int* failed;  // in shared memory; once set nobody in the CTA waits any more
  int* status;
  long long budget;
  // every 64 unsuccessful polls: whether to give up
  __device__ bool expired(int* spins, long long t0, int code) const {
    if ((++*spins & 63) != 0) return false;
    if (*failed == 0 && clock64() - t0 <= budget && ld_volatile_i32(status) == 0) return false;
    *failed = 1;
    atomicExch(status, code);
    return true;
  }
  // a barrier that this CTA, or (acquire at cluster scope) its cluster, completes
  template <bool kCluster>
  __device__ bool bar(uint64_t* b, uint32_t parity) const {
    if (kCluster ? mbar_try_wait_cluster(b, parity) : mbar_try_wait(b, parity)) return true;
    if (*failed) return false;
    int spins = 0;
    const long long t0 = clock64();
    while (!(kCluster ? mbar_try_wait_cluster(b, parity) : mbar_try_wait(b, parity)))
      if (expired(&spins, t0, 12)) return false;
    return true;
  }
  // the same for a whole warp: its lanes stay together when a wait runs out
  template <bool kCluster>
  __device__ bool warp_bar(uint64_t* b, uint32_t parity) const {
    return __all_sync(0xffffffffu, bar<kCluster>(b, parity));
  }
  __device__ bool warp_goes_on() const { return !__any_sync(0xffffffffu, *failed != 0); }
};

// Where a worker warp finds its k tiles of a step in the exchange buffer, and where they go.
struct Feed {
  const CUtensorMap* map;  // [2 slots][B][K] tagged words, box [1][NB][32]
  const uint32_t* x;       // the same
  char* b_tiles;
  uint64_t* tile_bar;      // [stages]: the copy of a tile has arrived
  uint64_t* full_bar;      // [stages]: it is whole, too
  long long K;
  int B, stages;
  int k0, sub;             // first word of this warp's first tile; from one of its P parts to the next
  uint32_t phases;         // of its tile_bars
};
// Brings this warp's tiles (warp and warp + 8) of one step: P parts of NB rows of 32 words each, in shared
// memory as the 128-byte swizzle that the UMMA descriptor expects.  A lane polls one chunk of four rows;
// when a tile's samples carry the step's number, all of it most likely does, and one lane has it copied by
// TMA (64 KB take 1600 clocks per SM; loads by the threads 2100 to 2400, and a round too early costs as
// much again).  Then every word is checked in shared memory, and a tile with a stale one copied again.
// The tag stays in the operand: the tensor core does not read those bits.  meanwhile() runs while the
// second tile, or the MMAs of the first, are in flight (before the first and after the second it costs 0.1
// to 0.8 us a step).
// kWhole: tiles whose words past the batch's rows and past K are zeros from the start; of up to eight rows they are
// stored by the lanes that polled them, without the copy and the second look at every word.  (One row of 1024
// units, 40 steps forward: 172 us by copies, 136 so; eight rows of a 320-unit GRU 114; nine rows are copied, 138.
// The backward pass, whose tiles start undefined, copies.)
template <bool kWhole, int P, int NB, typename Meanwhile>
__device__ __forceinline__ void bring_tiles(Feed& f, int slot, uint32_t tag, int warp, int lane,
                                            const Waits& w, int code, Meanwhile&& meanwhile) {
  constexpr int kTiles = kMaxTiles / kWorkers, kStep = kWorkers * kBK, kBytes = P * NB * 128;
  // kWhole, up to eight rows: the samples are all there is, and they are stored from where they are
  constexpr int kLoads = kTiles * P, kSets = kWhole ? 2 : 1;
  const bool direct = kWhole && f.B <= 4 * kSets;
  const int q = 4 * (lane & 7), row = (lane >> 3) * (direct ? 1 : (f.B + 3) / 4);
  const uint32_t* from = f.x + ((long long)slot * f.B + row) * f.K + f.k0 + q;
  auto copy = [&](int i) {
    const int s = warp + i * kWorkers;
    if (lane == 0) {
      asm volatile("fence.proxy.async.global;" ::: "memory");  // what the polls have seen, before the copy reads
      mbar_expect_tx(&f.tile_bar[s], kBytes);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        int c[3] = {f.k0 + i * kStep + p * f.sub, 0, slot};
        tma_load(f.map, &f.tile_bar[s], f.b_tiles + s * kBytes + p * (NB * 128), 3, c);
      }
    }
    __syncwarp();
  };
  uint32_t pending = 0, to_copy = 0;
  uint4 v[kSets * kLoads];  // the second set: four rows further down
#pragma unroll
  for (int i = 0; i < kTiles; ++i) {
    if (warp + i * kWorkers < f.stages) to_copy |= 1u << i;
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int h = 0; h < kSets; ++h)
        if (warp + i * kWorkers < f.stages && row + 4 * h < f.B && (h == 0 || direct) &&
            f.k0 + q + i * kStep + p * f.sub < f.K)
          pending |= 1u << (h * kLoads + i * P + p);
  }
  const uint32_t mine = to_copy, chunks = pending;
  int spins = 0;
  long long t0 = clock64();
  while (to_copy && w.warp_goes_on()) {
#pragma unroll
    for (int u = 0; u < kSets * kLoads; ++u)
      if (pending >> u & 1)
        v[u] = ld_relaxed_v4(from + (u / kLoads) * 4 * f.K + (u % kLoads / P) * kStep + (u % P) * f.sub);
#pragma unroll
    for (int u = 0; u < kSets * kLoads; ++u)
      if ((pending >> u & 1) && is_tagged(v[u], tag)) pending &= ~(1u << u);
#pragma unroll
    for (int i = 0; i < kTiles; ++i)
      if ((to_copy >> i & 1) && !__any_sync(0xffffffffu, (pending | pending >> kLoads) >> (i * P) & ((1u << P) - 1))) {
        if (direct) {
          const int s = warp + i * kWorkers;
#pragma unroll
          for (int u = 0; u < kSets * P; ++u) {
            const int h = u / P, p = u % P, b = row + 4 * h;
            if (chunks >> (h * kLoads + i * P + p) & 1)
              *reinterpret_cast<uint4*>(f.b_tiles + s * kBytes + p * (NB * 128) + b * 128 +
                                        (((lane & 7) ^ (b & 7)) << 4)) = v[h * kLoads + i * P + p];
          }
          fence_proxy_async();  // every lane's stores, before the MMAs read
          __syncwarp();
          if (lane == 0) mbar_arrive(&f.full_bar[s]);
        } else {
          copy(i);
        }
        to_copy &= ~(1u << i);
      }
    if (to_copy) w.expired(&spins, t0, code);
  }
  if (direct) {
#pragma unroll
    for (int i = 0; i < kTiles; ++i)  // (a wait ran out)
      if ((to_copy >> i & 1) && lane == 0) mbar_arrive(&f.full_bar[warp + i * kWorkers]);
    __syncwarp();
    meanwhile();
    return;
  }
  spins = 0;
  t0 = clock64();
#pragma unroll
  for (int i = 0; i < kTiles; ++i) {
    if (i == 1) meanwhile();
    if (!(mine >> i & 1)) continue;
    const int s = warp + i * kWorkers;
    for (;;) {
      if (!w.warp_bar<false>(&f.tile_bar[s], f.phases >> i & 1)) break;
      f.phases ^= 1u << i;
      bool whole = true;
#pragma unroll
      for (int u = 0; u < P * NB / 4; ++u) {
        const int p = u / (NB / 4), b = (lane >> 3) + 4 * (u % (NB / 4));
        const uint4 v = *reinterpret_cast<const uint4*>(f.b_tiles + s * kBytes + p * (NB * 128) + b * 128 +
                                                        (((lane & 7) ^ (b & 7)) << 4));
        if (b < f.B && f.k0 + q + i * kStep + p * f.sub < f.K) whole &= is_tagged(v, tag);
      }
      if (__all_sync(0xffffffffu, whole)) break;
      w.expired(&spins, t0, code);
      if (!w.warp_goes_on()) break;
      copy(i);
    }
    if (lane == 0) mbar_arrive(&f.full_bar[s]);
    __syncwarp();
  }
}
__device__ __forceinline__ uint32_t tagged(float v, uint32_t tag) {
  return (__float_as_uint(v) & ~kTagMask) | tag;
}

// Tensor memory: an accumulator per issuing warp, and k tiles of the weights: the A operand of an MMA may
// be in tensor memory, a lane per row, a column per k (K-major, 32 bits each).
__device__ __forceinline__ void umma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The MMAs of one k tile.  s: its place among the CTA's tiles, the first `in_smem` of which are in shared
// memory (a_desc0), the others in tensor memory from column a_tmem on.
template <bool kAMajorMn, int N>
__device__ __forceinline__ void issue_tile(uint32_t d, uint64_t a_desc0, uint32_t a_tmem, int in_smem,
                                           uint64_t b_desc0, int s, bool first) {
  const uint64_t b_desc = umma_desc_advance(b_desc0, s * N * 128);
  tc_fence_after();
  if (s < in_smem) {
    const uint32_t idesc = umma_idesc_tf32(N, kAMajorMn ? 1 : 0, 0);
    const uint64_t a_desc = umma_desc_advance(a_desc0, s * kABytes);
#pragma unroll
    for (int j = 0; j < kBK / kUmmaK; ++j)
      umma_tf32(d, umma_desc_advance(a_desc, j * (kAMajorMn ? 1024 : 32)), umma_desc_advance(b_desc, j * 32),
                idesc, first && j == 0 ? 0u : 1u);
  } else {
    const uint32_t idesc = umma_idesc_tf32(N, 0, 0);
    const uint32_t at = a_tmem + (uint32_t)((s - in_smem) * kBK);
#pragma unroll
    for (int j = 0; j < kBK / kUmmaK; ++j)
      umma_tf32_ts(d, at + j * kUmmaK, umma_desc_advance(b_desc, j * 32), idesc, first && j == 0 ? 0u : 1u);
  }
}
// 8 columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_st8(uint32_t addr, const float* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
               "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
               : "memory");
}
// All MMAs of one step, by one lane of an issuing warp: of every kIssuers-th tile as it becomes whole, tile s
// into accumulator s % accs (a power of two, at least kIssuers).
template <bool kAMajorMn, int N>
__device__ __forceinline__ bool issue_step(uint32_t d, uint32_t acc_stride, int accs, uint64_t a_desc0, uint32_t a_tmem, int in_smem,
                                           uint64_t b_desc0, int first, int stages, uint32_t parity,
                                           uint64_t* full_bar, uint64_t* done_bar, const Waits& w) {
  for (int s = first; s < stages; s += kIssuers) {
    if (!w.bar<false>(&full_bar[s], parity)) return false;
    issue_tile<kAMajorMn, N>(d + (uint32_t)(s & (accs - 1)) * acc_stride, a_desc0, a_tmem, in_smem, b_desc0, s,
                             s < accs);
  }
  umma_commit(done_bar);
  return true;
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld_async(uint32_t addr, uint32_t* r) {
  static_assert(N == 8 || N == 16, "");
  if constexpr (N == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(addr)
                 : "memory");
  else
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
        "%13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15])
        : "r"(addr)
        : "memory");
}
// N columns of this warp's rows: `accs` accumulators kStride columns apart, added in order.  Four are loaded
// together: eight take registers that the states of the batch need.
template <uint32_t kStride, int N>
__device__ __forceinline__ void read_sums(uint32_t at, int accs, float* v) {
  constexpr int kTogether = 4;
#pragma unroll
  for (int q0 = 0; q0 < kRnnAccs; q0 += kTogether) {
    if (q0 >= accs) break;
    uint32_t r[kTogether][N];
#pragma unroll
    for (int q = 0; q < kTogether; ++q)
      if (q0 + q < accs) tmem_ld_async<N>(at + (q0 + q) * kStride, r[q]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < kTogether; ++q) {
#pragma unroll
      for (int j = 0; j < N; ++j) asm volatile("" : "+r"(r[q][j]));  // read only after the wait
      if (q0 + q < accs) {
#pragma unroll
        for (int j = 0; j < N; ++j)
          v[j] = q0 + q == 0 ? __uint_as_float(r[0][j]) : v[j] + __uint_as_float(r[q][j]);
      }
    }
  }
}

template <typename Job>
struct Launch {
  CUtensorMap map[kMaxJobs];   // W_hh
  CUtensorMap xmap[kMaxJobs];  // xch
  Job job[kMaxJobs];
  uint32_t* xch[kMaxJobs];  // tagged states: [2][B][H], backward: gate gradients [2][B][G*H]
  int* status;
  long long wait_budget;
  long long out_stride, dy_stride;
  int T, B_total, H, act;
  int slice;    // states / gate rows of a CTA's k slice
  int stages;   // k tiles of a CTA, of 32 states or of P x 32 gate rows
  int in_smem;  // those whose weights are in shared memory; the others' are in tensor memory
  int accs;     // accumulators, of every accs-th k tile each
  int ctas;     // of one job
  int absent_cta;
};

// Shared memory: weights [in_smem][16 KB], states [stages][P * NB x 128 bytes], two slots of received
// partial sums, barriers.  Never less than half of an SM's: two CTAs of one SM would wait for each other's
// tensor memory.
// Received, forward: [KS][G][NB / 4][32 / KS units][4 rows of the batch].  Backward: [8 pieces of the gate rows]
// [NB / 4][outputs of the CTA][4].
template <int G, int NB>
struct Recv { static constexpr int kFloats = kUnits * G * NB; };
constexpr size_t kMostSmem = 227 * 1024;
constexpr size_t kSeqExtra = 512 + 1024;  // barriers, alignment
inline size_t seq_smem(int in_smem, int stages, int cols, int recv) {
  const size_t need = (size_t)in_smem * kABytes + (size_t)stages * cols * 128 + (size_t)2 * recv * 4 + kSeqExtra;
  return std::max(need, (size_t)120 * 1024);
}

// ---------------------------------------------------------------------------------- forward
//   pre[b][g*H + j] = gates[t][b][g*H + j] + sum_k W_hh[g*H + j][k] * h_{t-1}[b][k]
// A cluster owns 32 hidden units, all gates of them = up to 128 rows of one UMMA tile (gate-major;
// the rows of absent gates are zeros); its KS CTAs split K = H into slices of at most 256, or 512 with the
// weights of half the tiles in tensor memory.  Worker s brings the 32 states of k tile s (and of s + 8), two
// warps issue the MMAs (M = 128, N = batch), each of every other tile; tiles s and s + 8 share an accumulator.  The
// workers push the partial sums of each unit from tensor memory straight into the shared memory of the CTA
// that updates it (st.async: one trip, no cluster barrier), and every thread updates the same (unit,
// batch) pairs in all steps, with the cell state in a register.  What a step leaves for the backward pass is
// stored, and the next step's input projections are loaded, while its successor's tiles are in flight.
//
// Every worker counts for done_bar and for the received sums, whether or not it has a tile, row or pair to
// care for: one that only followed could fall behind by two phases and miss one, and a CTA's pushes of step
// s + 1 say that all its threads have read what they were sent in step s.
template <int KS, int G, int NB>
__global__ void __launch_bounds__(kSeqThreads, 1)
rnn_sequence_kernel(const __grid_constant__ Launch<SeqJob> a) {
  constexpr int kOwn = kUnits / KS;  // units this CTA updates
  constexpr int kHalf = NB / 2, kChunk = NB == 32 ? 16 : 8;
  constexpr uint32_t kAccStride = (NB + 31) / 32 * 32;
  constexpr int kItems = (kOwn * NB + kWorkThreads - 1) / kWorkThreads;
  extern __shared__ char smem_raw[];
  char* tiles = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const int stages = a.stages, in_smem = a.in_smem;
  char* a_tiles = tiles;
  char* b_tiles = tiles + in_smem * kABytes;
  float* recv = reinterpret_cast<float*>(b_tiles + stages * NB * 128);
  uint64_t* w_bar = reinterpret_cast<uint64_t*>(recv + 2 * Recv<G, NB>::kFloats);
  uint64_t* done_bar = w_bar + 1;
  uint64_t* recv_bar = done_bar + 1;         // [2]
  uint64_t* tile_bar = recv_bar + 2;         // [kMaxTiles]
  uint64_t* full_bar = tile_bar + kMaxTiles; // [kMaxTiles]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_bar + kMaxTiles);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int ji = blockIdx.x / a.ctas, cta = blockIdx.x - ji * a.ctas;
  const int group = cta / KS;
  const SeqJob& job = a.job[ji];
  const int H = a.H, B = job.B;
  const Waits waits{failed, a.status, a.wait_budget};

  if (threadIdx.x == 0) {
    mbar_init(w_bar, 1);
    mbar_init(done_bar, min(stages, kIssuers) + kWorkers);
    mbar_init(&recv_bar[0], 1 + kWorkers);  // the byte count's, the workers'
    mbar_init(&recv_bar[1], 1 + kWorkers);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&tile_bar[s], 1);
      mbar_init(&full_bar[s], 1);
    }
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemColumns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, a_tmem = tmem_base + a.accs * kAccStride;

  if (warp == 0) {  // the resident slice of W_hh
    if (lane == 0) mbar_expect_tx(w_bar, in_smem * G * (32 * 128));
    __syncwarp();
    for (int i = lane; i < in_smem * G; i += 32) {
      const int s = i / G, g = i - s * G;
      int c[2] = {rank * a.slice + s * kBK, g * H + group * kUnits};
      tma_load(&a.map[ji], w_bar, a_tiles + s * kABytes + g * (32 * 128), 2, c);
    }
  }
  if (G < 4) {  // rows 32 G .. 127 of every k tile belong to no gate
    constexpr int kPerStage = (4 - G) * (32 * 128 / 16);
    for (int i = threadIdx.x; i < in_smem * kPerStage; i += kSeqThreads) {
      const int s = i / (kPerStage > 0 ? kPerStage : 1), rem = i - s * kPerStage;
      *reinterpret_cast<float4*>(a_tiles + s * kABytes + G * (32 * 128) + rem * 16) =
          make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  // the tiles in tensor memory: this warp's 32 rows are the units of gate (warp & 3)
  if (warp < kWorkers && in_smem < stages) {
    const int g = warp & 3, unit = group * kUnits + lane;
    for (int s = in_smem + (warp >> 2); s < stages; s += 2) {
      const int k0 = rank * a.slice + s * kBK;
      const float* wp = job.w_hh + ((long long)g * H + unit) * H + k0;
#pragma unroll
      for (int c = 0; c < kBK; c += 8) {
        float v[8];
#pragma unroll
        for (int h = 0; h < 8; h += 4) {  // H is a multiple of 4
          const float4 x = g < G && unit < H && k0 + c + h < H ? *reinterpret_cast<const float4*>(wp + c + h)
                                                               : make_float4(0.f, 0.f, 0.f, 0.f);
          v[h] = x.x; v[h + 1] = x.y; v[h + 2] = x.z; v[h + 3] = x.w;
        }
        tmem_st8(a_tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((s - in_smem) * kBK + c), v);
      }
    }
    tmem_st_wait();
    tc_fence_before();
  }
  // the initial states, zeros past the end
  for (int i = threadIdx.x; i < stages * NB * 8; i += kSeqThreads) {
    const int s = i / (NB * 8), b = i / 8 % NB, k = rank * a.slice + s * kBK + 4 * (i & 7);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (b < B && k < H) {
      const float* hp = job.h0 + (long long)b * H + k;
      v = make_float4(hp[0], hp[1], hp[2], hp[3]);
    }
    *reinterpret_cast<float4*>(b_tiles + s * (NB * 128) + b * 128 + (((i & 7) ^ (b & 7)) << 4)) = v;
  }
  fence_proxy_async();
  if (threadIdx.x == 0) waits.bar<false>(w_bar, 0);
  __syncthreads();
  cluster_sync_all();  // every peer's barriers are initialised before anybody pushes

  if (warp >= kWorkers) {
    const int q = warp - kWorkers;
    if (q < stages && elect_one()) {
      const uint64_t a_desc0 = umma_desc(smem_u32(a_tiles), 16, 1024, 2);
      const uint64_t b_desc0 = umma_desc(smem_u32(b_tiles), 16, 1024, 2);
      for (int step = 0; step < a.T; ++step)
        if (!issue_step<false, NB>(tmem_base, kAccStride, a.accs, a_desc0, a_tmem, in_smem, b_desc0, q, stages,
                                   step & 1, full_bar, done_bar, waits))
          break;
    }
    __syncwarp();
  } else {
    int item_b[kItems], item_u[kItems];
    float state[kItems], b_hn[kItems];  // LSTM: c; GRU: h and the candidate's bias
    // this warp's with a row of the batch
    const int items = min(kItems, max(0, (B * kOwn - warp * 32 + kWorkThreads - 1) / kWorkThreads));
    bool live[kItems];
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      const int idx = threadIdx.x + it * kWorkThreads;
      item_b[it] = idx / kOwn;
      item_u[it] = idx - item_b[it] * kOwn;
      const int j = group * kUnits + rank * kOwn + item_u[it];
      live[it] = item_b[it] < B && j < H;
      state[it] = live[it] && G != 1 ? (G == 4 ? job.c0 : job.h0)[(long long)item_b[it] * H + j] : 0.f;
      b_hn[it] = live[it] && G == 3 ? job.b_hn[j] : 0.f;
    }
    Feed feed{&a.xmap[ji], a.xch[ji], b_tiles, tile_bar, full_bar, H, B, stages, rank * a.slice + warp * kBK, 0, 0};
    // this lane's row of the accumulator goes to the CTA that owns unit `lane`
    const int owner = lane / kOwn;
    const int quads = (B + 3) / 4;
    const uint32_t push_at = mapa_u32(
        smem_u32(recv) + (uint32_t)((((rank * G + (warp & 3)) * (NB / 4)) * kOwn + lane - owner * kOwn) * 16),
        (uint32_t)owner);
    const uint32_t push_bar = mapa_u32(smem_u32(recv_bar), (uint32_t)owner);
    const uint32_t recv_bytes = (uint32_t)(kUnits * G * quads * 16);

    // left by the step before: the activated gates (LSTM i f g o, GRU r z n, else h), h, cell state or q
    constexpr int kLeft = G == 1 ? 1 : G + 2;
    float left[kItems][kLeft], gin[kItems][G] = {};
    auto store_left = [&](int step) {
      const int t = job.reverse ? a.T - 1 - step : step;
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const int j = group * kUnits + rank * kOwn + item_u[it];
        const long long row = (long long)t * a.B_total + item_b[it];
        float* gp = job.gates + row * G * H + j;
#pragma unroll
        for (int g = 0; g < G; ++g) gp[(long long)g * H] = left[it][g];
        job.out[row * a.out_stride + j] = left[it][G == 1 ? 0 : G];
        if constexpr (G != 1) job.cells[row * H + j] = left[it][G + 1];
      }
    };
    auto load_gates = [&](int step) {
      const int t = job.reverse ? a.T - 1 - step : step;
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const float* gp = job.gates + ((long long)t * a.B_total + item_b[it]) * G * H + group * kUnits +
                          rank * kOwn + item_u[it];
#pragma unroll
        for (int g = 0; g < G; ++g) gin[it][g] = __ldcg(gp + (long long)g * H);
      }
    };

    int step = 0;
    for (; step < a.T && waits.warp_goes_on(); ++step) {
      const int slot = step & 1;
      if (threadIdx.x == 0) mbar_expect_tx(&recv_bar[slot], recv_bytes);
      if (step == 0) {
        for (int s = warp; s < stages; s += kWorkers)
          if (lane == 0) mbar_arrive(&full_bar[s]);
        load_gates(0);
      } else {
        // h of the step before, published with its step number
        bring_tiles<true, 1, NB>(feed, slot ^ 1, (uint32_t)step & kTagMask, warp, lane, waits, 13, [&] {
          store_left(step - 1);
          load_gates(step);
        });
      }
      if (lane == 0) mbar_arrive(done_bar);
      // (the accumulators are free: every worker has read the last step's sums before recv_bar was complete)
      if (waits.warp_bar<false>(done_bar, step & 1) && (warp & 3) < G) {
        tc_fence_after();
        const uint32_t at = push_at + (uint32_t)(slot * Recv<G, NB>::kFloats * 4);
        const uint32_t bar = push_bar + (uint32_t)(slot * 8);
#pragma unroll
        for (int i = 0; i < kHalf; i += kChunk) {
          const int c0 = (warp >> 2) * kHalf + i;  // warps w and w + 4 share the rows of tensor memory
          float v[kChunk];
          read_sums<kAccStride, kChunk>(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c0,
                                                  min(stages, a.accs), v);
#pragma unroll
          for (int j = 0; j < kChunk / 4; ++j)
            if (c0 / 4 + j < quads)
              st_async_v4(at + (uint32_t)((c0 / 4 + j) * (kOwn * 16)), bar, v[4 * j], v[4 * j + 1],
                          v[4 * j + 2], v[4 * j + 3]);
        }
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&recv_bar[slot]);
      if (!waits.warp_bar<true>(&recv_bar[slot], (step >> 1) & 1)) break;
      const float* rp = recv + slot * Recv<G, NB>::kFloats;
      uint32_t* h_x = a.xch[ji] + (long long)slot * B * H + group * kUnits + rank * kOwn;
      const uint32_t tag = (uint32_t)(step + 1) & kTagMask;
      auto update = [&](int it) {
        const int b = item_b[it], u = item_u[it];
        float pre[G];
#pragma unroll
        for (int g = 0; g < G; ++g) pre[g] = 0.f;
#pragma unroll
        for (int q = 0; q < KS; ++q)  // slices of 256: the order of lstm_step_kernel, the same bits
#pragma unroll
          for (int g = 0; g < G; ++g) pre[g] += rp[(((q * G + g) * (NB / 4) + (b >> 2)) * kOwn + u) * 4 + (b & 3)];
        float h;
        if constexpr (G == 4) {
          const float i = sigmoid_(pre[0] + gin[it][0]), f = sigmoid_(pre[1] + gin[it][1]);
          const float gg = tanhf(pre[2] + gin[it][2]), o = sigmoid_(pre[3] + gin[it][3]);
          const float c = f * state[it] + i * gg;
          state[it] = c;
          h = o * tanhf(c);
          left[it][0] = i; left[it][1] = f; left[it][2] = gg; left[it][3] = o; left[it][4] = h; left[it][5] = c;
        } else if constexpr (G == 1) {
          const float v = pre[0] + gin[it][0];
          h = a.act == 0 ? fmaxf(v, 0.f) : tanhf(v);
          left[it][0] = h;
        } else {
          const float r = sigmoid_(pre[0] + gin[it][0]), z = sigmoid_(pre[1] + gin[it][1]);
          const float q = pre[2] + b_hn[it];
          const float n = tanhf(gin[it][2] + r * q);
          h = (1.f - z) * n + z * state[it];
          state[it] = h;
          left[it][0] = r; left[it][1] = z; left[it][2] = n; left[it][3] = h; left[it][4] = q;
        }
        if (live[it] && cta != a.absent_cta) st_relaxed_u32(h_x + (long long)b * H + u, tagged(h, tag));
      };
      if (items == kItems) {  // the arithmetic of the pairs side by side
#pragma unroll
        for (int it = 0; it < kItems; ++it) update(it);
      } else {
#pragma unroll
        for (int it = 0; it < kItems; ++it)
          if (it < items) update(it);
      }
    }
    if (step > 0 && step == a.T) store_left(step - 1);
  }
  __syncthreads();
  if (*failed)  // what was copied or pushed, and the MMAs issued, before a wait ran out have ended after this
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {
    }
  cluster_sync_all();  // nobody leaves while a peer may still push into its shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemColumns);
  }
}

// --------------------------------------------------------------------------------- backward
//   dgates_t          = cell gradient of (dh_t + dy_t, dc_t)          (element-wise)
//   dh_{t-1}[b][k]    = sum_r dgates_t[b][r] * W_hh[r][k]             (r over the G*H gate rows)
// A cluster owns kOut = 128 / P of the H outputs k; its KC CTAs split the gate rows into slices, and each
// slice into P parts.  The 128 rows of a CTA's UMMA tile are (part, output), its P * NB columns (part,
// batch row): the blocks in which the two parts differ are computed and ignored (the time of an MMA of 32 or
// 64 columns is the reading of its A operand).  A CTA keeps its block of W_hh for all steps, in shared memory
// read straight from the forward weights as an MN-major operand (the output index k is the contiguous one),
// what does not fit there in tensor memory.  Per step: the thread that owns a (batch, unit) pair computes its
// dgates and publishes them as tagged words; tiles, MMAs and barriers as in the forward kernel; the sums go
// by st.async to the CTA of the cluster that
// finishes the output, where one thread adds them in slice order and runs the cell gradient of the
// next step (dh and dc of its pairs stay in registers).  So a step is one exchange through L2 and one
// inside the cluster.
template <int KC, int P, int G, int NB>
__global__ void __launch_bounds__(kSeqThreads, 1)
rnn_sequence_backward_kernel(const __grid_constant__ Launch<SeqBwdJob> a) {
  constexpr int kOut = kBM / P, kOwn = kOut / KC;  // outputs of the cluster, of this CTA
  constexpr int kCols = P * NB;                    // columns of an accumulator
  constexpr uint32_t kAccStride = (kCols + 31) / 32 * 32;
  constexpr int kItems = (kOwn * NB + kWorkThreads - 1) / kWorkThreads;
  constexpr int kRecv = kBM * NB;  // floats that a CTA receives per step: KC * P sums per pair
  extern __shared__ char smem_raw[];
  char* tiles = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const int stages = a.stages, in_smem = a.in_smem, sub = a.slice / P;
  char* a_tiles = tiles;
  char* b_tiles = tiles + in_smem * kABytes;
  float* recv = reinterpret_cast<float*>(b_tiles + stages * kCols * 128);
  uint64_t* w_bar = reinterpret_cast<uint64_t*>(recv + 2 * kRecv);
  uint64_t* done_bar = w_bar + 1;
  uint64_t* recv_bar = done_bar + 1;     // [2]
  uint64_t* tile_bar = recv_bar + 2;     // [kMaxTiles]
  uint64_t* full_bar = tile_bar + kMaxTiles;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_bar + kMaxTiles);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int ji = blockIdx.x / a.ctas, cta = blockIdx.x - ji * a.ctas;
  const int rank = (int)cluster_ctarank();
  const int group = cta / KC;
  const SeqBwdJob& job = a.job[ji];
  const int H = a.H, B = job.B, GH = G * H;
  const Waits waits{failed, a.status, a.wait_budget};

  if (threadIdx.x == 0) {
    mbar_init(w_bar, 1);
    mbar_init(done_bar, min(stages, kIssuers) + kWorkers);
    mbar_init(&recv_bar[0], 1 + kWorkers);  // the byte count's, the workers'
    mbar_init(&recv_bar[1], 1 + kWorkers);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&tile_bar[s], 1);
      mbar_init(&full_bar[s], 1);
    }
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemColumns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // stage s = gate rows 32 s .. 32 s + 31 of every part, box j = rows 32 j .. 32 j + 31 of the tile (the
    // layout of an MN-major A tile); gate rows and outputs past the end are zero-filled
    if (lane == 0) mbar_expect_tx(w_bar, in_smem * kABytes);
    __syncwarp();
    for (int i = lane; i < in_smem * 4; i += 32) {
      const int s = i >> 2, j = i & 3;
      int c[2] = {group * kOut + 32 * j % kOut, rank * a.slice + 32 * j / kOut * sub + s * kBK};
      tma_load(&a.map[ji], w_bar, a_tiles + s * kABytes + j * (kBK * 128), 2, c);
    }
  }
  // this warp's rows of the accumulator, and of the tiles in tensor memory: a part, 32 outputs of it
  const int part = (warp & 3) * 32 / kOut;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t a_tmem = tmem_base + a.accs * kAccStride;
  if (warp < kWorkers) {
    const int j = group * kOut + (warp & 3) * 32 % kOut + lane;
    for (int s = in_smem + (warp >> 2); s < stages; s += 2) {
      const int r0 = rank * a.slice + part * sub + s * kBK;
      const float* wp = job.w_hh + (long long)r0 * H + j;
#pragma unroll
      for (int c = 0; c < kBK; c += 8) {
        float v[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) v[h] = j < H && r0 + c + h < GH ? wp[(long long)(c + h) * H] : 0.f;
        tmem_st8(a_tmem + lanes + (uint32_t)((s - in_smem) * kBK + c), v);
      }
    }
    tmem_st_wait();
    tc_fence_before();
  }
  if (threadIdx.x == 0) waits.bar<false>(w_bar, 0);
  __syncthreads();
  cluster_sync_all();  // every peer's barriers are initialised before anybody pushes

  if (warp >= kWorkers) {
    const int q = warp - kWorkers;
    if (q < stages && elect_one()) {
      const uint64_t a_desc0 = umma_desc(smem_u32(a_tiles), kBK * 128, 512, 1);
      const uint64_t b_desc0 = umma_desc(smem_u32(b_tiles), 16, 1024, 2);
      for (int sb = 0; sb < a.T; ++sb)
        if (!issue_step<true, kCols>(tmem_base, kAccStride, a.accs, a_desc0, a_tmem, in_smem, b_desc0, q, stages,
                                     sb & 1, full_bar, done_bar, waits))
          break;
    }
    __syncwarp();
  } else {
    constexpr int kHalf = NB / 2, kChunk = NB == 32 ? 16 : 8;
    int item_b[kItems], item_u[kItems];
    float dh[kItems], dc[kItems];
    bool live[kItems];
    // what the cell gradient of a step reads: LSTM i f g o c c_prev; GRU r z n q h_prev; plain h; dy
    constexpr int kIn = G == 4 ? 7 : (G == 3 ? 6 : 2);
    float in[kItems][kIn] = {};
    auto fetch = [&](int sb) {
      const int step = a.T - 1 - sb;
      const int t = job.reverse ? a.T - 1 - step : step;
      const int t_prev = job.reverse ? t + 1 : t - 1;  // the forward pass's previous time
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const int b = item_b[it], j = group * kOut + rank * kOwn + item_u[it];
        const long long row = (long long)t * a.B_total + b, prow = (long long)t_prev * a.B_total + b;
        const float* g = job.gates + row * GH + j;
        in[it][0] = job.dy ? __ldcg(job.dy + row * a.dy_stride + j) : 0.f;
#pragma unroll
        for (int q = 0; q < G; ++q) in[it][1 + q] = __ldcg(g + (long long)q * H);
        if constexpr (G == 4) {
          in[it][5] = __ldcg(job.cells + row * H + j);
          in[it][6] = __ldcg(step == 0 ? job.first + (long long)b * H + j : job.cells + prow * H + j);
        } else if constexpr (G == 3) {
          in[it][4] = __ldcg(job.cells + row * H + j);
          in[it][5] = __ldcg(step == 0 ? job.first + (long long)b * H + j
                                       : job.out + prow * a.out_stride + j);
        }
      }
    };
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      const int idx = threadIdx.x + it * kWorkThreads;
      item_b[it] = idx / kOwn;
      item_u[it] = idx - item_b[it] * kOwn;
      const int j = group * kOut + rank * kOwn + item_u[it];
      live[it] = item_b[it] < B && j < H;
      const long long at = (long long)item_b[it] * H + j;
      dh[it] = live[it] && job.dh0 ? job.dh0[at] : 0.f;
      dc[it] = G == 4 && live[it] && job.dc0 ? job.dc0[at] : 0.f;
    }
    fetch(0);
    Feed feed{&a.xmap[ji], a.xch[ji], b_tiles, tile_bar, full_bar, GH, B, stages, rank * a.slice + warp * kBK, sub, 0};
    // this lane's row of the accumulator goes to the CTA that owns the output
    const int quads = (B + 3) / 4;
    const int out = ((warp & 3) * 32 + lane) % kOut, owner = out / kOwn;
    const uint32_t push_at = mapa_u32(
        smem_u32(recv) + (uint32_t)((((rank * P + part) * (NB / 4)) * kOwn + out - owner * kOwn) * 16),
        (uint32_t)owner);
    const uint32_t push_bar = mapa_u32(smem_u32(recv_bar), (uint32_t)owner);
    const uint32_t recv_bytes = (uint32_t)(kBM * quads * 16);

    float dg[kItems][G == 3 ? 4 : G];  // GRU: and dn * r, of the recurrent side
    auto store_grads = [&](int sb) {
      const int step = a.T - 1 - sb;
      const int t = job.reverse ? a.T - 1 - step : step;
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const long long at = ((long long)t * a.B_total + item_b[it]) * GH + group * kOut + rank * kOwn + item_u[it];
#pragma unroll
        for (int g = 0; g < G; ++g) job.dgates[at + (long long)g * H] = dg[it][g];
        if constexpr (G == 3) {
          job.dgh[at] = dg[it][0];
          job.dgh[at + H] = dg[it][1];
          job.dgh[at + 2 * H] = dg[it][3];
        }
      }
    };

    for (int sb = 0; sb < a.T && waits.warp_goes_on(); ++sb) {
      const int slot = sb & 1;
      const uint32_t tag = (uint32_t)(sb + 1) & kTagMask;
      uint32_t* x = a.xch[ji] + (long long)slot * B * GH;
      // ---- cell gradient of this step's time for this thread's (batch, unit) pairs
#pragma unroll
      for (int it = 0; it < kItems; ++it) {  // the arithmetic of all pairs side by side, live or not
        uint32_t* xo = x + (long long)item_b[it] * GH + group * kOut + rank * kOwn + item_u[it];
        const float d = dh[it] + in[it][0];
        if constexpr (G == 4) {
          const float gi = in[it][1], gf = in[it][2], gg = in[it][3], go = in[it][4];
          const float tc = tanhf(in[it][5]), cp = in[it][6];
          const float dct = dc[it] + d * go * (1.f - tc * tc);
          dg[it][0] = dct * gg * gi * (1.f - gi);
          dg[it][1] = dct * cp * gf * (1.f - gf);
          dg[it][2] = dct * gi * (1.f - gg * gg);
          dg[it][3] = d * tc * go * (1.f - go);
          dc[it] = dct * gf;
        } else if constexpr (G == 1) {
          const float h = in[it][1];
          dg[it][0] = a.act == 0 ? (h > 0.f ? d : 0.f) : d * (1.f - h * h);
        } else {
          const float r = in[it][1], z = in[it][2], n = in[it][3], q = in[it][4], hp = in[it][5];
          const float dn = d * (1.f - z) * (1.f - n * n);
          dg[it][0] = dn * q * r * (1.f - r);
          dg[it][1] = d * (hp - n) * z * (1.f - z);
          dg[it][2] = dn;
          dg[it][3] = dn * r;
          dc[it] = d * z;  // the direct part of the next dh
        }
#pragma unroll
        for (int g = 0; g < G; ++g)
          if (live[it]) st_relaxed_u32(xo + (long long)g * H, tagged(dg[it][G == 3 && g == 2 ? 3 : g], tag));
      }
      if (threadIdx.x == 0) mbar_expect_tx(&recv_bar[slot], recv_bytes);
      bring_tiles<false, P, NB>(feed, slot, tag, warp, lane, waits, 14, [&] {
        store_grads(sb);
        if (sb + 1 < a.T) fetch(sb + 1);
      });
      if (lane == 0) mbar_arrive(done_bar);
      if (waits.warp_bar<false>(done_bar, sb & 1)) {
        tc_fence_after();
        const uint32_t at = push_at + (uint32_t)(slot * kRecv * 4);
        const uint32_t bar = push_bar + (uint32_t)(slot * 8);
#pragma unroll
        for (int i = 0; i < kHalf; i += kChunk) {
          const int c0 = (warp >> 2) * kHalf + i;  // warps w and w + 4 share the rows of tensor memory
          float v[kChunk];
          read_sums<kAccStride, kChunk>(tmem_base + lanes + part * NB + c0, min(stages, a.accs), v);
#pragma unroll
          for (int j = 0; j < kChunk / 4; ++j)
            if (c0 / 4 + j < quads)
              st_async_v4(at + (uint32_t)((c0 / 4 + j) * (kOwn * 16)), bar, v[4 * j], v[4 * j + 1],
                          v[4 * j + 2], v[4 * j + 3]);
        }
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&recv_bar[slot]);
      if (!waits.warp_bar<true>(&recv_bar[slot], (sb >> 1) & 1)) break;
      // ---- dh_{t-1} of this thread's pairs: the partial sums, in slice order
      const float* rp = recv + slot * kRecv;
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        const int b = min(item_b[it], NB - 1);
        float sum = 0.f;
#pragma unroll
        for (int q = 0; q < KC * P; ++q)
          sum += rp[((q * (NB / 4) + (b >> 2)) * kOwn + item_u[it]) * 4 + (b & 3)];
        dh[it] = G == 3 ? dc[it] + sum : sum;
      }
    }
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      if (!live[it]) continue;
      const long long at = (long long)item_b[it] * H + group * kOut + rank * kOwn + item_u[it];
      job.dh_out[at] = dh[it];
      if (G == 4) job.dc_out[at] = dc[it];
    }
  }
  __syncthreads();
  if (*failed)  // what was copied or pushed, and the MMAs issued, before a wait ran out have ended after this
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {
    }
  cluster_sync_all();  // nobody leaves while a peer may still push into its shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemColumns);
  }
}

// ------------------------------------------------------------------------------------- host
typedef void (*FwdKernel)(const Launch<SeqJob>);
typedef void (*BwdKernel)(const Launch<SeqBwdJob>);

// One way to run a job: `rows` of the batch, a cluster of CTAs per group of units or outputs.
struct Plan {
  int rows;  // of the batch per job; 0: not possible
  int nb, cluster, slice, stages, in_smem, accs, ctas;
  size_t smem;
  const void* kernel;
};
void set_rows(Plan* p, int B, int nb) {
  p->nb = nb;
  const int parts = (B + nb - 1) / nb;
  p->rows = (B + parts - 1) / parts;
}
bool wants_48(int B) { return B > 32 && B <= 48; }  // where 48 rows save a second job

// Accumulators, `cols` wide: one per k tile up to kRnnAccs.  Beside them tensor memory takes what it holds of the
// weights (an MMA of 32 / 64 columns takes 28 / 41 clocks with A in tensor memory, 49 / 57 with A in shared
// memory), shared memory the rest; where that is too much, half as many accumulators, of chains twice as long.
// Sums of positive products are 5.9e-7 too small in chains of 128 products, below 2.2e-7 in chains of 32.
// (Two accumulators everywhere, and all the weights that fit in tensor memory: 61 steps of a 320-unit GRU 337
// us, so 354, with tiles of few rows stored by those who poll 301; 3 layers of both directions of a 1024-unit LSTM, 500 steps, with gradients 21.6 ms, so 22.0.)
void place_tiles(Plan* p, int cols, int recv) {
  p->accs = kIssuers;
  while (p->accs < std::min(p->stages, kRnnAccs)) p->accs *= 2;
  for (;; p->accs /= 2) {
    const int fit = (kTmemColumns - p->accs * ((cols + 31) / 32 * 32)) / kBK;
    p->in_smem = std::max(0, p->stages - fit);
    p->smem = seq_smem(p->in_smem, p->stages, cols, recv);
    if (p->smem <= kMostSmem || p->accs == kIssuers) return;
  }
}

template <int G, int NB>
const void* fwd_kernel(int ks) {
  FwdKernel k = ks == 1 ? rnn_sequence_kernel<1, G, NB>
                        : (ks == 2 ? rnn_sequence_kernel<2, G, NB> : rnn_sequence_kernel<4, G, NB>);
  return reinterpret_cast<const void*>(k);
}
// K slices per cluster: of at most 256 states as few as fit (each takes another partial sum through the
// cluster), equal in length.  wide: of at most 512, half the CTAs.
Plan forward_plan(int B, int H, int G, int nb, bool wide) {
  Plan p{};
  if (wide && H <= 512) return p;
  p.cluster = H <= 256 ? 1 : (H <= 512 || wide ? 2 : 4);
  p.slice = ((H + p.cluster - 1) / p.cluster + kBK - 1) / kBK * kBK;
  p.ctas = (H + kUnits - 1) / kUnits * p.cluster;
  p.stages = p.slice / kBK;
  place_tiles(&p, nb, kUnits * G * nb);
  if (p.smem > kMostSmem) return p;
  set_rows(&p, B, nb);
  if (nb == 32)
    p.kernel = G == 1 ? fwd_kernel<1, 32>(p.cluster) : (G == 3 ? fwd_kernel<3, 32>(p.cluster) : fwd_kernel<4, 32>(p.cluster));
  else
    p.kernel = G == 1 ? fwd_kernel<1, 48>(p.cluster) : (G == 3 ? fwd_kernel<3, 48>(p.cluster) : fwd_kernel<4, 48>(p.cluster));
  return p;
}
// Gate rows in KC * P = 8 equal pieces either way.
template <int KC, int P, int NB>
Plan backward_plan(int B, int H, int G) {
  Plan p{};
  const int GH = G * H, out = kBM / P;
  const int sub = ((GH + KC * P - 1) / (KC * P) + kBK - 1) / kBK * kBK;
  p.cluster = KC;
  p.slice = sub * P;
  p.ctas = (H + out - 1) / out * KC;
  p.stages = sub / kBK;
  place_tiles(&p, P * NB, kBM * NB);
  if (p.stages > kMaxTiles || p.smem > kMostSmem) return p;
  set_rows(&p, B, NB);
  p.kernel = reinterpret_cast<const void*>(G == 1   ? rnn_sequence_backward_kernel<KC, P, 1, NB>
                                           : G == 3 ? rnn_sequence_backward_kernel<KC, P, 3, NB>
                                                    : rnn_sequence_backward_kernel<KC, P, 4, NB>);
  return p;
}

// How many CTAs (clusters, where cluster > 1) of this launch the device holds at once.
int resident(const void* kernel, int cluster, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, size_t>, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(dev, kernel, smem);
  const auto it = known.find(key);
  if (it != known.end()) return it->second;
  int n = 0;
  bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) ==
            cudaSuccess;
  if (ok && cluster > 1) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)cluster);
    cfg.blockDim = dim3(kSeqThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ok = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess;
  } else if (ok) {
    ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kSeqThreads, smem) == cudaSuccess;
    n *= device_info().sm_count;
  }
  if (!ok) {
    (void)cudaGetLastError();
    n = 0;
  }
  known[key] = n;
  return n;
}
int jobs_at_once(const Plan& p) {
  return std::min(resident(p.kernel, p.cluster, p.smem) / (p.ctas / p.cluster), kMaxJobs);
}
int jobs_of(const SeqShape& s, const Plan& p) { return s.dirs * ((s.B + p.rows - 1) / p.rows); }

// The first of the ways in the order of their speed for one job, unless a later one takes fewer launches
// one after another.  (1024 units, four gates: a direction in clusters of 8 needs 8 of them and the device
// holds 15, so both directions together take clusters of 4.)
Plan plan_for(const SeqShape& s, bool backward) {
  Plan ways[4];
  int n = 0;
  if (!backward) {
    if (wants_48(s.B)) ways[n++] = forward_plan(s.B, s.H, s.G, 48, false);
    ways[n++] = forward_plan(s.B, s.H, s.G, 32, false);
    ways[n++] = forward_plan(s.B, s.H, s.G, 32, true);
  } else {
    if (wants_48(s.B)) {
      ways[n++] = backward_plan<8, 1, 48>(s.B, s.H, s.G);
      ways[n++] = backward_plan<4, 2, 48>(s.B, s.H, s.G);
    }
    ways[n++] = backward_plan<8, 1, 32>(s.B, s.H, s.G);
    ways[n++] = backward_plan<4, 2, 32>(s.B, s.H, s.G);
  }
  Plan best{};
  int fewest = 0;
  for (int i = 0; i < n; ++i) {
    const int at_once = ways[i].rows > 0 ? jobs_at_once(ways[i]) : 0;
    if (at_once < 1) continue;
    const int launches = (jobs_of(s, ways[i]) + at_once - 1) / at_once;
    if (fewest == 0 || launches < fewest) best = ways[i], fewest = launches;
  }
  return best;
}
size_t up256(size_t v) { return (v + 255) / 256 * 256; }
size_t xch_bytes(const SeqShape& s, int rows, bool backward) {
  return up256((size_t)2 * rows * s.H * (backward ? s.G : 1) * 4);
}

template <typename Job>
int launch(const char* name, const SeqShape& s, const Plan& p, const Job* jobs, int n, bool backward,
           void* scratch, cudaStream_t st, long long wait_budget, int absent_cta) {
  FLB200_REQUIRE(p.rows > 0, "%s: the device does not hold this launch", name);
  const int at_once = jobs_at_once(p);
  const size_t xb = xch_bytes(s, p.rows, backward);
  FLB200_CUDA_CHECK(cudaMemsetAsync(scratch, 0, xb * (size_t)n, st));  // step number 0
  for (int first = 0; first < n; first += at_once) {
    const int m = std::min(at_once, n - first);
    Launch<Job> a{};
    for (int i = 0; i < m; ++i) {
      const Job& j = jobs[first + i];
      const uint64_t dims[2] = {(uint64_t)s.H, (uint64_t)s.G * s.H};
      const uint64_t strides[1] = {(uint64_t)s.H * 4};
      const uint32_t box[2] = {32, 32};
      if (int rc = tc::make_tensor_map(&a.map[i], j.w_hh, 2, dims, strides, box,
                                       backward ? tc::kMapMnMajor : tc::kMapKMajor))
        return rc;
      a.job[i] = j;
      a.xch[i] = reinterpret_cast<uint32_t*>(static_cast<char*>(scratch) + xb * (size_t)(first + i));
      const uint64_t words = (uint64_t)(backward ? s.G : 1) * s.H;
      const uint64_t xdims[3] = {words, (uint64_t)j.B, 2};
      const uint64_t xstrides[2] = {words * 4, words * 4 * (uint64_t)j.B};
      const uint32_t xbox[3] = {32, (uint32_t)p.nb, 1};
      if (int rc = tc::make_tensor_map(&a.xmap[i], a.xch[i], 3, xdims, xstrides, xbox, tc::kMapKMajor)) return rc;
    }
    a.status = tc::status_ptr();
    a.wait_budget = wait_budget > 0 ? wait_budget : tc::kWaitBudget;
    a.out_stride = s.out_stride;
    a.dy_stride = s.dy_stride;
    a.T = s.T; a.B_total = s.B; a.H = s.H; a.act = s.act;
    a.slice = p.slice; a.stages = p.stages; a.in_smem = p.in_smem; a.accs = p.accs; a.ctas = p.ctas;
    a.absent_cta = absent_cta;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(m * p.ctas));
    cfg.blockDim = dim3(kSeqThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[1] = {&a};
    FLB200_CUDA_CHECK(cudaLaunchKernelExC(&cfg, p.kernel, args));
    FLB200_AFTER_LAUNCH(name);
    tc::count_tc_launch();
  }
  return FLB200_OK;
}

}  // namespace

int rnn_sequence_rows(int math_mode, const SeqShape& s, const float* w_hh, bool backward) {
  if (math_mode != FLB200_MATH_TF32 || !flb200_has_tensor_core_path()) return 0;
  if (s.B < 1 || s.H < 4 || s.H % 4 != 0 || s.H > 1024 || (s.G != 1 && s.G != 3 && s.G != 4)) return 0;
  if ((reinterpret_cast<uintptr_t>(w_hh) & 15) != 0) return 0;
  const Plan p = plan_for(s, backward);
  if (p.rows == 0) return 0;
  const int n = jobs_at_once(p);
  // a large batch in many launches one after another would lose to a kernel per step
  return (jobs_of(s, p) + n - 1) / n <= 8 ? p.rows : 0;
}

// Enough for every way that plan_for may choose: 48 rows a job, or equal parts of up to 32.
size_t rnn_sequence_scratch_bytes(const SeqShape& s, bool backward) {
  if (s.B < 1 || s.H < 4 || s.H % 4 != 0 || s.H > 1024) return 0;
  const int parts = (s.B + 31) / 32;
  const size_t split = xch_bytes(s, (s.B + parts - 1) / parts, backward) * (size_t)(parts * s.dirs);
  return wants_48(s.B) ? std::max(split, xch_bytes(s, s.B, backward) * (size_t)s.dirs) : split;
}

int rnn_sequence_forward(const SeqShape& s, const SeqJob* jobs, int n, void* scratch, cudaStream_t st,
                         long long wait_budget, int absent_cta) {
  return launch("rnn_sequence_forward", s, plan_for(s, false), jobs, n, false, scratch, st, wait_budget,
                absent_cta);
}
int rnn_sequence_backward(const SeqShape& s, const SeqBwdJob* jobs, int n, void* scratch,
                          cudaStream_t st) {
  return launch("rnn_sequence_backward", s, plan_for(s, true), jobs, n, true, scratch, st, 0, -1);
}

}  // namespace flb200
