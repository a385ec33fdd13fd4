// The recurrence of a layer as one persistent kernel: all T steps, with the recurrent weights
// resident in shared memory, and both directions (or several parts of a large batch) side by side
// as jobs of one launch where the device holds them.
//
// What bounds a step is latency: between two steps every unit's new state has to reach all CTAs.
// The states travel without barriers, fences or counters: each one is a 4-byte word of an exchange
// buffer whose low 13 bits, which a TF32 operand does not use, carry the step's number, and a reader
// polls the words themselves.  A word is complete the moment it is visible, so a step costs one
// write to L2 and one read back.  (Values that keep all their bits, the partial sums of the
// backward pass, travel as 8-byte pairs of value and step number.)  Two slots, used in turn, are
// enough: a CTA can only be asked to write step s + 2 once everybody has consumed step s, which the
// data dependence itself ensures (each state needs all states of the step before).
// With a grid-wide barrier per step (release counter, fence, cluster barrier) a step of a 1024-unit
// LSTM over 32 rows took 7.2 us forward and 8.0 us backward; now 3.9 and 6.9, and the two directions
// of a 512-unit one run together in 4.4 and 6.0.  Loads complete in order, yet neither prefetching
// the next step's gates nor loading them after the polls measured faster.
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
constexpr int kMaxStages = kRnnTiles;       // k tiles a CTA keeps: one per warp
constexpr int kSeqThreads = 256;
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
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_v2(unsigned long long* p, unsigned long long a,
                                              unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
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

// The k tile of one warp: NB batch rows of 32 tagged words, in shared memory as the 128-byte
// swizzle that the UMMA descriptor expects.  src: the row of batch 0, this lane's 16-byte chunk.
template <int NB>
__device__ __forceinline__ void load_tagged_tile(const uint32_t* src, long long row_stride, int B,
                                                 bool live, uint32_t tag, char* tile, int lane,
                                                 const Waits& w, int code) {
  constexpr int N = NB / 4;
  const int q = lane & 7, r = lane >> 3;
  uint4 v[N];
  uint32_t pending = 0;
#pragma unroll
  for (int u = 0; u < N; ++u)
    if (live && r + 4 * u < B) pending |= 1u << u;
  const uint32_t mine = pending;
  if (*w.failed) pending = 0;
  int spins = 0;
  const long long t0 = clock64();
  while (pending) {
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (pending >> u & 1) v[u] = ld_relaxed_v4(src + (long long)(r + 4 * u) * row_stride);
#pragma unroll
    for (int u = 0; u < N; ++u)
      if ((pending >> u & 1) && (((v[u].x ^ tag) | (v[u].y ^ tag) | (v[u].z ^ tag) | (v[u].w ^ tag)) &
                                 kTagMask) == 0)
        pending &= ~(1u << u);
    if (pending && w.expired(&spins, t0, code)) break;
  }
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const int b = r + 4 * u;
    if (mine >> u & 1)
      *reinterpret_cast<uint4*>(tile + b * 128 + ((q ^ (b & 7)) << 4)) =
          make_uint4(v[u].x & ~kTagMask, v[u].y & ~kTagMask, v[u].z & ~kTagMask, v[u].w & ~kTagMask);
  }
}
__device__ __forceinline__ uint32_t tagged(float v, uint32_t tag) {
  return (__float_as_uint(v) & ~kTagMask) | tag;
}

// Tensor memory: an accumulator of kAccCols columns per k tile.  Every warp issues the MMAs of the
// tile that it loaded.  From one thread that waits for tile after tile each tile's chain of descriptor
// moves starts anew, 540 clocks per tile and 4300 for eight; eight warps overlap theirs.
template <int NB>
struct Acc {
  static constexpr uint32_t kCols = NB <= 32 ? 32 : 64;
};
template <bool kAMajorMn, int NB>
__device__ __forceinline__ void issue_tile(uint32_t tmem, uint64_t a_desc0, uint64_t b_desc0, int s,
                                           uint64_t* done_bar) {
  const uint32_t idesc = umma_idesc_tf32(NB, kAMajorMn ? 1 : 0, 0);
  tc_fence_after();
#pragma unroll
  for (int j = 0; j < kBK / kUmmaK; ++j)
    umma_tf32(tmem + s * Acc<NB>::kCols, umma_desc_advance(a_desc0, s * kABytes + j * (kAMajorMn ? 1024 : 32)),
              umma_desc_advance(b_desc0, s * NB * 128 + j * 32), idesc, j ? 1u : 0u);
  umma_commit(done_bar);
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
// N columns of this warp's rows: the accumulators of all k tiles, loaded together, added in order
template <int NB, int N>
__device__ __forceinline__ void read_sums(uint32_t at, int stages, float* v) {
  uint32_t r[kMaxStages][N];
#pragma unroll
  for (int q = 0; q < kMaxStages; ++q)
    if (q < stages) tmem_ld_async<N>(at + q * Acc<NB>::kCols, r[q]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < kMaxStages; ++q) {
#pragma unroll
    for (int j = 0; j < N; ++j) asm volatile("" : "+r"(r[q][j]));  // read only after the wait
    if (q < stages) {
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = q == 0 ? __uint_as_float(r[0][j]) : v[j] + __uint_as_float(r[q][j]);
    }
  }
}

template <typename Job>
struct Launch {
  CUtensorMap map[kMaxJobs];
  Job job[kMaxJobs];
  uint32_t* xch[kMaxJobs];             // tagged states: [2][B][H], backward: [2][B][G*H]
  unsigned long long* part[kMaxJobs];  // backward: partial sums of two steps
  int* status;
  long long wait_budget;
  long long out_stride, dy_stride;
  int T, B_total, H, act;
  int slice, units;  // gate rows / states of a CTA's k slice; backward: outputs a CTA finishes
  int ctas;          // of one job
  int split;         // backward: slices of the gate rows
  int absent_cta;
};

// Shared memory: weights [stages][16 KB], states [stages][NB x 128 bytes], forward: two slots of
// received partial sums [KS][G][NB / 4][32 / KS units][4 rows of the batch], barriers.  Never less
// than half of an SM's: two CTAs of one SM would wait for each other's tensor memory.
template <int G, int NB>
struct Recv { static constexpr int kFloats = kUnits * G * NB; };
inline size_t seq_smem(int stages, int NB, int recv) {
  const size_t need = (size_t)stages * (kABytes + NB * 128) + (size_t)2 * recv * 4 + 256 + 1024;
  return std::max(need, (size_t)120 * 1024);
}

// ---------------------------------------------------------------------------------- forward
//   pre[b][g*H + j] = gates[t][b][g*H + j] + sum_k W_hh[g*H + j][k] * h_{t-1}[b][k]
// A cluster owns 32 hidden units, all gates of them = up to 128 rows of one UMMA tile (gate-major;
// the rows of absent gates are zeros); its KS CTAs split K = H into slices of at most 256.  Warp s
// brings the 32 states of k tile s and issues that tile's MMAs (M = 128, N = batch), all warps push the
// partial sums of each unit from tensor memory straight into the shared memory of the CTA that
// updates it (st.async: one trip, no cluster barrier), and every thread updates the same (unit,
// batch) pairs in all steps, with the cell state in a register.
template <int KS, int G, int NB>
__global__ void __launch_bounds__(kSeqThreads, 1)
rnn_sequence_kernel(const __grid_constant__ Launch<SeqJob> a) {
  constexpr int kOwn = kUnits / KS;  // units this CTA updates
  constexpr int kHalf = NB / 2, kChunk = NB == 32 ? 16 : 8;
  constexpr int kItems = (kOwn * NB + kSeqThreads - 1) / kSeqThreads;
  extern __shared__ char smem_raw[];
  char* tiles = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const int stages = a.slice / kBK;
  char* a_tiles = tiles;
  char* b_tiles = tiles + stages * kABytes;
  float* recv = reinterpret_cast<float*>(b_tiles + stages * NB * 128);
  uint64_t* w_bar = reinterpret_cast<uint64_t*>(recv + 2 * Recv<G, NB>::kFloats);
  uint64_t* done_bar = w_bar + 1;
  uint64_t* recv_bar = done_bar + 1;         // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(recv_bar + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int ji = blockIdx.x / a.ctas, cta = blockIdx.x - ji * a.ctas;
  const int group = cta / KS;
  const SeqJob& job = a.job[ji];
  const int H = a.H, B = job.B;
  const Waits waits{failed, a.status, a.wait_budget};

  if (threadIdx.x == 0) {
    mbar_init(w_bar, 1);
    mbar_init(done_bar, stages);
    mbar_init(&recv_bar[0], 1 + kSeqThreads / 32);  // the byte count's, the warps'
    mbar_init(&recv_bar[1], 1 + kSeqThreads / 32);
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kMaxStages * Acc<NB>::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {  // the resident slice of W_hh
    if (lane == 0) mbar_expect_tx(w_bar, stages * G * (32 * 128));
    __syncwarp();
    for (int i = lane; i < stages * G; i += 32) {
      const int s = i / G, g = i - s * G;
      int c[2] = {rank * a.slice + s * kBK, g * H + group * kUnits};
      tma_load(&a.map[ji], w_bar, a_tiles + s * kABytes + g * (32 * 128), 2, c);
    }
  }
  if (G < 4) {  // rows 32 G .. 127 of every k tile belong to no gate
    constexpr int kPerStage = (4 - G) * (32 * 128 / 16);
    for (int i = threadIdx.x; i < stages * kPerStage; i += kSeqThreads) {
      const int s = i / (kPerStage > 0 ? kPerStage : 1), rem = i - s * kPerStage;
      *reinterpret_cast<float4*>(a_tiles + s * kABytes + G * (32 * 128) + rem * 16) =
          make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  // batch rows and states past the end stay zero
  for (int i = threadIdx.x; i < stages * NB * 8; i += kSeqThreads)
    *reinterpret_cast<float4*>(b_tiles + i * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
  fence_proxy_async();
  if (threadIdx.x == 0) waits.bar<false>(w_bar, 0);
  __syncthreads();
  cluster_sync_all();  // every peer's barriers are initialised before anybody pushes

  const uint64_t a_desc0 = umma_desc(smem_u32(a_tiles), 16, 1024, 2);
  const uint64_t b_desc0 = umma_desc(smem_u32(b_tiles), 16, 1024, 2);
  {
    int item_b[kItems], item_u[kItems];
    float state[kItems];  // LSTM: c; GRU: h
    bool live[kItems];
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      const int idx = threadIdx.x + it * kSeqThreads;
      item_b[it] = idx / kOwn;
      item_u[it] = idx - item_b[it] * kOwn;
      const int j = group * kUnits + rank * kOwn + item_u[it];
      live[it] = item_b[it] < B && j < H;
      state[it] = live[it] && G != 1 ? (G == 4 ? job.c0 : job.h0)[(long long)item_b[it] * H + j] : 0.f;
    }
    // this warp's k tile: 8 lanes cover a row's 128 bytes
    const int k0 = rank * a.slice + warp * kBK + 4 * (lane & 7);
    const bool k_live = warp < stages && k0 < H;
    // this lane's row of the accumulator goes to the CTA that owns unit `lane`
    const int owner = lane / kOwn;
    const int quads = (B + 3) / 4;
    const uint32_t push_at = mapa_u32(
        smem_u32(recv) + (uint32_t)((((rank * G + (warp & 3)) * (NB / 4)) * kOwn + lane - owner * kOwn) * 16),
        (uint32_t)owner);
    const uint32_t push_bar = mapa_u32(smem_u32(recv_bar), (uint32_t)owner);
    const uint32_t recv_bytes = (uint32_t)(kUnits * G * quads * 16);

    for (int step = 0; step < a.T && waits.warp_goes_on(); ++step) {
      const int t = job.reverse ? a.T - 1 - step : step;
      const int slot = step & 1;
      float* g_t = job.gates + (long long)t * a.B_total * G * H + group * kUnits + rank * kOwn;
      // input projections of this step: in flight during the wait
      float gin[kItems][G];
#pragma unroll
      for (int it = 0; it < kItems; ++it)
        if (live[it]) {
          const float* gp = g_t + (long long)item_b[it] * G * H + item_u[it];
#pragma unroll
          for (int g = 0; g < G; ++g) gin[it][g] = __ldcg(gp + (long long)g * H);
        }
      if (threadIdx.x == 0) mbar_expect_tx(&recv_bar[slot], recv_bytes);
      if (warp < stages) {
        char* tile = b_tiles + warp * NB * 128;
        if (step == 0) {
          for (int b = lane >> 3; b < B; b += 4)
            if (k_live) {
              const float* hp = job.h0 + (long long)b * H + k0;
              *reinterpret_cast<float4*>(tile + b * 128 + (((lane & 7) ^ (b & 7)) << 4)) =
                  make_float4(hp[0], hp[1], hp[2], hp[3]);
            }
        } else {
          // h of the step before, published with its step number
          load_tagged_tile<NB>(a.xch[ji] + (long long)(slot ^ 1) * B * H + k0, H, B, k_live,
                               (uint32_t)step & kTagMask, tile, lane, waits, 13);
        }
        fence_proxy_async();  // generic-proxy writes, read by the tensor core next
        __syncwarp();
        // (the sums of the step before have been read: this CTA's own pushes were part of what this
        // warp has waited for)
        if (lane == 0) issue_tile<false, NB>(tmem_base, a_desc0, b_desc0, warp, done_bar);
        __syncwarp();
      }
      if ((warp & 3) < G && waits.warp_bar<false>(done_bar, step & 1)) {
        tc_fence_after();
        const uint32_t at = push_at + (uint32_t)(slot * Recv<G, NB>::kFloats * 4);
        const uint32_t bar = push_bar + (uint32_t)(slot * 8);
#pragma unroll
        for (int i = 0; i < kHalf; i += kChunk) {
          const int c0 = (warp >> 2) * kHalf + i;  // warps w and w + 4 share the rows of tensor memory
          float v[kChunk];
          read_sums<NB, kChunk>(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c0, stages, v);
#pragma unroll
          for (int j = 0; j < kChunk / 4; ++j)
            if (c0 / 4 + j < quads)
              st_async_v4(at + (uint32_t)((c0 / 4 + j) * (kOwn * 16)), bar, v[4 * j], v[4 * j + 1],
                          v[4 * j + 2], v[4 * j + 3]);
        }
        tc_fence_before();
      }
      // Every warp counts for the step's barrier, those too that had no tile, row or pair to care for:
      // one that only followed could fall behind by two phases and miss one.
      if (lane == 0) mbar_arrive(&recv_bar[slot]);
      if (!waits.warp_bar<true>(&recv_bar[slot], (step >> 1) & 1)) break;
      const float* rp = recv + slot * Recv<G, NB>::kFloats;
      uint32_t* h_x = a.xch[ji] + (long long)slot * B * H + group * kUnits + rank * kOwn;
      const uint32_t tag = (uint32_t)(step + 1) & kTagMask;
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const int b = item_b[it], u = item_u[it];
        float pre[G];
#pragma unroll
        for (int g = 0; g < G; ++g) pre[g] = 0.f;
#pragma unroll
        for (int q = 0; q < KS; ++q)  // same order as lstm_step_kernel: bit-identical sums
#pragma unroll
          for (int g = 0; g < G; ++g) pre[g] += rp[(((q * G + g) * (NB / 4) + (b >> 2)) * kOwn + u) * 4 + (b & 3)];
        const int j = group * kUnits + rank * kOwn + u;
        float* gp = g_t + (long long)b * G * H + u;
        const long long row = (long long)t * a.B_total + b;
        float h;
        if constexpr (G == 4) {
          const float i = sigmoid_(pre[0] + gin[it][0]), f = sigmoid_(pre[1] + gin[it][1]);
          const float gg = tanhf(pre[2] + gin[it][2]), o = sigmoid_(pre[3] + gin[it][3]);
          const float c = f * state[it] + i * gg;
          state[it] = c;
          h = o * tanhf(c);
          if (cta != a.absent_cta) st_relaxed_u32(h_x + (long long)b * H + u, tagged(h, tag));
          gp[0] = i; gp[H] = f; gp[2 * H] = gg; gp[3 * H] = o;
          job.cells[row * H + j] = c;
        } else if constexpr (G == 1) {
          const float v = pre[0] + gin[it][0];
          h = a.act == 0 ? fmaxf(v, 0.f) : tanhf(v);
          if (cta != a.absent_cta) st_relaxed_u32(h_x + (long long)b * H + u, tagged(h, tag));
          gp[0] = h;
        } else {
          const float r = sigmoid_(pre[0] + gin[it][0]), z = sigmoid_(pre[1] + gin[it][1]);
          const float q = pre[2] + job.b_hn[j];
          const float n = tanhf(gin[it][2] + r * q);
          h = (1.f - z) * n + z * state[it];
          state[it] = h;
          if (cta != a.absent_cta) st_relaxed_u32(h_x + (long long)b * H + u, tagged(h, tag));
          gp[0] = r; gp[H] = z; gp[2 * H] = n;
          job.cells[row * H + j] = q;
        }
        job.out[row * a.out_stride + j] = h;
      }
    }
  }
  __syncthreads();
  if (*failed)  // what was pushed, and the MMAs issued, before a wait ran out have ended after this
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {
    }
  cluster_sync_all();  // nobody leaves while a peer may still push into its shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kMaxStages * Acc<NB>::kCols);
  }
}

// --------------------------------------------------------------------------------- backward
//   dgates_t          = cell gradient of (dh_t + dy_t, dc_t)          (element-wise)
//   dh_{t-1}[b][k]    = sum_r dgates_t[b][r] * W_hh[r][k]             (r over the G*H gate rows)
// The H outputs k form tiles of 128 (M of one UMMA, N = batch), the gate rows are split into
// slices of up to 256; one CTA per (tile, slice), no clusters.  A CTA keeps its block of W_hh for
// all steps, read straight from the forward weights as an MN-major operand (the output index k is
// the contiguous one).  Per step: the thread that owns a (batch, unit) pair computes its dgates and
// publishes them as tagged words; warp s brings k tile s and contracts it, all warps publish the
// tile's partial sums as (value, step) pairs, laid out for the threads that finish them: each pair
// of the tile is finished by one thread, which adds the partial sums in slice order and runs the cell
// gradient of the next step (dh and dc of its pairs stay in registers).
template <int kItems, int G, int NB>
__global__ void __launch_bounds__(kSeqThreads, 1)
rnn_sequence_backward_kernel(const __grid_constant__ Launch<SeqBwdJob> a) {
  extern __shared__ char smem_raw[];
  char* tiles = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const int stages = a.slice / kBK;
  char* a_tiles = tiles;
  char* b_tiles = tiles + stages * kABytes;
  uint64_t* w_bar = reinterpret_cast<uint64_t*>(b_tiles + stages * NB * 128);
  uint64_t* done_bar = w_bar + 1;
  uint64_t* read_bar = done_bar + 1;  // a step's sums have left tensor memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(read_bar + 1);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ji = blockIdx.x / a.ctas, cta = blockIdx.x - ji * a.ctas;
  const int SL = a.split, units = a.units;
  const int mt = cta / SL, rank = cta - mt * SL;  // tile of 128 outputs, slice of the gate rows
  const SeqBwdJob& job = a.job[ji];
  const int H = a.H, B = job.B, GH = G * H;
  const Waits waits{failed, a.status, a.wait_budget};

  if (threadIdx.x == 0) {
    mbar_init(w_bar, 1);
    mbar_init(done_bar, stages);
    mbar_init(read_bar, kSeqThreads / 32);
    *failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kMaxStages * Acc<NB>::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // stage s = gate rows 32 s .. 32 s + 31 of the slice, box j = outputs 32 j .. 32 j + 31 (the
    // layout of an MN-major A tile); rows and outputs past the end are zero-filled
    if (lane == 0) mbar_expect_tx(w_bar, stages * kABytes);
    __syncwarp();
    for (int i = lane; i < stages * 4; i += 32) {
      const int s = i >> 2, j = i & 3;
      int c[2] = {mt * kBM + 32 * j, rank * a.slice + s * kBK};
      tma_load(&a.map[ji], w_bar, a_tiles + s * kABytes + j * (kBK * 128), 2, c);
    }
  }
  for (int i = threadIdx.x; i < stages * NB * 8; i += kSeqThreads)
    *reinterpret_cast<float4*>(b_tiles + i * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
  fence_proxy_async();
  if (threadIdx.x == 0) waits.bar<false>(w_bar, 0);
  __syncthreads();

  const uint64_t a_desc0 = umma_desc(smem_u32(a_tiles), kBK * 128, 512, 1);
  const uint64_t b_desc0 = umma_desc(smem_u32(b_tiles), 16, 1024, 2);
  constexpr int kHalf = NB / 2, kChunk = NB == 32 ? 16 : 8;
  {
    int item_b[kItems], item_u[kItems];
    float dh[kItems], dc[kItems];
    bool live[kItems];
    // what the cell gradient of a step reads: LSTM i f g o c c_prev; GRU r z n q h_prev; plain h; dy
    constexpr int kPull = kItems == 1 ? 16 : 8;  // partial sums in flight
    constexpr int kIn = G == 4 ? 7 : (G == 3 ? 6 : 2);
    float in[kItems][kIn];
    auto fetch = [&](int sb) {
      const int step = a.T - 1 - sb;
      const int t = job.reverse ? a.T - 1 - step : step;
      const int t_prev = job.reverse ? t + 1 : t - 1;  // the forward pass's previous time
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const int b = item_b[it], j = mt * kBM + rank * units + item_u[it];
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
      const int idx = threadIdx.x + it * kSeqThreads;
      item_b[it] = idx / units;
      item_u[it] = idx - item_b[it] * units;
      const int unit = rank * units + item_u[it], j = mt * kBM + unit;
      live[it] = item_b[it] < B && unit < kBM && j < H;
      const long long at = (long long)item_b[it] * H + j;
      dh[it] = live[it] && job.dh0 ? job.dh0[at] : 0.f;
      dc[it] = G == 4 && live[it] && job.dc0 ? job.dc0[at] : 0.f;
    }
    fetch(0);
    const int r0 = rank * a.slice + warp * kBK + 4 * (lane & 7);
    const bool r_live = warp < stages && r0 < GH;
    // partial sums: [slot][tile][finishing CTA][slice][batch / 2][units][2 rows of the batch]: the
    // 16-byte stores of neighbouring lanes fill whole sectors (in groups of 4 rows each store wrote
    // every other half sector, 2900 clocks per step for 32 KB)
    const int quads = (B + 3) / 4;
    const long long block = (long long)4 * quads * units;
    const long long tile_at = (long long)mt * SL * SL * block;
    const long long slot_size = (long long)a.ctas * SL * block;
    const int row = (warp & 3) * 32 + lane;  // accumulator row = output of the tile
    const bool row_live = mt * kBM + row < H;
    unsigned long long* push = a.part[ji] + tile_at + ((long long)(row / units) * SL + rank) * block + 2 * (row % units);
    const unsigned long long* pull = a.part[ji] + tile_at + (long long)rank * SL * block;

    for (int sb = 0; sb < a.T && waits.warp_goes_on(); ++sb) {
      const int step = a.T - 1 - sb;
      const int t = job.reverse ? a.T - 1 - step : step;
      const int slot = sb & 1;
      const uint32_t tag = (uint32_t)(sb + 1) & kTagMask;
      uint32_t* x = a.xch[ji] + (long long)slot * B * GH;
      // ---- cell gradient of time t for this thread's (batch, unit) pairs
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const int b = item_b[it], j = mt * kBM + rank * units + item_u[it];
        uint32_t* xo = x + (long long)b * GH + j;
        float* o = job.dgates + ((long long)t * a.B_total + b) * GH + j;
        const float d = dh[it] + in[it][0];
        if constexpr (G == 4) {
          const float gi = in[it][1], gf = in[it][2], gg = in[it][3], go = in[it][4];
          const float tc = tanhf(in[it][5]), cp = in[it][6];
          const float dct = dc[it] + d * go * (1.f - tc * tc);
          const float di = dct * gg * gi * (1.f - gi), df = dct * cp * gf * (1.f - gf);
          const float dg = dct * gi * (1.f - gg * gg), dgo = d * tc * go * (1.f - go);
          st_relaxed_u32(xo, tagged(di, tag));
          st_relaxed_u32(xo + H, tagged(df, tag));
          st_relaxed_u32(xo + 2 * H, tagged(dg, tag));
          st_relaxed_u32(xo + 3 * H, tagged(dgo, tag));
          o[0] = di; o[H] = df; o[2 * H] = dg; o[3 * H] = dgo;
          dc[it] = dct * gf;
        } else if constexpr (G == 1) {
          const float h = in[it][1];
          const float da = a.act == 0 ? (h > 0.f ? d : 0.f) : d * (1.f - h * h);
          st_relaxed_u32(xo, tagged(da, tag));
          o[0] = da;
        } else {
          const float r = in[it][1], z = in[it][2], n = in[it][3], q = in[it][4], hp = in[it][5];
          const float dn = d * (1.f - z) * (1.f - n * n);
          const float dz = d * (hp - n) * z * (1.f - z);
          const float dr = dn * q * r * (1.f - r);
          st_relaxed_u32(xo, tagged(dr, tag));
          st_relaxed_u32(xo + H, tagged(dz, tag));
          st_relaxed_u32(xo + 2 * H, tagged(dn * r, tag));
          float* oh = job.dgh + ((long long)t * a.B_total + b) * GH + j;
          o[0] = dr; o[H] = dz; o[2 * H] = dn;
          oh[0] = dr; oh[H] = dz; oh[2 * H] = dn * r;
          dc[it] = d * z;  // the direct part of the next dh
        }
      }
      if (sb + 1 < a.T) fetch(sb + 1);  // in flight during the exchange
      if (warp < stages) {
        load_tagged_tile<NB>(x + r0, GH, B, r_live, tag, b_tiles + warp * NB * 128, lane, waits, 14);
        fence_proxy_async();
        __syncwarp();
        if (sb > 0 && !waits.warp_bar<false>(read_bar, (sb - 1) & 1)) break;
        if (lane == 0) issue_tile<true, NB>(tmem_base, a_desc0, b_desc0, warp, done_bar);
        __syncwarp();
      }
      // the operand tiles may be overwritten, and the accumulators read, once the MMAs are done
      if (!waits.warp_bar<false>(done_bar, sb & 1)) break;
      const unsigned long long stamp = (unsigned long long)(sb + 1) << 32;
      // (all warps, those too whose rows lie past the end: one that only followed done_bar could fall two
      // steps behind it and miss a phase)
      {
        tc_fence_after();
        unsigned long long* to = push + slot * slot_size;
#pragma unroll
        for (int i = 0; i < kHalf; i += kChunk) {
          const int c0 = (warp >> 2) * kHalf + i;
          float v[kChunk];
          read_sums<NB, kChunk>(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c0, stages, v);
#pragma unroll
          for (int j = 0; j < kChunk / 4; ++j)
            if (row_live && c0 / 4 + j < quads) {
              unsigned long long* at = to + (long long)(c0 / 4 + j) * 4 * units;  // two pairs
              st_relaxed_v2(at, stamp | __float_as_uint(v[4 * j]), stamp | __float_as_uint(v[4 * j + 1]));
              st_relaxed_v2(at + 2 * units, stamp | __float_as_uint(v[4 * j + 2]), stamp | __float_as_uint(v[4 * j + 3]));
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(read_bar);
      }
      // ---- dh_{t-1} of this thread's pairs: the partial sums, in slice order
#pragma unroll
      for (int it = 0; it < kItems; ++it) {
        if (!live[it]) continue;
        const unsigned long long* from = pull + slot * slot_size +
                                         ((long long)(item_b[it] >> 1) * units + item_u[it]) * 2 + (item_b[it] & 1);
        float sum = 0.f;
        for (int q0 = 0; q0 < SL; q0 += kPull) {
          unsigned long long v[kPull];
          uint32_t pending = SL - q0 >= kPull ? (1u << kPull) - 1u : (1u << (SL - q0)) - 1u;
          const uint32_t mine = pending;
          if (*failed) pending = 0;
          int spins = 0;
          const long long t0 = clock64();
          while (pending) {
#pragma unroll
            for (int q = 0; q < kPull; ++q)
              if (pending >> q & 1) v[q] = ld_relaxed_u64(from + (q0 + q) * block);
#pragma unroll
            for (int q = 0; q < kPull; ++q)
              if ((pending >> q & 1) && (v[q] ^ stamp) >> 32 == 0) pending &= ~(1u << q);
            if (pending && waits.expired(&spins, t0, 15)) break;
          }
#pragma unroll
          for (int q = 0; q < kPull; ++q)
            if (mine >> q & 1) sum += __uint_as_float((uint32_t)v[q]);
        }
        dh[it] = G == 3 ? dc[it] + sum : sum;
      }
    }
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      if (!live[it]) continue;
      const long long at = (long long)item_b[it] * H + mt * kBM + rank * units + item_u[it];
      job.dh_out[at] = dh[it];
      if (G == 4) job.dc_out[at] = dc[it];
    }
  }
  __syncthreads();
  if (*failed)
    for (const long long t0 = clock64(); clock64() - t0 < 100000;) {
    }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kMaxStages * Acc<NB>::kCols);
  }
}

// ------------------------------------------------------------------------------------- host
typedef void (*FwdKernel)(const Launch<SeqJob>);
typedef void (*BwdKernel)(const Launch<SeqBwdJob>);

template <int G, int NB>
FwdKernel fwd_kernel(int ks) {
  return ks == 1 ? rnn_sequence_kernel<1, G, NB>
                 : (ks == 2 ? rnn_sequence_kernel<2, G, NB> : rnn_sequence_kernel<4, G, NB>);
}
FwdKernel fwd_kernel_for(int ks, int G, int NB) {
  if (NB == 32) return G == 1 ? fwd_kernel<1, 32>(ks) : (G == 3 ? fwd_kernel<3, 32>(ks) : fwd_kernel<4, 32>(ks));
  return G == 1 ? fwd_kernel<1, 48>(ks) : (G == 3 ? fwd_kernel<3, 48>(ks) : fwd_kernel<4, 48>(ks));
}
template <int G, int NB>
BwdKernel bwd_kernel(int items) {
  return items == 1 ? rnn_sequence_backward_kernel<1, G, NB>
         : items == 2 ? rnn_sequence_backward_kernel<2, G, NB>
         : items == 4 ? rnn_sequence_backward_kernel<4, G, NB>
                      : rnn_sequence_backward_kernel<8, G, NB>;
}
BwdKernel bwd_kernel_for(int items, int G, int NB) {
  if (NB == 32) return G == 1 ? bwd_kernel<1, 32>(items) : (G == 3 ? bwd_kernel<3, 32>(items) : bwd_kernel<4, 32>(items));
  return G == 1 ? bwd_kernel<1, 48>(items) : (G == 3 ? bwd_kernel<3, 48>(items) : bwd_kernel<4, 48>(items));
}

struct Plan {
  int rows;      // of the batch per job; 0: not supported
  int nb, ks, slice, ctas, items, units, split;
  size_t smem;
};

// K slices per cluster: as few as fit (each takes another partial sum through the cluster), equal in
// length.
Plan forward_plan(int B, int H, int G) {
  Plan p{};
  p.ks = H <= 256 ? 1 : (H <= 512 ? 2 : 4);
  p.slice = ((H + p.ks - 1) / p.ks + kBK - 1) / kBK * kBK;
  p.ctas = (H + kUnits - 1) / kUnits * p.ks;
  const int stages = p.slice / kBK;
  // up to 32 rows a job; up to 48 where they save a second job and fit in shared memory
  const size_t most = 227 * 1024;
  p.nb = 32;
  if (B > 32 && B <= 48 && seq_smem(stages, 48, kUnits * G * 48) <= most) p.nb = 48;
  const int parts = (B + p.nb - 1) / p.nb;
  p.rows = (B + parts - 1) / parts;
  p.smem = seq_smem(stages, p.nb, kUnits * G * p.nb);
  return p;
}
// Gate-row slices: short ones shorten the chain of MMAs and leave few pairs per thread, as long as
// `jobs` jobs fit on the device together (and a slice at most fills shared memory).
Plan backward_plan(int B, int H, int G, int jobs) {
  Plan p{};
  const int GH = G * H, mt = (H + kBM - 1) / kBM, outputs = H < kBM ? H : kBM;
  p.nb = B > 32 && B <= 48 ? 48 : 32;
  const int parts = (B + p.nb - 1) / p.nb;
  p.rows = (B + parts - 1) / parts;
  int sm = device_info().sm_count > 0 ? device_info().sm_count : 148;
  const int fewest = (GH + 32 * kMaxStages - 1) / (32 * kMaxStages);
  int want = sm / (mt * jobs);
  if (want < fewest && jobs > 1) want = sm / mt;
  p.split = std::max(fewest, std::min(std::min(want, 16), (GH + 31) / 32));
  p.slice = ((GH + p.split - 1) / p.split + kBK - 1) / kBK * kBK;
  p.split = (GH + p.slice - 1) / p.slice;
  p.units = (outputs + p.split - 1) / p.split;
  const int items = (p.units * p.nb + kSeqThreads - 1) / kSeqThreads;
  p.items = items <= 2 ? items : (items <= 4 ? 4 : 8);
  if (items > 8) p.rows = 0;
  p.ctas = mt * p.split;
  p.smem = seq_smem(p.slice / kBK, p.nb, 0);
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
int jobs_at_once(const Plan& p, int G, bool backward) {
  const int n = backward
                    ? resident(reinterpret_cast<const void*>(bwd_kernel_for(p.items, G, p.nb)), 1, p.smem) / p.ctas
                    : resident(reinterpret_cast<const void*>(fwd_kernel_for(p.ks, G, p.nb)), p.ks, p.smem) /
                          (p.ctas / p.ks);
  return std::min(n, kMaxJobs);
}
int jobs_of(const SeqShape& s, const Plan& p) { return s.dirs * ((s.B + p.rows - 1) / p.rows); }

Plan plan_for(const SeqShape& s, bool backward) {
  if (!backward) return forward_plan(s.B, s.H, s.G);
  const int parts = s.B <= 48 ? 1 : (s.B + 31) / 32;
  return backward_plan(s.B, s.H, s.G, std::min(kMaxJobs, s.dirs * parts));
}
size_t up256(size_t v) { return (v + 255) / 256 * 256; }
size_t xch_bytes(const SeqShape& s, const Plan& p, bool backward) {
  return up256((size_t)2 * p.rows * s.H * (backward ? s.G : 1) * 4);
}
size_t part_bytes(const Plan& p) { return up256((size_t)2 * p.ctas * p.split * ((p.rows + 3) / 4 * 4) * p.units * 8); }

template <typename Job>
int launch(const char* name, const SeqShape& s, const Plan& p, const Job* jobs, int n, bool backward,
           const void* kernel, void* scratch, cudaStream_t st, long long wait_budget, int absent_cta) {
  const int at_once = jobs_at_once(p, s.G, backward);
  FLB200_REQUIRE(at_once > 0, "%s: the device does not hold this launch", name);
  const size_t xb = xch_bytes(s, p, backward), pb = backward ? part_bytes(p) : 0;
  FLB200_CUDA_CHECK(cudaMemsetAsync(scratch, 0, (xb + pb) * (size_t)n, st));  // step number 0
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
      char* at = static_cast<char*>(scratch) + (xb + pb) * (size_t)(first + i);
      a.xch[i] = reinterpret_cast<uint32_t*>(at);
      a.part[i] = reinterpret_cast<unsigned long long*>(at + xb);
    }
    a.status = tc::status_ptr();
    a.wait_budget = wait_budget > 0 ? wait_budget : tc::kWaitBudget;
    a.out_stride = s.out_stride;
    a.dy_stride = s.dy_stride;
    a.T = s.T; a.B_total = s.B; a.H = s.H; a.act = s.act;
    a.slice = p.slice; a.units = p.units; a.ctas = p.ctas; a.split = p.split;
    a.absent_cta = absent_cta;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(m * p.ctas));
    cfg.blockDim = dim3(kSeqThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(backward ? 1 : p.ks);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[1] = {&a};
    FLB200_CUDA_CHECK(cudaLaunchKernelExC(&cfg, kernel, args));
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
  const int n = jobs_at_once(p, s.G, backward);
  // a large batch in many launches one after another would lose to a kernel per step
  return n > 0 && (jobs_of(s, p) + n - 1) / n <= 8 ? p.rows : 0;
}

size_t rnn_sequence_scratch_bytes(const SeqShape& s, bool backward) {
  if (s.B < 1 || s.H < 4 || s.H % 4 != 0 || s.H > 1024) return 0;
  const Plan p = plan_for(s, backward);
  if (p.rows == 0) return 0;
  return (xch_bytes(s, p, backward) + (backward ? part_bytes(p) : 0)) * (size_t)jobs_of(s, p);
}

int rnn_sequence_forward(const SeqShape& s, const SeqJob* jobs, int n, void* scratch, cudaStream_t st,
                         long long wait_budget, int absent_cta) {
  const Plan p = plan_for(s, false);
  return launch("rnn_sequence_forward", s, p, jobs, n, false,
                reinterpret_cast<const void*>(fwd_kernel_for(p.ks, s.G, p.nb)), scratch, st, wait_budget,
                absent_cta);
}
int rnn_sequence_backward(const SeqShape& s, const SeqBwdJob* jobs, int n, void* scratch,
                          cudaStream_t st) {
  const Plan p = plan_for(s, true);
  return launch("rnn_sequence_backward", s, p, jobs, n, true,
                reinterpret_cast<const void*>(bwd_kernel_for(p.items, s.G, p.nb)), scratch, st, 0, -1);
}

}  // namespace flb200
