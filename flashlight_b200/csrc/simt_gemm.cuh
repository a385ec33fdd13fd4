// fp32-FMA tiled contraction used by the STRICT (fp32 parity) mode of matmul and of the three
// convolution passes.  One kernel template; the operands are described by small "loader"
// functors, so a plain strided matrix, an im2col view of an image or a packed filter are all the
// same main loop.
//
//   C[z][m][n] = sum_k A[z](m,k) * B[z](k,n)
//
// What bounds it: the FP32 pipe, 128 FMA per clock and SM.  A loop of scalar FFMAs spends every
// issue slot on that pipe, so each load, address and shared-memory read costs arithmetic (the
// kernel this one replaces reached 18 TFLOP/s on ResNet-50: element-wise im2col gathers through
// registers, two barriers per 16 of K).  Here
//   * the arithmetic is packed, fma.rn.f32x2: half the issue slots for the same pipe time;
//   * an operand whose rows run contiguously stays [k][row] in shared memory: the halves of a
//     packed FMA are two neighbouring rows, the other side is broadcast.  Where k runs
//     contiguously in both they stay [row][k] and the halves are even and odd k, summed at the
//     end; that takes twice the accumulator registers and with them warps (9472 x 512 x 2304:
//     42 TFLOP/s against 49 with one side [k][row] and 55 with both);
//   * everything arrives by cp.async (16 bytes where the layout allows, else 4) in a ring of four
//     stages of 16 k, zero-filled at borders and tails;
//   * a product too small for 148 SMs splits K over a thread-block cluster of up to 8 CTAs and
//     adds the partial tiles through distributed shared memory, in rank order; only what still
//     leaves SMs idle after that goes through partial tiles in scratch and a second kernel.
// ResNet-50 forward, 29 images of 161 x 161: 7.8 -> 4.7 ms of contraction time; one MNIST digit:
// 167 -> 49 us.
//
// Loader concept (operand A indexes rows by m, operand B by n):
//   static constexpr int kKind;
//   kVecK  16-byte chunks along k:    Row row(r, z); Iter iter(k, z); advance(Iter&) by kBKf;
//                                     const float* at(Row, Iter) (null: zeros); k in chunks of 4
//   kVecRow  16-byte chunks along the row index, same interface (r a multiple of 4, advance by
//                                     kBKf as well)
//   kElemRows / kElemK  single elements, lanes along the rows / along k:
//                                     Row row(r, z); Kk kk(k, z); const float* at(Row, Kk)
//   const float* base() const;        any readable address (source of zero-size copies)
//
// Epilogue concept: element offsets of a row and of a column (-1: not stored) and
//   float* out; const float* bias (per column, may be null); float alpha, beta;
//   int along_m (consecutive rows are adjacent in memory, else consecutive columns);
//   int vec (the adjacent ones may be stored four at a time).
#pragma once
#include "common.cuh"
#include "tc_core.cuh"

namespace flb200 {

constexpr int kBKf = 16;       // k per stage
constexpr int kRingStages = 4;
constexpr int kRowPitch = 20;  // floats per [row][k] row: 16 k + 4, conflict-free 16-byte reads

enum { kVecK, kVecRow, kElemRows, kElemK };
constexpr bool k_layout(int kind) { return kind != kVecRow; }

// An 8 x 8 thread tile reads 16 floats per 64 FMA: 128 bytes a clock at full FMA rate, just what
// shared memory delivers; 8 x 4 is bound by it.  MINB: CTAs per SM to fit the registers to.
template <int BM_, int BN_, int TM_, int TN_, int MINB>
struct FfmaTile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, kMinBlocks = MINB;
  static constexpr int TX = BN / TN, TY = BM / TM;  // threads across columns / rows
  static constexpr int kThreads = TX * TY;
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src),
               "r"(live ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc::smem_u32(dst)), "l"(src),
               "r"(live ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
typedef unsigned long long f32x2;
__device__ __forceinline__ void ffma2(f32x2& d, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 both(float v) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float2 halves(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// Fills one operand's part of a stage; one instance per thread.
template <class L, int ROWS, int THREADS, int KIND = L::kKind>
struct Feeder;

template <class L, int ROWS, int THREADS>
struct Feeder<L, ROWS, THREADS, kVecK> {
  static constexpr int PASSES = ROWS * 4 / THREADS, STEP = THREADS / 4;
  static constexpr int kTableBytes = 0;
  typename L::Row rows[PASSES];
  typename L::Iter it;
  int k;
  __device__ void begin(const L& l, char*, int r0, int, int k0, int z) {
    const int t = threadIdx.x;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) rows[p] = l.row(r0 + t / 4 + STEP * p, z);
    k = k0 + 4 * (t & 3);
    it = l.iter(k, z);
  }
  __device__ void prepare(const L&, char*, int, int, int, int) {}
  __device__ void issue(const L& l, char*, float* dst, int, int kend) {
    const int t = threadIdx.x;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      const float* src = k < kend ? l.at(rows[p], it) : nullptr;
      cp_async16(dst + (t / 4 + STEP * p) * kRowPitch + 4 * (t & 3), src ? src : l.base(), src != nullptr);
    }
    k += kBKf;
    l.advance(it);
  }
};

template <class L, int ROWS, int THREADS>
struct Feeder<L, ROWS, THREADS, kVecRow> {
  static constexpr int CHUNKS = ROWS / 4, STEP = THREADS / CHUNKS, PASSES = kBKf / STEP;
  static constexpr int kTableBytes = 0;
  typename L::Row row;
  typename L::Iter it[PASSES];
  int k;
  __device__ void begin(const L& l, char*, int r0, int, int k0, int z) {
    const int t = threadIdx.x;
    row = l.row(r0 + 4 * (t % CHUNKS), z);
    k = k0 + t / CHUNKS;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) it[p] = l.iter(k + STEP * p, z);
  }
  __device__ void prepare(const L&, char*, int, int, int, int) {}
  __device__ void issue(const L& l, char*, float* dst, int, int kend) {
    const int t = threadIdx.x;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      const float* src = k + STEP * p < kend ? l.at(row, it[p]) : nullptr;
      cp_async16(dst + (t / CHUNKS + STEP * p) * ROWS + 4 * (t % CHUNKS), src ? src : l.base(), src != nullptr);
      l.advance(it[p]);
    }
    k += kBKf;
  }
};

// Single elements.  The decoded k of a stage (lanes along rows: 16 of them, made by 16 threads one
// stage ahead) or the decoded rows (lanes along k) sit in a shared table.  Rows past the last one are
// left as they are: nothing that they meet is stored.
template <class L, int ROWS, int THREADS>
struct Feeder<L, ROWS, THREADS, kElemRows> {
  static constexpr int KSTEP = THREADS / ROWS, PASSES = kBKf / KSTEP;
  static constexpr int kTableBytes = 2 * kBKf * (int)sizeof(typename L::Kk);
  typename L::Row row;
  bool live;
  __device__ void begin(const L& l, char*, int r0, int rows, int, int z) {
    row = l.row(r0 + threadIdx.x % ROWS, z);
    live = (int)(threadIdx.x % ROWS) < rows;
  }
  __device__ void prepare(const L& l, char* table, int k0, int slot, int kend, int z) {
    if (threadIdx.x < kBKf && k0 + (int)threadIdx.x < kend)
      reinterpret_cast<typename L::Kk*>(table)[(slot & 1) * kBKf + threadIdx.x] = l.kk(k0 + threadIdx.x, z);
  }
  __device__ void issue(const L& l, char* table, float* dst, int slot, int kleft) {
    if (!live) return;
    const int t = threadIdx.x;
    const typename L::Kk* kt = reinterpret_cast<const typename L::Kk*>(table) + (slot & 1) * kBKf;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      const int kl = t / ROWS + KSTEP * p;
      const float* src = kl < kleft ? l.at(row, kt[kl]) : nullptr;
      cp_async4(dst + (t % ROWS) * kRowPitch + kl, src ? src : l.base(), src != nullptr);
    }
  }
};
template <class L, int ROWS, int THREADS>
struct Feeder<L, ROWS, THREADS, kElemK> {
  static constexpr int RSTEP = THREADS / kBKf, PASSES = ROWS / RSTEP;
  static constexpr int kTableBytes = ROWS * (int)sizeof(typename L::Row);
  int k, z, live_rows;
  __device__ void begin(const L& l, char* table, int r0, int rows, int k0, int z_) {
    live_rows = rows < ROWS ? rows : ROWS;
    for (int r = threadIdx.x; r < live_rows; r += THREADS)
      reinterpret_cast<typename L::Row*>(table)[r] = l.row(r0 + r, z_);
    k = k0 + threadIdx.x % kBKf;
    z = z_;
  }
  __device__ void prepare(const L&, char*, int, int, int, int) {}
  __device__ void issue(const L& l, char* table, float* dst, int, int kend) {
    const int t = threadIdx.x;
    const typename L::Row* rows = reinterpret_cast<const typename L::Row*>(table);
    const bool live = k < kend;
    const typename L::Kk kk = l.kk(live ? k : 0, z);
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
      const int r = t / kBKf + RSTEP * p;
      if (r >= live_rows) break;
      const float* src = live ? l.at(rows[r], kk) : nullptr;
      cp_async4(dst + r * kRowPitch + t % kBKf, src ? src : l.base(), src != nullptr);
    }
    k += kBKf;
  }
};

template <class T, class AL, class BL>
struct FfmaSmem {
  static constexpr int kA = k_layout(AL::kKind) ? T::BM * kRowPitch : T::BM * kBKf;
  static constexpr int kB = k_layout(BL::kKind) ? T::BN * kRowPitch : T::BN * kBKf;
  static constexpr int kRing = kRingStages * (kA + kB) * 4;
  static constexpr int kTile = T::BM * (T::BN + 8) * 4;
  static_assert(kTile >= T::BN * (T::BM + 4) * 4, "both orders of the tile fit");
  static constexpr int kMain = kRing > kTile ? kRing : kTile;
  static constexpr int kTabA = (Feeder<AL, T::BM, T::kThreads>::kTableBytes + 15) / 16 * 16;
  static constexpr int kTabB = (Feeder<BL, T::BN, T::kThreads>::kTableBytes + 15) / 16 * 16;
  static constexpr int kTotal = kMain + kTabA + kTabB + (T::BM + T::BN) * 8;
};

// `splits` CTAs of a cluster (grid z, fastest) and psplits groups of them share the K range.
template <class T, class AL, class BL, class EP>
__global__ void __launch_bounds__(T::kThreads, T::kMinBlocks)
ffma_gemm_kernel(const AL al, const BL bl, const EP ep, int M, int N, int K, int tiles_n,
                 int csplits, int psplits, int k_per_split, float* __restrict__ partial) {
  chain_begin();
  constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, TX = T::TX, TY = T::TY;
  constexpr bool AK = k_layout(AL::kKind), BK = k_layout(BL::kKind);
  using S = FfmaSmem<T, AL, BL>;
  extern __shared__ __align__(16) char smem[];
  float* ring = reinterpret_cast<float*>(smem);
  char* tab_a = smem + S::kMain;
  char* tab_b = tab_a + S::kTabA;
  long long* roff = reinterpret_cast<long long*>(tab_b + S::kTabB);
  long long* coff = roff + BM;

  const int t = threadIdx.x;
  const int m0 = (int)(blockIdx.x / tiles_n) * BM, n0 = (int)(blockIdx.x % tiles_n) * BN;
  const int rank = (int)blockIdx.z % csplits, rest = (int)blockIdx.z / csplits;
  const int ps = rest % psplits, z = rest / psplits;
  const int kbeg = (ps * csplits + rank) * k_per_split;
  const int kend = min(kbeg + k_per_split, K);
  const int blocks = kbeg < kend ? (kend - kbeg + kBKf - 1) / kBKf : 0;

  Feeder<AL, BM, T::kThreads> fa;
  Feeder<BL, BN, T::kThreads> fb;
  constexpr bool kTables = AL::kKind >= kElemRows || BL::kKind >= kElemRows;
  fa.begin(al, tab_a, m0, M - m0, kbeg, z);
  fb.begin(bl, tab_b, n0, N - n0, kbeg, z);
  for (int r = t; r < BM; r += T::kThreads) roff[r] = m0 + r < M ? ep.row(m0 + r, z) : -1;
  for (int c = t; c < BN; c += T::kThreads) coff[c] = n0 + c < N ? ep.col(n0 + c, z) : -1;
  // the element feeders take what is left of the stage, the vector feeders their own k
  auto left_a = [&](int kb) { return AL::kKind == kElemRows ? kend - kb : kend; };
  auto left_b = [&](int kb) { return BL::kKind == kElemRows ? kend - kb : kend; };
  auto issue = [&](int b) {
    if (b < blocks) {
      float* dst = ring + (b % kRingStages) * (S::kA + S::kB);
      const int kb = kbeg + b * kBKf;
      fa.issue(al, tab_a, dst, b, left_a(kb));
      fb.issue(bl, tab_b, dst + S::kA, b, left_b(kb));
    }
    cp_async_commit();
  };
  auto prepare = [&](int b) {
    fa.prepare(al, tab_a, kbeg + b * kBKf, b, kend, z);
    fb.prepare(bl, tab_b, kbeg + b * kBKf, b, kend, z);
  };
  if (kTables) { prepare(0); __syncthreads(); }
#pragma unroll
  for (int b = 0; b < kRingStages - 1; ++b) {
    issue(b);
    if (kTables && b + 1 < blocks) { prepare(b + 1); __syncthreads(); }
  }

  // acc: even / odd k of (i, j) when both operands are [row][k]; else neighbouring columns (B
  // [k][row]) or neighbouring rows (only A is)
  constexpr int kAcc = (AK && BK) ? TM * TN : TM * TN / 2;
  f32x2 acc[kAcc];
#pragma unroll
  for (int i = 0; i < kAcc; ++i) acc[i] = 0ull;
  // a warp is 8 columns by 4 rows of threads
  const int lane = t & 31, warp = t >> 5;
  const int tx = lane % 8 + 8 * (warp % (TX / 8)), ty = lane / 8 + 4 * (warp / (TX / 8));

  for (int b = 0; b < blocks; ++b) {
    cp_async_wait<kRingStages - 2>();
    __syncthreads();
    issue(b + kRingStages - 1);
    if (kTables) prepare(b + kRingStages);
    const float* As = ring + (b % kRingStages) * (S::kA + S::kB);
    const float* Bs = As + S::kA;
#pragma unroll
    for (int q = 0; q < kBKf / 4; ++q) {
      if constexpr (AK && BK) {
        ulonglong2 a[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i)
          a[i] = *reinterpret_cast<const ulonglong2*>(As + (ty + TY * i) * kRowPitch + 4 * q);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Bs + (tx + TX * j) * kRowPitch + 4 * q);
#pragma unroll
          for (int i = 0; i < TM; ++i) ffma2(acc[i * TN + j], a[i].x, v.x);
#pragma unroll
          for (int i = 0; i < TM; ++i) ffma2(acc[i * TN + j], a[i].y, v.y);
        }
      } else if constexpr (!BK) {
        float4 a4[TM];
        if constexpr (AK) {
#pragma unroll
          for (int i = 0; i < TM; ++i)
            a4[i] = *reinterpret_cast<const float4*>(As + (ty + TY * i) * kRowPitch + 4 * q);
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          ulonglong2 v[TN / 4];
#pragma unroll
          for (int j = 0; j < TN / 4; ++j)
            v[j] = *reinterpret_cast<const ulonglong2*>(Bs + (4 * q + kk) * BN + 4 * (tx + TX * j));
          float a[TM];
          if constexpr (AK) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
              a[i] = kk == 0 ? a4[i].x : (kk == 1 ? a4[i].y : (kk == 2 ? a4[i].z : a4[i].w));
          } else {
#pragma unroll
            for (int i = 0; i < TM / 4; ++i)
              *reinterpret_cast<float4*>(a + 4 * i) =
                  *reinterpret_cast<const float4*>(As + (4 * q + kk) * BM + 4 * (ty + TY * i));
          }
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const f32x2 d = both(a[i]);
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) {
              ffma2(acc[(i * TN + 4 * j) / 2], d, v[j].x);
              ffma2(acc[(i * TN + 4 * j) / 2 + 1], d, v[j].y);
            }
          }
        }
      } else {
        float4 b4[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j)
          b4[j] = *reinterpret_cast<const float4*>(Bs + (tx + TX * j) * kRowPitch + 4 * q);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          ulonglong2 v[TM / 4];
#pragma unroll
          for (int i = 0; i < TM / 4; ++i)
            v[i] = *reinterpret_cast<const ulonglong2*>(As + (4 * q + kk) * BM + 4 * (ty + TY * i));
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const f32x2 d = both(kk == 0 ? b4[j].x : (kk == 1 ? b4[j].y : (kk == 2 ? b4[j].z : b4[j].w)));
#pragma unroll
            for (int i = 0; i < TM / 4; ++i) {
              ffma2(acc[(j * TM + 4 * i) / 2], v[i].x, d);
              ffma2(acc[(j * TM + 4 * i) / 2 + 1], v[i].y, d);
            }
          }
        }
      }
    }
  }

  // ---- the tile through shared memory: summed over the cluster, stored in memory order
  cp_async_wait<0>();
  __syncthreads();
  // (column after column where consecutive rows are adjacent in memory)
  const int pitch_r = ep.along_m ? 1 : BN + 8, pitch_c = ep.along_m ? BM + 4 : 1;
  float* tile = ring;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      float v;
      const int r = AK ? ty + TY * i : 4 * (ty + TY * (i / 4)) + i % 4;
      const int c = BK ? tx + TX * j : 4 * (tx + TX * (j / 4)) + j % 4;
      if constexpr (AK && BK) {
        const float2 h = halves(acc[i * TN + j]);
        v = h.x + h.y;
      } else if constexpr (!BK) {
        const float2 h = halves(acc[(i * TN + j) / 2]);
        v = j % 2 ? h.y : h.x;
      } else {
        const float2 h = halves(acc[(j * TM + i) / 2]);
        v = i % 2 ? h.y : h.x;
      }
      tile[r * pitch_r + c * pitch_c] = v;
    }
  if (csplits > 1) tc::cluster_sync_all();
  else __syncthreads();

  const int rows_here = BM / csplits, r_first = rank * rows_here;
  const uint32_t tile_u = tc::smem_u32(tile);
  const bool raw = psplits > 1;
  float* pbase = raw ? partial + ((long long)(z * psplits + ps) * M) * N : nullptr;
  // one or four adjacent values of the tile, summed over the cluster in rank order
  auto sum1 = [&](int at) {
    if (csplits == 1) return tile[at];
    float v = 0.f;
    for (int q = 0; q < csplits; ++q) {
      float u;
      asm volatile("ld.shared::cluster.f32 %0, [%1];"
                   : "=f"(u)
                   : "r"(tc::mapa_u32(tile_u + at * 4, (uint32_t)q)));
      v += u;
    }
    return v;
  };
  auto sum4 = [&](int at) {
    if (csplits == 1) return *reinterpret_cast<const float4*>(tile + at);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < csplits; ++q) {
      float4 u;
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(u.x), "=f"(u.y), "=f"(u.z), "=f"(u.w)
                   : "r"(tc::mapa_u32(tile_u + at * 4, (uint32_t)q)));
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    return v;
  };
  auto store4 = [&](float* to, float4 v, float4 bias) {
    float4* dst = reinterpret_cast<float4*>(to);
    v.x = ep.alpha * v.x + bias.x; v.y = ep.alpha * v.y + bias.y;
    v.z = ep.alpha * v.z + bias.z; v.w = ep.alpha * v.w + bias.w;
    if (ep.beta != 0.f) {
      const float4 o = *dst;
      v.x += ep.beta * o.x; v.y += ep.beta * o.y; v.z += ep.beta * o.z; v.w += ep.beta * o.w;
    }
    *dst = v;
  };
  if (raw ? !ep.along_m && (N & 3) == 0 : !ep.along_m && ep.vec != 0) {
    for (int idx = t; idx < rows_here * (BN / 4); idx += T::kThreads) {
      const int r = r_first + idx / (BN / 4), c = 4 * (idx % (BN / 4));
      const float4 v = sum4(r * pitch_r + c);
      if (roff[r] < 0 || coff[c] < 0) continue;
      if (raw) {
        *reinterpret_cast<float4*>(pbase + (long long)(m0 + r) * N + n0 + c) = v;
        continue;
      }
      float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ep.bias) {
        const float* bp = ep.bias + ep.bias_at(n0 + c, z);
        bias = make_float4(bp[0], bp[1], bp[2], bp[3]);
      }
      store4(ep.out + roff[r] + coff[c], v, bias);
    }
  } else if (!raw && ep.along_m && ep.vec != 0) {
    // four rows of a column per thread (one at a time, 16 x 28 x 28 x 256 -> 512 channels in fl's order
    // took 153 us, so 100)
    const int quads = rows_here / 4, shift = __ffs(quads) - 1;
    for (int idx = t; idx < quads * BN; idx += T::kThreads) {
      const int r = r_first + 4 * (idx & (quads - 1)), c = idx >> shift;
      const float4 v = sum4(r + c * pitch_c);
      if (roff[r] < 0 || coff[c] < 0) continue;
      const float b = ep.bias ? ep.bias[ep.bias_at(n0 + c, z)] : 0.f;
      store4(ep.out + roff[r] + coff[c], v, make_float4(b, b, b, b));
    }
  } else {
    // lanes along the rows where those are adjacent, or the columns too few to fill a warp
    const int cols = min(BN, N - n0), shift = __ffs(rows_here) - 1;
    const bool by_row = ep.along_m || cols < 16;
    for (int idx = t; idx < rows_here * (by_row ? cols : BN); idx += T::kThreads) {
      const int r = r_first + (by_row ? idx & (rows_here - 1) : idx / BN);
      const int c = by_row ? idx >> shift : idx % BN;
      float v = sum1(r * pitch_r + c * pitch_c);
      if (roff[r] < 0 || coff[c] < 0) continue;
      if (raw) {
        pbase[(long long)(m0 + r) * N + n0 + c] = v;
        continue;
      }
      float* dst = ep.out + roff[r] + coff[c];
      v = ep.alpha * v + (ep.bias ? ep.bias[ep.bias_at(n0 + c, z)] : 0.f);
      if (ep.beta != 0.f) v += ep.beta * *dst;
      *dst = v;
    }
  }
  if (csplits > 1) tc::cluster_sync_all();  // nobody leaves while a peer may read its tile
}

// Adds the partial tiles of the psplits groups in order and applies the epilogue.
template <class EP>
__global__ void __launch_bounds__(256)
ffma_reduce_kernel(const float* __restrict__ partial, const EP ep, int M, int N, int Z, int psplits) {
  chain_begin();
  const long long mn = (long long)M * N;
  const long long total = mn * Z;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int z = (int)(i / mn);
    const long long r = i - (long long)z * mn;
    const int m = (int)(r / N), n = (int)(r - (long long)m * N);
    const float* src = partial + (long long)z * psplits * mn + r;
    float s = 0.f;
#pragma unroll 8
    for (int sp = 0; sp < psplits; ++sp) s += src[(long long)sp * mn];
    float* dst = ep.out + ep.row(m, z) + ep.col(n, z);
    float v = ep.alpha * s + (ep.bias ? ep.bias[ep.bias_at(n, z)] : 0.f);
    if (ep.beta != 0.f) v += ep.beta * *dst;
    *dst = v;
  }
}

// ------------------------------------------------------------------ strided matrices
// A(row, k) = p[row * row_stride + k * k_stride + z * z_stride]; rows beyond `rows` read as 0.
template <int KIND>
struct StridedLoader {
  static constexpr int kKind = KIND;
  const float* p;
  long long row_stride, k_stride, z_stride;
  int rows;
  struct Row { long long off; };
  typedef long long Iter;
  typedef long long Kk;
  __device__ const float* base() const { return p; }
  __device__ Row row(int r, int z) const {
    return Row{r < rows ? r * row_stride + z * z_stride : -1};
  }
  __device__ Iter iter(int k, int) const { return k * k_stride; }
  __device__ Kk kk(int k, int) const { return k * k_stride; }
  __device__ void advance(Iter& it) const { it += kBKf * k_stride; }
  __device__ const float* at(const Row& r, long long k) const {
    return r.off >= 0 ? p + r.off + k : nullptr;
  }
};

struct StridedEpilogue {
  float* out;
  const float* bias;
  float alpha, beta;
  int along_m, vec;
  long long row_stride, col_stride, z_stride;
  __device__ long long row(int m, int z) const { return m * row_stride + z * z_stride; }
  __device__ long long col(int n, int) const { return n * col_stride; }
  __device__ int bias_at(int n, int) const { return n; }
};

// ------------------------------------------------------------------------- launch
struct SimtPlan {
  int tile;  // 0: 128 x 64, 1: 64 x 64, 2: 32 x 32
  int csplits, psplits;
  int k_per_split;
  size_t workspace_bytes;
};

// Clocks of one SM for the launch: FMA time at 128 per clock over the padded tiles (wider tiles
// read less shared memory per FMA), spread over rounds of the SMs, plus what a split costs.
inline SimtPlan plan_simt(long long M, long long N, long long K, long long Z) {
  struct Tile { int bm, bn; double slack, alone; };
  // slack: clocks per ideal clock of a full SM; alone: of one CTA by itself (four warps do not
  // cover their own latencies, and two of them feed two of the four schedulers)
  static const Tile tiles[3] = {{128, 64, 1.25, 1.8}, {64, 64, 1.35, 2.0}, {32, 32, 2.0, 3.5}};
  const long long sm = device_info().sm_count > 0 ? device_info().sm_count : 148;
  SimtPlan best{};
  double best_cost = -1.0;
  if (K < 1) K = 1;
  for (int i = 0; i < 3; ++i) {
    const Tile& t = tiles[i];
    const long long n = ((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn) * Z;
    for (int c = 1; c <= 8; c *= 2) {
      if (c > 1 && (K < 64LL * c || Z * c > 65535)) break;  // batches and splits share grid z
      for (int p = 1; p <= 64; p *= 2) {
        if (p > 1 && (c < 8 || K < 256LL * c * p || Z * c * p > 65535)) break;
        const long long kps = (K + (long long)c * p - 1) / ((long long)c * p);
        const long long ctas = n * c * p;
        const double ideal = (double)t.bm * t.bn * kps / 128.0;
        double time = ideal * t.slack * (double)((ctas + sm - 1) / sm);
        if (time < ideal * t.alone) time = ideal * t.alone;
        double cost = 3000.0 + time + (c > 1 ? 1500.0 : 0.0);
        if (p > 1) cost += 5000.0 + (double)M * N * Z * 4.0 * (2 * p) / 2500.0;
        if (best_cost < 0 || cost < best_cost) {
          best_cost = cost;
          best.tile = i;
          best.csplits = c;
          best.psplits = p;
        }
      }
    }
  }
  const long long s = (long long)best.csplits * best.psplits;
  best.k_per_split = (int)(((K + s - 1) / s + kBKf - 1) / kBKf * kBKf);
  best.workspace_bytes =
      best.psplits > 1 ? (size_t)(Z * best.psplits * M * N) * sizeof(float) : 0;
  return best;
}
template <class T, class AL, class BL, class EP>
int launch_ffma(const char* name, const AL& al, const BL& bl, const EP& ep, long long M, long long N,
                long long K, long long Z, const SimtPlan& p, float* partial, cudaStream_t st) {
  using S = FfmaSmem<T, AL, BL>;
  auto* kernel = ffma_gemm_kernel<T, AL, BL, EP>;
  static bool configured[64] = {false};
  int dev = 0;
  FLB200_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    FLB200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal));
    configured[dev] = true;
  }
  const long long tiles_m = (M + T::BM - 1) / T::BM, tiles_n = (N + T::BN - 1) / T::BN;
  FLB200_REQUIRE(tiles_m * tiles_n < 0x7fffffffLL && Z * p.csplits * p.psplits <= 65535,
                 "%s: extent out of range", name);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles_m * tiles_n), 1, (unsigned)(Z * p.csplits * p.psplits));
  cfg.blockDim = dim3(T::kThreads);
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (launch_chained)
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = (unsigned)p.csplits;
  cfg.attrs = attr;
  cfg.numAttrs = p.csplits > 1 ? 2 : 1;
  FLB200_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, al, bl, ep, (int)M, (int)N, (int)K, (int)tiles_n,
                                       p.csplits, p.psplits, p.k_per_split, partial));
  FLB200_AFTER_LAUNCH(name);
  return FLB200_OK;
}

template <class AL, class BL, class EP>
int launch_simt_gemm(const char* name, const AL& al, const BL& bl, const EP& ep, long long M,
                     long long N, long long K, long long Z, void* workspace,
                     size_t workspace_bytes, cudaStream_t st) {
  if (M <= 0 || N <= 0 || Z <= 0) return FLB200_OK;
  FLB200_REQUIRE(M < 0x7fffffffLL && N < 0x7fffffffLL && K >= 0 && K < 0x7fffff00LL,
                 "%s: extent out of range", name);
  constexpr bool kBothK = k_layout(AL::kKind) && k_layout(BL::kKind);
  constexpr bool kElem = AL::kKind >= kElemRows || BL::kKind >= kElemRows;
  SimtPlan p = plan_simt(M, N, K, Z);
  if (p.psplits > 1 && (!workspace || !aligned16(workspace) || workspace_bytes < p.workspace_bytes)) {
    // no scratch from the caller: the clusters alone share the K range
    p.psplits = 1;
    p.k_per_split = (int)(((K + p.csplits - 1) / p.csplits + kBKf - 1) / kBKf * kBKf);
    if (p.k_per_split < kBKf) p.k_per_split = kBKf;
  }
  FLB200_REQUIRE(Z * p.csplits * p.psplits <= 65535, "%s: too many batches", name);
  float* partial = static_cast<float*>(workspace);
  int rc;
  if constexpr (kElem) {
    // more threads for the same tile: single elements cost a dozen instructions each, and half as many
    // per thread hide twice the latency
    if (p.tile == 2)
      rc = launch_ffma<std::conditional_t<AL::kKind == kVecRow, FfmaTile<32, 32, 4, 2, 6>, FfmaTile<32, 32, 2, 4, 6>>>(
          name, al, bl, ep, M, N, K, Z, p, partial, st);
    else if (p.tile == 1)
      rc = launch_ffma<FfmaTile<64, 64, 8, 4, 4>>(name, al, bl, ep, M, N, K, Z, p, partial, st);
    else
      rc = launch_ffma<FfmaTile<128, 64, 8, 4, 2>>(name, al, bl, ep, M, N, K, Z, p, partial, st);
  } else if (p.tile == 2) {
    rc = launch_ffma<FfmaTile<32, 32, 4, 4, 8>>(name, al, bl, ep, M, N, K, Z, p, partial, st);
  } else if constexpr (kBothK) {
    rc = p.tile == 1
             ? launch_ffma<FfmaTile<64, 64, 8, 8, 4>>(name, al, bl, ep, M, N, K, Z, p, partial, st)
             : launch_ffma<FfmaTile<128, 64, 8, 8, 2>>(name, al, bl, ep, M, N, K, Z, p, partial, st);
  } else {
    rc = p.tile == 1
             ? launch_ffma<FfmaTile<64, 64, 8, 4, 4>>(name, al, bl, ep, M, N, K, Z, p, partial, st)
             : launch_ffma<FfmaTile<128, 64, 8, 8, 3>>(name, al, bl, ep, M, N, K, Z, p, partial, st);
  }
  if (rc) return rc;
  if (p.psplits > 1) {
    launch_chained(ffma_reduce_kernel<EP>, grid_for(M * N * Z, 256), 256, 0, st, partial, ep, (int)M, (int)N,
                                                                      (int)Z, p.psplits);
    FLB200_AFTER_LAUNCH("ffma_reduce");
  }
  return FLB200_OK;
}

}  // namespace flb200
