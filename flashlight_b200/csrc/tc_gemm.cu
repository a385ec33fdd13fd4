// Host side of the tcgen05 contraction: turns a strided matmul description into
// TMA tensor maps + operand plans, picks the tile width and the split-K factor,
// and launches tc_gemm_kernel (tc_core.cuh).  Used by flb200_matmul / the linear
// gradients in TF32 mode, by the convolution paths in tc_conv.cu and by rnn.cu.
#include <cuda_bf16.h>

#include "tc_gemm.cuh"

#include <cstdlib>
#include <cstring>
#include <mutex>

#include "tc_pair.cuh"

namespace flb200 {
namespace tc {

// ------------------------------------------------------- driver entry point
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    (void)cudaGetLastError();
  });
  return fn;
}

// Tensor map of fp32 or 16-bit elements (`operand`); dims[0] is the contiguous dimension,
// strides_bytes[i] belongs to dims[i+1], box[0] is 128 bytes.  K-major operand tiles use the
// 128-byte swizzle of 16-byte chunks, MN-major ones the swizzle of 32-byte chunks.
int make_tensor_map(CUtensorMap* map, const void* base, int rank, const uint64_t* dims,
                    const uint64_t* strides_bytes, const uint32_t* box, int mode,
                    const uint32_t* elem_strides, int operand) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(FLB200_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
  cuuint64_t gd[5];
  cuuint64_t gs[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gd[i] = dims[i];
    bx[i] = box[i];
    es[i] = elem_strides ? elem_strides[i] : 1;
    if (i > 0) gs[i - 1] = strides_bytes[i - 1];
  }
  // Encoding a map is work of the host alone and depends on these values only: each thread keeps the
  // last ones that it made.
  struct Key {
    const void* base;
    cuuint64_t gd[5], gs[4];
    cuuint32_t bx[5], es[5];
    int rank, mode, operand, used;
  };
  struct Entry { Key key; CUtensorMap map; };
  static thread_local Entry known[512] = {};
  Key key;
  memset(&key, 0, sizeof(key));
  key.base = base;
  key.rank = rank; key.mode = mode; key.operand = operand; key.used = 1;
  unsigned long long h = reinterpret_cast<uintptr_t>(base) >> 4;
  for (int i = 0; i < rank; ++i) {
    key.gd[i] = gd[i]; key.bx[i] = bx[i]; key.es[i] = es[i];
    if (i > 0) key.gs[i - 1] = gs[i - 1];
    h = h * 31 + gd[i] + 17 * bx[i];
  }
  Entry& e = known[(h * 0x9e3779b97f4a7c15ull) >> 55];
  if (memcmp(&e.key, &key, sizeof(key)) == 0) {
    *map = e.map;
    return FLB200_OK;
  }
  CUresult r = fn(map,
                  operand == kOperandBf16   ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                  : operand == kOperandF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                           : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                  (cuuint32_t)rank, const_cast<void*>(base),
                  gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  mode == kMapStaging ? CU_TENSOR_MAP_SWIZZLE_NONE
                                      : (mode == kMapMnMajor ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                                                             : CU_TENSOR_MAP_SWIZZLE_128B),
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(FLB200_INVALID_ARG, "cuTensorMapEncodeTiled failed with code %d (rank %d)", (int)r,
                rank);
  e.key = key;
  e.map = *map;
  return FLB200_OK;
}

namespace {
thread_local bool t_x3 = false;
}
bool x3_enabled() { return t_x3; }
X3Scope::X3Scope(bool on) : prev(t_x3) { t_x3 = on; }
X3Scope::~X3Scope() { t_x3 = prev; }

std::atomic<long long> g_tc_launches{0};
void count_tc_launch() { g_tc_launches.fetch_add(1, std::memory_order_relaxed); }

// ------------------------------------------------------------ status flag
__device__ int g_tc_status = 0;

int* status_ptr() {
  // one address per device, looked up with that device current
  static int* ptrs[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!ptrs[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_tc_status) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    ptrs[dev] = static_cast<int*>(p);
  }
  return ptrs[dev];
}

// ---------------------------------------------------------------- launch
// Sums split-K partial tiles in split order, then applies the epilogue.
static __global__ void __launch_bounds__(256)
tc_splitk_reduce_kernel(const float* __restrict__ partial, EpiloguePlan ep, int M, int N, int Z,
                        int splits) {
  chain_begin();
  const long long mn = (long long)M * N;
  const long long total = mn * Z;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int z = (int)(i / mn);
    const long long r = i - (long long)z * mn;
    const int m = (int)(r / N), n = (int)(r - (long long)m * N);
    if (ep.m_valid != 0 && ep.m_div != 0 && (m % ep.m_div) >= ep.m_valid) continue;
    float s = 0.f;
    for (int sp = 0; sp < splits; ++sp) s += partial[((long long)z * splits + sp) * mn + r];
    const long long off = epi_off(m, ep.m_div, ep.m_stride, ep.m_outer) +
                          epi_off(n, ep.n_div, ep.n_stride, ep.n_outer) + (long long)z * ep.z_stride;
    float v = ep.alpha * s + (ep.bias_m ? ep.bias_m[m] : 0.f) + (ep.bias_n ? ep.bias_n[n] : 0.f);
    if (ep.out16 == kOperandBf16) {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.out) + off;
      if (ep.beta != 0.f) v += ep.beta * __bfloat162float(*dst);
      *dst = __float2bfloat16(v);
    } else if (ep.out16 == kOperandF16) {
      __half* dst = reinterpret_cast<__half*>(ep.out) + off;
      if (ep.beta != 0.f) v += ep.beta * __half2float(*dst);
      *dst = __float2half_rn(v);
    } else {
      float* dst = ep.out + off;
      if (ep.beta != 0.f) v += ep.beta * *dst;
      *dst = v;
    }
  }
}

// The same for a row-major result (unit column stride, no row / column regrouping) of a
// multiple of 4 columns: four columns per thread, 16-byte loads of every split's partial sums,
// and the activation of a fused linear layer (pre-activation rounded to T first, as the store
// of an unsplit product does).  G = 8: the warps of a CTA share the splits of 32 such quads, for many
// splits of a small result (72 x 36 of 100: a thread that takes them one after another waits 19 us, so 3.6).
template <typename T, int G>
static __global__ void __launch_bounds__(256)
tc_splitk_reduce_vec_kernel(const float4* __restrict__ partial, EpiloguePlan ep, int M, int N4,
                            int Z, int splits) {
  chain_begin();
  constexpr int kItems = 256 / G;
  __shared__ float4 shared_sum[G > 1 ? 256 : 1];
  const int item = threadIdx.x % kItems, g = threadIdx.x / kItems;
  const long long mn4 = (long long)M * N4;
  const long long total = mn4 * Z;
  for (long long i0 = (long long)blockIdx.x * kItems; i0 < total; i0 += (long long)gridDim.x * kItems) {
    const long long i = i0 + item < total ? i0 + item : total - 1;
    const int z = (int)(i / mn4);
    const long long r = i - (long long)z * mn4;
    const int m = (int)(r / N4), n = 4 * (int)(r - (long long)m * N4);
    const float4* src = partial + (long long)z * splits * mn4 + r;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int sp = g; sp < splits; sp += G) {
      const float4 p = src[(long long)sp * mn4];
      s.x += p.x; s.y += p.y; s.z += p.z; s.w += p.w;
    }
    if constexpr (G > 1) {
      __syncthreads();  // the sums of the quads before have been read
      shared_sum[threadIdx.x] = s;
      __syncthreads();
      if (g > 0) continue;
#pragma unroll
      for (int q = 1; q < G; ++q) {
        const float4 p = shared_sum[q * kItems + item];
        s.x += p.x; s.y += p.y; s.z += p.z; s.w += p.w;
      }
    }
    if (i0 + item >= total) continue;
    const long long off = (long long)m * ep.m_stride + n + (long long)z * ep.z_stride;
    const float bm = ep.bias_m ? ep.bias_m[m] : 0.f;
    float4 v = make_float4(ep.alpha * s.x + bm, ep.alpha * s.y + bm, ep.alpha * s.z + bm,
                           ep.alpha * s.w + bm);
    if (ep.bias_n) {
      const float4 b = *reinterpret_cast<const float4*>(ep.bias_n + n);
      v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    T* dst = reinterpret_cast<T*>(ep.out) + off;
    if (ep.beta != 0.f) {
      v.x += ep.beta * Num<T>::to_f(dst[0]); v.y += ep.beta * Num<T>::to_f(dst[1]);
      v.z += ep.beta * Num<T>::to_f(dst[2]); v.w += ep.beta * Num<T>::to_f(dst[3]);
    }
    if (ep.act) {
      v = epi_round<T>(v);
      if (ep.pre) epi_store4(static_cast<T*>(ep.pre) + off, v);
      v = make_float4(epi_gelu(v.x), epi_gelu(v.y), epi_gelu(v.z), epi_gelu(v.w));
    }
    epi_store4(dst, v);
  }
}

template <typename T>
static void launch_reduce_vec(const float4* partial, const EpiloguePlan& ep, long long M, long long N4, long long Z,
                              int splits, cudaStream_t st) {
  const long long total = M * N4 * Z;
  if (splits >= 16 && total < 148 * 256)
    launch_chained(tc_splitk_reduce_vec_kernel<T, 8>, grid_for(total, 32), 256, 0, st, partial, ep, (int)M,
                   (int)N4, (int)Z, splits);
  else
    launch_chained(tc_splitk_reduce_vec_kernel<T, 1>, grid_for(total, 256), 256, 0, st, partial, ep, (int)M,
                   (int)N4, (int)Z, splits);
}

static long long env_ll(const char* name, long long dflt) {
  const char* v = getenv(name);
  return v && *v ? atoll(v) : dflt;
}

template <int BN>
static int launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, const OperandPlan& pa,
                       const OperandPlan& pb, const EpiloguePlan& ep, long long M, long long N,
                       long long k_iters, long long Z, const Launch& L, float* partial,
                       cudaStream_t st, int operand) {
  GemmProblem<BN> p;
  p.operand = operand;
  p.a = make_coords(pa); p.b = make_coords(pb); p.ep = ep;
  p.a_mn_major = pa.mn_major; p.b_mn_major = pb.mn_major;
  p.M = (int)M; p.N = (int)N; p.k_iters = (int)k_iters;
  p.splits = L.splits; p.iters_per_split = L.iters_per_split;
  p.tiles_m = (int)((M + kBM - 1) / kBM);
  // Pair tiles walk the column tiles of one pair of row tiles first: the row operand (the
  // large one of a tall product) is then fetched from DRAM once and found in L2 by the other
  // column tiles, instead of being streamed once per column tile with the output written in
  // between (1 x 1 layers that widen 4x: 11-15 % faster; FLB200_PAIR_N_FAST=0: rows first).
  static const long long n_fast = env_ll("FLB200_PAIR_N_FAST", 1);
  p.pair_n_fast = (int)n_fast;
  p.tiles_n = (int)((N + BN - 1) / BN);
  p.Z = (int)Z;
  p.partial = partial;
  p.set_store_mode();
  const long long tiles = (long long)p.tiles_m * p.tiles_n * Z * L.splits;
  FLB200_REQUIRE(tiles < 0x7fffffffLL, "tc_gemm: too many tiles");
  if constexpr (BN >= 256) {
    if (L.pairs) {
      const long long pair_tiles = (long long)((p.tiles_m + 1) / 2) * p.tiles_n * Z * L.splits;
      return launch_pair_problem<GemmProblem<BN>, BN>("tc_gemm_pair", ma, mb, p, pair_tiles, st);
    }
  }
  return launch_problem<GemmProblem<BN>, BN>("tc_gemm", ma, mb, p, tiles, st);
}

// Wider tiles re-read the 128-row operand less often (the contraction is fed from L2):
// 256 columns as soon as there are enough of them to fill most of such a tile.
int pick_bn(long long N) {
  if (N <= 32) return 32;
  if (N <= 64) return 64;
  if (N < 192) return 128;
  return 256;
}

void plan_splits(long long tiles, long long k_iters, long long min_ips, int* splits_out,
                 int* ips_out) {
  // The persistent grid hands tile i to CTA i % grid, so the launch lasts
  // ceil(tiles * splits / SMs) rounds of one tile each.  Pick the split count with the
  // shortest critical path, charging every tile a fixed cost (pipeline fill, writing and
  // re-reading its partial sums) expressed in stage iterations.
  const long long sm = device_info().sm_count > 0 ? device_info().sm_count : 148;
  if (tiles < 1) tiles = 1;
  if (k_iters < 1) k_iters = 1;
  long long smax = k_iters / (min_ips > 0 ? min_ips : 1);
  const long long by_waves = (4 * sm + tiles - 1) / tiles;
  if (smax > by_waves) smax = by_waves;
  if (smax > 1024) smax = 1024;
  if (smax < 1) smax = 1;
  long long best_s = 1, best_ips = k_iters, best_cost = -1;
  for (long long s = 1; s <= smax; ++s) {
    const long long ips = (k_iters + s - 1) / s;
    const long long se = (k_iters + ips - 1) / ips;
    const long long rounds = (tiles * se + sm - 1) / sm;
    const long long cost = rounds * (ips + (se > 1 ? 16 : 4));
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best_s = se;
      best_ips = ips;
    }
  }
  *splits_out = (int)best_s;
  *ips_out = (int)best_ips;
}

// The launch lasts `rounds` tiles per CTA (or CTA pair), so the plan weighs the clocks of a tile
// against how evenly the tiles fill the 148 SMs.  Clocks of one stage (128 bytes of K), measured
// before a lane of the producers and issuers did nothing but add, and kept since (their order decides):
// a tile sits at the shared-memory port, 2 x (16 KB + BN x 128 B) per stage at 128 B/clock, and
// above ~420 of barrier hand-over; a pair halves the B half of that and runs at the tensor
// pipe's own 512.  A small product wants narrow tiles and a split of K for the sake of the
// idle SMs: a 128-row bf16 product of 2304 columns ran on 9 CTAs of 148 with 256-column tiles,
// 17 us; on 72 with 32-column ones, 7 us.
static Launch compute_launch(long long M, long long N, long long k_iters, long long Z, bool a_mn_major,
                             bool b_mn_major, int operand, bool split_k, long long sm, bool x3) {
  const int box = operand == kOperandTf32 ? 32 : 64;
  const long long tiles_m = (M + kBM - 1) / kBM;
  Launch best{};
  double best_cost = -1.0;
  struct Width { int bn, pairs, clocks; };
  static const Width widths[5] = {
      {256, 1, 530}, {256, 0, 780}, {128, 0, 520}, {64, 0, 440}, {32, 0, 420}};
  int widest = pick_bn(N);
  if (operand != kOperandTf32 && b_mn_major && widest < box) widest = box;
  for (const Width& w : widths) {
    if (w.bn > widest) continue;
    if (operand != kOperandTf32 && b_mn_major && w.bn < box) continue;  // one box at least
    if (w.pairs) {
      if (x3 || M <= kBM) continue;
      // TF32 pairs, measured: both operands MN-major win 4 % on the largest products and lose on others, and
      // a short K loop loses more to the cross-CTA hand-offs than it gains
      if (operand == kOperandTf32 && (b_mn_major || k_iters < (a_mn_major ? 8 : 4))) continue;
      if (k_iters < 4) continue;
    }
    double clocks = w.clocks * (x3 ? 2.5 : 1.0);
    // issuing a TMA copy took a producer warp ~120 clocks, and there are two of them.  (The boxes of a grouped
    // MN-major operand are one copy now, which counts as its boxes here still: counting it so changed no time
    // by more than noise.)
    const int copies = (a_mn_major ? kBM / box : 1) +
                       (b_mn_major ? (w.pairs ? w.bn / 2 : w.bn) / box : 1);
    if (clocks < copies * 65.0) clocks = copies * 65.0;
    const double drain = 600.0 + 8.0 * w.bn;  // storing one tile, hidden behind the next
    const long long units = w.pairs ? sm / 2 : sm;
    const long long tiles = (w.pairs ? (tiles_m + 1) / 2 : tiles_m) * ((N + w.bn - 1) / w.bn) * Z;
    const long long by_k = k_iters / 4;
    long long tries[3] = {1, units / (tiles > 0 ? tiles : 1), 2 * units / (tiles > 0 ? tiles : 1)};
    for (int i = 0; i < 3; ++i) {
      long long s = tries[i] < by_k ? tries[i] : by_k;
      if (i > 0 && (!split_k || s < 2)) continue;
      if (s < 1) s = 1;
      const long long ips = (k_iters + s - 1) / s;
      s = (k_iters + ips - 1) / ips;
      const long long rounds = (tiles * s + units - 1) / units;
      const double loop = ips * clocks > drain ? ips * clocks : drain;
      double cost = 4000.0 + rounds * loop + drain;
      // the partial sums and the second launch that adds them
      if (s > 1) cost += 4500.0 + (double)M * N * Z * 4.0 * (2 * s + 1) / 2500.0;
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best.bn = w.bn;
        best.pairs = w.pairs;
        best.splits = (int)s;
        best.iters_per_split = (int)ips;
      }
    }
  }
  best.workspace_bytes = best.splits > 1 ? (size_t)(Z * best.splits * M * N) * sizeof(float) : 0;
  return best;
}

// Weighing a plan takes 0.3 us and an operator asks for several (its workspace, its launch): each
// thread remembers the plans of the last sizes it saw.
Launch plan_launch(long long M, long long N, long long k_iters, long long Z, bool a_mn_major,
                   bool b_mn_major, int operand, bool split_k) {
  struct Entry { long long m, n, k, z, rest; Launch plan; };
  static thread_local Entry known[256] = {};
  const long long sm = device_info().sm_count > 0 ? device_info().sm_count : 148;
  const bool x3 = x3_enabled();
  if (k_iters < 1) k_iters = 1;
  const long long rest = 1 + (a_mn_major ? 2 : 0) + (b_mn_major ? 4 : 0) + (split_k ? 8 : 0) +
                         (x3 ? 16 : 0) + operand * 32LL + sm * 256;
  const unsigned long long h = ((unsigned long long)(M * 31 + N) * 31 + k_iters * 7 + Z) * 31 + rest;
  Entry& e = known[(h * 0x9e3779b97f4a7c15ull) >> 56];
  if (e.m != M || e.n != N || e.k != k_iters || e.z != Z || e.rest != rest)
    e = Entry{M, N, k_iters, Z, rest,
              compute_launch(M, N, k_iters, Z, a_mn_major, b_mn_major, operand, split_k, sm, x3)};
  return e.plan;
}

int run(const CUtensorMap& ma, const CUtensorMap& mb, const OperandPlan& pa, const OperandPlan& pb,
        const EpiloguePlan& ep, long long M, long long N, long long k_iters, long long Z, Launch L,
        void* ws, size_t ws_bytes, cudaStream_t st, int operand) {
  const uintptr_t out_addr = reinterpret_cast<uintptr_t>(ep.out);
  const bool rows_of_4 = ep.m_div == 0 && ep.n_div == 0 && ep.m_valid == 0 && ep.n_stride == 1 &&
                         N % 4 == 0 && ep.m_stride % 4 == 0 && ep.z_stride % 4 == 0 &&
                         out_addr % (ep.out16 ? 8 : 16) == 0 &&
                         (!ep.bias_n || aligned16(ep.bias_n));
  if (L.splits > 1) {
    // split-K partials are written with 16-byte vectors: an unaligned workspace is not used
    // (nor are the column statistics of the output taken from partial sums)
    const size_t one = (size_t)(Z * M * N) * sizeof(float);
    long long s = ws && aligned16(ws) ? (long long)(ws_bytes / one) : 0;
    if (s > L.splits) s = L.splits;
    if (s < 2 || ep.stats || (ep.act && !rows_of_4)) s = 1;
    L.iters_per_split = (int)((k_iters + s - 1) / s);
    L.splits = (int)((k_iters + L.iters_per_split - 1) / L.iters_per_split);
  }
  float* partial = static_cast<float*>(ws);
  int rc;
  if (L.bn == 32) rc = launch_gemm<32>(ma, mb, pa, pb, ep, M, N, k_iters, Z, L, partial, st, operand);
  else if (L.bn == 64) rc = launch_gemm<64>(ma, mb, pa, pb, ep, M, N, k_iters, Z, L, partial, st, operand);
  else if (L.bn == 128) rc = launch_gemm<128>(ma, mb, pa, pb, ep, M, N, k_iters, Z, L, partial, st, operand);
  else rc = launch_gemm<256>(ma, mb, pa, pb, ep, M, N, k_iters, Z, L, partial, st, operand);
  if (rc) return rc;
  if (L.splits > 1) {
    if (rows_of_4) {
      const float4* p4 = reinterpret_cast<const float4*>(partial);
      if (ep.out16 == kOperandBf16) launch_reduce_vec<__nv_bfloat16>(p4, ep, M, N / 4, Z, L.splits, st);
      else if (ep.out16 == kOperandF16) launch_reduce_vec<__half>(p4, ep, M, N / 4, Z, L.splits, st);
      else launch_reduce_vec<float>(p4, ep, M, N / 4, Z, L.splits, st);
    } else {
      const int rgrid = grid_for(M * N * Z, 256);
      launch_chained(tc_splitk_reduce_kernel, rgrid, 256, 0, st, partial, ep, (int)M, (int)N, (int)Z,
                                                     L.splits);
    }
    FLB200_AFTER_LAUNCH("tc_splitk_reduce");
  }
  return FLB200_OK;
}

}  // namespace tc

// ----------------------------------------------------- strided matmul entry
namespace {

struct Side {
  bool ok, mn_major;
  long long ld;  // stride (elements) of the non-contiguous dimension
};

// op(r, k) at base[r*row + k*col]: decide the major and the leading dimension.
// `vec` = elements per 16 bytes (4 for fp32, 8 for bf16): leading dimensions must keep every
// row 16-byte aligned.
Side classify(long long row, long long col, long long rows, long long K, long long vec) {
  Side s{false, false, 0};
  if (col == 1 && (row % vec == 0 || rows == 1) && row >= 1) {
    s = Side{true, false, rows == 1 ? (K + vec - 1) / vec * vec : row};
  } else if (row == 1 && (col % vec == 0 || K == 1) && col >= 1) {
    s = Side{true, true, K == 1 ? (rows + vec - 1) / vec * vec : col};
  }
  return s;
}

struct Prepared {
  bool ok = false;
  bool swap = false;
  Side a, b;
};

Prepared prepare(const flb200_matmul_desc* d, const void* a, const void* b, const void* c) {
  Prepared p;
  const bool bf16 = d->dtype == FLB200_BF16;
  if ((d->dtype != FLB200_F32 && !bf16) || d->m < 1 || d->n < 1 || d->k < 1) return p;
  const long long vec = bf16 ? 8 : 4;
  if (!aligned16(a) || !aligned16(b) || !c) return p;
  if (d->batch > 1 && (d->a_batch % vec != 0 || d->b_batch % vec != 0)) return p;
  // too little work to pay for a tensor-core launch: leave it to the fp32 kernel (bf16 has
  // no other kernel and always comes here)
  if (!bf16 && (double)d->m * (double)d->n * (double)d->k < 262144.0) return p;
  p.a = classify(d->a_row, d->a_col, d->m, d->k, vec);
  // B(k, n): "row" of the operand is n with stride b_col; k stride is b_row
  p.b = classify(d->b_col, d->b_row, d->n, d->k, vec);
  if (!p.a.ok || !p.b.ok) return p;
  p.swap = d->m < 64 && d->n > d->m;  // put the long extent on the 128-row side of the MMA
  p.ok = true;
  return p;
}

// Tensor map + plan of one operand: rows x K matrix (+ batch).
int build_operand(const Side& s, const void* base, long long rows, long long K, long long batch,
                  long long batch_stride, int tile_rows, CUtensorMap* map, tc::OperandPlan* plan,
                  int operand) {
  const bool half = operand != tc::kOperandTf32;
  const uint32_t kstage = tc::stage_k(operand);  // elements of K per stage (128 bytes)
  const uint64_t esize = half ? 2 : 4;
  uint64_t dims[4], strides[3];
  uint32_t box[4];
  *plan = tc::OperandPlan{};
  plan->k_inner = 0;
  plan->k2_dim = -1;
  int rank = 2;
  if (s.mn_major) {
    box[0] = half ? 64 : 32; box[1] = kstage;
    dims[0] = (uint64_t)rows; dims[1] = (uint64_t)K;
    plan->mn_major = 1; plan->mn_dim = 0; plan->k_dim = 1;
    if (rows % box[0] == 0) {
      dims[0] = box[0]; dims[2] = (uint64_t)rows / box[0];
      strides[1] = box[0] * esize;
      box[2] = (uint32_t)tile_rows / box[0];
      plan->mn_dim = 2;
      plan->mn_grouped = half ? 6 : 5;
      rank = 3;
    }
  } else {
    dims[0] = (uint64_t)K; dims[1] = (uint64_t)rows;
    box[0] = kstage; box[1] = (uint32_t)tile_rows;
    plan->mn_major = 0; plan->mn_dim = 1; plan->k_dim = 0;
  }
  plan->k_elems = (int)kstage;
  strides[0] = (uint64_t)s.ld * esize;
  plan->z_dim = -1;
  if (batch > 1) {
    dims[rank] = (uint64_t)batch;
    strides[rank - 1] = (uint64_t)batch_stride * esize;
    box[rank] = 1;
    plan->z_dim = rank++;
  }
  plan->rank = rank;
  // 16-bit tiles use the plain 128-byte swizzle for both majors
  return tc::make_tensor_map(map, base, rank, dims, strides, box,
                             s.mn_major && !half ? tc::kMapMnMajor : tc::kMapKMajor, nullptr,
                             operand);
}

}  // namespace

bool tc_gemm_supported(const flb200_matmul_desc* d, const void* a, const void* b, const void* c) {
  if (device_info().cc_major != 10) return false;
  if (!tc::encode_tiled_fn()) return false;
  return prepare(d, a, b, c).ok;
}

size_t tc_gemm_workspace_bytes(const flb200_matmul_desc* d) {
  if (!d || d->m < 1 || d->n < 1 || d->k < 1) return 0;
  // What the call will want depends on things that this query does not know (operand alignment,
  // and for the linear layers the type): the largest of the plans it may choose in this mode.
  size_t need = 0;
  for (int operand : {(int)tc::kOperandTf32, (int)tc::kOperandBf16}) {
    tc::X3Scope x3(operand == tc::kOperandTf32 && d->math_mode == FLB200_MATH_F32X3);
    const long long k_iters = (d->k + tc::stage_k(operand) - 1) / tc::stage_k(operand);
    for (int mn = 0; mn < 2; ++mn)
      for (int swap = 0; swap < 2; ++swap) {
        const size_t w = tc::plan_launch(swap ? d->n : d->m, swap ? d->m : d->n, k_iters, d->batch,
                                         mn != 0, mn != 0, operand, true)
                             .workspace_bytes;
        if (w > need) need = w;
      }
  }
  return need;
}

size_t tc_gemm_call_workspace_bytes(const flb200_matmul_desc* d, const void* a, const void* b, const void* c) {
  const Prepared p = prepare(d, a, b, c);
  if (!p.ok) return 0;
  const int operand = tc::operand_of(d->dtype);
  const long long kstage = tc::stage_k(operand);
  return tc::plan_launch(p.swap ? d->n : d->m, p.swap ? d->m : d->n, (d->k + kstage - 1) / kstage, d->batch,
                         (p.swap ? p.b : p.a).mn_major, (p.swap ? p.a : p.b).mn_major, operand, true)
      .workspace_bytes;
}

int tc_gemm_run(const flb200_matmul_desc* d, const void* a, const void* b, void* c, void* ws,
                size_t ws_bytes, cudaStream_t st, const float* bias_n, int act, void* pre,
                bool wide) {
  const Prepared p = prepare(d, a, b, c);
  if (!p.ok) return fail(FLB200_UNSUPPORTED, "tc_gemm: layout not covered");
  const bool fused = bias_n != nullptr || act != 0 || pre != nullptr;
  if (fused && (p.swap || d->c_col != 1 || d->beta != 0.f || d->n % 32 != 0 || d->batch != 1 ||
                (d->c_row & 7) != 0 || !aligned16(c) || (pre && !aligned16(pre))))
    return fail(FLB200_UNSUPPORTED,
                "tc_gemm: bias / activation are fused only into a row-major, 16-byte aligned "
                "result of a multiple of 32 columns");
  const int operand = tc::operand_of(d->dtype);
  const long long kstage = tc::stage_k(operand);
  const long long k_iters = (d->k + kstage - 1) / kstage;
  CUtensorMap ma, mb;
  tc::OperandPlan pa, pb;
  tc::EpiloguePlan ep{};
  ep.out = static_cast<float*>(c);
  ep.out16 = wide ? 0 : operand;
  ep.alpha = d->alpha;
  ep.beta = d->beta;
  ep.z_stride = d->c_batch;
  ep.bias_n = bias_n;
  ep.act = act;
  ep.pre = pre;
  // swapped, C^T = B^T A^T: the kernel's rows are the caller's columns
  const Side &sa = p.swap ? p.b : p.a, &sb = p.swap ? p.a : p.b;
  const long long M = p.swap ? d->n : d->m, N = p.swap ? d->m : d->n;
  ep.m_stride = p.swap ? d->c_col : d->c_row;
  ep.n_stride = p.swap ? d->c_row : d->c_col;
  const tc::Launch L =
      tc::plan_launch(M, N, k_iters, d->batch, sa.mn_major, sb.mn_major, operand, ws != nullptr);
  if (int rc = build_operand(sa, p.swap ? b : a, M, d->k, d->batch, p.swap ? d->b_batch : d->a_batch,
                             tc::kBM, &ma, &pa, operand))
    return rc;
  if (int rc = build_operand(sb, p.swap ? a : b, N, d->k, d->batch, p.swap ? d->a_batch : d->b_batch,
                             L.b_box_rows(), &mb, &pb, operand))
    return rc;
  return tc::run(ma, mb, pa, pb, ep, M, N, k_iters, d->batch, L, ws, ws_bytes, st, operand);
}

}  // namespace flb200

extern "C" {

int flb200_has_tensor_core_path(void) {
  return flb200::device_info().cc_major == 10 && flb200::tc::encode_tiled_fn() != nullptr ? 1 : 0;
}

long long flb200_tc_kernel_launches(void) {
  return flb200::tc::g_tc_launches.load(std::memory_order_relaxed);
}

// Reads (and clears) the device flag that a bounded wait inside a tensor-core kernel raises when
// it runs out.  Synchronises the stream.  Returns FLB200_TIMEOUT if the flag was set.
int flb200_tc_poll_status(void* stream) {
  using namespace flb200;
  int* p = tc::status_ptr();
  if (!p) return FLB200_OK;
  int v = 0;
  cudaStream_t st = as_stream(stream);
  FLB200_CUDA_CHECK(cudaMemcpyAsync(&v, p, sizeof(int), cudaMemcpyDeviceToHost, st));
  FLB200_CUDA_CHECK(cudaStreamSynchronize(st));
  if (v != 0) {
    FLB200_CUDA_CHECK(cudaMemsetAsync(p, 0, sizeof(int), st));
    return fail(FLB200_TIMEOUT, "a tensor-core kernel gave up waiting (stage %d)", v);
  }
  return FLB200_OK;
}

}  // extern "C"
