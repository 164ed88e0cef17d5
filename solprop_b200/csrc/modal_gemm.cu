// The modal transform as dense products: the GEMM route of the source evaluation.
//
// The reference synthesises the node field E[i, t] = tau sum_m S[i, m] a[m, t] and projects
// the node streams back, P_m(t) = sum_i W[m, i] P_i(t) / tau, as matrix products
// (src/solprop/backends/numpy_ref/passes/transforms.py:87-187; the native backend's
// synthesis provider native/src/general/trial.cpp:181-315 and its GEMM wrapper
// native/include/solprop_native/transforms/gemm.hpp:55-275).  On the fused route the
// response column synthesises and projects on CUDA cores from a modal window in shared
// memory; this route takes the products out of the column, so that any number of modes
// and nodes fits:
//
//   plain form (FP64):   k_gemm_f64, a tiled FP64 product, k summed in order;
//   mixed form (FP32):   each operand split into three BF16 parts x = hi + mid + lo
//                        (hi = bf16(x), mid = bf16(x - hi), lo = bf16(x - hi - mid)), and
//                        the six leading cross products hi.hi, mid.hi, hi.mid, lo.hi,
//                        mid.mid, hi.lo accumulated in FP32 by tcgen05.mma in tensor
//                        memory -- the K loop walks the six (A part, B part) pairs, so no
//                        operand is duplicated -- which keeps the product to FP32 accuracy
//                        (the terms left out are below 2^-24 of the leading one).
//
// The tcgen05 kernels put time along the accumulator's 128 lanes, so that its rows leave (and,
// for the projection, its operand's rows arrive) as coalesced rows of the FP32 node arrays:
// k_synthesis_split3, persistent, and k_project_split3, which splits the node streams into
// their BF16 parts on the way into tensor memory.  Every wait is bounded and a give-up marks
// *status (the column's status slot, which the host reads with the norms); tensor memory is
// freed on every path.  No load is multicast.
#include <cuda_bf16.h>

#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace sp {
namespace {

using namespace tc;

constexpr int kGM = 128, kGK = 64;
constexpr int kSynThreads = 384;  // warp 0: loads, warp 1: products, warps 4 .. 11: two groups of 128 lanes
constexpr int kProThreads = 512;  // ... warps 4 .. 15: three groups
constexpr uint32_t kPartBytes = kGM * kGK * 2;  // a 128 x 64 BF16 slice: 16 KB

// the six (A part, B part) pairs; the last, hi hi, has an accumulator of its own: the tensor
// core's FP32 accumulation does not round to nearest, so every product added to a large sum
// costs it accuracy, and the five small products are summed apart from the large one
__device__ constexpr int kTerms[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};

struct SplitMaps {
  CUtensorMap a[3];
  CUtensorMap b[3];
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc_all(uint32_t* slot) {  // every column, by one whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(512u)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_all(uint32_t tmem) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// ---- synthesis: E[row, t] = f sum_k S[row, k] a[k, t], f = *scale; accumulator lanes = 128
// samples t, columns = 128 rows of S.  A persistent CTA walks tiles t-major; a ring stage is
// one 64-wide K slice of the three parts of both operands (96 KB, two stages); the products of
// tile i go to accumulators i % 2, which eight warps drain -- lane t of column c is one element
// of row c, so a warp stores 128 contiguous bytes per column with no staging.
// What bounds it: the FP32 node field it writes.  32 768 rows x 32 768 samples, 30 modes:
// 0.86 ms (5.0 TB/s written); 2.04 ms with a CTA per 128 x 256 tile, drained through shared memory.
constexpr int kSynStages = 2, kSynAcc = 2;
constexpr uint32_t kSynStage = 6 * kPartBytes;
constexpr size_t kSynSmem = (size_t)kSynStages * kSynStage + 1024 + 256;

__global__ void __launch_bounds__(kSynThreads, 1)
    k_synthesis_split3(const __grid_constant__ SplitMaps maps, float* __restrict__ E, int n_rows, int n_t, int K,
                       int k_last, const double* scale, double* status) {
  extern __shared__ __align__(1024) unsigned char g_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)g_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + (size_t)kSynStages * kSynStage);
  uint64_t* empty = full + kSynStages;
  uint64_t* acc_full = empty + kSynStages;
  uint64_t* acc_empty = acc_full + kSynAcc;
  uint64_t* drain = acc_empty + kSynAcc;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  __shared__ volatile int failed;
  __shared__ volatile int consumed;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n_k = K / kGK, row_tiles = (n_rows + 127) / 128, tiles = (n_t / kGM) * row_tiles;
  // this CTA's tiles: consecutive, so that the samples' slices stay in L2
  const int first = (int)((long)blockIdx.x * tiles / gridDim.x), last = (int)((long)(blockIdx.x + 1) * tiles / gridDim.x);
  if (threadIdx.x == 0) {
    failed = 0;
    consumed = 0;
    for (int s = 0; s < kSynStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kSynAcc; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);
    }
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) tmem_alloc_all(tmem_slot);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  int loads = 0;  // K slices asked for (thread 0)
  if (threadIdx.x == 0) {
    int& g = loads;
    for (int tile = first; tile < last && !failed; ++tile) {
      const int t0 = (tile / row_tiles) * kGM, r0 = (tile % row_tiles) * 128;
      for (int k = 0; k < n_k; ++k, ++g) {
        const int s = g % kSynStages;
        if (g >= kSynStages && !mbar_wait(&empty[s], (uint32_t)(g / kSynStages - 1) & 1)) {
          failed = 1;
          break;
        }
        unsigned char* stage = ring + (size_t)s * kSynStage;
        mbar_expect_tx(&full[s], kSynStage);
        for (int p = 0; p < 3; ++p) {
          tma_load_2d(stage + p * kPartBytes, &maps.a[p], &full[s], k * kGK, t0);
          tma_load_2d(stage + (3 + p) * kPartBytes, &maps.b[p], &full[s], k * kGK, r0);
        }
      }
    }
  } else if (threadIdx.x == 32) {
    constexpr uint32_t kIdescN = idesc_bf16(kGM, 128);
    int g = 0, it = 0;
    for (int tile = first; tile < last && !failed; ++tile, ++it) {
      const int b = it % kSynAcc;
      if (it >= kSynAcc && !mbar_wait(&acc_empty[b], (uint32_t)(it / kSynAcc - 1) & 1)) {
        failed = 1;
        break;
      }
      for (int k = 0; k < n_k; ++k, ++g) {
        const int s = g % kSynStages;
        if (!mbar_wait(&full[s], (uint32_t)(g / kSynStages) & 1)) {
          failed = 1;
          break;
        }
        fence_after();
        const unsigned char* stage = ring + (size_t)s * kSynStage;
        const int steps = k == n_k - 1 ? k_last : kGK / 16;  // the last slice's padding is left out
#pragma unroll
        for (int term = 0; term < 6; ++term) {
          const uint64_t da = sw128_desc(stage + kTerms[term][1] * kPartBytes);  // the field's part
          const uint64_t db = sw128_desc(stage + (3 + kTerms[term][0]) * kPartBytes);
          for (int kk = 0; kk < steps; ++kk)
            umma_bf16(tmem + (uint32_t)b * 256 + (term < 5 ? 128 : 0), da + 2ull * kk, db + 2ull * kk, kIdescN,
                      (k | kk) != 0 || (term > 0 && term < 5) ? 1u : 0u);
        }
        umma_commit(&empty[s]);
        consumed = g + 1;
      }
      if (failed) break;
      umma_commit(&acc_full[b]);
    }
    umma_commit(drain);
  } else if (warp >= 4) {
    const int quarter = warp % 4, half = (warp - 4) / 4;
    const float f = scale ? (float)*scale : 1.0f;
    int it = 0;
    for (int tile = first; tile < last; ++tile, ++it) {
      const int b = it % kSynAcc;
      if (!warp_agrees(mbar_wait(&acc_full[b], (uint32_t)(it / kSynAcc) & 1) && !failed)) {
        failed = 1;
        break;
      }
      fence_after();
      const int t = (tile / row_tiles) * kGM + quarter * 32 + lane, r0 = (tile % row_tiles) * 128 + half * 64;
      float* out = E + (size_t)r0 * n_t + t;
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t v[32], low[32];
        __syncwarp();
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * 256 + half * 64 + c);
        tmem_load_32(acc, v);
        tmem_load_32(acc + 128, low);
        if (c == 32) {  // read: the accumulator may be filled again
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[b]);
        }
        if (r0 + c + 32 <= n_rows) {
#pragma unroll
          for (int j = 0; j < 32; ++j) out[(size_t)(c + j) * n_t] = f * (__uint_as_float(low[j]) + __uint_as_float(v[j]));
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (r0 + c + j < n_rows) out[(size_t)(c + j) * n_t] = f * (__uint_as_float(low[j]) + __uint_as_float(v[j]));
        }
      }
    }
  }
  __syncwarp();
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!mbar_wait(drain, 0)) failed = 1;
    if (failed)  // the loads in flight land before the CTA leaves
      for (int h = consumed; h < loads; ++h) mbar_wait(&full[h % kSynStages], (uint32_t)(h / kSynStages) & 1);
  }
  fence_before();
  __syncthreads();
  if (warp == 0) tmem_free_all(tmem);
  if (threadIdx.x == 0 && failed) *status = 1.0;
}

// ---- projection: partial[z][m, t] = sum over split z's nodes of W[m, i] P[i, t].  Accumulator
// lanes = 128 samples t, columns = BN modes.  The streams are the A operand, and it lives in
// tensor memory: a thread owns one sample, loads 64 nodes' values of it (coalesced along t),
// splits them into the three BF16 parts in registers and stores the parts as packed K pairs
// (lane t, 32 columns a part), three groups of four warps taking the slices in turn; W's parts
// come by TMA.  So the FP32 streams are read once and no BF16 copy of them touches memory.
// What bounds it: those reads and the slices' conversion.  32 768 rows x 32 768 samples, 30
// modes: 1.33 ms (3.2 TB/s read); 3.04 ms of split transpose and 1.90 ms of product before, when
// the parts went through memory.
constexpr int kProStages = 4;
constexpr uint32_t kProACols = 96;  // three parts of 64 BF16 in packed pairs
template <int BN> constexpr uint32_t project_stage() { return 3u * BN * kGK * 2; }
template <int BN> constexpr size_t project_smem() { return (size_t)kProStages * project_stage<BN>() + 1024 + 256; }
static_assert(kProStages * kProACols + 2 * 64 <= 512, "the stages and the accumulators fit tensor memory");

__device__ __forceinline__ void tmem_store_32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
// the product with its A operand in tensor memory
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the next BF16 part of 64 values as packed pairs; the values keep what is left of them
__device__ __forceinline__ void next_part(float (&v)[kGK], uint32_t (&packed)[kGK / 2]) {
#pragma unroll
  for (int i = 0; i < kGK / 2; ++i) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    packed[i] = *reinterpret_cast<const uint32_t*>(&pair);
    v[2 * i] -= __uint_as_float(packed[i] << 16);
    v[2 * i + 1] -= __uint_as_float(packed[i] & 0xffff0000u);
  }
}

template <int BN>
__global__ void __launch_bounds__(kProThreads, 1)
    k_project_split3(const __grid_constant__ SplitMaps maps, const float* __restrict__ streams, int n_nodes, int n_t,
                     int kpad, float* __restrict__ partial, int n_modes, size_t split_stride, double* status) {
  constexpr uint32_t kStage = project_stage<BN>();
  extern __shared__ __align__(1024) unsigned char g_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)g_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* w_full = reinterpret_cast<uint64_t*>(ring + (size_t)kProStages * kStage);
  uint64_t* a_full = w_full + kProStages;
  uint64_t* empty = a_full + kProStages;
  uint64_t* done = empty + kProStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  __shared__ volatile int failed;
  __shared__ volatile int consumed;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int t0 = blockIdx.x * kGM, m0 = blockIdx.y * BN;
  const int n_all = kpad / kGK;
  const int ks0 = (int)((long)blockIdx.z * n_all / gridDim.z), ks1 = (int)((long)(blockIdx.z + 1) * n_all / gridDim.z);
  const int total = ks1 - ks0;
  if (threadIdx.x == 0) {
    failed = 0;
    consumed = 0;
    for (int s = 0; s < kProStages; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&a_full[s], 4);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) tmem_alloc_all(tmem_slot);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;  // the accumulators' BN columns (hi hi, the rest), then the stages'

  int loads = 0;  // slices of W asked for (thread 0)
  if (threadIdx.x == 0) {
    int& g = loads;
    for (; g < total && !failed; ++g) {
      const int s = g % kProStages;
      if (g >= kProStages && !mbar_wait(&empty[s], (uint32_t)(g / kProStages - 1) & 1)) {
        failed = 1;
        break;
      }
      unsigned char* stage = ring + (size_t)s * kStage;
      mbar_expect_tx(&w_full[s], kStage);
      for (int p = 0; p < 3; ++p) tma_load_2d(stage + p * (BN * kGK * 2), &maps.b[p], &w_full[s], (ks0 + g) * kGK, m0);
    }
  } else if (threadIdx.x == 32) {
    constexpr uint32_t kIdescN = idesc_bf16(kGM, BN);
    for (int g = 0; g < total && !failed; ++g) {
      const int s = g % kProStages;
      const uint32_t parity = (uint32_t)(g / kProStages) & 1;
      if (!mbar_wait(&w_full[s], parity)) {
        failed = 1;
        break;
      }
      consumed = g + 1;
      if (!mbar_wait(&a_full[s], parity)) {
        failed = 1;
        break;
      }
      fence_after();
      const unsigned char* stage = ring + (size_t)s * kStage;
      const uint32_t a = tmem + 2 * BN + (uint32_t)s * kProACols;
#pragma unroll
      for (int term = 0; term < 6; ++term) {
        const uint64_t db = sw128_desc(stage + kTerms[term][1] * (BN * kGK * 2));
#pragma unroll
        for (int kk = 0; kk < kGK / 16; ++kk)
          umma_bf16_ts(tmem + (term < 5 ? BN : 0), a + (uint32_t)(kTerms[term][0] * 32 + kk * 8), db + 2ull * kk,
                       kIdescN, (g | kk) != 0 || (term > 0 && term < 5) ? 1u : 0u);
      }
      umma_commit(&empty[s]);
    }
    umma_commit(done);
  } else if (warp >= 4) {
    const int quarter = warp % 4, group = (warp - 4) / 4;
    const float* column = streams + t0 + quarter * 32 + lane;
    for (int g = group; g < total; g += 3) {
      const int s = g % kProStages, k0 = (ks0 + g) * kGK;
      float v[kGK];
#pragma unroll
      for (int i = 0; i < kGK; ++i) v[i] = k0 + i < n_nodes ? __ldcs(column + (size_t)(k0 + i) * n_t) : 0.0f;
      if (!warp_agrees((g < kProStages || mbar_wait(&empty[s], (uint32_t)(g / kProStages - 1) & 1)) && !failed)) {
        failed = 1;
        break;
      }
      fence_after();
      const uint32_t a = tmem + ((uint32_t)(quarter * 32) << 16) + 2 * BN + (uint32_t)s * kProACols;
      uint32_t packed[kGK / 2];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        next_part(v, packed);
        tmem_store_32(a + (uint32_t)p * 32, packed);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[s]);
    }
  }
  __syncwarp();
  __syncthreads();
  const bool ok = mbar_wait(done, 0);
  if (threadIdx.x == 0 && (!ok || failed))  // the loads in flight land before the CTA leaves
    for (int h = consumed; h < loads; ++h) mbar_wait(&w_full[h % kProStages], (uint32_t)(h / kProStages) & 1);
  __syncwarp();
  fence_after();
  if (warp >= 4 && warp < 8) {
    const int quarter = warp % 4;
    float* out = partial + (size_t)blockIdx.z * split_stride + t0 + quarter * 32 + lane;
#pragma unroll
    for (int c = 0; c < BN; c += 32) {
      uint32_t r[32], low[32];
      __syncwarp();
      tmem_load_32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c, r);
      tmem_load_32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(BN + c), low);
      const bool good = total > 0 && ok && !failed;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (m0 + c + j < n_modes)
          out[(size_t)(m0 + c + j) * n_t] = good ? __uint_as_float(low[j]) + __uint_as_float(r[j]) : 0.0f;
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 0) tmem_free_all(tmem);
  if (threadIdx.x == 0 && (!ok || failed)) *status = 1.0;
}

// out[i] = f sum_z partials[z][i], the splits added in order; f = *scale or 1 / *scale
template <class T>
__global__ void k_reduce_splits(const T* __restrict__ partials, int splits, size_t count, size_t stride,
                                T* __restrict__ out, size_t out_stride, int rows, const double* scale,
                                int divide) {
  // `rows` blocks of `count` values, block r at r * stride in each split and r * out_stride out
  const T f = (T)(divide ? 1.0 / *scale : *scale);
  const size_t total = (size_t)rows * count;
  for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < total; g += (size_t)gridDim.x * blockDim.x) {
    const size_t r = g / count, i = g % count;
    T acc = T(0);
    for (int z = 0; z < splits; ++z) acc += partials[(size_t)z * rows * stride + r * stride + i];
    out[r * out_stride + i] = f * acc;
  }
}

// the three BF16 parts of x, in the order hi, mid, lo
template <class T>
__device__ __forceinline__ void split3(T x, __nv_bfloat16 (&p)[3]) {
  const float v = (float)x;
  p[0] = __float2bfloat16_rn(v);
  const float r1 = v - __bfloat162float(p[0]);
  p[1] = __float2bfloat16_rn(r1);
  p[2] = __float2bfloat16_rn(r1 - __bfloat162float(p[1]));
}

// out[p][r][c] = part p of src[c][r] (c < C; 0 for C <= c < ld_out), r < R; 64 (c) x 32 (r)
// tiles through shared memory: the source is read in 128-byte rows, and each warp stores a
// part's 64 columns of one row as 32 BF16 pairs, a 128-byte row.  src rows have pitch
// ld_src; ld_out is even.
template <class T>
__global__ void __launch_bounds__(256) k_split3_transpose(const T* __restrict__ src, int C, int R, int ld_src,
                                                          __nv_bfloat16* __restrict__ out, int ld_out) {
  __shared__ T tile[64][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 64;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;  // 32 x 8
  for (int j = ty; j < 64; j += 8) {
    const int c = c0 + j, r = r0 + tx;
    tile[j][tx] = (c < C && r < R) ? src[(size_t)c * ld_src + r] : T(0);
  }
  __syncthreads();
  const size_t panel = (size_t)R * ld_out;
  for (int j = ty; j < 32; j += 8) {
    const int r = r0 + j, c = c0 + 2 * tx;
    if (r >= R || c >= ld_out) continue;
    __nv_bfloat16 a[3], b[3];
    split3(tile[2 * tx][j], a);
    split3(tile[2 * tx + 1][j], b);
    const size_t at = (size_t)r * ld_out + c;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      __nv_bfloat162 v;
      v.x = a[p];
      v.y = b[p];
      *reinterpret_cast<__nv_bfloat162*>(out + p * panel + at) = v;
    }
  }
}

// C[M, N] = f (A[M, K] B[K, N]), row-major, f = *scale or 1 / *scale, N even; 32 x 256 tiles:
// a thread takes 16 rows of two neighbouring columns, k summed in order.  Per k it reads its
// columns' pair and eight broadcast pairs of A from shared memory for 32 fused multiply-adds;
// slabs of 16 k arrive by cp.async while the last one is multiplied.
// What bounds it: FP64 issue (32 DFMA to 12 shared-memory wavefronts).  4 050 rows x 16 384
// complex samples, 30 modes: projection 598 -> 246 us, synthesis 280 -> 262 us against 64 x 64
// tiles of four by four outputs a thread, whose operands came as 8-byte reads.
constexpr int kFM = 32, kFN = 256, kFK = 16, kFPitch = kFM + 2;
constexpr size_t kF64Smem = sizeof(double) * 2 * kFK * (kFN + kFPitch);

template <int kBytes>
__device__ __forceinline__ void copy_async(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(smem)), "l"(gmem), "n"(kBytes),
               "r"(valid ? kBytes : 0)
               : "memory");
}

__global__ void __launch_bounds__(256, 2) k_gemm_f64(const double* __restrict__ A, int lda, const double* __restrict__ B,
                                                     int ldb, double* __restrict__ C, int ldc, int M, int N, int K,
                                                     const double* scale, int divide, size_t split_stride) {
  extern __shared__ __align__(16) double gf_raw[];
  double* Bs = gf_raw;                           // [2][kFK][kFN]
  double* As = gf_raw + (size_t)2 * kFK * kFN;   // [2][kFK][kFPitch], transposed
  const int tx = threadIdx.x % 128, rows = threadIdx.x / 128 * 16;
  const int m0 = blockIdx.y * kFM, n0 = blockIdx.x * kFN;
  // split K over gridDim.z: this CTA's slabs of kFK, its partial tile at C + z split_stride
  const int n_all = (K + kFK - 1) / kFK;
  const int kb0 = (int)((long)blockIdx.z * n_all / gridDim.z), kb1 = (int)((long)(blockIdx.z + 1) * n_all / gridDim.z);
  C += (size_t)blockIdx.z * split_stride;
  auto load = [&](int slab) {
    double* b = Bs + (size_t)(slab & 1) * kFK * kFN;
    double* a = As + (size_t)(slab & 1) * kFK * kFPitch;
    const int k0 = slab * kFK;
#pragma unroll
    for (int i = 0; i < kFK * kFN / 2 / 256; ++i) {
      const int kk = 2 * i + threadIdx.x / 128, c = 2 * tx;
      const bool in = k0 + kk < K && n0 + c < N;
      copy_async<16>(b + kk * kFN + c, in ? B + (size_t)(k0 + kk) * ldb + n0 + c : B, in);
    }
#pragma unroll
    for (int i = 0; i < kFK * kFM / 256; ++i) {
      const int at = i * 256 + threadIdx.x, kk = at % kFK, mm = at / kFK;
      const bool in = k0 + kk < K && m0 + mm < M;
      copy_async<8>(a + kk * kFPitch + mm, in ? A + (size_t)(m0 + mm) * lda + k0 + kk : A, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[16][2] = {};
  if (kb0 < kb1) load(kb0);
  for (int slab = kb0; slab < kb1; ++slab) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // this slab has arrived; the other buffer's readers are done
    if (slab + 1 < kb1) load(slab + 1);
    const double* b = Bs + (size_t)(slab & 1) * kFK * kFN + 2 * tx;
    const double* a = As + (size_t)(slab & 1) * kFK * kFPitch + rows;
    const int depth = min(kFK, K - slab * kFK);
#pragma unroll 4
    for (int kk = 0; kk < depth; ++kk) {
      const double2 v = *reinterpret_cast<const double2*>(b + kk * kFN);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const double2 w = *reinterpret_cast<const double2*>(a + kk * kFPitch + 2 * i);
        acc[2 * i][0] = fma(w.x, v.x, acc[2 * i][0]);
        acc[2 * i][1] = fma(w.x, v.y, acc[2 * i][1]);
        acc[2 * i + 1][0] = fma(w.y, v.x, acc[2 * i + 1][0]);
        acc[2 * i + 1][1] = fma(w.y, v.y, acc[2 * i + 1][1]);
      }
    }
  }
  const int n = n0 + 2 * tx;
  if (n >= N) return;
  const double s = scale ? *scale : 1.0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int m = m0 + rows + i;
    if (m >= M) continue;
    const double2 v = make_double2(!scale ? acc[i][0] : divide ? acc[i][0] / s : s * acc[i][0],
                                   !scale ? acc[i][1] : divide ? acc[i][1] / s : s * acc[i][1]);
    *reinterpret_cast<double2*>(C + (size_t)m * ldc + n) = v;
  }
}

// the FP64 projection's split-K factor: two waves of the 148 SMs' two CTAs each, as nearly as the
// tiles divide them, each split at least 8 slabs long; where that leaves SMs without a CTA, one CTA
// an SM of splits of 2 slabs at least (64 nodes, rows of 1 024, 8 tiles of 4 slabs: 12.1 -> 7.9 us)
int f64_splits(int tiles, int slabs) {
  const int s = std::min(4 * 148 / tiles, slabs / 8);
  return std::max(1, tiles * s >= 148 ? s : std::max(s, std::min(148 / tiles, slabs / 2)));
}
int f64_tiles(int n_modes, int n_to) { return ((n_to + kFN - 1) / kFN) * ((n_modes + kFM - 1) / kFM); }
// the tcgen05 projection's: CTAs for four waves of at least 4 slices, and no accumulator longer
// than 32 slices (2 048 nodes): its error grows with the length of the sum (kTerms).  Two waves are
// as fast, but their sums are twice as long: 1.0e-6 from 64 bits on a fibre where four leave
// about 5e-7 (3 600 nodes, rows of 4 096: 5.0e-7).
int split3_splits(int tiles, int k_slices) {
  int s = 1;
  while ((tiles * s < 4 * 148 && k_slices / (2 * s) >= 4) || k_slices > 32 * s) s *= 2;
  return s;
}
int mode_tile(int n_modes) { return n_modes <= 32 ? 32 : 64; }
int split3_tiles(int n_modes, int n_to) {
  const int bn = mode_tile(n_modes);
  return (n_modes + bn - 1) / bn * ((n_to + kGM - 1) / kGM);
}

// parts (rows, kpad) of an operand as tiles of box_rows x 64
bool part_maps(CUtensorMap (&maps)[3], const uint16_t* parts, int rows, int kpad, int box_rows) {
  for (int p = 0; p < 3; ++p)
    if (!make_bf16_map(&maps[p], parts + p * (size_t)rows * kpad, rows, kpad, kpad, box_rows, kGK)) return false;
  return true;
}

template <class T>
cudaError_t split_transpose(const T* src, int C, int R, int ld_src, uint16_t* out, int ld_out, cudaStream_t s) {
  const dim3 grid((R + 31) / 32, (ld_out + 63) / 64);
  k_split3_transpose<T><<<grid, 256, 0, s>>>(src, C, R, ld_src, reinterpret_cast<__nv_bfloat16*>(out), ld_out);
  return cudaGetLastError();
}

}  // namespace

int modal_kpad(int k) { return ((k + kGK - 1) / kGK) * kGK; }

cudaError_t configure_modal_gemm() {
  cudaError_t e = cudaFuncSetAttribute(k_synthesis_split3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSynSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_gemm_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF64Smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_project_split3<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)project_smem<32>());
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_project_split3<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)project_smem<64>());
}

void split3_host(const double* src, int rows, int cols, int ld_out, std::vector<uint16_t>& out) {
  out.assign((size_t)3 * rows * ld_out, 0);
  const size_t panel = (size_t)rows * ld_out;
  for (int r = 0; r < rows; ++r)
    for (int c = 0; c < cols; ++c) {
      const float v = (float)src[(size_t)r * cols + c];
      const __nv_bfloat16 hi = __float2bfloat16_rn(v);
      const float r1 = v - __bfloat162float(hi);
      const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
      const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
      const size_t at = (size_t)r * ld_out + c;
      out[at] = __bfloat16_as_ushort(hi);
      out[panel + at] = __bfloat16_as_ushort(mid);
      out[2 * panel + at] = __bfloat16_as_ushort(lo);
    }
}

cudaError_t modal_synthesis_f64(const double* S, const double* modal, double* E, int n_nodes, int n_modes,
                                int n_to, const double* taper, cudaStream_t s) {
  const dim3 grid((n_to + kFN - 1) / kFN, (n_nodes + kFM - 1) / kFM);
  k_gemm_f64<<<grid, 256, kF64Smem, s>>>(S, n_modes, modal, n_to, E, n_to, n_nodes, n_to, n_modes, taper, 0, 0);
  return cudaGetLastError();
}

size_t modal_projection_scratch(int n_modes, int n_nodes, int n_to) {
  const int s = std::max(f64_splits(f64_tiles(n_modes, n_to), (n_nodes + kFK - 1) / kFK),
                         split3_splits(split3_tiles(n_modes, n_to), modal_kpad(n_nodes) / kGK));
  return (size_t)s * n_modes * n_to;
}

cudaError_t modal_projection_f64(const double* W, const double* node_streams, double* out, int n_streams,
                                 int n_modes, int n_nodes, int n_to, size_t out_stride, const double* taper,
                                 double* scratch, cudaStream_t s) {
  const int splits = f64_splits(f64_tiles(n_modes, n_to), (n_nodes + kFK - 1) / kFK);
  const size_t part = (size_t)n_modes * n_to;
  const dim3 grid((n_to + kFN - 1) / kFN, (n_modes + kFM - 1) / kFM, splits);
  for (int st = 0; st < n_streams; ++st) {
    k_gemm_f64<<<grid, 256, kF64Smem, s>>>(W, n_nodes, node_streams + (size_t)st * n_nodes * n_to, n_to, scratch, n_to,
                                    n_modes, n_to, n_nodes, nullptr, 1, part);
    k_reduce_splits<double><<<592, 256, 0, s>>>(scratch, splits, part, part, out + st * out_stride, part, 1,
                                                taper, 1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t modal_synthesis_split3(const uint16_t* s_parts, const double* modal, uint16_t* modal_parts, float* E,
                                   int n_nodes, int n_modes, int n_to, int kpad, const double* taper,
                                   double* status, cudaStream_t s) {
  // A = the modal field transposed, (n_to, kpad) in three parts
  cudaError_t e = split_transpose<double>(modal, n_modes, n_to, n_to, modal_parts, kpad, s);
  if (e != cudaSuccess) return e;
  SplitMaps maps;
  if (!part_maps(maps.a, modal_parts, n_to, kpad, kGM) || !part_maps(maps.b, s_parts, n_nodes, kpad, 128))
    return cudaErrorInvalidValue;
  const int tiles = n_to / kGM * ((n_nodes + 127) / 128);
  const int k_last = (n_modes - (kpad - kGK) + 15) / 16;  // 16-wide steps of the last slice that hold modes
  k_synthesis_split3<<<std::min(tiles, 148), kSynThreads, kSynSmem, s>>>(maps, E, n_nodes, n_to, kpad, k_last, taper,
                                                                       status);
  return cudaGetLastError();
}

cudaError_t modal_projection_split3(const uint16_t* w_parts, const float* node_streams, float* out, int n_streams,
                                    int n_modes, int n_nodes, int n_to, int kpad, size_t out_stride,
                                    const double* taper, double* status, float* scratch, cudaStream_t s) {
  const int bn = mode_tile(n_modes);
  const int splits = split3_splits(split3_tiles(n_modes, n_to), kpad / kGK);
  const size_t part = (size_t)n_modes * n_to;
  SplitMaps maps;
  if (!part_maps(maps.b, w_parts, n_modes, kpad, bn)) return cudaErrorInvalidValue;
  const dim3 grid(n_to / kGM, (n_modes + bn - 1) / bn, splits);
  for (int st = 0; st < n_streams; ++st) {
    const float* streams = node_streams + (size_t)st * n_nodes * n_to;
    if (bn == 32)
      k_project_split3<32><<<grid, kProThreads, project_smem<32>(), s>>>(maps, streams, n_nodes, n_to, kpad, scratch,
                                                                       n_modes, part, status);
    else
      k_project_split3<64><<<grid, kProThreads, project_smem<64>(), s>>>(maps, streams, n_nodes, n_to, kpad, scratch,
                                                                       n_modes, part, status);
    k_reduce_splits<float><<<592, 256, 0, s>>>(scratch, splits, part, part, out + st * out_stride, part, 1, taper,
                                               1);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace sp
