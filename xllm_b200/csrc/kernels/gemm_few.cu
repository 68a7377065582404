// Products of few rows (decode: up to 64), C[M, N] (bf16) = A[M, K] W[N, K]^T, whose time is the weights' way from HBM:
//
//   bf16               (+ bias), the contract of xllm_gemm_bf16
//   block-scaled fp8   sum over 128-wide K blocks of (A_q . W_q^T) a_scale[m, kb] w_scale[n / 128, kb], A_q, W_q e4m3, sums in
//                      fp32: that of xllm_gemm_fp8_block
//   grouped (experts)  either, rows of A sorted by expert in tiles of TN rows, tile_expert as in gemm_tcgen05.cu; bf16 also
//                      with the gated activation of interleaved gate and up rows
//
// The operands are swapped: 128 WEIGHT rows are the rows of the tcgen05 tile and 16, 32 or 64 token rows its columns, so what
// is read back (per K block for fp8, whose blocks differ in scale) is the tokens there are, not 128 columns of weights for a
// tile of mostly absent rows, and an expert with four rows costs no loads and stores of 128.  A CTA needs half an SM, and two
// of them cover each other's start and end.  The first weights of an ungrouped product start for L2 before the wait for the
// kernel in front.  Where the tiles alone leave SMs idle:
//
//   bf16  a cluster of up to eight CTAs cuts K: every CTA sums its slice, the slices meet through distributed shared memory, in a
//         fixed order.  (Split-K in gemm_tcgen05.cu meets in scratch memory by reduce-adds, a round trip of some 6 us.)
//   fp8   narrower tiles, of 64 or 32 weight rows (instructions of 64 rows; of 32 weight rows, the others are whatever lies behind
//         and are not read back), and more of them side by side for more rows of A.  K stays whole, so that the scaled blocks
//         are added one after the other as in gemm_fp8_block_kernel and a row comes out with the same bits however many rows
//         there are: the e4m3 rounding in front of the next product turns other last bits into other values (K cut over
//         clusters: a step of two latent layers 0.02 to 0.03 from the same rows' among many).
//
// Measured (one B200, 16 rows, before: gemm_fp8_block_kernel): 7168 x 16384 fp8 (117 MB of weights, 18 us at the copy rate)
// 56 -> 29 us, 1536 x 7168 25 -> 10 us, 7168 x 18432 63 -> 32 us; 32 experts, of which every row chose eight, 4096 x 7168 214 -> 163
// us (143 at the copy rate) and 7168 x 2048 186 -> 92 us (72).  bf16, one row (before: split-K in gemm_tcgen05.cu, and the
// activation's own kernel): 4096 x 4096 13 -> 9 us, gated 24576 x 4096 44 -> 39 us (31 at the copy rate), 4096 x 12288 26 -> 20 us.
//
// Every mbarrier wait is bounded; on expiry all roles leave, tensor memory is released and an error word is set
// (xllm_gemm_few_error_status).
#include "tc_common.cuh"
#include <atomic>
#include <mutex>

namespace xllm {
namespace few {

using namespace tc;

constexpr int kMaxSplit = 8, kPrefetchBlocks = 8;
constexpr int kFp8MaxK = 49152;        // the scales of a whole K lie in shared memory: 98 KB at most

// WR: weight rows of a tile; G: K blocks of a stage of the ring, which are also read back together
template <int TN, bool FP8, int WR, int G>
struct Smem {
  static constexpr int acc = FP8 ? (256 / (G * TN) < 4 ? 256 / (G * TN) : 4) : 1;     // groups of G accumulators
  static constexpr int cols = FP8 ? acc * G * TN : (TN < 32 ? 32 : TN);               // of tensor memory
  static constexpr int w_bytes = WR * 128, x_bytes = TN * 128, block = w_bytes + x_bytes, stage = G * block;
  static constexpr int stages = FP8 ? 100 * 1024 / stage : (TN == 64 ? 3 : 4);
  static constexpr int rows = WR < 128 ? 64 : 128;                                    // of an instruction
  static constexpr int behind = rows * 128 - block > 0 ? rows * 128 - block : 0;      // rows the last block's instructions read beyond it
  static constexpr int readers = WR < 128 ? WR / 16 : 4;                              // warps with rows of the tile
  static constexpr int bars = stages * stage + behind, scales = bars + (2 * stages + 2 * acc) * 8 + 16;
  static constexpr int total(int k_blocks) { return scales + (FP8 ? k_blocks * (TN + 1) * 4 : 0) + 1024; }
  static_assert(WR % 32 == 0 && block % 1024 == 0 && cols <= 256 && acc >= 2 - !FP8, "swizzled tiles, and two CTAs an SM");
  static_assert(FP8 || (WR == 128 && G == 1 && 2 * TN * 128 * 4 <= stages * stage), "the sums meet where the ring was");
};

struct Params {
  bf16* c;
  int64_t ldc;
  const float *a_scale, *w_scale;      // fp8
  const bf16* bias;                    // bf16, or null
  int M, N, k_blocks, x_rows, sliced;  // k_blocks of 128 bytes; x_rows: rows of a copy of A
  const int32_t* tile_expert;
  int act;                             // 0, or as in GemmMode: W's rows are [64 gate | 64 up], C has N / 2 columns
  float limit, alpha;
  int* err;
};

// kind::f8f6f4, A = B = e4m3 (both K-major), D = f32, M = 128
__device__ __forceinline__ void umma_fp8(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void prefetch_2d(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, uint32_t rank) {
  float v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
               : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}

__device__ __forceinline__ void copy_f32(float* dst, const float* src, bool in) {      // zero where not
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}

__device__ __forceinline__ float gated(float x, float y, int act, float limit, float alpha) {
  if (act == 4) return clamped_glu(x, y, limit, alpha);
  if (act == 1) return x / (1.f + __expf(-x)) * y;
  if (act == 2) return 0.5f * x * (1.f + erff(x * 0.70710678f)) * y;
  return 0.5f * x * (1.f + tanhf(0.7978845608f * (x + 0.044715f * x * x * x))) * y;
}

// grid: row tiles x tiles of WR weight rows; with slices of K, which make the cluster, (slices, tiles)
template <int TN, bool FP8, int WR, int G>
__global__ void __launch_bounds__(192, 2)
gemm_few_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w, const Params p) {
  using S = Smem<TN, FP8, WR, G>;
  constexpr int kAcc = S::acc;
  constexpr int KE = FP8 ? 128 : 64;                                  // elements of a K block
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem), bar0 = sbase + S::bars;
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (S::stages + s); };
  auto tfull = [&](int a) { return bar0 + 8u * (2 * S::stages + a); };
  auto tempty = [&](int a) { return bar0 + 8u * (2 * S::stages + kAcc + a); };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + S::bars + (2 * S::stages + 2 * kAcc) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* scales = reinterpret_cast<float*>(smem + S::scales);         // [K block of the slice][row]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (The number of slices from the grid, which is known to be positive: the loop over the rows they share is unrolled by it.  From a
  // parameter, 64 rows of 6144 x 4096 take 20.7 us instead of 19.2.)
  const int splits = p.sliced ? gridDim.x : 1, rank = p.sliced ? blockIdx.x : 0, tile = p.sliced ? blockIdx.y : blockIdx.x;
  const int m_tiles = (p.M + TN - 1) / TN, mt = tile % m_tiles, nt = tile / m_tiles;
  const int kb0 = (int)((int64_t)rank * p.k_blocks / splits), kb1 = (int)((int64_t)(rank + 1) * p.k_blocks / splits);
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::stages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int a = 0; a < kAcc; ++a) {
      mbar_init(tfull(a), 1);
      mbar_init(tempty(a), S::readers);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (p.tile_expert == nullptr && warp == 0) {
    if (lane < kPrefetchBlocks && kb0 + lane < kb1) prefetch_2d(&tma_w, (kb0 + lane) * KE, nt * WR);
    __syncwarp();
  }
  pdl_wait();
  int expert = 0;
  if (p.tile_expert != nullptr) {
    expert = p.tile_expert[mt];
    if (expert < 0) return;            // uniform for the cluster: nothing allocated yet
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(S::cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Not before the allocation: a dependent block that came first could take this SM's tensor memory and keep it in its own wait
  // for this grid, which would then wait for it without end.
  pdl_launch_dependents();
  const uint32_t tmem = *tmem_holder;
  const int m0 = mt * TN, n0 = nt * WR;
  const int live = min(TN, p.M - m0);
  float acc[TN];
  bool ok = true;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    const int wy = expert * p.N + n0;
    for (int kb = kb0, i = 0; kb < kb1; kb += G, ++i) {
      const int st = i % S::stages;
      if (!mbar_wait_warp(empty(st), ((i / S::stages) & 1) ^ 1, abort_flag)) { ok = false; break; }
      const uint32_t dst = sbase + st * S::stage;
      if (elect_one()) {
        mbar_expect_tx(full(st), min(G, kb1 - kb) * (S::w_bytes + p.x_rows * 128));
#pragma unroll
        for (int b = 0; b < G; ++b)
          if (kb + b < kb1) {
            tma_load_2d(dst + b * S::block, &tma_w, (kb + b) * KE, wy, full(st));
            tma_load_2d(dst + b * S::block + S::w_bytes, &tma_x, (kb + b) * KE, m0, full(st));
          }
      }
      __syncwarp();
    }
    if (!ok) {
      const long long t0 = clock64();
      while (clock64() - t0 < 20000000LL) {}          // bounded grace period for copies in flight
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t ID = FP8 ? (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(S::rows >> 4) << 24) : idesc(false, TN);
    for (int kb = kb0, i = 0; kb < kb1; kb += G, ++i) {
      const int st = i % S::stages, a = i % kAcc;
      if (FP8 && !mbar_wait_warp(tempty(a), ((i / kAcc) & 1) ^ 1, abort_flag)) break;
      if (!mbar_wait_warp(full(st), (i / S::stages) & 1, abort_flag)) break;
      tc_fence_after();
      const uint64_t wd = smem_desc(sbase + st * S::stage, 16, 1024), xd = smem_desc(sbase + st * S::stage + S::w_bytes, 16, 1024);
      if (elect_one()) {
        // the blocks of a stage in turn: a product waits for the one in front that adds to the same accumulator
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int b = 0; b < G; ++b)
            if (G == 1 || kb + b < kb1) {
              const uint64_t at = b * (S::block >> 4) + 2 * k;
              if constexpr (FP8) umma_fp8(tmem + (a * G + b) * TN, wd + at, xd + at, ID, k != 0);
              else umma(tmem, wd + at, xd + at, ID, (i | k) != 0);
            }
        umma_commit(empty(st));        // the ring slot is free once these MMAs have read it
        if (FP8) umma_commit(tfull(a));                // ... and the blocks' products are complete
        else if (kb + 1 == kb1) umma_commit(tfull(0));
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ scale and add (warps 2..5): a thread owns a weight row
    const int t = threadIdx.x - 64, n_kb = kb1 - kb0;
    const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    constexpr int C = TN < 32 ? 16 : 32;
    if constexpr (FP8) {
      // All of them in flight together, then each times its block's: a load at a time, they took longer than the weights.
      const float* ws = p.w_scale + ((int64_t)expert * p.N + n0) / 128 * p.k_blocks + kb0;
      const int at_k = n_kb * TN;                       // the weights' scales lie behind the rows'
      for (int r = warp - 2; r < TN; r += 4)
        for (int k = lane; k < n_kb; k += 32)
          copy_f32(scales + k * TN + r, p.a_scale + (int64_t)(m0 + (r < live ? r : 0)) * p.k_blocks + kb0 + k, r < live);
      for (int k = t; k < n_kb; k += 128) copy_f32(scales + at_k + k, ws + k, true);
      asm volatile("cp.async.wait_all;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");
      for (int i = t; i < at_k / 4; i += 128) {
        float4* v = reinterpret_cast<float4*>(scales) + i;
        const float f = scales[at_k + i / (TN / 4)];
        float4 x = *v;
        x.x *= f; x.y *= f; x.z *= f; x.w *= f;
        *v = x;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[j] = 0.f;
      const int groups = (warp & 3) < S::readers ? (n_kb + G - 1) / G : 0;
      constexpr int B = G * TN <= 64 ? G : 1;                                   // blocks read at a time
      for (int i = 0; i < groups; ++i) {
        const int a = i % kAcc;
        ok = ok && mbar_wait(tfull(a), (i / kAcc) & 1, abort_flag);
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int b0 = 0; b0 < G; b0 += B) {
          if (G > 1 && i * G + b0 >= n_kb) break;
          uint32_t r[B * TN];
#pragma unroll
          for (int j = 0; j < B * TN; j += C) {          // (of blocks behind the last one: what is there, and not used)
            if constexpr (C == 16) tmem_ld16(at + (a * G + b0) * TN + j, r + j);
            else tmem_ld32(at + (a * G + b0) * TN + j, r + j);
          }
          tmem_ld_wait();
          if (b0 + B >= G || i * G + b0 + B >= n_kb) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty(a));       // handed back before the arithmetic
          }
#pragma unroll
          for (int b = 0; b < B; ++b) {
            if (B > 1 && i * G + b >= n_kb) break;
            const float4* sc = reinterpret_cast<const float4*>(scales + (i * G + b0 + b) * TN);
            const uint32_t* v = r + b * TN;
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
              const float4 f = sc[j >> 2];
              acc[j] = fmaf(__uint_as_float(v[j]), f.x, acc[j]);
              acc[j + 1] = fmaf(__uint_as_float(v[j + 1]), f.y, acc[j + 1]);
              acc[j + 2] = fmaf(__uint_as_float(v[j + 2]), f.z, acc[j + 2]);
              acc[j + 3] = fmaf(__uint_as_float(v[j + 3]), f.w, acc[j + 3]);
            }
          }
        }
      }
    } else {
      ok = mbar_wait(tfull(0), 0, abort_flag);
      __syncwarp();
      tc_fence_after();
      uint32_t r[TN];
#pragma unroll
      for (int j = 0; j < TN; j += C) {
        if constexpr (C == 16) tmem_ld16(at + j, r + j);
        else tmem_ld32(at + j, r + j);
      }
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[j] = __uint_as_float(r[j]);
    }
  }
  // warps 2..5: the weight row of the tile at this tensor memory lane (of instructions of 64 rows, 16 lie in every 32 lanes)
  const int row = S::rows == 128 ? (warp & 3) * 32 + lane : (lane < 16 ? (warp & 3) * 16 + lane : WR);
  const bool stores = warp >= 2 && row < WR && n0 + row < p.N;
  const float bias = !FP8 && stores && p.bias != nullptr ? __bfloat162float(p.bias[n0 + row]) : 0.f;
  float* red = reinterpret_cast<float*>(smem);        // [row of A][weight row]: every copy of the ring has been consumed
  float* fin = splits > 1 ? red + TN * 128 : red;     // what the activation reads
  if (FP8 || splits == 1) {
    if (!FP8 && p.act != 0) {
      if (warp >= 2) {
#pragma unroll
        for (int j = 0; j < TN; ++j) fin[j * 128 + row] = acc[j];
      }
    } else if (stores && ok) {
      bf16* dst = p.c + (int64_t)m0 * p.ldc + n0 + row;
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (j < live) dst[j * p.ldc] = __float2bfloat16(acc[j] + bias);
    }
  } else {
    if (warp >= 2)
#pragma unroll
      for (int j = 0; j < TN; ++j) red[j * 128 + row] = acc[j];
    __syncwarp();
    cluster_sync();
    if (warp >= 2)
      for (int j = rank; j < live; j += splits) {
        const uint32_t at = sbase + (uint32_t)(j * 128 + row) * 4;
        float v[kMaxSplit], sum = 0.f;
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s) v[s] = s < splits ? ld_cluster(at, s) : 0.f;
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s) sum += v[s];
        if (p.act != 0) fin[j * 128 + row] = sum;
        else if (stores && ok) p.c[(int64_t)(m0 + j) * p.ldc + n0 + row] = __float2bfloat16(sum + bias);
      }
    __syncwarp();
  }
  if (!FP8 && p.act != 0 && warp >= 2) {              // N a multiple of 128
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const int f = row & 63;
    const auto rounded = [](float x) { return __bfloat162float(__float2bfloat16(x)); };   // as the two-launch form stores them
    if (ok)
      for (int j = rank + splits * (row >> 6); j < live; j += 2 * splits)
        p.c[(int64_t)(m0 + j) * p.ldc + nt * 64 + f] =
            __float2bfloat16(gated(rounded(fin[j * 128 + f]), rounded(fin[j * 128 + 64 + f]), p.act, p.limit, p.alpha));
  }
  if (!FP8 && splits > 1) cluster_sync();             // nobody leaves while its sums are being read
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.err != nullptr) atomicExch(p.err, 1);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::cols));
  }
}

static std::atomic<int*> g_err[64] = {};

// The error word of a device, made at its first launch or by xllm_gemm_few_prepare (a capture allows no allocation), or null.
static int* error_word(int dev) {
  static std::mutex making;
  int* word = g_err[dev & 63].load(std::memory_order_acquire);
  if (word != nullptr) return word;
  const std::lock_guard<std::mutex> lock(making);
  word = g_err[dev & 63].load(std::memory_order_acquire);
  if (word != nullptr) return word;
  if (cudaMalloc(&word, sizeof(int)) != cudaSuccess || cudaMemset(word, 0, sizeof(int)) != cudaSuccess) return nullptr;
  g_err[dev & 63].store(word, std::memory_order_release);
  return word;
}

// [rows, cols] with row stride ld elements; box = [box_rows, 128 bytes], 128-byte swizzle
static bool make_map_of(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows, bool fp8) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * (fp8 ? 1 : 2)};
  cuuint32_t box[2] = {fp8 ? 128u : 64u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides,
            box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How many CTAs cut K: an SM works through ceil(tiles x s / 148) slices of ceil(k_blocks / s) blocks, each with a start and
// an end worth about three blocks of its bandwidth; meeting costs about two more.
static int choose_split(int tiles, int k_blocks) {
  int best = 1;
  double cost = 1e30;
  for (int s = 1; s <= kMaxSplit && s <= k_blocks; ++s) {
    const int waves = (tiles * s + 147) / 148;
    const double c = waves * ((k_blocks + s - 1) / s + 3.0) + (s > 1 ? 2.0 : 0.0);
    if (c < cost - 1e-9) { cost = c; best = s; }
  }
  return best;
}

template <int TN, bool FP8, int WR, int G>
static int launch(const void* a, const void* w, const Params& p, int K, int64_t lda, int64_t ldw, int n_experts, int splits,
                  int dev, cudaStream_t s) {
  using S = Smem<TN, FP8, WR, G>;
  static std::atomic<int> attr_bytes[64] = {};
  const int per = (p.k_blocks + splits - 1) / splits, smem = S::total(per);
  if (smem > 232448) return (int)cudaErrorInvalidValue;
  if (attr_bytes[dev & 63].load(std::memory_order_acquire) < smem) {
    // once and for all sizes: a kernel may use what its launch asks for, up to this
    const cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<TN, FP8, WR, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return (int)e;
    attr_bytes[dev & 63].store(232448, std::memory_order_release);
  }
  CUtensorMap tx, tw;
  if (!make_map_of(&tx, a, p.M, K, lda, p.x_rows, FP8) || !make_map_of(&tw, w, (int64_t)p.N * n_experts, K, ldw, WR, FP8))
    return (int)cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  const unsigned tiles = (unsigned)(((p.M + TN - 1) / TN) * ((p.N + WR - 1) / WR));
  cfg.gridDim = p.sliced ? dim3(splits, tiles) : dim3(tiles);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_few_kernel<TN, FP8, WR, G>, tx, tw, p);
  return e != cudaSuccess ? (int)e : XLLM_LAUNCH_CHECK();
}

// Tile of an ungrouped fp8 product, {rows of A, weight rows}: the smallest of which an SM has one or, here and there, two.  A CTA
// goes through K block by block, and a block takes it what the instructions need (some 170 ns of 128 weight rows, 85 ns of 64 or
// fewer) or what its sums take to read back (some 65 ns per 16 rows of A, 32 at a time and lane quarter), whichever is longer,
// while the weights' way from HBM only counts from two thirds of the SMs on.  Measured (one B200, us; 16, 32, 64 rows of A):
//   {16, 32}   1536 x 7168 10, 10, 13   4096 x 7168 11, 14, 25   7168 x 16384 28, 50, 91
//   {16, 64}               13, 13, 13               13, 14, 18                29, 36, 66   12288 x 4096 14, 20, 32
//   {32, 64}                   15, 15                   15, 16                    33, 62                    15, 22
//   {32, 128}                  19, 19                   20, 20                    46, 45                    16, 17   24576 x 1536 11, 17
//   {64, 128}                      26                       27                        55                        19           11, 14
static void fp8_tile(int M, int N, int& tile, int& wr) {
  constexpr int kTiles = 200;
  const auto count = [&](int t, int w) { return (int64_t)((M + t - 1) / t) * ((N + w - 1) / w); };
  tile = 16;
  if (count(16, wr = 32) <= kTiles || count(16, wr = 64) <= kTiles) return;
  if (M > 16) {
    tile = 32;
    if (count(32, wr = 64) <= kTiles) return;
  }
  wr = 128;
  if (M > 32 && count(32, 128) > kTiles) tile = 64;
}

// Grouped: `tile` rows of A at a time, which belong to one expert; M a multiple of it.
template <bool FP8>
static int run(const void* a, const void* w, Params p, int n_experts, int tile, int K, int64_t lda, int64_t ldw, cudaStream_t s) {
  constexpr int KE = FP8 ? 128 : 64;
  int wr = 128;
  if (FP8 && p.tile_expert == nullptr) fp8_tile(p.M, p.N, tile, wr);
  if ((tile != 16 && tile != 32 && tile != 64) || n_experts < 1 || (p.tile_expert != nullptr && (p.M % tile || p.N % 128)) ||
      (((uintptr_t)a | (uintptr_t)w | (uintptr_t)p.c) & 15))
    return (int)cudaErrorInvalidValue;
  p.k_blocks = (K + KE - 1) / KE;
  p.x_rows = p.M >= tile ? tile : ((p.M + 7) & ~7);
  const int64_t tiles = (int64_t)((p.M + tile - 1) / tile) * ((p.N + wr - 1) / wr);
  if (tiles > INT32_MAX) return (int)cudaErrorInvalidValue;
  int dev = 0;
  cudaGetDevice(&dev);
  p.err = error_word(dev);
  if (p.err == nullptr) return (int)cudaErrorMemoryAllocation;
  // a grouped launch holds tiles of experts nobody chose: how many are live is not known here, and there are many
  const int splits = FP8 || p.tile_expert != nullptr || tiles > 65535 ? 1 : choose_split((int)tiles, p.k_blocks);
  p.sliced = splits > 1;
  const auto go = [&](auto kernel) { return kernel(a, w, p, K, lda, ldw, n_experts, splits, dev, s); };
  if constexpr (FP8) {
    if (wr == 32) return go(launch<16, true, 32, 4>);
    if (wr == 64) return go(tile == 16 ? launch<16, true, 64, 2> : launch<32, true, 64, 2>);
    return go(tile == 16 ? launch<16, true, 128, 2> : (tile == 32 ? launch<32, true, 128, 2> : launch<64, true, 128, 2>));
  } else {
    return go(tile == 16 ? launch<16, false, 128, 1> : (tile == 32 ? launch<32, false, 128, 1> : launch<64, false, 128, 1>));
  }
}

static Params make_params(void* c, int64_t ldc, int M, int N, const void* tile_expert) {
  Params p{};
  p.c = (bf16*)c; p.ldc = ldc; p.M = M; p.N = N; p.tile_expert = (const int32_t*)tile_expert;
  return p;
}

}  // namespace few
}  // namespace xllm

// C[M, N] = A[M, K] W[N, K]^T (+ bias[N]) for up to 64 rows.  K, N, lda, ldw % 8 == 0, 16-byte aligned bases.
XLLM_API int xllm_gemm_bf16_few(const void* a, const void* w, void* c, const void* bias, int M, int N, int K, int64_t lda,
                                int64_t ldw, int64_t ldc, void* stream) {
  using namespace xllm::few;
  if (M == 0 || N == 0) return 0;
  if (M > 64 || K <= 0 || K % 8 || N % 8 || lda % 8 || ldw % 8) return (int)cudaErrorInvalidValue;
  Params p = make_params(c, ldc, M, N, nullptr);
  p.bias = (const xllm::bf16*)bias;
  return run<false>(a, w, p, 1, M <= 16 ? 16 : (M <= 32 ? 32 : 64), K, lda, ldw, (cudaStream_t)stream);
}

// The same for xllm_gemm_bf16_act_mul's contract: N rows of interleaved gate and up, N % 128 == 0, C [M, N / 2], act 1 .. 4.
XLLM_API int xllm_gemm_bf16_act_mul_few(const void* a, const void* w, void* c, int M, int N, int K, int64_t lda, int64_t ldw,
                                        int64_t ldc, int act, float limit, float alpha, void* stream) {
  using namespace xllm::few;
  if (M == 0 || N == 0) return 0;
  if (M > 64 || K <= 0 || K % 8 || N % 128 || lda % 8 || ldw % 8 || act < 1 || act > 4) return (int)cudaErrorInvalidValue;
  Params p = make_params(c, ldc, M, N, nullptr);
  p.act = act; p.limit = limit; p.alpha = alpha;
  return run<false>(a, w, p, 1, M <= 16 ? 16 : (M <= 32 ? 32 : 64), K, lda, ldw, (cudaStream_t)stream);
}

// xllm_gemm_bf16_grouped and (act != 0) xllm_gemm_bf16_grouped_act_mul over tiles of `tile` rows (16, 32, 64); N % 128 == 0.
XLLM_API int xllm_gemm_bf16_grouped_few(const void* a, const void* w, void* c, const void* tile_expert, int tile, int M, int N,
                                        int K, int n_experts, int64_t lda, int64_t ldc, int act, float limit, float alpha,
                                        void* stream) {
  using namespace xllm::few;
  if (M == 0 || N == 0) return 0;
  if (tile_expert == nullptr || K <= 0 || K % 8 || lda % 8 || act < 0 || act > 4) return (int)cudaErrorInvalidValue;
  Params p = make_params(c, ldc, M, N, tile_expert);
  p.act = act; p.limit = limit; p.alpha = alpha;
  return run<false>(a, w, p, n_experts, tile, K, lda, K, (cudaStream_t)stream);
}

// The contracts of xllm_gemm_fp8_block, for up to 64 rows, and (tile_expert not null) xllm_gemm_fp8_block_grouped, `tile` rows of A
// (16, 32 or 64) at a time, with the same sums in the same order.  K of at most 49152.
XLLM_API int xllm_gemm_fp8_few(const void* a, const void* w, void* c, const void* a_scale, const void* w_scale,
                               const void* tile_expert, int n_experts, int tile, int M, int N, int K, int64_t lda, int64_t ldw,
                               int64_t ldc, void* stream) {
  using namespace xllm::few;
  if (M == 0 || N == 0) return 0;
  if (K % 128 || K <= 0 || K > kFp8MaxK || N % 8 || lda % 16 || ldw % 16 || (tile_expert == nullptr && M > 64)) return (int)cudaErrorInvalidValue;
  Params p = make_params(c, ldc, M, N, tile_expert);
  p.a_scale = (const float*)a_scale; p.w_scale = (const float*)w_scale;
  return run<true>(a, w, p, n_experts, tile, K, lda, ldw, (cudaStream_t)stream);
}

// What launches on this device need, ahead of a capture.
XLLM_API int xllm_gemm_few_prepare() {
  int dev = 0;
  cudaGetDevice(&dev);
  return xllm::few::error_word(dev) != nullptr ? 0 : (int)cudaErrorMemoryAllocation;
}

// 0 = no bounded wait expired in these kernels on this device since the last call.
XLLM_API int xllm_gemm_few_error_status() {
  int dev = 0;
  cudaGetDevice(&dev);
  int* word = xllm::few::g_err[dev & 63].load(std::memory_order_acquire);
  if (word == nullptr) return 0;
  int v = 0;
  cudaMemcpy(&v, word, sizeof(int), cudaMemcpyDeviceToHost);
  if (v != 0) cudaMemset(word, 0, sizeof(int));
  return v;
}
