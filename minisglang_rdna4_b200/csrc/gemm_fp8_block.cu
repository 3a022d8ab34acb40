// Block-scaled fp8 GEMM (W8A8 with 128 x 128 weight blocks and 1 x 128 activation groups), dense
// and grouped (mixture of experts):
//
//   C[m, n] = sum over K blocks kb of  a_s[m, kb] * w_s[n / 128, kb] * ( Aq[m, kb] . Bq[n, kb] )
//
// with Aq / Bq e4m3, a_s fp32 [M, K/128] and w_s fp32 [N/128, K/128] (grouped: [E, N/128, K/128]).
// This is the checkpoint format "block fp8" (DeepSeek / compressed-tensors `strategy: block`,
// `block_structure [128, 128]`) that the reference serves through its Fp8Block linear method and
// its w8a8 expert kernels (python/minisgl/quant/method.py:846-897,
// python/minisgl/quant/kernels.py:1181-1331).
//
// The scales change every 128 elements of K and are arbitrary fp32 numbers, so they cannot ride
// on the block-scaled MMA kinds (those take power-of-two UE8M0 scales). Instead every K block
// (= one pipeline stage, four tcgen05.mma kind::f8f6f4 of K = 32) is accumulated on its own
// into one of four 128-column tensor-memory buffers; the four promotion warps pull a finished
// block out with tcgen05.ld, multiply by the block's scale product and add it to a 128-float
// register accumulator per row while the tensor core already works on the next blocks in the
// other buffers. Every row's sum runs over K in ascending order and does not depend on M.
//
// Structure as in gemm_tcgen05.cu: persistent CTAs, warp 0 = TMA producer, warp 1 = MMA issuer
// and tensor-memory owner, warps 2-5 = promotion + store. All waits are bounded.
//
// Bound of many rows: what an SM takes in from L2, 32 KB for each K block of a tile (with the MMAs, the promotion and the stores all
// left out a block still takes 0.49 us, 65 GB/s an SM). On top of that came the stores: a lane wrote 16 bytes of its own row at a time,
// a quarter of the time of the first product and 30 % of the second. A warp now packs its 32 x 64 results into shared memory and
// leaves them to one TMA store, whose end it waits for before the next tile's. Eight promotion warps of 64 columns each were 2
// to 4 % slower than four (4096 x 4096, 100 rows 17.1 us, 16.5 with four; 24576 x 4096, 1024 rows 159, 154), two partial buffers
// and six stages up to 5 % slower than four and five for many rows.
// B200, us, stores of the lanes -> this, weights not in L2: 24576 x 4096, 4096 rows 650 -> 576, 1024 rows 178 -> 158, 100 rows
// 36.5 -> 34.5; 1536 x 2048, 4096 rows 29.5 -> 25.6, 128 rows 11.2 -> 10.1; 4096 x 4096, 4096 rows 111 -> 100, 128 rows 17.1 -> 17.0. Up to 16
// rows it costs 3 % (1536 x 2048 9.3 -> 9.7, 4096 x 4096 16.0 -> 16.5): the end of a store is waited for.
#include "common.cuh"
#include "ptx.cuh"

#include <mutex>
#include <string>
#include <unordered_map>

using namespace msgl;
using namespace msgl::ptx;

int msgl_b_static_level();   // gemm_tcgen05.cu: level set by msgl_gemm_static_weights

namespace {

constexpr int BM = 128, BN = 128, BK = 128;
constexpr int kThreads = 192;      // TMA, MMA, four promotion warps
constexpr int PARTS = 4;           // partial buffers
constexpr int STAGES = 5;
constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK;
constexpr int off_a = 0;
constexpr int off_b = off_a + STAGES * A_BYTES;
constexpr int PATCH_BYTES = 32 * 128;   // half of a promotion warp's results: 32 rows of 64 16-bit columns
constexpr int off_patch = off_b + STAGES * B_BYTES;
constexpr int off_bar = off_patch + 8 * PATCH_BYTES;
constexpr int n_bars = 2 * STAGES + 2 * PARTS;  // full / empty per stage, pfull / pempty per partial buffer
constexpr int smem_total = off_bar + n_bars * 8 + 16;
constexpr int NCOLS = PARTS * BN;

struct BlockArgs {
  int M, N, K;
  int m_tiles, n_tiles, k_blocks;
  const float* a_scale;   // [M, k_blocks]
  const float* w_scale;   // [experts, n_tiles, k_blocks]
  void* c;
  long long ldc;
  int out_dtype;
  const int32_t* tile_expert;  // grouped: expert of M tile m (negative: tile past the live rows)
  int tma_out;                 // results leave through tma_c
  int l2_ahead;                // request a work item's weight stream into L2 one item ahead
  int* status;
};

__device__ int g_block_status = 0;

__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                      const __grid_constant__ CUtensorMap tma_c, const BlockArgs args) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar_base = s_base + off_bar;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto pfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
  auto pempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + PARTS + s); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + off_bar + n_bars * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + off_bar + n_bars * 8 + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total_tiles = args.m_tiles * args.n_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < PARTS; ++s) {
      mbar_init(pfull_bar(s), 1);
      mbar_init(pempty_bar(s), 4);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tma_a);
    prefetch_tensormap(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), NCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_enter();  // nothing above touched global memory

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      // A weight tile that only one or two row tiles use (grouped experts, decode-sized dense calls) is
      // streamed once: its whole K range is requested into L2 one work item ahead, so the ring in
      // shared memory covers L2 latency instead of HBM latency.
      const bool l2_ahead = args.l2_ahead && (args.tile_expert != nullptr || args.m_tiles <= 2);
      auto prefetch_item = [&](int tile) {
        const int m_tile = tile % args.m_tiles, n_tile = tile / args.m_tiles;
        const int expert = args.tile_expert != nullptr ? args.tile_expert[m_tile] : 0;
        if (expert < 0) return;
        for (int kb = 0; kb < args.k_blocks; ++kb) tma_prefetch_2d(&tma_b, kb * BK, expert * args.N + n_tile * BN);
      };
      if (l2_ahead && (int)blockIdx.x < total_tiles) prefetch_item(blockIdx.x);
      for (int tile = blockIdx.x; tile < total_tiles && !*abort_flag; tile += gridDim.x) {
        const int m_tile = tile % args.m_tiles, n_tile = tile / args.m_tiles;
        if (l2_ahead && tile + (int)gridDim.x < total_tiles) prefetch_item(tile + gridDim.x);
        int expert = 0;
        if (args.tile_expert != nullptr) {
          expert = args.tile_expert[m_tile];
          if (expert < 0) continue;
        }
        for (int kb = 0; kb < args.k_blocks; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, args.status, 121)) break;
          mbar_expect_tx(full_bar(stage), A_BYTES + B_BYTES);
          tma_load_2d(s_base + off_a + stage * A_BYTES, &tma_a, full_bar(stage), kb * BK, m_tile * BM);
          tma_load_2d(s_base + off_b + stage * B_BYTES, &tma_b, full_bar(stage), kb * BK,
                      expert * args.N + n_tile * BN);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (*abort_flag) {  // give copies that are still in flight time to land before the CTA exits
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0, pb = 0;
      uint32_t phase = 0, pphase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok && !*abort_flag; tile += gridDim.x) {
        if (args.tile_expert != nullptr && args.tile_expert[tile % args.m_tiles] < 0) continue;
        for (int kb = 0; kb < args.k_blocks; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, args.status, 123)) { ok = false; break; }
          if (!mbar_wait(pempty_bar(pb), pphase ^ 1u, abort_flag, args.status, 122)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_s = s_base + off_a + stage * A_BYTES;
          const uint32_t b_s = s_base + off_b + stage * B_BYTES;
          const uint32_t d_tmem = tmem_base + pb * BN;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f8f6f4(d_tmem, smem_desc_sw128(a_s + k * 32), smem_desc_sw128(b_s + k * 32),
                       idesc_dense(0, 0, BM, BN), k != 0 ? 1u : 0u);
          tc_commit(empty_bar(stage));  // the stage is free once these MMAs have read it
          tc_commit(pfull_bar(pb));     // and this K block's partial sums are complete
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
          if (++pb == PARTS) { pb = 0; pphase ^= 1u; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ promotion + store (warps 2..5)
    constexpr int W = BN / 2;   // columns that are read at once
    const int q = warp & 3;     // tensor-memory lane quarter this warp may read
    int pb = 0;
    uint32_t pphase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      const int m_tile = tile % args.m_tiles, n_tile = tile / args.m_tiles;
      int expert = 0;
      if (args.tile_expert != nullptr) {
        expert = args.tile_expert[m_tile];
        if (expert < 0) continue;
      }
      const int row = m_tile * BM + q * 32 + lane;
      const bool row_ok = row < args.M;
      const float* as_row = args.a_scale + (size_t)(row_ok ? row : 0) * args.k_blocks;
      const float* ws_row = args.w_scale + ((size_t)expert * args.n_tiles + n_tile) * args.k_blocks;
      float acc[2][W];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < W; ++e) acc[h][e] = 0.f;
      float as_next = row_ok ? __ldg(as_row) : 0.f, ws_next = row_ok ? __ldg(ws_row) : 0.f;
      for (int kb = 0; kb < args.k_blocks; ++kb) {
        const float s = as_next * ws_next;
        if (kb + 1 < args.k_blocks && row_ok) {
          as_next = __ldg(as_row + kb + 1);
          ws_next = __ldg(ws_row + kb + 1);
        }
        if (!mbar_wait(pfull_bar(pb), pphase, abort_flag, args.status, 124)) { ok = false; break; }
        tc_fence_after();
        const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(pb * BN);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r0[32], r1[32];
          tmem_ld_32x32b_x32(t_addr + h * W, r0);
          tmem_ld_32x32b_x32(t_addr + h * W + 32, r1);
          tmem_ld_wait();
          if (h == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(pempty_bar(pb));
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            acc[h][e] = fmaf(__uint_as_float(r0[e]), s, acc[h][e]);
            acc[h][32 + e] = fmaf(__uint_as_float(r1[e]), s, acc[h][32 + e]);
          }
        }
        if (++pb == PARTS) { pb = 0; pphase ^= 1u; }
      }
      if (!ok) break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int colbase = n_tile * BN + h * W;
        auto pack = [&](int i) {   // columns 2i and 2i + 1
          if (args.out_dtype == MSGL_BF16) {
            __nv_bfloat162 v = __floats2bfloat162_rn(acc[h][2 * i], acc[h][2 * i + 1]);
            return *reinterpret_cast<uint32_t*>(&v);
          }
          __half2 v = __floats2half2_rn(acc[h][2 * i], acc[h][2 * i + 1]);
          return *reinterpret_cast<uint32_t*>(&v);
        };
        if (args.tma_out) {
          uint8_t* const patch = smem + off_patch + (q * 2 + h) * PATCH_BYTES;
          if (h == 0 && lane == 0) bulk_wait_group_read<0>();   // the tile before this one has left the patch
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 8; ++u)   // 128-byte swizzle: 16-byte unit u of row r lives at unit u ^ (r & 7)
            *reinterpret_cast<uint4*>(patch + lane * 128 + ((u ^ (lane & 7)) << 4)) =
                make_uint4(pack(u * 4), pack(u * 4 + 1), pack(u * 4 + 2), pack(u * 4 + 3));
          fence_proxy_async();
          __syncwarp();
          const int row0 = m_tile * BM + q * 32;
          if (lane == 0 && row0 < args.M && colbase < args.N) {
            tma_store_2d(&tma_c, s_base + off_patch + (q * 2 + h) * PATCH_BYTES, colbase, row0);
            bulk_commit_group();
          }
        } else if (row_ok) {
          if (args.out_dtype == MSGL_F32) {
            float* crow = reinterpret_cast<float*>(args.c) + (size_t)row * args.ldc + colbase;
#pragma unroll
            for (int g = 0; g < W / 4; ++g)
              if (colbase + g * 4 < args.N)
                *reinterpret_cast<float4*>(crow + g * 4) =
                    make_float4(acc[h][g * 4], acc[h][g * 4 + 1], acc[h][g * 4 + 2], acc[h][g * 4 + 3]);
          } else {
            uint16_t* crow = reinterpret_cast<uint16_t*>(args.c) + (size_t)row * args.ldc + colbase;
#pragma unroll
            for (int g = 0; g < W / 8; ++g)
              if (colbase + g * 8 < args.N)
                *reinterpret_cast<uint4*>(crow + g * 8) = make_uint4(pack(g * 4), pack(g * 4 + 1), pack(g * 4 + 2), pack(g * 4 + 3));
          }
        }
      }
    }
    if (lane == 0) bulk_wait_group<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, NCOLS);
  }
}

// ------------------------------------------------------------------------------------------
// SiLU(gate) * up followed by per-group (128 outputs) e4m3 quantisation: the producer of the second
// expert GEMM's activations. Sixteen lanes per (row, group), 16-byte loads. sorted_pair (or null): rows
// that no (token, expert) pair was given (negative) are left out; of a decode step's rows, which are padded to whole tiles
// for each expert, that is nearly all of them.
// B200, us, 768 columns: 16640 rows, 384 of them live, 19.1 -> 8.0; 52096 rows, 35840 live, 59.4 -> 36.9.
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) silu_mul_quant_group_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q,
                                                                   float* __restrict__ out_scale,
                                                                   const int32_t* __restrict__ sorted_pair, int inter,
                                                                   int groups_per_row, size_t total_groups) {
  pdl_enter();
  const size_t gidx = (size_t)blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4);
  const size_t row = gidx / groups_per_row;
  const bool live = gidx < total_groups && (sorted_pair == nullptr || sorted_pair[row] >= 0);
  const int lane = threadIdx.x & 15;
  const int i = (int)(gidx % groups_per_row) * 128 + lane * 8;
  float v[8];
  float amax = 0.f;
  if (live) {
    float g[8], u[8];
    load8(x + row * 2 * inter + i, g);
    load8(x + row * 2 * inter + inter + i, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float h = 0.5f * g[e];
      float t;
      asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
      v[e] = to_float(from_float<T>(fmaf(h, t, h) * u[e]));
      amax = fmaxf(amax, fabsf(v[e]));
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (!live) return;
  const float scale = fmaxf(amax, 1e-8f) / kFp8Max;
  if (lane == 0) out_scale[gidx] = scale;
  *reinterpret_cast<uint2*>(out_q + row * inter + i) = pack8_e4m3(v, scale);
}

// ------------------------------------------------------------------------------------------
// Grouped form for few rows per expert (decode steps): the product is a read of the experts' weights.
//
// Bound: HBM bytes of the weights. The kernel above stages 128 rows of tokens, nearly all of them padding, beside every 128 weight
// rows, which leaves half of the ring to weights, and its promotion is 128 columns wide. Here the weights are the 128-row side
// of the MMA and an expert's rows come in tiles of NB = 16 or 32, the columns: 12 or 10 stages of weights are
// in flight, and a thread promotes the NB columns of its weight row. Every K block is still promoted on its own with
// the product of its two scales, in ascending order: the same sums. GLU: a work item is 128 gate rows and
// the 128 up rows that belong to them, so SiLU(gate) * up, and its maximum over the group of 128 outputs, are at hand in the
// registers of one warpgroup, and e4m3 rows leave the kernel in the place of 16-bit ones that a kernel of its own read again.
// B200, us of a whole expert layer (8 of 128 experts, 2048 columns, 768 wide; the weights alone take 92), 128-row tiles -> this:
// 1 token 30.7 -> 31.2, 4: 60.4 -> 56.8, 16: 135 -> 98, 48: 172 -> 124, 128: 179 -> 137, 256 (NB 32): 188 -> 152, 320: 183 -> 154. The epilogue
// of GLU is a chain that the ring covers up to NB = 32 only (the divisions by one thread a column and the maxima in one
// instruction took 30 us off at NB = 32): tiles of 64 rows took 280.
// ------------------------------------------------------------------------------------------
constexpr int kFewBlocks = 32;     // K blocks, at most

template <int NB> struct FewCfg {
  static constexpr int X_BYTES = NB * BK;
  static constexpr int SCALE_BYTES = NB * kFewBlocks * 4;
  static constexpr int FIT = (232448 - 1024 - 2 * SCALE_BYTES - 4 * NB * 4 - 512) / (B_BYTES + X_BYTES);
  static constexpr int STAGES = FIT > 12 ? 12 : FIT;
  static constexpr int NCOLS = PARTS * NB;                   // 64 or 128
  static constexpr int off_x = STAGES * B_BYTES;
  static constexpr int off_scale = off_x + STAGES * X_BYTES;
  static constexpr int off_max = off_scale + 2 * SCALE_BYTES;
  static constexpr int off_bar = off_max + 4 * NB * 4;
  static constexpr int total = off_bar + (2 * STAGES + 2 * PARTS) * 8 + 16;
};

struct FewArgs {
  int n_items, k_blocks;       // work items of a row tile, K blocks
  int experts_n;               // weight rows of an expert
  int scale_rows;              // rows of an expert's weight scales
  int up_tiles;                // GLU: 128-row tiles from a gate tile to its up tile
  const float* x_scale;        // [M, k_blocks]
  const float* w_scale;        // [experts, scale_rows, k_blocks]
  void* c;                     // 16-bit [M, ldc], or GLU: e4m3 [M, ldc]
  float* c_scale;              // GLU: [M, n_items]
  int ldc, bf16;
  const int32_t* tile_expert;  // [M / NB]
  const int32_t* live;         // row tiles that have rows
  int* status;
};

template <int NB, bool GLU>
__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_block_few_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x, const FewArgs args) {
  using C = FewCfg<NB>;
  constexpr int STAGES_ = C::STAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar_base = s_base + C::off_bar;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES_ + s); };
  auto pfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES_ + s); };
  auto pempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES_ + PARTS + s); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + C::off_bar + (2 * STAGES_ + 2 * PARTS) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = args.k_blocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES_; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < PARTS; ++s) {
      mbar_init(pfull_bar(s), 1);
      mbar_init(pempty_bar(s), 4);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tma_w);
    prefetch_tensormap(&tma_x);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::NCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_enter();
  // neighbouring CTAs have neighbouring row tiles of the same weight tiles: an expert of several tiles is read once
  const int live = *args.live, items = live * args.n_items;
  constexpr int HALVES = GLU ? 2 : 1;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int item = blockIdx.x; item < items && !*abort_flag; item += gridDim.x) {
        const int m = item % live, n = item / live;
        const int expert = args.tile_expert[m];
        if (expert < 0) break;   // (none among the live tiles)
        for (int half = 0; half < HALVES; ++half) {
          const int row = expert * args.experts_n + (n + half * args.up_tiles) * BN;
          for (int kb = 0; kb < KB; ++kb) {
            if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, args.status, 125)) break;
            mbar_expect_tx(full_bar(stage), B_BYTES + C::X_BYTES);
            tma_load_2d(s_base + stage * B_BYTES, &tma_w, full_bar(stage), kb * BK, row);
            tma_load_2d(s_base + C::off_x + stage * C::X_BYTES, &tma_x, full_bar(stage), kb * BK, m * NB);
            if (++stage == STAGES_) { stage = 0; phase ^= 1u; }
          }
        }
      }
      if (*abort_flag) {  // give copies that are still in flight time to land before the CTA exits
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0, pb = 0;
      uint32_t phase = 0, pphase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok && !*abort_flag; item += gridDim.x) {
        if (args.tile_expert[item % live] < 0) break;
        for (int kb = 0; kb < HALVES * KB; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, args.status, 126)) { ok = false; break; }
          if (!mbar_wait(pempty_bar(pb), pphase ^ 1u, abort_flag, args.status, 127)) { ok = false; break; }
          tc_fence_after();
          const uint32_t w_s = s_base + stage * B_BYTES, x_s = s_base + C::off_x + stage * C::X_BYTES, d = tmem_base + pb * NB;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f8f6f4(d, smem_desc_sw128(w_s + k * 32), smem_desc_sw128(x_s + k * 32), idesc_dense(0, 0, BN, NB), k != 0 ? 1u : 0u);
          tc_commit(empty_bar(stage));
          tc_commit(pfull_bar(pb));
          if (++stage == STAGES_) { stage = 0; phase ^= 1u; }
          if (++pb == PARTS) { pb = 0; pphase ^= 1u; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ promotion + store (warps 2..5)
    const int q = warp & 3, r = q * 32 + lane, tid = threadIdx.x - 64;   // tensor-memory lane = weight row of the tile
    int pb = 0, buf = 0;
    uint32_t pphase = 0;
    bool ok = true;
    // the row scales of a tile, [K block][NB], one work item ahead
    auto ask_scales = [&](int item, int to) {
      if (item < items) {
        const float* src = args.x_scale + (size_t)(item % live) * NB * KB;
        const uint32_t dst = s_base + C::off_scale + to * C::SCALE_BYTES;
        for (int i = tid; i < NB * KB; i += 128) {
          const int m = i / KB, kb = i - m * KB;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + (kb * NB + m) * 4), "l"(src + i) : "memory");
        }
      }
    };
    ask_scales(blockIdx.x, 0);
    // After a wait that gave up, the items are still walked through, so that the four warps meet at every barrier.
    for (int item = blockIdx.x; item < items; item += gridDim.x, buf ^= 1) {
      const int m = item % live, n = item / live;
      const int expert = args.tile_expert[m];
      if (expert < 0) break;
      asm volatile("cp.async.wait_all;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");   // the scales are there, and the other buffer has been read
      ask_scales(item + gridDim.x, buf ^ 1);
      const float4* xs = reinterpret_cast<const float4*>(smem + C::off_scale + buf * C::SCALE_BYTES);
      float acc[HALVES][NB];
#pragma unroll
      for (int half = 0; half < HALVES; ++half) {
#pragma unroll
        for (int e = 0; e < NB; ++e) acc[half][e] = 0.f;
        const float* ws_row = args.w_scale + ((size_t)expert * args.scale_rows + n + half * args.up_tiles) * KB;
        float w_next = __ldg(ws_row);
        for (int kb = 0; kb < KB && ok; ++kb) {
          const float w = w_next;
          if (kb + 1 < KB) w_next = __ldg(ws_row + kb + 1);
          float sw[NB];   // ready before the block is
#pragma unroll
          for (int e = 0; e < NB; e += 4) {
            const float4 x = xs[kb * (NB / 4) + e / 4];
            sw[e] = x.x * w; sw[e + 1] = x.y * w; sw[e + 2] = x.z * w; sw[e + 3] = x.w * w;
          }
          if (!mbar_wait(pfull_bar(pb), pphase, abort_flag, args.status, 128)) { ok = false; break; }
          tc_fence_after();
          const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(pb * NB);
          uint32_t v[NB];
          if constexpr (NB == 16) tmem_ld_32x32b_x16(t_addr, v);
          else tmem_ld_32x32b_x32(t_addr, v);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(pempty_bar(pb));
#pragma unroll
          for (int e = 0; e < NB; ++e) acc[half][e] = fmaf(__uint_as_float(v[e]), sw[e], acc[half][e]);
          if (++pb == PARTS) { pb = 0; pphase ^= 1u; }
        }
      }
      if (GLU) {
        // rounded where the 16-bit form rounds; one maximum per column over the four warps
        float* red = reinterpret_cast<float*>(smem + C::off_max);
        auto round16 = [&](float x) {
          return args.bf16 ? __bfloat162float(__float2bfloat16_rn(x)) : __half2float(__float2half_rn(x));
        };
#pragma unroll
        for (int e = 0; e < NB; ++e) {
          const float g = round16(acc[0][e]), u = round16(acc[HALVES - 1][e]), h = 0.5f * g;
          float t;
          asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
          acc[0][e] = round16(fmaf(h, t, h) * u);
          // (bits of magnitudes sort as the magnitudes do; fmaxf would leave a NaN out too)
          const float a = fabsf(acc[0][e]);
          const uint32_t mx = __reduce_max_sync(0xffffffffu, a == a ? __float_as_uint(a) : 0u);
          if (lane == (e & 31)) red[q * NB + e] = __uint_as_float(mx);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (tid < NB) {   // one thread per column divides
          const float mx = fmaxf(fmaxf(red[tid], red[NB + tid]), fmaxf(red[2 * NB + tid], red[3 * NB + tid]));
          const float scale = fmaxf(mx, 1e-8f) / kFp8Max;
          if (ok) args.c_scale[((size_t)m * NB + tid) * args.n_items + n] = scale;
          red[tid] = 1.0f / scale;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        uint8_t* const out = reinterpret_cast<uint8_t*>(args.c) + (size_t)m * NB * args.ldc + n * BN + r;
        if (ok) {
#pragma unroll
          for (int e = 0; e < NB; ++e) out[(size_t)e * args.ldc] = float_to_e4m3(acc[0][e] * red[e]);
        }
        // (the next item writes `red` behind another barrier)
      } else if (ok) {
        // neighbouring lanes swap every other value, so that a lane stores two neighbouring columns of C at once
        const int odd = lane & 1;
        uint16_t* const p = reinterpret_cast<uint16_t*>(args.c) + (size_t)(m * NB + odd) * args.ldc + n * BN + (r & ~1);
#pragma unroll
        for (int e = 0; e < NB; e += 2) {
          const float other = __shfl_xor_sync(0xffffffffu, odd ? acc[0][e] : acc[0][e + 1], 1);
          const float lo = odd ? other : acc[0][e], hi = odd ? acc[0][e + 1] : other;
          uint32_t w;
          if (args.bf16) {
            const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
            w = *reinterpret_cast<const uint32_t*>(&v);
          } else {
            const __half2 v = __floats2half2_rn(lo, hi);
            w = *reinterpret_cast<const uint32_t*>(&v);
          }
          *reinterpret_cast<uint32_t*>(p + (size_t)e * args.ldc) = w;
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::NCOLS);
  }
}

struct MapKey {
  const void* ptr;
  uint64_t inner, rows;
  uint32_t box_rows;
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && inner == o.inner && rows == o.rows && box_rows == o.box_rows;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = std::hash<const void*>()(k.ptr);
    h ^= std::hash<uint64_t>()(k.inner * 1315423911ull + k.rows) + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
    return h ^ k.box_rows;
  }
};
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;
std::mutex g_maps_mutex;

// K-major e4m3 matrix [rows, inner] with contiguous rows of `row_bytes`; box 128 x box_rows, 128B swizzle
int make_map(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t rows, uint64_t row_bytes, uint32_t box_rows,
             bool cache) {
  MapKey key{ptr, inner, rows, box_rows};
  if (cache) {
    std::lock_guard<std::mutex> g(g_maps_mutex);
    auto it = g_maps.find(key);
    if (it != g_maps.end()) { *out = it->second; return MSGL_OK; }
  }
  msgl_encode_tiled_fn enc = msgl_get_encode_tiled();
  if (enc == nullptr) return MSGL_CUDA_ERROR;
  cuuint64_t dims[2] = {inner, rows};
  cuuint64_t strides[1] = {row_bytes};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    msgl_set_error_text(("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r)).c_str());
    return MSGL_CUDA_ERROR;
  }
  if (cache) {
    std::lock_guard<std::mutex> g(g_maps_mutex);
    if (g_maps.size() > 8192) g_maps.clear();
    g_maps[key] = *out;
  }
  return MSGL_OK;
}

}  // namespace

// a [M, K] e4m3 (row stride lda bytes), b [experts * N, K] e4m3, a_scale [M, ceil(K/128)] fp32,
// w_scale [experts, ceil(N/128), ceil(K/128)] fp32, c [M, N] (ldc elements) of out_dtype.
// tile_expert == nullptr: dense (experts = 1). Grouped: M % 128 == 0 and tile_expert[M / 128].
MSGL_API int msgl_gemm_fp8_block(const void* a, long long lda, const void* b, void* c, long long ldc, int M, int N,
                                 int K, const void* a_scale, const void* w_scale, const void* tile_expert,
                                 int num_experts, int out_dtype, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || N % 8 || K % 16 || lda % 16 || a_scale == nullptr || w_scale == nullptr)
    return MSGL_BAD_ARG;
  if (out_dtype != MSGL_BF16 && out_dtype != MSGL_F16 && out_dtype != MSGL_F32) return MSGL_BAD_ARG;
  if (tile_expert != nullptr && (M % 128 || num_experts <= 0)) return MSGL_BAD_ARG;
  if (tile_expert != nullptr && N % 128) return MSGL_BAD_ARG;  // a tile must not straddle two experts' rows
  if (M == 0) return MSGL_OK;
  BlockArgs args;
  args.M = M; args.N = N; args.K = K;
  args.m_tiles = (M + BM - 1) / BM;
  args.n_tiles = (N + BN - 1) / BN;
  args.k_blocks = (K + BK - 1) / BK;
  args.a_scale = (const float*)a_scale;
  args.w_scale = (const float*)w_scale;
  args.c = c;
  args.ldc = ldc;
  args.out_dtype = out_dtype;
  args.tile_expert = (const int32_t*)tile_expert;
  args.l2_ahead = msgl_b_static_level() >= 2 ? 1 : 0;
  int* status = nullptr;
  cudaGetSymbolAddress((void**)&status, g_block_status);
  args.status = status;
  const uint64_t b_rows = (uint64_t)N * (uint64_t)(tile_expert != nullptr ? num_experts : 1);
  CUtensorMap ma, mb;
  int rc = make_map(&ma, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BM, false);
  if (rc) return rc;
  rc = make_map(&mb, b, (uint64_t)K, b_rows, (uint64_t)K, BN, true);
  if (rc) return rc;
  // 16-bit results whose rows a tensor map can describe leave as 32 x 64 boxes
  CUtensorMap mc = ma;
  args.tma_out = out_dtype != MSGL_F32 && ldc % 8 == 0 && ldc >= N && (uintptr_t)c % 16 == 0;
  if (args.tma_out) {
    msgl_encode_tiled_fn enc = msgl_get_encode_tiled();
    cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M}, strides[1] = {(cuuint64_t)ldc * 2};
    cuuint32_t box[2] = {64, 32}, estr[2] = {1, 1};
    args.tma_out = enc != nullptr &&
                   enc(&mc, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, c, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  constexpr int smem = smem_total + 1024;
  static_assert(smem <= 232448, "shared memory");
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_fp8_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) { msgl_set_error("fp8 block gemm smem attribute", e); return MSGL_CUDA_ERROR; }
    configured = true;
  }
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  int grid = args.m_tiles * args.n_tiles;
  if (grid > sms) grid = sms;
  cudaError_t e = msgl_launch(gemm_fp8_block_kernel, dim3(grid), dim3(kThreads), smem, stream, ma, mb, mc, args);
  if (e != cudaSuccess) { msgl_set_error("gemm_fp8_block launch", e); return MSGL_CUDA_ERROR; }
  return MSGL_OK;
}

namespace {
template <int NB, bool GLU>
int launch_few(const CUtensorMap& mw, const CUtensorMap& mx, const FewArgs& args, int ctas, cudaStream_t stream) {
  constexpr int smem = FewCfg<NB>::total + 1024;
  static_assert(smem <= 232448, "shared memory");
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm_fp8_block_few_kernel<NB, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaError_t e = configured;
  if (e == cudaSuccess) e = msgl_launch(gemm_fp8_block_few_kernel<NB, GLU>, dim3(ctas), dim3(kThreads), smem, stream, mw, mx, args);
  if (e != cudaSuccess) { msgl_set_error("gemm_fp8_block_few", e); return MSGL_CUDA_ERROR; }
  return MSGL_OK;
}
}  // namespace

// Grouped, few rows per expert: rows of a [M, K] e4m3 sorted by expert in tiles of nb = 16 or 32, live [1] the number of
// tiles that have rows. glu 0: c 16-bit [M, N]. glu 1: N = 2 * inter rows of gate, then up; c e4m3 [M, inter] of
// SiLU(gate) * up with c_scale [M, inter / 128]; dtype: the 16-bit type that gate, up and their product are rounded to.
// N (inter) a multiple of 128, K of 128 up to 4096.
MSGL_API int msgl_gemm_fp8_block_few(const void* a, const void* b, void* c, void* c_scale, int M, int N, int K, const void* a_scale,
                                     const void* w_scale, const void* tile_expert, const void* live, int num_experts, int nb, int glu,
                                     int dtype, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || K % 128 || K > 128 * kFewBlocks || N % (glu ? 256 : 128) || num_experts <= 0) return MSGL_BAD_ARG;
  if ((nb != 16 && nb != 32) || M % nb || (glu && c_scale == nullptr)) return MSGL_BAD_ARG;
  if (dtype != MSGL_BF16 && dtype != MSGL_F16) return MSGL_BAD_ARG;
  if ((uintptr_t)a % 16 || (uintptr_t)b % 16 || (uintptr_t)c % 16) return MSGL_BAD_ARG;
  if (M == 0) return MSGL_OK;
  FewArgs args;
  args.n_items = N / (glu ? 256 : 128);
  args.k_blocks = K / 128;
  args.experts_n = N;
  args.scale_rows = N / 128;
  args.up_tiles = args.n_items;
  args.x_scale = (const float*)a_scale;
  args.w_scale = (const float*)w_scale;
  args.c = c;
  args.c_scale = (float*)c_scale;
  args.ldc = glu ? N / 2 : N;
  args.bf16 = dtype == MSGL_BF16;
  args.tile_expert = (const int32_t*)tile_expert;
  args.live = (const int32_t*)live;
  int* status = nullptr;
  cudaGetSymbolAddress((void**)&status, g_block_status);
  args.status = status;
  CUtensorMap mw, mx;
  int rc = make_map(&mw, b, (uint64_t)K, (uint64_t)N * num_experts, (uint64_t)K, BN, true);
  if (rc == MSGL_OK) rc = make_map(&mx, a, (uint64_t)K, (uint64_t)M, (uint64_t)K, nb, false);
  if (rc) return rc;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  const long long most = (long long)(M / nb) * args.n_items;
  const int ctas = most < sms ? (int)most : sms;
  if (glu) return nb == 16 ? launch_few<16, true>(mw, mx, args, ctas, stream) : launch_few<32, true>(mw, mx, args, ctas, stream);
  return nb == 16 ? launch_few<16, false>(mw, mx, args, ctas, stream) : launch_few<32, false>(mw, mx, args, ctas, stream);
}

// 0 when no bounded wait of the block-fp8 GEMM has run out since the last reset; else 121 producer /
// 122 partial buffer / 123 stage / 124 promotion wait (few rows: 125 / 127 / 126 / 128).
MSGL_API int msgl_gemm_fp8_block_status(int reset) {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_block_status, sizeof(int));
  if (reset && v != 0) {
    int z = 0;
    cudaMemcpyToSymbol(g_block_status, &z, sizeof(int));
  }
  return v;
}

// x [rows, 2 * inter] (gate columns then up columns) -> e4m3 [rows, inter] + fp32 scales [rows, inter / 128];
// sorted_pair [rows] or null: rows with a negative entry are not written
MSGL_API int msgl_silu_mul_quant_group(const void* x, void* out_q, void* out_scale, const void* sorted_pair, int rows, int inter,
                                       int dtype, cudaStream_t stream) {
  if (inter % 128 || rows < 0) return MSGL_BAD_ARG;
  if (rows == 0) return MSGL_OK;
  const int gpr = inter / 128;
  const size_t total = (size_t)rows * gpr;
  const unsigned blocks = (unsigned)((total + 15) / 16);
  cudaError_t e;
  if (dtype == MSGL_BF16)
    e = msgl_launch(silu_mul_quant_group_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, (const __nv_bfloat16*)x,
                    (uint8_t*)out_q, (float*)out_scale, (const int32_t*)sorted_pair, inter, gpr, total);
  else if (dtype == MSGL_F16)
    e = msgl_launch(silu_mul_quant_group_kernel<__half>, dim3(blocks), dim3(256), 0, stream, (const __half*)x, (uint8_t*)out_q,
                    (float*)out_scale, (const int32_t*)sorted_pair, inter, gpr, total);
  else
    return MSGL_BAD_ARG;
  if (e != cudaSuccess) { msgl_set_error("silu_mul_quant_group", e); return MSGL_CUDA_ERROR; }
  return MSGL_OK;
}
