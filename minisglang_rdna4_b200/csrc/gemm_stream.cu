// C[M,N] = A[M,K] * B[N,K]^T for decode steps: few rows, so the product is a read of the weights B.
//
// Bound: HBM bytes of B. Every SM has to pull its share at its own limit (about 45 GB/s x 148), all the
// time: a CTA that has no tile, or a second one while the others have finished, is bandwidth lost.
// So the weights are the 128-row side of the MMA (D^T[128 weight rows, NB columns] with NB = 16 .. 128
// columns for the rows of A), which leaves nearly all of the shared-memory ring to weights in flight (11
// stages of 16 KB at NB = 16, against 6 where 128 rows of A were staged with them), and the
// (tile, K block) units of the whole product are dealt to the CTAs in equal contiguous ranges: each
// has the same bytes to read, whatever N is. A tile whose K is shared by several CTAs is summed
// in ascending order of K, by the CTA that finishes last or, as unreduced planes, by the reader; the
// deal depends on N and K alone, so a row's result does not depend on how many rows there are.
//
// B200, us a product, weights not in L2 (the bytes alone at 6.65 TB/s); gemm_tcgen05.cu, which stages 128 rows of A and
// deals whole tiles -> this kernel, finished sums (planes):
//   N x K, type            bytes    1 row                   16 rows                 64 rows
//   24576 x 4096 bf16      30.3     59.3 -> 37.1            47.3 -> 38.0            48.7 -> 42.7
//   4096 x 12288 bf16      15.1     77.4 -> 22.5 (19.0)     56.2 -> 23.5 (19.8)     56.4 -> 29.9 (21.7)
//   151936 x 2560 bf16    117.0    173.6 -> 128.5          186.7 -> 129.7          137.7 -> 135.0
//   57344 x 8192 e4m3      70.6    105.5 -> 80.0            94.2 -> 81.2            96.9 -> 86.5
//   2560 x 9728 mxfp4       2.0     27.9 -> 12.3 (7.8)      27.8 -> 13.6 (8.1)      28.0 -> 20.5 (9.2)
//   6144 x 2560 mxfp4       1.3     13.0 -> 9.6             12.2 -> 10.0            10.4 -> 14.5
// Where the bytes are few, what is left is the summing of shared tiles (a store, a ticket and a load through L2, about
// 4 us and 0.05 us a row): up to how many rows a product is taken follows its tiles and K blocks (ops/cuda.py, _stream_rows).
#include "common.cuh"
#include "ptx.cuh"

#include <string>

using namespace msgl;
using namespace msgl::ptx;

int msgl_b_static_level();   // gemm_tcgen05.cu: level set by msgl_gemm_static_weights

namespace {

constexpr int kThreads = 192;   // TMA, MMA, four epilogue warps
constexpr int kTile = 128;      // weight rows of a tile
constexpr int kMaxPlanes = 8;

enum Kind : int { KIND_F16 = 0, KIND_BF16 = 1, KIND_F8 = 2, KIND_MXF4 = 3 };

struct StreamArgs {
  int M, N;
  int k_blocks, units;       // K blocks of a tile (128 bytes of a weight row), tiles * k_blocks
  const float* a_scale;      // [M] or null
  const float* b_scale;      // [N] or null
  const void* bias;          // [N] or null
  int bias_dtype, out_dtype;
  void* c;                   // [M, ldc], or planes [planes][M][ldc] fp32
  long long ldc;
  int planes;                // 0: finished sums
  const uint8_t* sf;         // kind 3: scale atoms [N / 128][k_blocks][512]
  float* ws;                 // [2 * CTAs][NB][128] partial tiles
  uint32_t* count;           // [tiles], zero between calls
  int b_static;
  int* status;
};

__device__ int g_stream_status = 0;

template <int KIND, int NB> struct Cfg {
  static constexpr int A_BYTES = kTile * 128, B_BYTES = NB * 128, SF_BYTES = KIND == KIND_MXF4 ? 512 : 0;
  static constexpr int STAGES_FIT = (232448 - 1024 - 4096) / (A_BYTES + B_BYTES + SF_BYTES);
  static constexpr int STAGES = STAGES_FIT > 11 ? 11 : STAGES_FIT;
  static constexpr int off_b = STAGES * A_BYTES;
  static constexpr int off_sf = off_b + STAGES * B_BYTES;
  static constexpr int off_ones = off_sf + STAGES * SF_BYTES;
  static constexpr int off_scale = off_ones + 512;
  static constexpr int off_bar = off_scale + NB * 4;
  static constexpr int total = off_bar + (2 * STAGES + 4) * 8 + 16;
  static constexpr int need = 2 * NB + (KIND == KIND_MXF4 ? 8 : 0);
  static constexpr int NCOLS = need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512;
};

__device__ __forceinline__ uint32_t pack2(int out_dtype, float x0, float x1) {
  if (out_dtype == MSGL_BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(x0, x1);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __half2 v = __floats2half2_rn(x0, x1);
  return *reinterpret_cast<uint32_t*>(&v);
}

// `n` (16 or 32) consecutive columns of the warp's lanes
template <int N> __device__ __forceinline__ void load_cols(uint32_t addr, float (&v)[N]) {
  if constexpr (N == 32) {
    uint32_t r[32];
    tmem_ld_32x32b_x32(addr, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
  } else {
    uint32_t r[16];
    tmem_ld_32x32b_x16(addr, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
  }
}

// The epilogue of N columns (rows m0 .. m0 + N of C) of one weight row per lane. 16-bit results: neighbouring
// lanes swap every other value, so that a lane stores two neighbouring columns of C at once.
template <int N>
__device__ __forceinline__ void store_cols(const StreamArgs& a, const float* row_scale, float (&v)[N], int m0, int n, float b_s,
                                           float bias) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = fmaf(v[i] * row_scale[m0 + i], b_s, bias);
  if (a.out_dtype == MSGL_F32) {
    float* p = reinterpret_cast<float*>(a.c) + (size_t)m0 * a.ldc + n;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (m0 + i < a.M && n < a.N) p[(size_t)i * a.ldc] = v[i];
  } else {
    const int odd = threadIdx.x & 1;
    uint16_t* p = reinterpret_cast<uint16_t*>(a.c) + (size_t)(m0 + odd) * a.ldc + (n & ~1);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float other = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
      const uint32_t w = odd ? pack2(a.out_dtype, other, v[i + 1]) : pack2(a.out_dtype, v[i], other);
      if (m0 + i + odd < a.M && n < a.N) *reinterpret_cast<uint32_t*>(p + (size_t)i * a.ldc) = w;
    }
  }
}

// The sum of a tile's parts, in ascending order of K, and its epilogue: a lane has four neighbouring columns of C, a warp
// every fourth row, so that up to 16 loads of 16 bytes a thread are under way (one value a lane and 32 rows at a time, the
// layout of the parts' stores, took 2.4x as long for this at 64 rows).
template <int NB>
__device__ __forceinline__ void finish_tile(const StreamArgs& a, const float* row_scale, int tile, int first, int final) {
  constexpr int R = NB / 4 < 16 ? NB / 4 : 16;
  constexpr size_t SLOT = (size_t)NB * kTile;
  const int lane = threadIdx.x & 31, n = tile * kTile + lane * 4;
  if (n >= a.N) return;
  float4 b_s = make_float4(1.f, 1.f, 1.f, 1.f);
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  if (a.b_scale != nullptr) b_s = make_float4(a.b_scale[n], a.b_scale[n + 1], a.b_scale[n + 2], a.b_scale[n + 3]);
  if (a.bias != nullptr)
    for (int i = 0; i < 4; ++i)
      bias[i] = a.bias_dtype == MSGL_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[n + i])
                : a.bias_dtype == MSGL_F16 ? __half2float(reinterpret_cast<const __half*>(a.bias)[n + i])
                                           : reinterpret_cast<const float*>(a.bias)[n + i];
#pragma unroll 1
  for (int m0 = (threadIdx.x >> 5) - 2; m0 < a.M; m0 += 4 * R) {
    float4 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int c = first; c <= final; ++c) {
      const float* p = a.ws + ((size_t)c * 2 + (c == first ? 1 : 0)) * SLOT + (size_t)m0 * kTile + lane * 4;
      float4 t[R];
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (m0 + 4 * i < a.M) t[i] = __ldcg(reinterpret_cast<const float4*>(p + (size_t)i * 4 * kTile));
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (m0 + 4 * i < a.M) { v[i].x += t[i].x; v[i].y += t[i].y; v[i].z += t[i].z; v[i].w += t[i].w; }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int m = m0 + 4 * i;
      if (m >= a.M) break;
      const float s = row_scale[m];
      const float x0 = fmaf(v[i].x * s, b_s.x, bias[0]), x1 = fmaf(v[i].y * s, b_s.y, bias[1]);
      const float x2 = fmaf(v[i].z * s, b_s.z, bias[2]), x3 = fmaf(v[i].w * s, b_s.w, bias[3]);
      if (a.out_dtype == MSGL_F32)
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.c) + (size_t)m * a.ldc + n) = make_float4(x0, x1, x2, x3);
      else
        *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(a.c) + (size_t)m * a.ldc + n) =
            make_uint2(pack2(a.out_dtype, x0, x1), pack2(a.out_dtype, x2, x3));
    }
  }
}

// units [range(cta), range(cta + 1)) are this CTA's
__device__ __forceinline__ int range_of(int units, int cta, int ctas) { return (int)((long long)units * cta / ctas); }
__device__ __forceinline__ int cta_of(int units, int unit, int ctas) {
  return (int)((((long long)unit + 1) * ctas - 1) / units);
}

template <int KIND, int NB>
__global__ void __launch_bounds__(kThreads, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                   const StreamArgs args) {
  using C = Cfg<KIND, NB>;
  constexpr int STAGES = C::STAGES;
  constexpr int BKE = (KIND == KIND_F16 || KIND == KIND_BF16) ? 64 : 128;
  // TMA counts the packed source bytes of a 4-bit tile
  constexpr uint32_t STAGE_TX = (KIND == KIND_MXF4 ? C::A_BYTES / 2 : C::A_BYTES) + C::B_BYTES + C::SF_BYTES;
  constexpr int COLS = NB < 32 ? 16 : 32;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar_base = s_base + C::off_bar;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
  auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + 2 + s); };
  volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem + C::off_bar + (2 * STAGES + 4) * 8);
  volatile uint32_t* tmem_slot = words;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(words + 1);
  volatile uint32_t* last = words + 2;
  float* row_scale = reinterpret_cast<float*>(smem + C::off_scale);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = args.k_blocks;
  const int u_begin = range_of(args.units, blockIdx.x, gridDim.x), u_end = range_of(args.units, blockIdx.x + 1, gridDim.x);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull_bar(s), 1);
      mbar_init(tempty_bar(s), 4);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tma_w);
    prefetch_tensormap(&tma_x);
  }
  if (KIND == KIND_MXF4) {
    // block scales of the rows of A: 2^0 (their fp32 scale is applied in the epilogue)
    for (int i = threadIdx.x; i < 128; i += blockDim.x) reinterpret_cast<uint32_t*>(smem + C::off_ones)[i] = 0x7F7F7F7Fu;
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::NCOLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!(warp == 0 && lane == 0)) pdl_enter();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      auto load_weights = [&](int u, int s) {
        const int tile = u / KB, kb = u - tile * KB;
        mbar_expect_tx(full_bar(s), STAGE_TX);
        tma_load_2d(s_base + s * C::A_BYTES, &tma_w, full_bar(s), kb * BKE, tile * kTile);
        if (KIND == KIND_MXF4) bulk_load(s_base + C::off_sf + s * C::SF_BYTES, args.sf + (size_t)u * 512, 512, full_bar(s));
      };
      // weights that no kernel in flight writes: the whole ring fills while the kernel ahead still runs
      const int pre = args.b_static ? min(STAGES, u_end - u_begin) : 0;
      for (int s = 0; s < pre; ++s) load_weights(u_begin + s, s);
      pdl_enter();
      int stage = 0;
      uint32_t phase = 0;
      for (int u = u_begin; u < u_end; ++u) {
        if (u - u_begin >= pre) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, args.status, 131)) break;
          load_weights(u, stage);
        }
        tma_load_2d(s_base + C::off_b + stage * C::B_BYTES, &tma_x, full_bar(stage), (u % KB) * BKE, 0);
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (*abort_flag) {  // give copies that are still in flight time to land before the CTA exits
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t sfw = tmem_base + 2 * NB, sfx = sfw + 4;
      if (KIND == KIND_MXF4) tmem_cp_32x128b_warpx4(sfx, smem_desc_sf(s_base + C::off_ones));
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int u = u_begin; u < u_end && ok;) {
        const int kb0 = u % KB, kb1 = min(KB, kb0 + u_end - u);
        if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag, args.status, 132)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * NB;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, args.status, 133)) { ok = false; break; }
          tc_fence_after();
          const uint32_t w_s = s_base + stage * C::A_BYTES, x_s = s_base + C::off_b + stage * C::B_BYTES;
          if (KIND == KIND_MXF4) tmem_cp_32x128b_warpx4(sfw, smem_desc_sf(s_base + C::off_sf + stage * C::SF_BYTES));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t wd = smem_desc_sw128(w_s + k * 32), xd = smem_desc_sw128(x_s + k * 32);
            const uint32_t accum = (kb != kb0 || k != 0) ? 1u : 0u;
            if (KIND == KIND_F16) mma_f16(d, wd, xd, idesc_dense(0, 0, kTile, NB), accum);
            else if (KIND == KIND_BF16) mma_f16(d, wd, xd, idesc_dense(1, 1, kTile, NB), accum);
            else if (KIND == KIND_F8) mma_f8f6f4(d, wd, xd, idesc_dense(0, 0, kTile, NB), accum);
            else mma_mxf8f6f4(d, wd, xd, idesc_block_scaled(5, 0, kTile, NB, (uint32_t)k, 0), accum, sfw, sfx);
          }
          tc_commit(empty_bar(stage));
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        tc_commit(tfull_bar(acc));
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        u += kb1 - kb0;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3, r = q * 32 + lane;   // tensor-memory lane = weight row of the tile
    for (int m = threadIdx.x - 64; m < NB; m += 128) row_scale[m] = args.a_scale != nullptr && m < args.M ? args.a_scale[m] : 1.f;
    asm volatile("bar.sync 1, 128;" ::: "memory");
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int u = u_begin; u < u_end;) {
      const int tile = u / KB, kb0 = u - tile * KB, kb1 = min(KB, kb0 + u_end - u);
      const int n = tile * kTile + r;
      float b_s = 1.f, bias = 0.f;
      const bool whole = kb1 - kb0 == KB;
      const int first = cta_of(args.units, tile * KB, gridDim.x), final = cta_of(args.units, tile * KB + KB - 1, gridDim.x);
      if (n < args.N) {
        if (args.b_scale != nullptr) b_s = __ldg(args.b_scale + n);
        if (args.bias != nullptr && (args.planes == 0 || kb0 == 0))
          bias = args.bias_dtype == MSGL_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(args.bias)[n])
                 : args.bias_dtype == MSGL_F16 ? __half2float(reinterpret_cast<const __half*>(args.bias)[n])
                                               : reinterpret_cast<const float*>(args.bias)[n];
      }
      // after a wait that gave up, the range is still walked through, so that the four warps meet at every barrier
      ok = ok && mbar_wait(tfull_bar(acc), acc_phase, abort_flag, args.status, 134);
      tc_fence_after();
      const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * NB);
      if (args.planes > 0) {
        // plane i of a tile: the i-th CTA that has a part of its K; the planes that are left are zero
        StreamArgs plane = args;
        float* const c0 = reinterpret_cast<float*>(args.c);
        const size_t stride = (size_t)args.M * args.ldc;
        plane.c = c0 + ((int)blockIdx.x - first) * stride;
#pragma unroll 1
        for (int m0 = 0; m0 < NB && m0 < args.M; m0 += COLS) {
          float v[COLS];
          load_cols<COLS>(t_addr + m0, v);
          store_cols<COLS>(plane, row_scale, v, m0, n, b_s, bias);
        }
        if (kb0 == 0 && n < args.N)
          for (int p = final - first + 1; p < args.planes; ++p)
            for (int m = 0; m < args.M; ++m) c0[p * stride + (size_t)m * args.ldc + n] = 0.f;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));
      } else if (whole) {
#pragma unroll 1
        for (int m0 = 0; m0 < NB && m0 < args.M; m0 += COLS) {
          float v[COLS];
          load_cols<COLS>(t_addr + m0, v);
          store_cols<COLS>(args, row_scale, v, m0, n, b_s, bias);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));
      } else {
        // A CTA has at most two parts of tiles: the end of one (slot 0) and the start of another (slot 1).
        constexpr size_t SLOT = (size_t)NB * kTile;
        float* mine = args.ws + ((size_t)blockIdx.x * 2 + (kb0 == 0 ? 1 : 0)) * SLOT + r;
#pragma unroll 1
        for (int m0 = 0; m0 < NB && m0 < args.M; m0 += COLS) {
          float v[COLS];
          load_cols<COLS>(t_addr + m0, v);
#pragma unroll
          for (int i = 0; i < COLS; ++i)
            if (m0 + i < args.M) mine[(size_t)(m0 + i) * kTile] = v[i];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));
        __threadfence();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (threadIdx.x == 64) {
          uint32_t seen;
          asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(seen) : "l"(args.count + tile), "r"(1u) : "memory");
          const uint32_t is_last = seen + 1u == (uint32_t)(final - first + 1) ? 1u : 0u;
          if (is_last) args.count[tile] = 0u;
          *last = is_last;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (*last) {
          __threadfence();
          finish_tile<NB>(args, row_scale, tile, first, final);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");   // `last` is written again
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      u += kb1 - kb0;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::NCOLS);
  }
}

int make_map(CUtensorMap* out, const void* ptr, CUtensorMapDataType dt, uint64_t inner, uint64_t rows, uint64_t row_bytes,
             uint32_t box_inner, uint32_t box_rows) {
  msgl_encode_tiled_fn enc = msgl_get_encode_tiled();
  if (enc == nullptr) return MSGL_CUDA_ERROR;
  cuuint64_t dims[2] = {inner, rows}, strides[1] = {row_bytes};
  cuuint32_t box[2] = {box_inner, box_rows}, estr[2] = {1, 1};
  CUresult r = enc(out, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS) return MSGL_OK;
  msgl_set_error_text(("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r)).c_str());
  return MSGL_CUDA_ERROR;
}

template <int KIND, int NB>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const StreamArgs& args, int ctas, cudaStream_t stream) {
  constexpr int smem = Cfg<KIND, NB>::total + 1024;
  static_assert(smem <= 232448, "shared memory");
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm_stream_kernel<KIND, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaError_t e = configured;
  if (e == cudaSuccess)
    e = msgl_launch(gemm_stream_kernel<KIND, NB>, dim3(ctas), dim3(kThreads), smem, stream, mw, mx, args);
  if (e != cudaSuccess) { msgl_set_error("gemm_stream", e); return MSGL_CUDA_ERROR; }
  return MSGL_OK;
}

template <int KIND>
int launch_nb(int nb, const CUtensorMap& mw, const CUtensorMap& mx, const StreamArgs& args, int ctas, cudaStream_t stream) {
  switch (nb) {
    case 16: return launch<KIND, 16>(mw, mx, args, ctas, stream);
    case 32: return launch<KIND, 32>(mw, mx, args, ctas, stream);
    case 64: return launch<KIND, 64>(mw, mx, args, ctas, stream);
    default: return launch<KIND, 128>(mw, mx, args, ctas, stream);
  }
}

int k_blocks_of(int kind, int K) { return (K + (kind <= KIND_BF16 ? 63 : 127)) / (kind <= KIND_BF16 ? 64 : 128); }
int columns_of(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }

// CTAs that share the K of one tile, at most
int widest_tile(int tiles, int kb, int ctas) {
  const long long units = (long long)tiles * kb;
  int most = 1;
  for (int t = 0; t < tiles; ++t) {
    const int a = (int)(((long long)t * kb + 1) * ctas - 1 < 0 ? 0 : (((long long)t * kb + 1) * ctas - 1) / units);
    const int b = (int)((((long long)(t + 1) * kb) * ctas - 1) / units);
    most = b - a + 1 > most ? b - a + 1 : most;
  }
  return most;
}

}  // namespace

// The deal of C[., N] over K: CTAs, and in *planes the most that share a tile. One CTA per SM; fewer where a CTA would
// have less than four K blocks (a product this short is latency, and more partial sums only add to it) or where `limit`
// planes would not do.
MSGL_API int msgl_gemm_stream_plan(int kind, int N, int K, int limit, int* planes) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  const int kb = k_blocks_of(kind, K), tiles = (N + kTile - 1) / kTile;
  const long long units = (long long)tiles * kb;
  int ctas = (int)(units / 4 < sms ? (units / 4 > 0 ? units / 4 : 1) : sms);
  int most = widest_tile(tiles, kb, ctas);
  while (limit > 0 && most > limit && ctas > 1) most = widest_tile(tiles, kb, --ctas);
  if (planes != nullptr) *planes = most;
  return ctas;
}

// M <= 128 rows. kind and operands as msgl_gemm. planes == 0: c [M, ldc] of out_dtype, ws fp32
// [2 * ctas][16 | 32 | 64 | 128][128], count [N / 128] zero on entry and on exit. planes > 0: c is fp32 [planes][M][N], the
// parts of the sum in ascending order of K (the bias in the first), neither ws nor count. ctas (and planes) from
// msgl_gemm_stream_plan.
MSGL_API int msgl_gemm_stream(int kind, const void* a, long long lda, const void* b, void* c, long long ldc, int M, int N, int K,
                              const void* a_scale, const void* b_scale, const void* bias, int bias_dtype, const void* sf_atoms,
                              int out_dtype, int planes, int ctas, void* ws, void* count, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || M > 128 || ctas <= 0 || planes < 0 || planes > kMaxPlanes) return MSGL_BAD_ARG;
  const int esize = kind <= KIND_BF16 ? 2 : 1;
  if (N % 8 || ldc % 8 || (K * esize) % 16 || (lda * esize) % 16 || (uintptr_t)a % 16 || (uintptr_t)b % 16 || (uintptr_t)c % 16) {
    msgl_set_error_text("gemm_stream: operands must be 16-byte aligned with 16-byte row strides, N a multiple of 8");
    return MSGL_BAD_ARG;
  }
  if (kind == KIND_MXF4 && (K % 32 || sf_atoms == nullptr || (uintptr_t)sf_atoms % 16 || (uintptr_t)b % 32)) return MSGL_BAD_ARG;
  if (planes == 0 ? (ws == nullptr || count == nullptr) : out_dtype != MSGL_F32) return MSGL_BAD_ARG;
  StreamArgs args;
  args.M = M; args.N = N;
  args.k_blocks = k_blocks_of(kind, K);
  args.units = (N + kTile - 1) / kTile * args.k_blocks;
  args.a_scale = (const float*)a_scale;
  args.b_scale = (const float*)b_scale;
  args.bias = bias;
  args.bias_dtype = bias_dtype;
  args.out_dtype = out_dtype;
  args.c = c;
  args.ldc = ldc;
  args.planes = planes;
  args.sf = (const uint8_t*)sf_atoms;
  args.ws = (float*)ws;
  args.count = (uint32_t*)count;
  args.b_static = msgl_b_static_level();
  if (ctas > args.units) ctas = args.units;
  int* status = nullptr;
  cudaGetSymbolAddress((void**)&status, g_stream_status);
  args.status = status;
  const int nb = columns_of(M);
  CUtensorMap mw, mx;
  int rc;
  if (kind == KIND_F16 || kind == KIND_BF16) {
    const CUtensorMapDataType dt = kind == KIND_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    rc = make_map(&mw, b, dt, K, N, (uint64_t)K * 2, 64, kTile);
    if (!rc) rc = make_map(&mx, a, dt, K, M, (uint64_t)lda * 2, 64, nb);
  } else {
    // 4-bit rows are stored in whole 128-element K blocks (zero codes past K)
    const uint64_t k4 = (uint64_t)args.k_blocks * 128;
    rc = kind == KIND_MXF4 ? make_map(&mw, b, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, k4, N, k4 / 2, 128, kTile)
                           : make_map(&mw, b, CU_TENSOR_MAP_DATA_TYPE_UINT8, K, N, (uint64_t)K, 128, kTile);
    if (!rc) rc = make_map(&mx, a, CU_TENSOR_MAP_DATA_TYPE_UINT8, K, M, (uint64_t)lda, 128, nb);
  }
  if (rc) return rc;
  switch (kind) {
    case KIND_F16: return launch_nb<KIND_F16>(nb, mw, mx, args, ctas, stream);
    case KIND_BF16: return launch_nb<KIND_BF16>(nb, mw, mx, args, ctas, stream);
    case KIND_F8: return launch_nb<KIND_F8>(nb, mw, mx, args, ctas, stream);
    case KIND_MXF4: return launch_nb<KIND_MXF4>(nb, mw, mx, args, ctas, stream);
    default: return MSGL_BAD_ARG;
  }
}

// Number of the capture that a stream is in, 0 where it is in none: no two captures of a process have the same.
MSGL_API unsigned long long msgl_capture_id(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(stream, &status, &id) != cudaSuccess) {   // the legacy stream while another one captures
    cudaGetLastError();
    return 0;
  }
  return status == cudaStreamCaptureStatusActive ? id : 0;
}

// 0 when no bounded wait has run out since the last reset; else 131 producer / 132 accumulator / 133 stage / 134 epilogue.
MSGL_API int msgl_gemm_stream_status(int reset) {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_stream_status, sizeof(int));
  if (reset && v != 0) {
    int z = 0;
    cudaMemcpyToSymbol(g_stream_status, &z, sizeof(int));
  }
  return v;
}
