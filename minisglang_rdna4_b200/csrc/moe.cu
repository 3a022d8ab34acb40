// Mixture-of-experts routing and data movement around the grouped tcgen05 GEMMs.
//
//   moe_route      : scores (softmax or sigmoid) -> top-k -> renormalise, one warp per token,
//                    plus per-expert counts (the reference's moe_route_align / moe_topk_*;
//                    python/minisgl/quant/kernels.py:423-481)
//   moe_align      : pad every expert's row count to the 128-row GEMM tile, assign each
//                    (token, k) pair a row in the expert-sorted order, record the expert of
//                    every tile (sgl_kernel.moe_align_block_size in the reference's CUDA path,
//                    python/minisgl/moe/fused.py:96-117)
//   moe_quant_rows : quantise token rows to e4m3 once each and write them to all their rows in expert-sorted order
//   moe_permute    : gather token rows into expert-sorted order, times their weight where that acts on the input
//   moe_combine    : out[t] = sum_k w[t,k] * y[row_of(t,k)] in a fixed k order
//                    (mmq_fp8_moe_gather_reduce, python/minisgl/quant/kernels.py:877)
//   moe_combine32  : the same sum in fp32 for an fp32 residual stream, with a shared expert's
//                    output, behind a sigmoid gate per token where it has one
//
// Shapes are static for CUDA graphs: the sorted buffers are sized for the worst case
// T*k + E*127 rows and tiles past the live count carry expert id -1, which the GEMM skips.
#include "common.cuh"

using namespace msgl;

namespace {

constexpr int kMaxExperts = 512;
constexpr int kMaxTopK = 16;
constexpr int kSmallPairs = 4096;   // (token, expert) pairs that one CTA aligns: eight a thread

// one warp per token; PER values per lane: E <= 32 PER. Each of the k rounds walks all PER values.
// B200, us, 8 of 128 experts: 48 tokens 5.7 -> 3.5, 4480 tokens 16.0 -> 9.4; of 256: 5.8 -> 4.2, 16.1 -> 11.9; of 512 as before.
template <typename T, int PER>
__global__ void moe_route_kernel(const T* __restrict__ logits, const float* __restrict__ bias,
                                 float* __restrict__ topk_w, int32_t* __restrict__ topk_ids,
                                 int32_t* __restrict__ counts, int tokens, int E, int k, int renorm, int sigmoid,
                                 float scale, int e_start, int e_local, long long ld, int groups, int keep) {
  pdl_enter();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= tokens) return;
  const int lane = threadIdx.x & 31;
  float v[PER];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    v[i] = e < E ? to_float(logits[t * ld + e]) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
  if (sigmoid) {
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = (lane + 32 * i) < E ? 1.f / (1.f + expf(-v[i])) : -INFINITY;
  } else {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      v[i] = (lane + 32 * i) < E ? expf(v[i] - mx) : 0.f;
      sum += v[i];
    }
    sum = warp_sum(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = (lane + 32 * i) < E ? v[i] * inv : -INFINITY;
  }
  // experts are chosen by score + selection bias (when given); the weights are the scores themselves
  float c[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    c[i] = (bias != nullptr && e < E) ? v[i] + bias[e] : v[i];
  }
  if (groups > 1) {
    // only experts of the best `keep` groups stay eligible; a group's score is its best member's
    const int size = E / groups;
    float g0 = -INFINITY, g1 = -INFINITY;      // lane l holds the groups l and l + 32
    for (int g = 0; g < groups; ++g) {
      float best = -INFINITY;
#pragma unroll
      for (int i = 0; i < PER; ++i)
        if ((lane + 32 * i) / size == g) best = fmaxf(best, c[i]);
      best = warp_max(best);
      if (lane == (g & 31)) (g < 32 ? g0 : g1) = best;
    }
    unsigned long long open = 0;
    for (int kk = 0; kk < keep; ++kk) {
      float best = g0 >= g1 ? g0 : g1;
      int bi = g0 >= g1 ? lane : lane + 32;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      open |= 1ull << bi;
      if ((bi & 31) == lane) (bi < 32 ? g0 : g1) = -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      if (e < E && !(open >> (e / size) & 1)) c[i] = -INFINITY;
    }
  }
  float wsel[kMaxTopK];
  int isel[kMaxTopK];
  float total = 0.f;
  for (int kk = 0; kk < k; ++kk) {
    // arg-max over the remaining choice scores, lowest expert id on ties
    float best = -INFINITY, bw = 0.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      if (c[i] > best || (c[i] == best && e < bi)) { best = c[i]; bi = e; bw = v[i]; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const float ow = __shfl_xor_sync(0xffffffffu, bw, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; bw = ow; }
    }
    wsel[kk] = bw;
    isel[kk] = bi;
    total += bw;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i == bi) c[i] = -INFINITY;
  }
  if (lane == 0) {
    const float norm = renorm ? 1.f / fmaxf(total, 1e-20f) : 1.f;
    for (int kk = 0; kk < k; ++kk) {
      topk_w[(size_t)t * k + kk] = wsel[kk] * norm * scale;
      topk_ids[(size_t)t * k + kk] = isel[kk];
      const int local = isel[kk] - e_start;
      if (counts != nullptr && local >= 0 && local < e_local) atomicAdd(counts + local, 1);
    }
  }
}

// exclusive padded offsets of the experts' rows in s_off [0, e_local], one thread per expert
__device__ __forceinline__ void padded_offsets(int count, int* s_off, int e_local, int block) {
  __shared__ int s_warp[32];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  int v = e < e_local ? (count + block - 1) / block * block : 0;
  int sum = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += up;
  }
  if (lane == 31) s_warp[warp] = sum;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += s_warp[w];
  if (e < e_local) s_off[e] = before + sum - v;
  if (e == e_local - 1) s_off[e_local] = before + sum;
  __syncthreads();
}

// expert of a tile's rows, -1 past the live ones
__device__ __forceinline__ int tile_owner(const int* s_off, int e_local, int row) {
  if (row >= s_off[e_local]) return -1;
  int lo = 0, hi = e_local;   // the last expert whose range starts at or before the row (empty ones have no rows)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s_off[mid] <= row) lo = mid; else hi = mid;
  }
  return lo;
}

// single CTA of kMaxExperts threads: padded offsets + tile -> expert map
__global__ void __launch_bounds__(kMaxExperts) moe_offsets_kernel(const int32_t* __restrict__ counts, int32_t* __restrict__ offsets,
                                                                  int32_t* __restrict__ cursor, int32_t* __restrict__ tile_expert,
                                                                  int32_t* __restrict__ meta, int e_local, int max_tiles, int block) {
  pdl_enter();
  __shared__ int s_off[kMaxExperts + 1];
  padded_offsets((int)threadIdx.x < e_local ? counts[threadIdx.x] : 0, s_off, e_local, block);
  if (threadIdx.x == 0) {
    meta[0] = s_off[e_local] / block;   // live tiles
    meta[1] = s_off[e_local];           // live (padded) rows
  }
  for (int e = threadIdx.x; e <= e_local; e += blockDim.x) {
    offsets[e] = s_off[e];
    if (e < e_local) cursor[e] = 0;
  }
  for (int m = threadIdx.x; m < max_tiles; m += blockDim.x) tile_expert[m] = tile_owner(s_off, e_local, m * block);
}

// The whole alignment of few pairs in one CTA: counters and cursors in shared memory, so that nothing of it needs a memset
// or a second launch. 48 tokens of 8 experts: two memsets and two kernels took about 16 us of a layer, this one 6.
__global__ void __launch_bounds__(kMaxExperts) moe_align_small_kernel(
    const int32_t* __restrict__ topk_ids, int32_t* __restrict__ offsets, int32_t* __restrict__ tile_expert,
    int32_t* __restrict__ meta, int32_t* __restrict__ sorted_pair, int32_t* __restrict__ pair_row, int pairs, int e_start,
    int e_local, int max_rows, int block) {
  pdl_enter();
  __shared__ int s_off[kMaxExperts + 1], s_count[kMaxExperts];
  for (int i = threadIdx.x * 4; i < max_rows; i += blockDim.x * 4)   // max_rows: a multiple of `block`
    *reinterpret_cast<int4*>(sorted_pair + i) = make_int4(-1, -1, -1, -1);
  s_count[threadIdx.x] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int local = topk_ids[p] - e_start;
    if (local >= 0 && local < e_local) atomicAdd(s_count + local, 1);
  }
  __syncthreads();
  padded_offsets(s_count[threadIdx.x], s_off, e_local, block);
  s_count[threadIdx.x] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int local = topk_ids[p] - e_start;
    int row = -1;
    if (local >= 0 && local < e_local) {
      row = s_off[local] + atomicAdd(s_count + local, 1);
      sorted_pair[row] = p;
    }
    pair_row[p] = row;
  }
  if (threadIdx.x == 0) {
    meta[0] = s_off[e_local] / block;
    meta[1] = s_off[e_local];
  }
  for (int e = threadIdx.x; e <= e_local; e += blockDim.x) offsets[e] = s_off[e];
  for (int m = threadIdx.x; m < max_rows / block; m += blockDim.x) tile_expert[m] = tile_owner(s_off, e_local, m * block);
}

// one thread per (token, k) pair: claim a row in the expert's range
__global__ void moe_scatter_kernel(const int32_t* __restrict__ topk_ids, const int32_t* __restrict__ offsets,
                                   int32_t* __restrict__ cursor, int32_t* __restrict__ sorted_pair,
                                   int32_t* __restrict__ pair_row, int pairs, int e_start, int e_local) {
  pdl_enter();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= pairs) return;
  const int local = topk_ids[p] - e_start;
  if (local < 0 || local >= e_local) {
    pair_row[p] = -1;
    return;
  }
  const int row = offsets[local] + atomicAdd(cursor + local, 1);
  sorted_pair[row] = p;
  pair_row[p] = row;
}

// x [tokens, hidden] -> e4m3 rows in expert-sorted order with one scale per `group` elements (128, or hidden: one per
// row). A CTA per token: its row is read and quantised once and written to its k rows. Rows that belong to no pair are not
// written: a row of the grouped GEMMs depends on its own operand row alone and nothing reads the others' results.
// B200, us, with the alignment, 8 of 128 experts, 2048 columns in groups of 128, against a gather of 16-bit rows (padding
// rows too) that were quantised after it: 48 tokens 77.4 -> 5.9, 4480 tokens 235 -> 27.6.
template <typename T>
__global__ void __launch_bounds__(256) moe_quant_rows_kernel(const T* __restrict__ x, const int32_t* __restrict__ pair_row,
                                                             uint8_t* __restrict__ out_q, float* __restrict__ out_scale,
                                                             int hidden, int k, int per_row) {
  pdl_enter();
  __shared__ float scratch[32];
  const int t = blockIdx.x;
  const T* src = x + (size_t)t * hidden;
  const int32_t* rows = pair_row + (size_t)t * k;
  if (per_row) {
    float amax = 0.f;
    for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
      float v[8];
      load8(src + i, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
    }
    const float scale = fmaxf(block_max(amax, scratch), 1e-8f) / kFp8Max;
    for (int j = threadIdx.x; j < k; j += blockDim.x)
      if (rows[j] >= 0) out_scale[rows[j]] = scale;
    for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
      float v[8];
      load8(src + i, v);
      const uint2 q = pack8_e4m3(v, scale);
#pragma unroll 4
      for (int j = 0; j < k; ++j) {
        const int row = rows[j];
        if (row >= 0) *reinterpret_cast<uint2*>(out_q + (size_t)row * hidden + i) = q;
      }
    }
    return;
  }
  const int groups = hidden / 128;
  for (int base = 0; base < hidden; base += blockDim.x * 8) {   // hidden % 128 == 0: sixteen lanes are in or out together
    const int i = base + threadIdx.x * 8;
    float v[8];
    float amax = 0.f;
    if (i < hidden) {
      load8(src + i, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (i >= hidden) continue;
    const float scale = fmaxf(amax, 1e-8f) / kFp8Max;
    const uint2 q = pack8_e4m3(v, scale);
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
      const int row = rows[j];
      if (row < 0) continue;
      *reinterpret_cast<uint2*>(out_q + (size_t)row * hidden + i) = q;
      if ((threadIdx.x & 15) == 0) out_scale[(size_t)row * groups + i / 128] = scale;
    }
  }
}

template <typename T>
__global__ void moe_permute_kernel(const T* __restrict__ x, const int32_t* __restrict__ sorted_pair,
                                   T* __restrict__ out, int hidden, int k, int rows, const float* __restrict__ topk_w) {
  pdl_enter();
  const int row = blockIdx.x;
  if (row >= rows) return;
  const int pair = sorted_pair[row];
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row * hidden);
  const int vecs = hidden / (16 / (int)sizeof(T));
  if (pair < 0) {
    for (int i = threadIdx.x; i < vecs; i += blockDim.x) dst[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  if (topk_w != nullptr) {
    const float w = topk_w[pair];
    for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
      float v[8];
      load8(x + (size_t)(pair / k) * hidden + i, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] *= w;
      store8(out + (size_t)row * hidden + i, v);
    }
    return;
  }
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(pair / k) * hidden);
  for (int i = threadIdx.x; i < vecs; i += blockDim.x) dst[i] = src[i];
}

template <typename T>
__global__ void moe_combine_kernel(const T* __restrict__ y, const float* __restrict__ topk_w,
                                   const int32_t* __restrict__ pair_row, T* __restrict__ out, int hidden, int k) {
  // four rows' loads at a time: one after the other they were a round trip to memory each
  pdl_enter();
  const int t = blockIdx.x;
  for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int k0 = 0; k0 < k; k0 += 4) {
      Vec8<T> r[4];
      int row[4];
      float w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        row[j] = k0 + j < k ? pair_row[(size_t)t * k + k0 + j] : -1;
        w[j] = k0 + j < k ? topk_w[(size_t)t * k + k0 + j] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (row[j] >= 0) r[j] = *reinterpret_cast<const Vec8<T>*>(y + (size_t)row[j] * hidden + i);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (row[j] >= 0) {
          float v[8];
          unpack8(r[j], v);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += w[j] * v[e];
        }
    }
    store8(out + (size_t)t * hidden + i, acc);
  }
}

// out [tokens, cols] fp32; topk_w null: every weight is one (it acted on the input); shared [tokens, shared_cols]
// (columns past that: no shared part), shared_gate: one logit per token, ldg elements apart, or null
template <typename T>
__global__ void __launch_bounds__(256) moe_combine32_kernel(const T* __restrict__ y, const float* __restrict__ topk_w,
                                                            const int32_t* __restrict__ pair_row,
                                                            const T* __restrict__ shared, int shared_cols,
                                                            const float* __restrict__ shared_gate, long long ldg,
                                                            float* __restrict__ out, int cols, int k) {
  pdl_enter();
  const int t = blockIdx.x;
  const float sg = shared_gate != nullptr ? 1.f / (1.f + expf(-shared_gate[t * ldg])) : 1.f;
  for (int i = threadIdx.x * 8; i < cols; i += blockDim.x * 8) {
    float acc[8], v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    if (shared != nullptr && i < shared_cols) {
      load8(shared + (size_t)t * shared_cols + i, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = sg * v[e];
    }
    for (int kk = 0; kk < k; ++kk) {
      const int row = pair_row[(size_t)t * k + kk];
      if (row < 0) continue;
      const float w = topk_w != nullptr ? topk_w[(size_t)t * k + kk] : 1.f;
      load8(y + (size_t)row * cols + i, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(w, v[e], acc[e]);
    }
    store8(out + (size_t)t * cols + i, acc);
  }
}

}  // namespace

MSGL_API int msgl_moe_combine32(const void* y, const void* topk_w, const void* pair_row, const void* shared,
                                int shared_cols, const void* shared_gate, long long ldg, void* out, int tokens, int cols,
                                int k, int dtype, cudaStream_t stream) {
  if (tokens == 0) return MSGL_OK;
  if (tokens < 0 || cols % 8 || shared_cols % 8) return MSGL_BAD_ARG;
  const int threads = cols / 8 < 256 ? ((cols / 8 + 31) / 32) * 32 : 256;
#define COMBINE32(T)                                                                                                 \
  msgl_launch(moe_combine32_kernel<T>, dim3(tokens), dim3(threads), 0, stream, (const T*)y, (const float*)topk_w,    \
              (const int32_t*)pair_row, (const T*)shared, shared_cols, (const float*)shared_gate, ldg, (float*)out,  \
              cols, k)
  if (dtype == MSGL_BF16) COMBINE32(__nv_bfloat16);
  else if (dtype == MSGL_F32) COMBINE32(float);
  else return MSGL_BAD_ARG;
#undef COMBINE32
  MSGL_CHECK_LAUNCH("moe_combine32");
  return MSGL_OK;
}

// logits [tokens, E] with row stride ld. groups > 1: experts are chosen among the best `keep` of that many groups of
// neighbours, a group scoring as its best member (up to 64 groups)
MSGL_API int msgl_moe_route(const void* logits, const void* bias, void* topk_w, void* topk_ids, void* counts,
                            int tokens, int E, int k, int renorm, int sigmoid, float scale, int e_start, int e_local,
                            long long ld, int groups, int keep, int dtype, cudaStream_t stream) {
  if (E > kMaxExperts || k > kMaxTopK || k > E) {
    msgl_set_error_text("moe_route: up to 512 experts, 16 per token");
    return MSGL_BAD_ARG;
  }
  if (groups > 1 && (groups > 64 || E % groups || keep <= 0 || keep > groups || k > E / groups * keep)) return MSGL_BAD_ARG;
  // counts (optional): tokens per local expert, for the alignment step; zeroed here
  if (counts != nullptr) cudaMemsetAsync(counts, 0, sizeof(int32_t) * e_local, stream);
  if (tokens == 0) return MSGL_OK;
  const int warps = 4;
  const int blocks = (tokens + warps - 1) / warps;
#define ROUTE(T)                                  \
  do {                                            \
    if (E <= 128) ROUTE_PER(T, 4);                \
    else if (E <= 256) ROUTE_PER(T, 8);           \
    else ROUTE_PER(T, 16);                        \
  } while (0)
#define ROUTE_PER(T, PER)                                                                                            \
  msgl_launch(moe_route_kernel<T, PER>, dim3(blocks), dim3(warps * 32), 0, stream, (const T*)logits, (const float*)bias, \
              (float*)topk_w, (int32_t*)topk_ids, (int32_t*)counts, tokens, E, k, renorm, sigmoid, scale, e_start,   \
              e_local, ld, groups, keep)
  if (dtype == MSGL_F32) ROUTE(float);
  else if (dtype == MSGL_BF16) ROUTE(__nv_bfloat16);
  else if (dtype == MSGL_F16) ROUTE(__half);
  else return MSGL_BAD_ARG;
#undef ROUTE
#undef ROUTE_PER
  MSGL_CHECK_LAUNCH("moe_route");
  return MSGL_OK;
}

// counts [e_local] (from msgl_moe_route) -> offsets [e_local+1], tile_expert [max_tiles], meta [2],
// sorted_pair [max_rows] (filled with -1 first), pair_row [tokens*k]
MSGL_API int msgl_moe_align(const void* topk_ids, const void* counts, void* offsets, void* cursor, void* tile_expert,
                            void* meta, void* sorted_pair, void* pair_row, int tokens, int k, int e_start,
                            int e_local, int max_rows, int block, cudaStream_t stream) {
  if (tokens == 0) return MSGL_OK;
  if (e_local <= 0 || e_local > kMaxExperts || max_rows % block) return MSGL_BAD_ARG;
  const int few = tokens * k;
  if (few <= kSmallPairs && block % 4 == 0 && (uintptr_t)sorted_pair % 16 == 0) {
    msgl_launch(moe_align_small_kernel, dim3(1), dim3(kMaxExperts), 0, stream, (const int32_t*)topk_ids, (int32_t*)offsets,
                (int32_t*)tile_expert, (int32_t*)meta, (int32_t*)sorted_pair, (int32_t*)pair_row, few, e_start, e_local,
                max_rows, block);
    MSGL_CHECK_LAUNCH("moe_align");
    return MSGL_OK;
  }
  if (counts == nullptr) return MSGL_BAD_ARG;
  cudaMemsetAsync(sorted_pair, 0xff, sizeof(int32_t) * (size_t)max_rows, stream);
  msgl_launch(moe_offsets_kernel, dim3(1), dim3(kMaxExperts), 0, stream, (const int32_t*)counts, (int32_t*)offsets, (int32_t*)cursor,
                                            (int32_t*)tile_expert, (int32_t*)meta, e_local, max_rows / block, block);
  const int pairs = tokens * k;
  msgl_launch(moe_scatter_kernel, dim3((pairs + 255) / 256), dim3(256), 0, stream, (const int32_t*)topk_ids, (const int32_t*)offsets,
                                                              (int32_t*)cursor, (int32_t*)sorted_pair,
                                                              (int32_t*)pair_row, pairs, e_start, e_local);
  MSGL_CHECK_LAUNCH("moe_align");
  return MSGL_OK;
}

// x [tokens, hidden] (16-bit) -> out_q e4m3 [max_rows, hidden], out_scale [max_rows, hidden / group] at the rows of pair_row
// [tokens, k] that are not negative; group 128, or 0: one scale per row
MSGL_API int msgl_moe_quant_rows(const void* x, const void* pair_row, void* out_q, void* out_scale, int tokens, int hidden, int k,
                                 int group, int dtype, cudaStream_t stream) {
  if (tokens == 0) return MSGL_OK;
  if (tokens < 0 || hidden <= 0 || k <= 0 || (group != 0 && group != 128) || hidden % (group ? 128 : 8)) return MSGL_BAD_ARG;
  const int threads = hidden / 8 < 256 ? (hidden / 8 + 31) / 32 * 32 : 256;
#define QUANT_ROWS(T)                                                                                                   \
  msgl_launch(moe_quant_rows_kernel<T>, dim3(tokens), dim3(threads), 0, stream, (const T*)x, (const int32_t*)pair_row, \
              (uint8_t*)out_q, (float*)out_scale, hidden, k, (int)(group == 0))
  if (dtype == MSGL_BF16) QUANT_ROWS(__nv_bfloat16);
  else if (dtype == MSGL_F16) QUANT_ROWS(__half);
  else return MSGL_BAD_ARG;
#undef QUANT_ROWS
  MSGL_CHECK_LAUNCH("moe_quant_rows");
  return MSGL_OK;
}

// topk_w (optional): the weight of every (token, expert) pair, multiplied into its row
MSGL_API int msgl_moe_permute(const void* x, const void* sorted_pair, void* out, int hidden, int k, int rows,
                              const void* topk_w, int dtype, cudaStream_t stream) {
  if (rows == 0) return MSGL_OK;
  if (hidden % 8) return MSGL_BAD_ARG;
  int threads = hidden / 8 < 256 ? ((hidden / 8 + 31) / 32) * 32 : 256;
  if (dtype == MSGL_BF16)
    msgl_launch(moe_permute_kernel<__nv_bfloat16>, dim3(rows), dim3(threads), 0, stream, (const __nv_bfloat16*)x, (const int32_t*)sorted_pair,
                                                                   (__nv_bfloat16*)out, hidden, k, rows, (const float*)topk_w);
  else if (dtype == MSGL_F16)
    msgl_launch(moe_permute_kernel<__half>, dim3(rows), dim3(threads), 0, stream, (const __half*)x, (const int32_t*)sorted_pair,
                                                            (__half*)out, hidden, k, rows, (const float*)topk_w);
  else if (dtype == MSGL_F32)
    msgl_launch(moe_permute_kernel<float>, dim3(rows), dim3(threads), 0, stream, (const float*)x, (const int32_t*)sorted_pair,
                                                           (float*)out, hidden, k, rows, (const float*)topk_w);
  else
    return MSGL_BAD_ARG;
  MSGL_CHECK_LAUNCH("moe_permute");
  return MSGL_OK;
}

MSGL_API int msgl_moe_combine(const void* y, const void* topk_w, const void* pair_row, void* out, int tokens,
                              int hidden, int k, int dtype, cudaStream_t stream) {
  if (tokens == 0) return MSGL_OK;
  if (hidden % 8) return MSGL_BAD_ARG;
  int threads = hidden / 8 < 256 ? ((hidden / 8 + 31) / 32) * 32 : 256;
  if (dtype == MSGL_BF16)
    msgl_launch(moe_combine_kernel<__nv_bfloat16>, dim3(tokens), dim3(threads), 0, stream, (const __nv_bfloat16*)y, (const float*)topk_w,
                                                                     (const int32_t*)pair_row, (__nv_bfloat16*)out,
                                                                     hidden, k);
  else if (dtype == MSGL_F16)
    msgl_launch(moe_combine_kernel<__half>, dim3(tokens), dim3(threads), 0, stream, (const __half*)y, (const float*)topk_w,
                                                              (const int32_t*)pair_row, (__half*)out, hidden, k);
  else
    return MSGL_BAD_ARG;
  MSGL_CHECK_LAUNCH("moe_combine");
  return MSGL_OK;
}
