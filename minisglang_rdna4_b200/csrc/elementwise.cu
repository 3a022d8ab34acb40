// Elementwise / row-wise kernels: embedding gather, RMSNorm (+residual add) (+per-token e4m3
// producer), gated activations (+quant), stand-alone activation quantisers.
//
// Replaces the reference's tail_hip package (rms_norm, rms_norm_add, rms_norm_quant,
// rms_norm_add_quant, silu_and_mul, gelu_and_mul; python/minisgl/layers/norm.py:16-168,
// python/minisgl/layers/activation.py:25-64) and its embedding gather
// (python/minisgl/kernel/csrc/jit/index.cu:31-96). All kernels are memory-bound: they read
// each input once with 16-byte accesses and keep the row in shared memory between the
// reduction and the write.
#include "common.cuh"

#include <string>

using namespace msgl;

static thread_local std::string g_last_error;
void msgl_set_error(const char* where, cudaError_t err) {
  g_last_error = std::string(where) + ": " + cudaGetErrorString(err);
}
void msgl_set_error_text(const char* text) { g_last_error = text; }
MSGL_API const char* msgl_last_error() { return g_last_error.c_str(); }

static int g_pdl = 1;
bool msgl_pdl_enabled() { return g_pdl != 0; }
// Programmatic dependent launch of every kernel of the library: 1 on (default), 0 off.
MSGL_API int msgl_set_pdl(int on) {
  const int prev = g_pdl;
  g_pdl = on;
  return prev;
}

// ------------------------------------------------------------------------------------------
// embedding: out[i, :] = (start <= ids[i] < start + len) ? W[ids[i] - start, :] : 0
// ------------------------------------------------------------------------------------------
__global__ void embedding_kernel(const int32_t* __restrict__ ids, const uint4* __restrict__ w,
                                 uint4* __restrict__ out, int row_vecs, int start, int len) {
  pdl_enter();
  int row = blockIdx.x;
  (void)MSGL_OOB(ids[row], 0x7fffffffLL);   // a negative token id
  int id = ids[row] - start;
  bool inside = id >= 0 && id < len;
  const uint4* src = w + (size_t)(inside ? id : 0) * row_vecs;
  uint4* dst = out + (size_t)row * row_vecs;
  for (int i = threadIdx.x; i < row_vecs; i += blockDim.x)
    dst[i] = inside ? __ldg(src + i) : make_uint4(0, 0, 0, 0);
}

MSGL_API int msgl_embedding(const void* ids, const void* w, void* out, int rows, int hidden_bytes,
                            int start, int len, cudaStream_t stream) {
  if (hidden_bytes % 16) return MSGL_BAD_ARG;
  if (rows == 0) return MSGL_OK;
  int vecs = hidden_bytes / 16;
  int threads = vecs < 256 ? ((vecs + 31) / 32) * 32 : 256;
  msgl_launch(embedding_kernel, dim3(rows), dim3(threads), 0, stream, (const int32_t*)ids, (const uint4*)w, (uint4*)out, vecs,
                                                 start, len);
  MSGL_CHECK_LAUNCH("embedding");
  return MSGL_OK;
}

// ------------------------------------------------------------------------------------------
// RMSNorm family. One CTA per row; every thread keeps its VPT 16-byte vectors of the (summed) row in
// registers between the reduction and the write, so the row is read once.
//   ADD   : residual += x (stored back, rounded to T), norm of the sum
//   QUANT : emit e4m3 row + fp32 scale (amax/448) instead of T
//   PLANES: x is fp32 [planes][rows][hidden], the K ranges of a split-K GEMM; they are summed in
//           ascending order and rounded to T, which is what an unsplit GEMM would have handed over
//
// Bound: HBM for many rows, one memory round trip for few. All loads of a row (x, residual, weight; of
// planes four at a time) are issued before the first store: with the residual's store between two
// vectors' loads each of up to eight vectors cost a round trip of its own. Threads and vectors a thread are
// chosen by the width and the form alone (never by the row count: the order of the sum, and with it a row's bits,
// would follow): two vectors a thread, so that a decode step's few rows have all their bytes under way too, four above 4096 columns,
// where 512 and more threads a row leave too few rows on an SM, and without a residual, which halves the bytes of a row, above 2560.
// B200, us, with the residual and e4m3 out, before -> after: 1 x 2560 3.9 -> 2.7, 64 x 4096 4.7 -> 3.1, 8190 x 2560 31.5 -> 30.3,
// 8190 x 8192 120 -> 107, 8190 x 12288 255 -> 200, 16 bits out 256 -> 140; without a residual 8190 x 8192 76 -> 64 (two
// vectors: 82), 8190 x 12288 117 -> 98 (157), 8190 x 4096 32.0 -> 32.7 (35.1), 16 x 4096 2.8 -> 2.0; 5 planes of 64 x 4096
// 7.6 -> 4.5, 3 of 32 x 8192 11.9 -> 4.9.
// ------------------------------------------------------------------------------------------
template <typename T, bool ADD, bool QUANT, int VPT, int MAXT, bool PLANES = false>
__global__ void __launch_bounds__(MAXT) rms_norm_kernel(const T* __restrict__ x, T* __restrict__ residual,
                                                        const T* __restrict__ w, T* __restrict__ out,
                                                        uint8_t* __restrict__ out_q, float* __restrict__ out_scale,
                                                        int hidden, float eps, float w_offset, int planes,
                                                        size_t plane_stride) {
  pdl_enter();
  __shared__ float scratch[32];
  const int row = blockIdx.x, step = blockDim.x * 8;
  const size_t at = (size_t)row * hidden;
  float v[VPT][8];
  Vec8<T> xv[VPT], rv[VPT], wv[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = j * step + threadIdx.x * 8;
    if (i < hidden) {
      if (!PLANES) xv[j] = *reinterpret_cast<const Vec8<T>*>(x + at + i);
      if (ADD) rv[j] = *reinterpret_cast<const Vec8<T>*>(residual + at + i);
      wv[j] = *reinterpret_cast<const Vec8<T>*>(w + i);
    }
  }
  if (PLANES) {
    const float* xp = reinterpret_cast<const float*>(x) + at;
#pragma unroll
    for (int j = 0; j < VPT; ++j)
#pragma unroll
      for (int k = 0; k < 8; ++k) v[j][k] = 0.f;
#pragma unroll 1
    for (int p0 = 0; p0 < planes; p0 += 4) {
      float4 t[4][VPT][2];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
          const int i = j * step + threadIdx.x * 8;
          if (p0 + p < planes && i < hidden) {
            t[p][j][0] = __ldg(reinterpret_cast<const float4*>(xp + (p0 + p) * plane_stride + i));
            t[p][j][1] = __ldg(reinterpret_cast<const float4*>(xp + (p0 + p) * plane_stride + i + 4));
          }
        }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int j = 0; j < VPT; ++j)
          if (p0 + p < planes && j * step + threadIdx.x * 8 < hidden)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              v[j][4 * h] += t[p][j][h].x; v[j][4 * h + 1] += t[p][j][h].y;
              v[j][4 * h + 2] += t[p][j][h].z; v[j][4 * h + 3] += t[p][j][h].w;
            }
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = j * step + threadIdx.x * 8;
    if (i < hidden) {
      if (PLANES) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j][k] = to_float(from_float<T>(v[j][k]));
      } else {
        unpack8(xv[j], v[j]);
      }
      if (ADD) {
        float r[8];
        unpack8(rv[j], r);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j][k] += r[k];
        store8(residual + at + i, v[j]);
        // the norm sees the rounded residual, exactly what the next layer will read
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j][k] = to_float(from_float<T>(v[j][k]));
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += v[j][k] * v[j][k];
    }
  }
  ss = block_sum(ss, scratch);
  const float rstd = rsqrtf(ss / (float)hidden + eps);
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = j * step + threadIdx.x * 8;
    if (i < hidden) {
      float wf[8];
      unpack8(wv[j], wf);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        // round to T as the unfused op would, so the quantised row matches norm -> quant
        v[j][k] = to_float(from_float<T>(v[j][k] * rstd * (wf[k] + w_offset)));
        if (QUANT) amax = fmaxf(amax, fabsf(v[j][k]));
      }
      if (!QUANT) store8(out + at + i, v[j]);
    }
  }
  if (QUANT) {
    amax = block_max(amax, scratch);
    const float scale = fmaxf(amax, 1e-8f) / kFp8Max;
    if (threadIdx.x == 0) out_scale[row] = scale;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = j * step + threadIdx.x * 8;
      if (i < hidden) *reinterpret_cast<uint2*>(out_q + at + i) = pack8_e4m3(v[j], scale);
    }
  }
}

constexpr int kMaxRow = 16384, kMaxPlanesRow = 8192;   // widest row of a norm, and of one that sums planes

// planes == 0: x is of type T
template <typename T, int VPT, int MAXT>
static void launch_rms_vpt(const void* x, int planes, void* residual, const void* w, void* out, void* out_q, void* out_scale,
                           int rows, int hidden, float eps, float off, cudaStream_t s) {
  const bool add = residual != nullptr, quant = out_q != nullptr;
  const int vecs = hidden / 8, threads = vecs > 0 ? ((vecs + VPT - 1) / VPT + 31) / 32 * 32 : 32;
  const size_t stride = (size_t)rows * hidden;
#define RMS_LAUNCH(A, Q, P)                                                                                                   \
  msgl_launch(rms_norm_kernel<T, A, Q, VPT, MAXT, P>, dim3(rows), dim3(threads), 0, s, (const T*)x, (T*)residual, (const T*)w, \
              (T*)out, (uint8_t*)out_q, (float*)out_scale, hidden, eps, off, planes, stride)
  if constexpr (MAXT * VPT * 8 <= kMaxPlanesRow && VPT < 4) {
    if (planes > 0) {
      if (quant) RMS_LAUNCH(true, true, true);
      else RMS_LAUNCH(true, false, true);
      return;
    }
  }
  if (add && quant) RMS_LAUNCH(true, true, false);
  else if (add) RMS_LAUNCH(true, false, false);
  else if (quant) RMS_LAUNCH(false, true, false);
  else RMS_LAUNCH(false, false, false);
#undef RMS_LAUNCH
}

template <typename T>
static int launch_rms(const void* x, int planes, void* residual, const void* w, void* out, void* out_q, void* out_scale, int rows,
                      int hidden, float eps, int plus_one, cudaStream_t s) {
  const float off = plus_one ? 1.f : 0.f;
  const int vecs = hidden / 8;
  const bool plain = residual == nullptr && out_q == nullptr;
#define RMS(V, TH) launch_rms_vpt<T, V, TH>(x, planes, residual, w, out, out_q, out_scale, rows, hidden, eps, off, s)
  if (vecs <= 128) RMS(1, 128);
  else if (vecs <= 512 && !(plain && vecs > 320)) RMS(2, 256);
  else if (vecs <= 512) RMS(4, 128);
  else if (planes > 0) RMS(2, 512);   // (whose loads of four planes are registers enough)
  else if (vecs <= 1024) RMS(4, 256);
  else RMS(4, 512);
#undef RMS
  MSGL_CHECK_LAUNCH("rms_norm");
  return MSGL_OK;
}

// residual += sum of the fp32 planes [planes][rows][hidden] of a split-K GEMM (ascending order,
// rounded to the 16-bit type first), then the norm of the sum; 16-bit or quantised output.
MSGL_API int msgl_rms_norm_planes(const void* x_planes, int planes, void* residual, const void* w, void* out,
                                  void* out_q, void* out_scale, int rows, int hidden, float eps, int plus_one,
                                  int dtype, cudaStream_t stream) {
  if (hidden % 8 || hidden > kMaxPlanesRow || planes < 1 || residual == nullptr) return MSGL_BAD_ARG;
  if (rows == 0) return MSGL_OK;
  if (dtype == MSGL_BF16)
    return launch_rms<__nv_bfloat16>(x_planes, planes, residual, w, out, out_q, out_scale, rows, hidden, eps, plus_one, stream);
  if (dtype == MSGL_F16)
    return launch_rms<__half>(x_planes, planes, residual, w, out, out_q, out_scale, rows, hidden, eps, plus_one, stream);
  return MSGL_BAD_ARG;
}

// residual == nullptr: plain norm. out_q != nullptr: quantised output (out may be nullptr).
MSGL_API int msgl_rms_norm(const void* x, void* residual, const void* w, void* out, void* out_q,
                           void* out_scale, int rows, int hidden, float eps, int plus_one, int dtype,
                           cudaStream_t stream) {
  if (hidden % 8 || hidden > kMaxRow) return MSGL_BAD_ARG;
  if (rows == 0) return MSGL_OK;
  if (dtype == MSGL_BF16)
    return launch_rms<__nv_bfloat16>(x, 0, residual, w, out, out_q, out_scale, rows, hidden, eps, plus_one, stream);
  if (dtype == MSGL_F16)
    return launch_rms<__half>(x, 0, residual, w, out, out_q, out_scale, rows, hidden, eps, plus_one, stream);
  return MSGL_BAD_ARG;
}

// ------------------------------------------------------------------------------------------
// gated activation: out[m, i] = act(x[m, i]) * x[m, I + i]
// ------------------------------------------------------------------------------------------
enum ActKind : int { ACT_SILU = 0, ACT_GELU = 1, ACT_GELU_TANH = 2, ACT_CLAMPED = 3 };
__device__ __forceinline__ float act_fn(float g, int kind) {
  if (kind == ACT_SILU) {
    // x * sigmoid(x) = h + h * tanh(h) with h = x / 2: one special-function op instead of two
    // (exp and reciprocal); tanh.approx is good to ~2^-11, below the 16-bit rounding of the result
    const float h = 0.5f * g;
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
    return fmaf(h, t, h);
  }
  if (kind == ACT_GELU) return 0.5f * g * (1.f + erff(g * 0.70710678118654752f));
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * g * (1.f + tanhf(k0 * (g + k1 * g * g * g)));
}

// g sigmoid(alpha g) (u + 1), g clamped at limit from above, u on both sides
template <typename T> __device__ __forceinline__ float clamped_glu(float g, float u, float alpha, float limit) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  const float z = -alpha * g;
  return g / (1.f + (sizeof(T) == 4 ? expf(z) : __expf(z))) * (u + 1.f);
}

template <typename T>
__global__ void act_mul_kernel(const T* __restrict__ x, T* __restrict__ out, int inter, size_t total_vecs,
                               int kind, float alpha, float limit) {
  pdl_enter();
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total_vecs) return;
  int vecs_per_row = inter / 8;
  size_t row = idx / vecs_per_row;
  int col = (int)(idx % vecs_per_row) * 8;
  const T* g = x + row * 2 * inter + col;
  float a[8], b[8], y[8];
  load8(g, a);
  load8(g + inter, b);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (kind == ACT_CLAMPED) y[k] = clamped_glu<T>(a[k], b[k], alpha, limit);
    else if (sizeof(T) == 4 && kind == ACT_SILU) y[k] = a[k] / (1.f + expf(-a[k])) * b[k];
    else y[k] = act_fn(a[k], kind) * b[k];
  }
  store8(out + row * inter + col, y);
}

// The product is rounded to T before its maximum is taken, so a thread keeps it as T between the two passes. Bound: HBM.
// KIND is a constant (a branch on it between two vectors' loads made each of up to 14 vectors a memory round trip of
// its own) and the loads of AHEAD vectors are issued together.
// B200, us, before -> after: 8192 x 28672 698 -> 310 (3.8 TB/s), 8190 x 9728 86 -> 74.5, 1 x 9728 3.3 -> 2.9.
template <typename T, int VPT, int THREADS, int KIND>
__global__ void __launch_bounds__(THREADS) act_mul_quant_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q,
                                                                float* __restrict__ out_scale, int inter) {
  constexpr int AHEAD = VPT < 4 ? VPT : 4;
  pdl_enter();
  __shared__ float scratch[32];
  const int row = blockIdx.x;
  const T* g = x + (size_t)row * 2 * inter;
  Vec8<T> kept[VPT];
  float amax = 0.f;
#pragma unroll
  for (int j0 = 0; j0 < VPT; j0 += AHEAD) {
    Vec8<T> a[AHEAD], b[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      const int i = ((j0 + j) * THREADS + threadIdx.x) * 8;
      if (j0 + j < VPT && i < inter) {
        a[j] = *reinterpret_cast<const Vec8<T>*>(g + i);
        b[j] = *reinterpret_cast<const Vec8<T>*>(g + inter + i);
      }
    }
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      const int i = ((j0 + j) * THREADS + threadIdx.x) * 8;
      if (j0 + j < VPT && i < inter) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 ga = to_float2(a[j].v[k]), up = to_float2(b[j].v[k]);
          const auto y = Pack2<T>::make(act_fn(ga.x, KIND) * up.x, act_fn(ga.y, KIND) * up.y);
          kept[j0 + j].v[k] = y;
          const float2 f = to_float2(y);
          amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
      }
    }
  }
  amax = block_max(amax, scratch);
  const float scale = fmaxf(amax, 1e-8f) / kFp8Max;
  if (threadIdx.x == 0) out_scale[row] = scale;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = (j * THREADS + threadIdx.x) * 8;
    if (i < inter) {
      float v[8];
      unpack8(kept[j], v);
      *reinterpret_cast<uint2*>(out_q + (size_t)row * inter + i) = pack8_e4m3(v, scale);
    }
  }
}

template <typename T, int KIND>
static int launch_act_quant(const void* x, void* out_q, void* out_scale, int rows, int inter, cudaStream_t s) {
  // the widest block that has a few vectors for every thread; a decode step's few rows take twice the threads, which have
  // more of a row under way at once (8190 x 1408: 11.3 us with 128 threads, 13.3 with 256; 1 x 1408 1.6 and 1.5)
  const int vecs = inter / 8;
#define ACT_LAUNCH(V, TH) \
  msgl_launch(act_mul_quant_kernel<T, V, TH, KIND>, dim3(rows), dim3(TH), 0, s, (const T*)x, (uint8_t*)out_q, (float*)out_scale, inter)
  if (vecs > 7 * 512) return MSGL_BAD_ARG;
  if (vecs > 5 * 256 || (rows <= 2048 && vecs > 512)) {
    const int vpt = (vecs + 511) / 512;
    if (vpt <= 2) ACT_LAUNCH(2, 512);
    else if (vpt <= 3) ACT_LAUNCH(3, 512);
    else if (vpt <= 4) ACT_LAUNCH(4, 512);
    else if (vpt <= 5) ACT_LAUNCH(5, 512);
    else ACT_LAUNCH(7, 512);
  } else {
    const int vpt = (vecs + 255) / 256;
    if (vecs <= 128) ACT_LAUNCH(1, 128);
    else if (vecs <= 256 && rows > 2048) ACT_LAUNCH(2, 128);
    else if (vpt <= 1) ACT_LAUNCH(1, 256);
    else if (vpt <= 2) ACT_LAUNCH(2, 256);
    else if (vpt <= 3) ACT_LAUNCH(3, 256);
    else ACT_LAUNCH(5, 256);
  }
#undef ACT_LAUNCH
  return MSGL_OK;
}

template <typename T>
static int launch_act_quant(const void* x, void* out_q, void* out_scale, int rows, int inter, int kind, cudaStream_t s) {
  if (kind == ACT_SILU) return launch_act_quant<T, ACT_SILU>(x, out_q, out_scale, rows, inter, s);
  if (kind == ACT_GELU) return launch_act_quant<T, ACT_GELU>(x, out_q, out_scale, rows, inter, s);
  return launch_act_quant<T, ACT_GELU_TANH>(x, out_q, out_scale, rows, inter, s);
}

// alpha, limit: constants of kind 3 (clamped), which has no quantised form
MSGL_API int msgl_act_and_mul(const void* x, void* out, void* out_q, void* out_scale, int rows, int inter,
                              int kind, float alpha, float limit, int dtype, cudaStream_t stream) {
  if (kind == ACT_CLAMPED && out_q != nullptr) return MSGL_BAD_ARG;
  if (inter % 8) return MSGL_BAD_ARG;
  if (rows == 0) return MSGL_OK;
  if (out_q == nullptr) {
    size_t vecs = (size_t)rows * (inter / 8);
    int threads = 256;
    unsigned blocks = (unsigned)((vecs + threads - 1) / threads);
    if (dtype == MSGL_BF16)
      msgl_launch(act_mul_kernel<__nv_bfloat16>, dim3(blocks), dim3(threads), 0, stream, (const __nv_bfloat16*)x, (__nv_bfloat16*)out,
                                                                    inter, vecs, kind, alpha, limit);
    else if (dtype == MSGL_F16)
      msgl_launch(act_mul_kernel<__half>, dim3(blocks), dim3(threads), 0, stream, (const __half*)x, (__half*)out, inter, vecs, kind,
                  alpha, limit);
    else if (dtype == MSGL_F32)
      msgl_launch(act_mul_kernel<float>, dim3(blocks), dim3(threads), 0, stream, (const float*)x, (float*)out, inter, vecs, kind,
                  alpha, limit);
    else
      return MSGL_BAD_ARG;
  } else {
    int rc;
    if (dtype == MSGL_BF16) rc = launch_act_quant<__nv_bfloat16>(x, out_q, out_scale, rows, inter, kind, stream);
    else if (dtype == MSGL_F16) rc = launch_act_quant<__half>(x, out_q, out_scale, rows, inter, kind, stream);
    else return MSGL_BAD_ARG;
    if (rc) return rc;
  }
  MSGL_CHECK_LAUNCH("act_and_mul");
  return MSGL_OK;
}

// ------------------------------------------------------------------------------------------
// stand-alone activation quantisers: per token (group == hidden) or per `group` elements
// ------------------------------------------------------------------------------------------
// A group is one row of up to 16384 elements (a CTA each, VPT 16-byte vectors a thread, read once), or a run of
// elements of any multiple of 8 (a power of two of lanes each, vectors 16 bytes a lane). Many short rows are runs too: a CTA of
// one or two warps for each costs more than it reads (8190 x 512 8.9 us, as runs 4.2; 8190 x 1024 9.0, 6.6; but 2397 x 1024 2.9, 3.5).
// B200, us, a warp for each group of any length and two passes over it -> now: 1 x 4096 3.7 -> 1.8, 256 x 4096 5.1 -> 2.7, 8192 x 8192 53 -> 38; 16640 x 2048 in groups of 128
// 51 -> 33.
template <typename T, int VPT>
__global__ void __launch_bounds__(512) quant_row_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q,
                                                        float* __restrict__ out_scale, int group) {
  pdl_enter();
  __shared__ float scratch[32];
  const size_t at = (size_t)blockIdx.x * group;
  const int step = blockDim.x * 8;
  Vec8<T> kept[VPT];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = j * step + threadIdx.x * 8;
    if (i < group) kept[j] = *reinterpret_cast<const Vec8<T>*>(x + at + i);
  }
#pragma unroll
  for (int j = 0; j < VPT; ++j)
    if (j * step + threadIdx.x * 8 < group) {
      float v[8];
      unpack8(kept[j], v);
#pragma unroll
      for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(v[k]));
    }
  amax = block_max(amax, scratch);
  const float scale = fmaxf(amax, 1e-8f) / kFp8Max;
  if (threadIdx.x == 0) out_scale[blockIdx.x] = scale;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = j * step + threadIdx.x * 8;
    if (i < group) {
      float v[8];
      unpack8(kept[j], v);
      *reinterpret_cast<uint2*>(out_q + at + i) = pack8_e4m3(v, scale);
    }
  }
}

template <typename T, int LANES>
__global__ void __launch_bounds__(256) quant_group_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_q,
                                                          float* __restrict__ out_scale, int group, size_t total_groups) {
  pdl_enter();
  const size_t gidx = ((size_t)blockIdx.x * 256 + threadIdx.x) / LANES;
  const bool live = gidx < total_groups;
  const int lane = threadIdx.x & (LANES - 1);
  const T* src = x + gidx * group;
  float amax = 0.f;
  for (int i = lane * 8; live && i < group; i += LANES * 8) {
    float v[8];
    load8(src + i, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(v[k]));
  }
#pragma unroll
  for (int o = LANES >> 1; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (!live) return;
  const float scale = fmaxf(amax, 1e-8f) / kFp8Max;
  if (lane == 0) out_scale[gidx] = scale;
  for (int i = lane * 8; i < group; i += LANES * 8) {
    float v[8];
    load8(src + i, v);
    *reinterpret_cast<uint2*>(out_q + gidx * group + i) = pack8_e4m3(v, scale);
  }
}

template <typename T>
static void launch_quant(const void* x, void* out_q, void* out_scale, size_t total, int group, cudaStream_t s) {
  const int vecs = group / 8;
  const bool runs = vecs <= 32 || (vecs <= 64 && total >= 2048) || (vecs <= 128 && total >= 4096);
  if (!runs && vecs <= 4 * 512) {
    const int vpt = vecs <= 64 ? 1 : vecs <= 1024 ? 2 : 4, threads = ((vecs + vpt - 1) / vpt + 31) / 32 * 32;
#define QUANT_ROW(V) \
  msgl_launch(quant_row_kernel<T, V>, dim3((unsigned)total), dim3(threads), 0, s, (const T*)x, (uint8_t*)out_q, (float*)out_scale, group)
    if (vpt == 1) QUANT_ROW(1);
    else if (vpt == 2) QUANT_ROW(2);
    else QUANT_ROW(4);
#undef QUANT_ROW
    return;
  }
#define QUANT_GROUPS(L)                                                                                                            \
  msgl_launch(quant_group_kernel<T, L>, dim3((unsigned)((total * L + 255) / 256)), dim3(256), 0, s, (const T*)x, (uint8_t*)out_q, \
              (float*)out_scale, group, total)
  if (vecs <= 1) QUANT_GROUPS(1);
  else if (vecs <= 2) QUANT_GROUPS(2);
  else if (vecs <= 4) QUANT_GROUPS(4);
  else if (vecs <= 8) QUANT_GROUPS(8);
  else if (vecs <= 16) QUANT_GROUPS(16);
  else QUANT_GROUPS(32);
#undef QUANT_GROUPS
}

MSGL_API int msgl_quant_fp8(const void* x, void* out_q, void* out_scale, int rows, int hidden, int group,
                            int dtype, cudaStream_t stream) {
  if (group <= 0) group = hidden;
  if (hidden % group || group % 8) return MSGL_BAD_ARG;
  if (rows == 0) return MSGL_OK;
  const size_t total = (size_t)rows * (hidden / group);
  if (dtype == MSGL_BF16) launch_quant<__nv_bfloat16>(x, out_q, out_scale, total, group, stream);
  else if (dtype == MSGL_F16) launch_quant<__half>(x, out_q, out_scale, total, group, stream);
  else return MSGL_BAD_ARG;
  MSGL_CHECK_LAUNCH("quant_fp8");
  return MSGL_OK;
}


// ---------------------------------------------------------------------------------- bounds-check report
#ifdef MSGL_CHECK_BOUNDS
namespace {
constexpr int kMaxCollectors = 64;
msgl_bounds_collect_fn g_collectors[kMaxCollectors];
int g_num_collectors = 0;
}  // namespace
void msgl_bounds_register(msgl_bounds_collect_fn fn) {
  if (g_num_collectors < kMaxCollectors) g_collectors[g_num_collectors++] = fn;
}
#endif

// 1 when this library was built with the device-side bounds checks.
MSGL_API int msgl_bounds_enabled() {
#ifdef MSGL_CHECK_BOUNDS
  return 1;
#else
  return 0;
#endif
}

// Collects (and clears) the out-of-range indices the kernels of this library have recorded on the
// current device since the last call. Writes up to `max_lines` text lines of `line_bytes` bytes each
// ("file.cu:LINE value V limit L") into `text`; returns the number of records. Synchronises the device.
MSGL_API int msgl_bounds_report(char* text, int max_lines, int line_bytes) {
#ifdef MSGL_CHECK_BOUNDS
  cudaDeviceSynchronize();
  int total = 0;
  for (int c = 0; c < g_num_collectors; ++c) {
    const char* file = "";
    msgl::BoundsRecord recs[msgl::kBoundsRing];
    const int n = g_collectors[c](&file, recs, msgl::kBoundsRing);
    const char* base = file;
    for (const char* p = file; *p; ++p)
      if (*p == '/') base = p + 1;
    for (int i = 0; i < n; ++i) {
      if (total < max_lines && text != nullptr)
        snprintf(text + (size_t)total * line_bytes, line_bytes, "%s:%d value %lld limit %lld", base, recs[i].line,
                 recs[i].value, recs[i].limit);
      ++total;
    }
  }
  return total;
#else
  (void)text; (void)max_lines; (void)line_bytes;
  return 0;
#endif
}
