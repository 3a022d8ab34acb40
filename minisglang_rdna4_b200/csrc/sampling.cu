// Sampling kernels: row-wise arg-max over fp32 logits (greedy decoding and speculative verify)
// and temperature / top-k / top-p / min-p sampling by bisection on the probability threshold.
//
// Replaces the reference's sampler_hip.top_k_top_p_sampling_from_logits_
// (python/minisgl/engine/_sampler_hip.py:42-63) and the torch arg-max of its greedy path.
// The sampling kernel never sorts the vocabulary: top-k and top-p both keep "every token
// whose probability is at least some pivot", so the pivot is found by bisection over
// probability values (each probe is one pass over the row held in shared memory or re-read
// from L2), then the token is drawn by an inverse-CDF scan in vocabulary order over the kept
// set. Semantics follow python/minisgl/engine/sample.py:108-142 (min-p floor, then top-k, then
// top-p over the surviving mass, renormalise, draw).
#include "common.cuh"
#include "ptx.cuh"

#include <cooperative_groups.h>

using namespace msgl;

namespace {

constexpr int kArgmaxCtas = 8;   // of a row's cluster

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  // larger value wins; on ties the lower index wins (matches torch.argmax on the first maximum)
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

// A cluster of gridDim.x CTAs per row, each with a contiguous share of it. Bound: for few rows the loads that one SM keeps in
// flight. argmax_plan has the times.
template <int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) argmax_kernel(const float* __restrict__ logits, int32_t* __restrict__ out,
                                                     int vocab, long long stride) {
  // A CTA's shared memory may be written by the others once it runs: each says so here, and waits for the others to have
  // said so in front of its store. The scan of the row lies in between.
  if (gridDim.x > 1) ptx::cluster_arrive_all();
  pdl_enter();
  __shared__ ArgMax red[THREADS / 32];
  __shared__ ArgMax all[kArgmaxCtas];
  const float* row = logits + (size_t)blockIdx.y * stride;
  ArgMax best{-INFINITY, 0x7fffffff};
  const int share = ((vocab + (int)gridDim.x - 1) / (int)gridDim.x + 3) / 4 * 4;   // a multiple of 4: shares stay aligned
  const int begin = min(vocab, (int)blockIdx.x * share), end = min(vocab, begin + share);
  if (((uintptr_t)row % 16) == 0) {
    const int vec_end = begin + (end - begin) / 4 * 4, step = blockDim.x * 4;
    for (int i0 = begin + threadIdx.x * 4; i0 < vec_end; i0 += 4 * step) {
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i0 + j * step < vec_end) v[j] = *reinterpret_cast<const float4*>(row + i0 + j * step);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + j * step;
        if (i >= vec_end) break;
        best = better(best, ArgMax{v[j].x, i});
        best = better(best, ArgMax{v[j].y, i + 1});
        best = better(best, ArgMax{v[j].z, i + 2});
        best = better(best, ArgMax{v[j].w, i + 3});
      }
    }
    for (int i = vec_end + threadIdx.x; i < end; i += blockDim.x) best = better(best, ArgMax{row[i], i});
  } else {
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) best = better(best, ArgMax{row[i], i});
  }
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = better(best, other);
    }
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  reduce();
  if (lane == 0) red[warp] = best;
  __syncthreads();
  if (warp == 0) {
    best = lane < (int)(blockDim.x >> 5) ? red[lane] : ArgMax{-INFINITY, 0x7fffffff};
    reduce();
  }
  if (gridDim.x > 1) {
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    ptx::cluster_wait_all();
    if (threadIdx.x == 0) *cluster.map_shared_rank(all + blockIdx.x, 0) = best;
    __syncwarp();
    ptx::cluster_sync_all();
    if (blockIdx.x != 0) return;
    if (warp == 0) {
      best = lane < (int)gridDim.x ? all[lane] : ArgMax{-INFINITY, 0x7fffffff};
      reduce();
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[blockIdx.y] = best.i == 0x7fffffff ? 0 : best.i;
}

// ---- sampling --------------------------------------------------------------------------
// count and mass of probabilities > pivot (strict) or >= pivot
__device__ __forceinline__ void probe(const float* __restrict__ row, int vocab, float mx, float inv_t, float inv_z,
                                      float pivot, bool strict, float* scratch, float& count, float& mass) {
  float c = 0.f, m = 0.f;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float p = __expf((row[i] - mx) * inv_t) * inv_z;
    if (strict ? (p > pivot) : (p >= pivot)) { c += 1.f; m += p; }
  }
  count = block_sum(c, scratch);
  mass = block_sum(m, scratch);
}

__global__ void __launch_bounds__(1024) sample_kernel(const float* __restrict__ logits, long long stride,
                                                      const float* __restrict__ temps, const int32_t* __restrict__ top_k,
                                                      const float* __restrict__ top_p, const float* __restrict__ min_p,
                                                      const float* __restrict__ uniform, int32_t* __restrict__ out,
                                                      int vocab) {
  pdl_enter();
  __shared__ float scratch[32];
  __shared__ ArgMax red[32];
  __shared__ float warp_mass[32];
  const int r = blockIdx.x;
  const float* row = logits + (size_t)r * stride;
  const float t = temps[r];
  // row maximum and arg-max
  ArgMax best{-INFINITY, 0x7fffffff};
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) best = better(best, ArgMax{row[i], i});
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) red[warp] = best;
  __syncthreads();
  best = red[0];
  for (int w = 1; w < nw; ++w) best = better(best, red[w]);
  if (t <= 0.f) {
    if (threadIdx.x == 0) out[r] = best.i;
    return;
  }
  const float mx = best.v, inv_t = 1.f / fmaxf(t, 1e-6f);
  float z = 0.f;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) z += __expf((row[i] - mx) * inv_t);
  z = block_sum(z, scratch);
  const float inv_z = 1.f / z;
  const float p_max = inv_z;  // probability of the arg-max token
  // pivot = smallest probability that is still kept
  float pivot = 0.f;
  if (min_p != nullptr && min_p[r] > 0.f) pivot = p_max * min_p[r];
  const int k = top_k != nullptr ? top_k[r] : 0;
  const float pp = top_p != nullptr ? top_p[r] : 1.f;
  if ((k > 0 && k < vocab) || pp < 1.f) {
    // A token of probability x survives iff fewer than k tokens are more probable and the mass of
    // the more probable tokens does not exceed top-p. Both tests are monotone in x, so the kept
    // set is {p >= x*}; bisect for x*. `hi` always passes the test, `lo` does not.
    float lo = 0.f, hi = p_max;
    for (int it = 0; it < 40; ++it) {
      const float mid = 0.5f * (lo + hi);
      if (mid <= lo || mid >= hi) break;
      float cnt, mass;
      probe(row, vocab, mx, inv_t, inv_z, mid, true, scratch, cnt, mass);
      const bool keep = !((k > 0 && k < vocab) && cnt >= (float)k) && !(pp < 1.f && mass > pp);
      if (keep) hi = mid; else lo = mid;
    }
    pivot = fmaxf(pivot, hi);
  }
  // kept mass
  float cnt, mass;
  probe(row, vocab, mx, inv_t, inv_z, pivot, false, scratch, cnt, mass);
  const float target = uniform[r] * mass;
  // inverse-CDF scan in vocabulary order over kept tokens: each thread owns a contiguous span
  const int per = (vocab + blockDim.x - 1) / blockDim.x;
  const int begin = min(threadIdx.x * per, vocab), end = min(begin + per, vocab);
  float local = 0.f;
  for (int i = begin; i < end; ++i) {
    const float p = __expf((row[i] - mx) * inv_t) * inv_z;
    if (p >= pivot) local += p;
  }
  // exclusive prefix over threads
  float incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) warp_mass[warp] = incl;
  __syncthreads();
  float warp_off = 0.f;
  for (int w = 0; w < warp; ++w) warp_off += warp_mass[w];
  const float excl = warp_off + incl - local;
  __shared__ int chosen;
  if (threadIdx.x == 0) chosen = -1;
  __syncthreads();
  if (local > 0.f && target >= excl && target < excl + local) {
    float run = excl;
    int pick = -1;
    for (int i = begin; i < end; ++i) {
      const float p = __expf((row[i] - mx) * inv_t) * inv_z;
      if (p >= pivot) {
        run += p;
        pick = i;
        if (target < run) break;
      }
    }
    if (pick >= 0) atomicMax(&chosen, pick);
  }
  __syncthreads();
  if (threadIdx.x == 0) out[r] = chosen >= 0 ? chosen : best.i;
}

}  // namespace

namespace {

struct ArgMaxPlan {
  int ctas, threads;   // of a row's cluster, of a CTA
  bool two;            // the form of which two CTAs of 1024 threads fit on an SM
};

// A share of less than 2048 values is one round of loads: nothing to split. Clusters of CTAs that do not all fit at once start in
// rounds, so a row has as many CTAs as keep the whole within the SMs; of wide rows up to four CTAs of 512 threads on an SM, whose loads
// make up for that. Up to two rows for each SM, one CTA a row of the form that fits twice.
// B200, us, 1024 threads a row -> this: 151936 columns, 1 row 13.7 -> 3.6, 16 14.2 -> 4.9, 37 14.3 -> 6.4, 64 14.4 -> 7.9 (clusters
// of 8: 10.5), 100 14.4 -> 9.6, 150 24.1 -> 19.0, 256 28.9 -> 27.2 (without the form for two: 34); 16384 columns, 1 row 2.6 -> 2.2,
// 64 2.9 -> 2.8 (clusters of 8: 5.4), 256 4.2 -> 4.1; 32000, 64 4.3 -> 3.5, 256 6.1 -> 6.2.
ArgMaxPlan argmax_plan(int rows, int vocab) {
  constexpr int sms = 148;
  const bool two = rows > sms && rows <= 2 * sms;
  if (vocab < kArgmaxCtas * 2048) return {1, 512, two};
  if (vocab < 65536) {
    if (rows <= sms / 2) return {rows <= sms / 8 ? 8 : rows <= sms / 4 ? 4 : 2, 512, false};
    return {1, 512, two};
  }
  if (rows <= 50) return {8, 512, false};
  if (rows <= sms / 2) return {2, 1024, true};
  if (rows <= sms) return {4, 512, false};
  if (rows <= sms * 3 / 2) return {2, 512, false};
  return {1, two ? 1024 : 512, two};
}

}  // namespace

MSGL_API int msgl_argmax(const void* logits, void* out, int rows, int vocab, long long stride, cudaStream_t stream) {
  if (rows == 0) return MSGL_OK;
  const ArgMaxPlan plan = argmax_plan(rows, vocab);
  auto* const kernel = plan.two ? argmax_kernel<1024, 2> : argmax_kernel<512, 3>;
  for (int r0 = 0; r0 < rows; r0 += 65535) {
    cudaLaunchAttribute attr[2] = {};
    int attrs = 0;
    if (msgl_pdl_enabled()) {
      attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (plan.ctas > 1) {
      attr[attrs].id = cudaLaunchAttributeClusterDimension;
      attr[attrs++].val.clusterDim = {(unsigned)plan.ctas, 1, 1};
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.ctas, rows - r0 < 65535 ? rows - r0 : 65535);
    cfg.blockDim = dim3(plan.threads);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = attrs;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, (const float*)logits + (size_t)r0 * stride, (int32_t*)out + r0,
                                             vocab, stride);
    if (e != cudaSuccess) { msgl_set_error("argmax", e); return MSGL_CUDA_ERROR; }
  }
  return MSGL_OK;
}

MSGL_API int msgl_sample(const void* logits, long long stride, const void* temps, const void* top_k,
                         const void* top_p, const void* min_p, const void* uniform, void* out, int rows, int vocab,
                         cudaStream_t stream) {
  if (rows == 0) return MSGL_OK;
  msgl_launch(sample_kernel, dim3(rows), dim3(1024), 0, stream, (const float*)logits, stride, (const float*)temps, (const int32_t*)top_k,
                                           (const float*)top_p, (const float*)min_p, (const float*)uniform,
                                           (int32_t*)out, vocab);
  MSGL_CHECK_LAUNCH("sample");
  return MSGL_OK;
}
