// Flat-buffer optimizer kernels: one launch per (decay / no-decay) region instead of one per tensor, the
// gradient scale (unscale x clip, or 0 = "skip this step") read from device memory so that the inf/NaN
// decision never round-trips through the host, and the 16-bit shadow weights written in the same pass.
// Arithmetic per element is the reference's k_adamw / k_lion (cuda/kernels.cu:1021-1066, see also
// core/ops_cpu_dense.cpp:997-1030); the squared-norm reduction replaces one launch + D2H per tensor
// (cuda/kernels.cu:1068-1128) by a two-stage deterministic reduction over the flat gradient.
#include "sm100_common.cuh"
#include "gb_api.h"

namespace gb {

struct OptConst { float scale, lr, bc1, bc2, beta1, beta2, eps, wd; };
template <int KIND>
__device__ __forceinline__ void opt_update(float& w, float g, float& m, float& v, const OptConst& c) {
  const float gi = g * c.scale;
  if (KIND == 0) {
    m = c.beta1 * m + (1.0f - c.beta1) * gi;
    v = c.beta2 * v + (1.0f - c.beta2) * gi * gi;
    float upd = (m / c.bc1) / (sqrtf(v / c.bc2) + c.eps);
    if (c.wd != 0.0f) upd += c.wd * w;
    w -= c.lr * upd;
  } else {
    const float d = c.beta1 * m + (1.0f - c.beta1) * gi;
    float upd = (d > 0.0f) ? 1.0f : ((d < 0.0f) ? -1.0f : 0.0f);
    if (c.wd != 0.0f) upd += c.wd * w;
    w -= c.lr * upd;
    m = c.beta2 * m + (1.0f - c.beta2) * gi;
  }
}

// Bound by memory: 30 bytes a parameter (Lion 22).  Four parameters a thread, one trip, as many blocks as that takes: 148 x 8 blocks that walk
// the buffers reach 6.1 TB/s here, this 6.9 (as long as the four values stay in registers: with a count in the loops over them they
// lived in local memory, 4.1 TB/s).  108 M parameters, AdamW: 785 -> 473 us.
template <typename T, int KIND>
__global__ void __launch_bounds__(256) opt_step_kernel(float* __restrict__ w, const float* __restrict__ g,
                                                       float* __restrict__ m, float* __restrict__ v, T* __restrict__ w16,
                                                       long long n, const float* __restrict__ hyper,
                                                       const float* __restrict__ scale_dev, float beta1, float beta2,
                                                       float eps, float wd) {
  const OptConst c{scale_dev[0], hyper[0], hyper[1], hyper[2], beta1, beta2, eps, wd};
  if (c.scale == 0.f) return;   // rejected step: weights, moments and shadows stay as they are
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * 4;
  if (i + 4 <= n) {
    float4 a = *reinterpret_cast<const float4*>(w + i), d = *reinterpret_cast<const float4*>(m + i), e = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 b = *reinterpret_cast<const float4*>(g + i);
    if (KIND == 0) e = *reinterpret_cast<const float4*>(v + i);
    opt_update<KIND>(a.x, b.x, d.x, e.x, c);
    opt_update<KIND>(a.y, b.y, d.y, e.y, c);
    opt_update<KIND>(a.z, b.z, d.z, e.z, c);
    opt_update<KIND>(a.w, b.w, d.w, e.w, c);
    *reinterpret_cast<float4*>(w + i) = a;
    *reinterpret_cast<float4*>(m + i) = d;
    if (KIND == 0) *reinterpret_cast<float4*>(v + i) = e;
    if (w16) *reinterpret_cast<uint2*>(w16 + i) = make_uint2(Cvt<T>::pack2(a.x, a.y), Cvt<T>::pack2(a.z, a.w));
  } else {
    for (long long k = i; k < n; ++k) {
      float x = w[k], y = m[k], z = KIND == 0 ? v[k] : 0.f;
      opt_update<KIND>(x, g[k], y, z, c);
      w[k] = x;
      m[k] = y;
      if (KIND == 0) v[k] = z;
      if (w16) w16[k] = Cvt<T>::from_f(x);
    }
  }
}

constexpr int SQ_THREADS = 256;
constexpr long long SQ_CHUNK = 1 << 16;   // elements per block

__global__ void __launch_bounds__(SQ_THREADS) sqnorm_partial_kernel(const float* __restrict__ g, long long n,
                                                                    double* __restrict__ partial) {
  __shared__ double s[SQ_THREADS];
  const long long lo = blockIdx.x * SQ_CHUNK, hi = min(n, lo + SQ_CHUNK);
  double acc = 0.0;
  long long i = lo + threadIdx.x * 4;
  for (; i + 7 * SQ_THREADS * 4 + 4 <= hi; i += 8 * SQ_THREADS * 4) {            // eight loads in flight, added in the order of the loop below
    float4 a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = *reinterpret_cast<const float4*>(g + i + u * SQ_THREADS * 4);
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += (double)a[u].x * a[u].x + (double)a[u].y * a[u].y + (double)a[u].z * a[u].z + (double)a[u].w * a[u].w;
  }
  for (; i < hi; i += SQ_THREADS * 4) {
    if (i + 4 <= hi) {
      const float4 a = *reinterpret_cast<const float4*>(g + i);
      acc += (double)a.x * a.x + (double)a.y * a.y + (double)a.z * a.z + (double)a.w * a.w;
    } else {
      for (long long k = i; k < hi; ++k) acc += (double)g[k] * g[k];
    }
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = SQ_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// out[0] = grad_scale * clip_factor, or 0 when the norm is not finite; out[1] = gnorm.
// extra_sq (optional): further squared-norm terms already reduced elsewhere (e.g. other ranks' shards).
__global__ void finish_norm_kernel(const double* __restrict__ partial, int n_partial, const float* __restrict__ gs_dev,
                                   float grad_scale, float clip, float* __restrict__ out) {
  __shared__ double s[256];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n_partial; i += 256) acc += partial[i];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float gs = gs_dev ? gs_dev[0] : grad_scale;
    const double gnorm = sqrt(s[0]) * (double)gs;
    float clip_scale = 1.0f;
    if (clip > 0.0f && gnorm > (double)clip) clip_scale = (float)((double)clip / (gnorm + 1e-6));
    const bool finite = isfinite(gnorm);
    out[0] = finite ? gs * clip_scale : 0.f;
    out[1] = (float)gnorm;
  }
}

__global__ void fill_f32_kernel(float* __restrict__ p, float v, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) p[i] = v;
}

}  // namespace gb

using namespace gb;

extern "C" int gb_optimizer_step(const gb_opt_args* a, cudaStream_t st) {
  if (!a || a->n < 0 || !a->w || !a->g || !a->m || !a->scale_dev || !a->hyper) return -1;
  if (a->kind == 0 && !a->v) return -1;
  if (a->n == 0) return 0;
  if ((reinterpret_cast<uintptr_t>(a->w) | reinterpret_cast<uintptr_t>(a->g) | reinterpret_cast<uintptr_t>(a->m)) & 15) return -2;
  const long long blocks = ((a->n + 3) / 4 + 255) / 256;
  if (blocks > 0x7fffffffll) return -3;
#define GB_OPT(T, KIND)                                                                                              \
  opt_step_kernel<T, KIND><<<(int)blocks, 256, 0, st>>>(a->w, a->g, a->m, a->v, (T*)a->w16, a->n, a->hyper, a->scale_dev, \
                                                        a->beta1, a->beta2, a->eps, a->wd)
  if (a->is_bf16) { if (a->kind == 0) GB_OPT(__nv_bfloat16, 0); else GB_OPT(__nv_bfloat16, 1); }
  else { if (a->kind == 0) GB_OPT(__half, 0); else GB_OPT(__half, 1); }
#undef GB_OPT
  return gb_launch_rc();
}

extern "C" int gb_sqnorm_blocks(long long n) { return (int)((n + SQ_CHUNK - 1) / SQ_CHUNK); }

extern "C" int gb_sqnorm_partial(const float* g, long long n, double* partial, cudaStream_t st) {
  if (n <= 0) return 0;
  if (reinterpret_cast<uintptr_t>(g) & 15) return -2;
  sqnorm_partial_kernel<<<gb_sqnorm_blocks(n), SQ_THREADS, 0, st>>>(g, n, partial);
  return gb_launch_rc();
}

extern "C" int gb_finish_norm(const double* partial, int n_partial, const float* grad_scale_dev, float grad_scale,
                              float clip, float* out, cudaStream_t st) {
  finish_norm_kernel<<<1, 256, 0, st>>>(partial, n_partial, grad_scale_dev, grad_scale, clip, out);
  return gb_launch_rc();
}

extern "C" int gb_fill_f32(float* p, float v, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  fill_f32_kernel<<<(int)blocks, 256, 0, st>>>(p, v, n);
  return gb_launch_rc();
}
