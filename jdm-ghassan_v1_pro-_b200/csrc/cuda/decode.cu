// Decode-time kernels (contract in gb_decode.h).  Batch-1 decoding reads every active weight once per token and
// does two flops per weight: it is bound by HBM bandwidth and launch count, not by the tensor cores.  So weights
// stay in their storage format (fp16 / bf16 / 8-bit / 4-bit blocks) and are expanded in registers inside the dot
// product; one warp owns one output row, lanes stride over 8-value units of the row, partial sums are fp32.
#include <type_traits>

#include "sm100_common.cuh"
#include "gb_decode.h"
#include "decode_fmt.cuh"

namespace gb {

constexpr int GV_WARPS = 8;            // output rows per CTA
constexpr int GV_THREADS = GV_WARPS * 32;

template <typename XT>
__device__ __forceinline__ float dot8(const float (&w)[8], const XT* __restrict__ x) {
  const uint4 q = *reinterpret_cast<const uint4*>(x);
  float s = 0.f;
  if constexpr (std::is_same<XT, __half>::value) {
    const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); s += w[2 * i] * f.x + w[2 * i + 1] * f.y; }
  } else {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); s += w[2 * i] * f.x + w[2 * i + 1] * f.y; }
  }
  return s;
}

// KS warps share one stored row: warp slice ks takes units ks*32 + lane, stepping by 32*KS.  Decoding one token is
// bound by load latency, not bandwidth (a row is a few hundred bytes), so the short rows are spread over more warps
// and every lane keeps several independent loads in flight; the slices meet in shared memory.
template <int FMT, int NB, int KS, typename XT>
__device__ __forceinline__ void row_partial(const uint8_t* __restrict__ wrow, int K, const XT* __restrict__ x, long long ldx,
                                            int nb, int ks, float (&acc)[NB]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 2
  for (int u = lane + 32 * ks; u < (K >> 3); u += 32 * KS) {
    float w[8];
    load8<FMT>(wrow, u, w);
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (j < nb) acc[j] += dot8<XT>(w, x + j * ldx + 8 * u);
  }
}

// sum over lanes, then over the KS warps of the row; the result is valid in lane 0 of slice 0
template <int KS>
__device__ __forceinline__ float row_finish(float v, float* __restrict__ sm, int row_in_cta, int ks) {
  v = warp_sum(v);
  if constexpr (KS == 1) return v;
  if ((threadIdx.x & 31) == 0) sm[row_in_cta * KS + ks] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < KS; ++i) t += sm[row_in_cta * KS + i];
  __syncthreads();
  return t;
}

template <int FMT, int NB, int KS, typename XT>
__global__ void __launch_bounds__(GV_THREADS) gemv_kernel(const uint8_t* __restrict__ W, long long row_bytes, int N, int K,
                                                         const XT* __restrict__ x, long long ldx, int B,
                                                         void* __restrict__ out, long long ldo, int out_f32,
                                                         const float* __restrict__ addend, long long ld_add) {
  pdl_wait();
  __shared__ float sm[GV_WARPS];
  const int warp = threadIdx.x >> 5, ric = warp / KS, ks = warp % KS;
  const int row = blockIdx.x * (GV_WARPS / KS) + ric;
  const bool live = row < N;                              // dead rows still take part in the block barriers
  const uint8_t* wrow = W + (size_t)(live ? row : 0) * row_bytes;
  for (int b0 = 0; b0 < B; b0 += NB) {
    float acc[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) acc[j] = 0.f;
    const int nb = min(NB, B - b0);
    if (live) row_partial<FMT, NB, KS, XT>(wrow, K, x + (long long)b0 * ldx, ldx, nb, ks, acc);
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const float v0 = row_finish<KS>(acc[j], sm, ric, ks);
      if (live && j < nb && ks == 0 && (threadIdx.x & 31) == 0) {
        float v = v0;
        if (addend) v += addend[(long long)(b0 + j) * ld_add + row];
        if (out_f32) reinterpret_cast<float*>(out)[(long long)(b0 + j) * ldo + row] = v;
        else reinterpret_cast<XT*>(out)[(long long)(b0 + j) * ldo + row] = Cvt<XT>::from_f(v);
      }
    }
  }
}

template <int FMT, int KS, typename XT>
__global__ void __launch_bounds__(GV_THREADS) expert_swiglu_kernel(const uint8_t* __restrict__ Wg, const uint8_t* __restrict__ Wu,
                                                                  long long row_bytes, int ne, int E, int d,
                                                                  const XT* __restrict__ x, const int* __restrict__ idx,
                                                                  int top_k, int slots, XT* __restrict__ act) {
  pdl_wait();
  __shared__ float sm[2 * GV_WARPS];
  const int warp = threadIdx.x >> 5, ric = warp / KS, ks = warp % KS;
  const int j = blockIdx.x * (GV_WARPS / KS) + ric;
  const int b = blockIdx.y / slots, slot = blockIdx.y % slots;
  const int e = slot < top_k ? idx[b * top_k + slot] : ne;
  const bool live = j < E && e >= 0 && e <= ne;
  float g[1] = {0.f}, u[1] = {0.f};
  if (live) {
    const size_t r = (size_t)e * E + j;
    row_partial<FMT, 1, KS, XT>(Wg + r * row_bytes, d, x + (long long)b * d, d, 1, ks, g);
    row_partial<FMT, 1, KS, XT>(Wu + r * row_bytes, d, x + (long long)b * d, d, 1, ks, u);
  }
  const float gs = row_finish<KS>(g[0], sm, ric, ks);
  const float us = row_finish<KS>(u[0], sm + GV_WARPS, ric, ks);
  if (live && ks == 0 && (threadIdx.x & 31) == 0)
    act[((long long)b * slots + slot) * E + j] = Cvt<XT>::from_f(gs / (1.f + __expf(-gs)) * us);
}

template <int FMT, int KS, typename XT>
__global__ void __launch_bounds__(GV_THREADS) expert_down_kernel(const uint8_t* __restrict__ Wd, long long row_bytes, int ne, int d,
                                                                int E, const XT* __restrict__ act, const int* __restrict__ idx,
                                                                const float* __restrict__ w, int top_k, int slots,
                                                                const float* __restrict__ resid, float* __restrict__ out) {
  pdl_wait();
  __shared__ float sm[GV_WARPS];
  const int warp = threadIdx.x >> 5, ric = warp / KS, ks = warp % KS;
  const int r = blockIdx.x * (GV_WARPS / KS) + ric;
  const int b = blockIdx.y;
  const bool live = r < d;
  // weighted sum over the slots taken per lane before any reduction: one reduction per output value, and the
  // loads of different slots do not wait for one another.  Slot order and lane order are fixed: reproducible.
  float total = 0.f;
  if (live) {
    for (int slot = 0; slot < slots; ++slot) {
      const int e = slot < top_k ? idx[b * top_k + slot] : ne;
      if (e < 0 || e > ne) continue;
      const float wgt = slot < top_k ? w[b * top_k + slot] : 1.f;
      float y[1] = {0.f};
      row_partial<FMT, 1, KS, XT>(Wd + ((size_t)e * d + r) * row_bytes, E, act + ((long long)b * slots + slot) * E, E, 1, ks, y);
      total += wgt * y[0];
    }
  }
  const float t = row_finish<KS>(total, sm, ric, ks);
  if (live && ks == 0 && (threadIdx.x & 31) == 0) out[(long long)b * d + r] = resid[(long long)b * d + r] + t;
}

// Router for decode: one block per token, one warp per expert (round robin), then a serial soft-max / top-k over at
// most 64 experts.  Same rules as the training router: bias steers the selection only, ties go to the lowest index,
// weights are the selected probabilities renormalised.
template <typename XT>
__global__ void __launch_bounds__(256) decode_route_kernel(const XT* __restrict__ x, const float* __restrict__ rw,
                                                          const float* __restrict__ bias, int d, int ne, int top_k,
                                                          int* __restrict__ idx, float* __restrict__ wout) {
  pdl_wait();
  __shared__ float lg[64];
  const int b = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const XT* xr = x + (long long)b * d;
  for (int e = warp; e < ne; e += 8) {
    const float* wr = rw + (size_t)e * d;
    float s = 0.f;
    for (int i = lane * 2; i < d; i += 64) {
      const float2 xv = Cvt<XT>::unpack2(*reinterpret_cast<const uint32_t*>(xr + i));
      const float2 wv = *reinterpret_cast<const float2*>(wr + i);
      s += xv.x * wv.x + xv.y * wv.y;
    }
    s = warp_sum(s);
    if (lane == 0) lg[e] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mx = -INFINITY;
    for (int e = 0; e < ne; ++e) mx = fmaxf(mx, lg[e]);
    float sum = 0.f;
    for (int e = 0; e < ne; ++e) { lg[e] = __expf(lg[e] - mx); sum += lg[e]; }
    const float inv = 1.f / sum;
    unsigned long long taken = 0ull;
    float psel[8], psum = 0.f;
    int esel[8];
    for (int k = 0; k < top_k; ++k) {
      float bv = -INFINITY;
      int bi = 0;
      for (int e = 0; e < ne; ++e) {
        if (taken >> e & 1ull) continue;
        const float sc = lg[e] * inv + (bias ? bias[e] : 0.f);
        if (sc > bv) { bv = sc; bi = e; }
      }
      taken |= 1ull << bi;
      esel[k] = bi;
      psel[k] = lg[bi] * inv;
      psum += psel[k];
    }
    const float invs = psum > 1e-8f ? 1.f / psum : 0.f;
    for (int k = 0; k < top_k; ++k) {
      idx[b * top_k + k] = esel[k];
      wout[b * top_k + k] = psel[k] * invs;
    }
  }
}

// ---------------------------------------------------------------------------------------------- KV cache
// Keys, values and positions of the first *n of T prompt rows per sequence into the cache: one warp per row.
template <typename T>
__global__ void __launch_bounds__(256) kv_rows_kernel(const T* __restrict__ k, long long ld_k, const T* __restrict__ v, long long ld_v,
                                                      T* __restrict__ cK, T* __restrict__ cV, int* __restrict__ slot_pos,
                                                      const int* __restrict__ n, int rows, int Tlen, int cap, int kv_dim) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int b = row / Tlen, t = row - b * Tlen;
  if (row >= rows || t >= min(*n, cap)) return;
  const long long dst = ((long long)b * cap + t) * kv_dim;
  for (int i = lane * 8; i < kv_dim; i += 256) {
    *reinterpret_cast<uint4*>(cK + dst + i) = *reinterpret_cast<const uint4*>(k + row * ld_k + i);
    *reinterpret_cast<uint4*>(cV + dst + i) = *reinterpret_cast<const uint4*>(v + row * ld_v + i);
  }
  if (lane == 0) slot_pos[(long long)b * cap + t] = t;
}

template <typename T>
__global__ void kv_append_kernel(const T* __restrict__ k, long long ld_k, const T* __restrict__ v, long long ld_v,
                                 T* __restrict__ cK, T* __restrict__ cV, int* __restrict__ slot_pos,
                                 const gb_seq_state* __restrict__ st, int cap, int pinned, int kv_dim) {
  pdl_wait();
  const int b = blockIdx.x;
  const gb_seq_state s = st[b];
  const int slot = s.cache_len < cap ? s.cache_len : pinned + s.ring_start;
  T* dk = cK + ((long long)b * cap + slot) * kv_dim;
  T* dv = cV + ((long long)b * cap + slot) * kv_dim;
  for (int i = threadIdx.x * 8; i < kv_dim; i += blockDim.x * 8) {
    *reinterpret_cast<uint4*>(dk + i) = *reinterpret_cast<const uint4*>(k + b * ld_k + i);
    *reinterpret_cast<uint4*>(dv + i) = *reinterpret_cast<const uint4*>(v + b * ld_v + i);
  }
  if (threadIdx.x == 0) slot_pos[(long long)b * cap + slot] = s.abs_pos;
}

__global__ void decode_advance_kernel(gb_seq_state* __restrict__ st, int* __restrict__ pos_out, int B, int cap, int pinned) {
  pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  gb_seq_state s = st[b];
  if (s.cache_len < cap) s.cache_len += 1;
  else s.ring_start = (s.ring_start + 1) % max(1, cap - pinned);
  s.abs_pos += 1;
  st[b] = s;
  pos_out[b] = s.abs_pos;
}

// ---------------------------------------------------------------------------------------------- decode attention
// grid (B*KV, splits), 4 warps.  A block serves the G = H/KV query heads that share one K/V head, so each cached
// row is read once per group.  HD / 8 lanes share a slot with one 16-byte load of its key and one of its value, so a warp works on
// 256 / HD slots side by side and a dot product is reduced over HD / 8 lanes; the loads of four slots per lane come before the
// first use.  Every group of lanes keeps an online softmax per query head; groups, warps and then the splits are merged
// with the usual (max, sum, weighted output) rule.
// Bound by the latency of a trip (load, reduce, exponentials, accumulate).  One slot a trip over all 32 lanes took sixteen trips where
// this takes one (32 sequences, 500 slots, 8 splits): 18.6 -> 11.4 us a launch,
// and its merge, which overlaps it, 17.9 -> 6.2.
template <typename T, int HD, int G>
__global__ void __launch_bounds__(128) decode_attn_kernel(const T* __restrict__ q, long long ld_q, const T* __restrict__ cK,
                                                         const T* __restrict__ cV, const int* __restrict__ slot_pos,
                                                         const gb_seq_state* __restrict__ st, float* __restrict__ scratch,
                                                         int splits, int H, int KV, int cap, int window, float scale,
                                                         int* __restrict__ ticket, T* __restrict__ out, long long ld_o) {
  pdl_wait();
  constexpr int LPS = HD / 8, SPW = 32 / LPS, U = G <= 4 ? 4 : 2;      // lanes per slot, slots side by side, slots in flight per lane
  const int b = blockIdx.x / KV, kvh = blockIdx.x % KV, split = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane / LPS, sub = lane % LPS;
  const gb_seq_state s = st[b];
  // the step's own token was appended before this kernel and is not counted in cache_len yet
  const int n_slots = min(cap, s.cache_len + 1);
  const bool wide = ((reinterpret_cast<uintptr_t>(cK) | reinterpret_cast<uintptr_t>(cV)) & 15) == 0;    // rows are whole 64 bytes
  auto load8 = [&](const T* p) {
    uint4 r;
    if (wide) r = *reinterpret_cast<const uint4*>(p);
    else {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = Cvt<T>::pack2(Cvt<T>::to_f(p[2 * i]), Cvt<T>::to_f(p[2 * i + 1]));
      r = make_uint4(w[0], w[1], w[2], w[3]);
    }
    return r;
  };
  auto unpack8 = [](const uint4& r, float (&f)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 x = Cvt<T>::unpack2(w[i]); f[2 * i] = x.x; f[2 * i + 1] = x.y; }
  };
  float qv[G][8], m[G], l[G], o[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const T* qp = q + b * ld_q + (long long)(kvh * G + g) * HD + sub * 8;
#pragma unroll
    for (int e = 0; e < 8; ++e) { qv[g][e] = Cvt<T>::to_f(qp[e]) * scale; o[g][e] = 0.f; }
    m[g] = -INFINITY;
    l[g] = 0.f;
  }
  const int per = (n_slots + splits - 1) / splits;
  const int lo = split * per, hi = min(n_slots, lo + per);
  const long long kvd = (long long)KV * HD;
  const T* kb = cK + (long long)b * cap * kvd + kvh * HD + sub * 8;
  const T* vb = cV + (long long)b * cap * kvd + kvh * HD + sub * 8;
  for (int j0 = lo + warp * SPW; j0 < hi; j0 += U * 4 * SPW) {         // the warp's first slot of the trip
    uint4 kr[U], vr[U];
    bool ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * 4 * SPW + grp;
      ok[u] = j < hi && !(window > 0 && s.abs_pos - slot_pos[(long long)b * cap + j] >= window);
      kr[u] = vr[u] = make_uint4(0u, 0u, 0u, 0u);
      if (ok[u]) {
        kr[u] = load8(kb + (long long)j * kvd);
        vr[u] = load8(vb + (long long)j * kvd);
      }
    }
    float d[U][G];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float kf[8];
      unpack8(kr[u], kf);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float x = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) x += qv[g][e] * kf[e];
        d[u][g] = x;
      }
    }
#pragma unroll
    for (int off = LPS / 2; off > 0; off >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int g = 0; g < G; ++g) d[u][g] += __shfl_xor_sync(0xffffffffu, d[u][g], off);
    float p[U][G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float mn = m[g];
#pragma unroll
      for (int u = 0; u < U; ++u) if (ok[u]) mn = fmaxf(mn, d[u][g]);
      const float mu = mn == -INFINITY ? 0.f : mn;                     // nothing seen so far in this group of lanes
      const float c = __expf(m[g] - mu);
      l[g] *= c;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[g][e] *= c;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        p[u][g] = ok[u] ? __expf(d[u][g] - mu) : 0.f;
        l[g] += p[u][g];
      }
      m[g] = mn;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float vf[8];
      unpack8(vr[u], vf);
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int e = 0; e < 8; ++e) o[g][e] += p[u][g] * vf[e];
    }
  }
  // the groups of a warp
#pragma unroll
  for (int off = LPS; off < 32; off <<= 1)
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[g], off), mm = fmaxf(m[g], mo);
      const float f = m[g] == -INFINITY ? 0.f : __expf(m[g] - mm);
      l[g] *= f;
      l[g] += __shfl_xor_sync(0xffffffffu, l[g], off);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        o[g][e] *= f;
        o[g][e] += __shfl_xor_sync(0xffffffffu, o[g][e], off);
      }
      m[g] = mm;
    }
  // merge the four warps through shared memory
  __shared__ float sm_m[4][G], sm_l[4][G];
  __shared__ __align__(16) float sm_o[4][G][HD];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) { sm_m[warp][g] = m[g]; sm_l[warp][g] = l[g]; }
    if (grp == 0) {
      float4* dst = reinterpret_cast<float4*>(&sm_o[warp][g][sub * 8]);
      dst[0] = make_float4(o[g][0], o[g][1], o[g][2], o[g][3]);
      dst[1] = make_float4(o[g][4], o[g][5], o[g][6], o[g][7]);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < G * HD; t += 128) {
    const int g = t / HD, c = t % HD;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) mm = fmaxf(mm, sm_m[w][g]);
    float ll = 0.f, oo = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = sm_m[w][g] == -INFINITY ? 0.f : __expf(sm_m[w][g] - mm);
      ll += sm_l[w][g] * f;
      oo += sm_o[w][g][c] * f;
    }
    float* dst = scratch + (((long long)b * H + kvh * G + g) * splits + split) * (HD + 2);
    dst[2 + c] = oo;
    if (c == 0) { dst[0] = mm; dst[1] = ll; }
  }
  if (ticket == nullptr) return;            // the splits are merged by decode_attn_merge_kernel
  // The last split of this (sequence, kv head) to get here merges all of them, in split order: same result whoever
  // it is.  The ticket returns to zero for the next launch.
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const int t = atomicAdd(&ticket[blockIdx.x], 1);
    s_last = (t == splits - 1);
    if (s_last) ticket[blockIdx.x] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int t = threadIdx.x; t < G * HD; t += 128) {
    const int g = t / HD, c = t % HD;
    const float* base = scratch + ((long long)b * H + kvh * G + g) * splits * (HD + 2);
    float mm = -INFINITY;
    for (int sp = 0; sp < splits; ++sp) mm = fmaxf(mm, __ldcg(base + sp * (HD + 2)));
    float ll = 0.f, oo = 0.f;
    for (int sp = 0; sp < splits; ++sp) {
      const float ms = __ldcg(base + sp * (HD + 2));
      const float f = ms == -INFINITY ? 0.f : __expf(ms - mm);
      ll += __ldcg(base + sp * (HD + 2) + 1) * f;
      oo += __ldcg(base + sp * (HD + 2) + 2 + c) * f;
    }
    out[b * ld_o + (long long)(kvh * G + g) * HD + c] = Cvt<T>::from_f(ll > 0.f ? oo / ll : 0.f);
  }
}

// The same for up to eight splits (1, 2, 4 or 8): the splits of a (sequence, kv head) are a cluster, whose CTAs exchange their results through
// distributed shared memory and write the output, so there is no merge kernel behind it.  Keys and values are loaded two slots a lane ahead of
// the ones being worked on, with `early` the first ones before the wait for the kernel ahead, which then writes the step's own row and the queries and
// nothing else that is read here (a full ring's next slot is not known here, so it loads behind the wait).
// Bound by the latency of the chain and the instructions of the scores at short caches, by memory at long ones: 32 sequences, 500 slots, 3 query
// heads a key head, 4 splits (16 MB, 2.5 us at the copy rate): 8.3 us of the step, before 9.9 with 8 splits and 2.4 for the merge.
template <typename T, int HD, int G>
__global__ void __launch_bounds__(128, G <= 4 ? 4 : 2) decode_attn_cluster_kernel(const T* __restrict__ q, long long ld_q, const T* __restrict__ cK,
                                                                     const T* __restrict__ cV, const int* __restrict__ slot_pos,
                                                                     const gb_seq_state* __restrict__ st, int splits, int H, int KV, int cap, int window,
                                                                     float scale, int early, T* __restrict__ out, long long ld_o) {
  if (!early) pdl_wait();                                               // the launch ahead may have written the state or the cache
  constexpr int LPS = HD / 8, SPW = 32 / LPS, TRIP = 2 * 4 * SPW;       // lanes per slot, slots side by side, slots of a trip of the CTA
  __shared__ __align__(16) float sm_q[G][HD];
  constexpr int PARTS = 4 * SPW;                                        // groups of lanes that share a slot, in the CTA
  __shared__ float sm_m[PARTS + 1][G], sm_l[PARTS + 1][G], sm_f[PARTS][G];      // theirs, and the CTA's
  __shared__ __align__(16) float sm_o[PARTS + 1][G][HD];
  const int split = (int)cluster_ctarank(), item = (int)cluster_id_x(), b = item / KV, kvh = item - b * KV;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane / LPS, sub = lane % LPS;
  const gb_seq_state s = st[b];
  // the step's own token was appended before this kernel and is not counted in cache_len yet
  const int n_slots = min(cap, s.cache_len + 1);
  const bool full = s.cache_len >= cap;
  const bool wide = ((reinterpret_cast<uintptr_t>(cK) | reinterpret_cast<uintptr_t>(cV)) & 15) == 0;    // rows are whole 64 bytes
  const int per = (n_slots + splits - 1) / splits, lo = split * per, hi = min(n_slots, lo + per);
  const long long kvd = (long long)KV * HD;
  const T* kb = cK + (long long)b * cap * kvd + kvh * HD + sub * 8;
  const T* vb = cV + (long long)b * cap * kvd + kvh * HD + sub * 8;
  auto load8 = [&](const T* p) {
    uint4 r;
    if (wide) r = __ldcg(reinterpret_cast<const uint4*>(p));
    else {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = Cvt<T>::pack2(Cvt<T>::to_f(__ldcg(p + 2 * i)), Cvt<T>::to_f(__ldcg(p + 2 * i + 1)));
      r = make_uint4(w[0], w[1], w[2], w[3]);
    }
    return r;
  };
  struct Pair { uint4 k[2], v[2]; bool ok[2]; };
  const int first = lo + warp * SPW + grp;                              // the lane's slot u of trip t: first + (2 t + u) * 4 SPW
  auto fetch = [&](Pair& x, int t, bool own, bool rest) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = first + (2 * t + u) * 4 * SPW;
      const bool mine = j == n_slots - 1;                               // the step's own slot, unless the ring is full
      if (rest) {
        x.ok[u] = j < hi;
        x.k[u] = x.v[u] = make_uint4(0u, 0u, 0u, 0u);
      }
      if (j < hi && (mine ? own : rest)) {
        x.k[u] = load8(kb + (long long)j * kvd);
        x.v[u] = load8(vb + (long long)j * kvd);
        if (window > 0) x.ok[u] = s.abs_pos - __ldcg(slot_pos + (long long)b * cap + j) < window;
      }
    }
  };
  Pair A, B2;
  const int trips = hi > lo ? (hi - lo + TRIP - 1) / TRIP : 0;
  if (!full) { fetch(A, 0, false, true); fetch(B2, 1, false, true); }
  pdl_wait();
  fetch(A, 0, true, full);
  fetch(B2, 1, true, full);
  for (int i = threadIdx.x; i < G * HD; i += 128) sm_q[i / HD][i % HD] = Cvt<T>::to_f(q[b * ld_q + (long long)kvh * G * HD + i]) * scale;
  __syncthreads();
  auto unpack8 = [](const uint4& r, float (&f)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 x = Cvt<T>::unpack2(w[i]); f[2 * i] = x.x; f[2 * i + 1] = x.y; }
  };
  // The scores of a trip are one to a lane: the sums over the lanes of a slot are exchanged so that lane `sub` ends up with sum number sub & (NS - 1)
  // (heads below, the two slots above), which takes its exponential; the lanes then pass the weights round.
  constexpr int GP = G <= 1 ? 1 : G <= 2 ? 2 : G <= 4 ? 4 : 8, NS = 2 * GP;
  static_assert(NS <= 2 * LPS, "a slot's lanes hold at most two sums each");
  constexpr int PER = NS > LPS ? 2 : 1, ND = NS / PER;                  // sums a lane ends up with, lanes that differ
  const int mine = sub & (ND - 1);
  float o[G][8], m[PER], l[PER];                                        // of the lane's heads: maximum, the lane's share of the sum
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int e = 0; e < 8; ++e) o[g][e] = 0.f;
#pragma unroll
  for (int r = 0; r < PER; ++r) { m[r] = -INFINITY; l[r] = 0.f; }
  // sum i = u * GP + g; after the exchange lane `mine` holds sums mine + r * ND
  auto work = [&](const Pair& x) {
    float s[NS];
    {
      float f[2][8];
#pragma unroll
      for (int u = 0; u < 2; ++u) unpack8(x.k[u], f[u]);
#pragma unroll
      for (int g = 0; g < GP; ++g) {
        if (g < G) {
          const float4 q0 = *reinterpret_cast<const float4*>(&sm_q[g][sub * 8]), q1 = *reinterpret_cast<const float4*>(&sm_q[g][sub * 8 + 4]);
#pragma unroll
          for (int u = 0; u < 2; ++u)
            s[u * GP + g] = q0.x * f[u][0] + q0.y * f[u][1] + q0.z * f[u][2] + q0.w * f[u][3] + q1.x * f[u][4] + q1.y * f[u][5] + q1.z * f[u][6] + q1.w * f[u][7];
        } else {
          s[g] = s[GP + g] = 0.f;
        }
      }
    }
#pragma unroll
    for (int off = LPS / 2; off >= ND; off >>= 1)
#pragma unroll
      for (int i = 0; i < NS; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], off);
#pragma unroll
    for (int off = ND / 2; off > 0; off >>= 1) {
      const bool up = (sub & off) != 0;
#pragma unroll
      for (int r = 0; r < PER; ++r)
#pragma unroll
        for (int i = 0; i < off; ++i) {
          const float keep = up ? s[r * ND + i + off] : s[r * ND + i], give = up ? s[r * ND + i] : s[r * ND + i + off];
          s[r * ND + i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
    }
    float c[PER], p[PER], mn[PER], sc[PER];
#pragma unroll
    for (int r = 0; r < PER; ++r) {
      const int i = mine + r * ND, u = i / GP;
      sc[r] = (u == 0 ? x.ok[0] : x.ok[1]) ? s[r * ND] : -INFINITY;
      mn[r] = fmaxf(m[r], sc[r]);
    }
    if constexpr (PER == 2) {                                          // the lane holds both slots of its head
      mn[0] = mn[1] = fmaxf(mn[0], mn[1]);
    } else {
      mn[0] = fmaxf(mn[0], __shfl_xor_sync(0xffffffffu, mn[0], GP));
    }
#pragma unroll
    for (int r = 0; r < PER; ++r) {
      const float mu = mn[r] == -INFINITY ? 0.f : mn[r];               // nothing seen so far in this group of lanes
      c[r] = __expf(m[r] - mu);
      p[r] = __expf(sc[r] - mu);
      l[r] = l[r] * c[r] + p[r];
      m[r] = mn[r];
    }
    float f[2][8];
#pragma unroll
    for (int u = 0; u < 2; ++u) unpack8(x.v[u], f[u]);
    const int lead = lane - sub;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float cg = __shfl_sync(0xffffffffu, c[0], lead + g);
      const float p0 = __shfl_sync(0xffffffffu, p[0], lead + g), p1 = __shfl_sync(0xffffffffu, p[PER - 1], PER == 2 ? lead + g : lead + GP + g);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[g][e] = o[g][e] * cg + p0 * f[0][e] + p1 * f[1][e];
    }
  };
#pragma unroll 1
  for (int t = 0; t < trips; t += 2) {
    work(A);
    if (t + 2 < trips) fetch(A, t + 2, true, true);
    if (t + 1 < trips) {
      work(B2);
      if (t + 3 < trips) fetch(B2, t + 3, true, true);
    }
  }
  float lt = l[0];
  if constexpr (PER == 2) lt += l[PER - 1];
  else lt += __shfl_xor_sync(0xffffffffu, lt, GP);
  // every group of lanes of every warp leaves its result, and the CTA adds them in their order
  const int part = warp * SPW + grp;
  if (sub < G) { sm_m[part][sub] = m[0]; sm_l[part][sub] = lt; }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float4* dst = reinterpret_cast<float4*>(&sm_o[part][g][sub * 8]);
    dst[0] = make_float4(o[g][0], o[g][1], o[g][2], o[g][3]);
    dst[1] = make_float4(o[g][4], o[g][5], o[g][6], o[g][7]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < PARTS * G; i += 128) {
    const int w0 = i / G, g = i - w0 * G;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < PARTS; ++w) mm = fmaxf(mm, sm_m[w][g]);
    sm_f[w0][g] = sm_m[w0][g] == -INFINITY ? 0.f : __expf(sm_m[w0][g] - mm);
    if (w0 == 0) sm_m[PARTS][g] = mm;
  }
  __syncthreads();
  if (threadIdx.x < G) {
    float ll = 0.f;
#pragma unroll
    for (int w = 0; w < PARTS; ++w) ll += sm_l[w][threadIdx.x] * sm_f[w][threadIdx.x];
    sm_l[PARTS][threadIdx.x] = ll;
  }
  for (int t = threadIdx.x; t < G * HD; t += 128) {
    const int g = t / HD, c = t % HD;
    float oo = 0.f;
#pragma unroll
    for (int w = 0; w < PARTS; ++w) oo += sm_o[w][g][c] * sm_f[w][g];
    sm_o[PARTS][g][c] = oo;
  }
  cluster_sync_all();
  auto remote = [](const float* p, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(mapa_shared(smem_u32(p), (uint32_t)rank)) : "memory");
    return v;
  };
  for (int t = split * 128 + (int)threadIdx.x; t < G * HD; t += splits * 128) {      // the splits, in their order
    const int g = t / HD, c = t % HD;
    float ms[8], ls[8], os[8], mm = -INFINITY;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      ms[r] = -INFINITY;
      ls[r] = os[r] = 0.f;
      if (r < splits) { ms[r] = remote(&sm_m[PARTS][g], r); ls[r] = remote(&sm_l[PARTS][g], r); os[r] = remote(&sm_o[PARTS][g][c], r); }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) mm = fmaxf(mm, ms[r]);
    float ll = 0.f, oo = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float f = ms[r] == -INFINITY ? 0.f : __expf(ms[r] - mm);
      ll += ls[r] * f;
      oo += os[r] * f;
    }
    out[b * ld_o + (long long)(kvh * G + g) * HD + c] = Cvt<T>::from_f(ll > 0.f ? oo / ll : 0.f);
  }
  cluster_sync_all();                                  // the other CTAs have read this one's shared memory
}

// One block of HD threads per (sequence, head).  The split maxima and sums are read by one thread per split and the
// per-split factors go through shared memory, so that the long loop over the splits carries no dependent load: the
// earlier form (every thread walking all splits twice, each step waiting for its load) took 12 us per launch, a
// fifth of a token step, for a few kilobytes.
template <typename T, int HD>
__global__ void decode_attn_merge_kernel(const float* __restrict__ scratch, int splits, T* __restrict__ out, long long ld_o, int H) {
  __shared__ float s_f[128];
  __shared__ float s_red[4];
  pdl_wait();
  const int b = blockIdx.x / H, h = blockIdx.x % H, c = threadIdx.x;
  const float* base = scratch + ((long long)b * H + h) * splits * (HD + 2);
  // maximum over the splits (splits <= 128: up to two per thread)
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  if (c < splits) { m0 = base[c * (HD + 2)]; l0 = base[c * (HD + 2) + 1]; }
  if (c + HD < splits) { m1 = base[(c + HD) * (HD + 2)]; l1 = base[(c + HD) * (HD + 2) + 1]; }
  float mm = warp_max(fmaxf(m0, m1));
  if ((c & 31) == 0) s_red[c >> 5] = mm;
  __syncthreads();
  mm = s_red[0];
  for (int w = 1; w < HD / 32; ++w) mm = fmaxf(mm, s_red[w]);
  const float f0 = m0 == -INFINITY ? 0.f : __expf(m0 - mm), f1 = m1 == -INFINITY ? 0.f : __expf(m1 - mm);
  if (c < splits) s_f[c] = f0;
  if (c + HD < splits) s_f[c + HD] = f1;
  __syncthreads();                       // also orders the reads of s_red above against the writes below
  float ll = warp_sum(l0 * f0 + l1 * f1);
  if ((c & 31) == 0) s_red[c >> 5] = ll;
  __syncthreads();
  ll = 0.f;
  for (int w = 0; w < HD / 32; ++w) ll += s_red[w];
  float oo = 0.f;
#pragma unroll 8
  for (int s = 0; s < splits; ++s) oo += base[s * (HD + 2) + 2 + c] * s_f[s];
  out[b * ld_o + (long long)h * HD + c] = Cvt<T>::from_f(ll > 0.f ? oo / ll : 0.f);
}

// ---------------------------------------------------------------------------------------------- fused decode step
// Fewer, fatter kernels for the token step: at batch 1 every kernel costs a few microseconds however little it does.
//   gemv_norm:            RMSNorm of the fp32 residual inside the GEMV (every block normalises the row it needs)
//   route_norm:           RMSNorm + router (soft-max, bias-steered top-k), one block per token
//   swiglu_norm:          RMSNorm + gate/up rows of the selected experts
//   qk_rope_append:       QK-norm + RoPE; k heads land in the cache slot, v heads are copied beside them
//   decode_attn (ticket): the last split to finish merges the partial results; measured slower than the separate
//                         merge launch (the merge is a serial tail of the longest block), so the engine does not use it
// Rounding points are those of the separate kernels (normalised activations pass through 16 bits), so both routes
// give the same numbers.

// Row b of x (fp32, d values) normalised into xs (16-bit) by one warp, as rmsnorm_fwd_kernel does it.
template <typename XT>
__device__ __forceinline__ void norm_row_to_smem(const float* __restrict__ x, const float* __restrict__ w, XT* __restrict__ xs,
                                                 int d, float eps) {
  const int lane = threadIdx.x & 31;
  const float4* xr = reinterpret_cast<const float4*>(x);
  float ss = 0.f;
  for (int i = lane; i < d / 4; i += 32) {
    const float4 v = xr[i];
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  ss = warp_sum(ss);
  float inv = rsqrtf(ss / (float)d + eps);
  if (!isfinite(inv)) inv = 0.f;
  const float4* wr = reinterpret_cast<const float4*>(w);
  for (int i = lane; i < d / 4; i += 32) {
    const float4 v = xr[i], g = wr[i];
    uint2 o;
    o.x = Cvt<XT>::pack2(v.x * inv * g.x, v.y * inv * g.y);
    o.y = Cvt<XT>::pack2(v.z * inv * g.z, v.w * inv * g.w);
    *reinterpret_cast<uint2*>(xs + 4 * i) = o;
  }
}

template <int FMT, int NB, int KS, typename XT>
__global__ void __launch_bounds__(GV_THREADS) gemv_norm_kernel(const uint8_t* __restrict__ W, long long row_bytes, int N, int K,
                                                              const float* __restrict__ x32, long long ldx32,
                                                              const float* __restrict__ norm_w, float eps, int B,
                                                              void* __restrict__ out, long long ldo, int out_f32) {
  pdl_wait();
  extern __shared__ __align__(16) uint8_t gv_dyn[];
  XT* xs = reinterpret_cast<XT*>(gv_dyn);                 // [B][K]
  __shared__ float sm[GV_WARPS];
  const int warp = threadIdx.x >> 5, ric = warp / KS, ks = warp % KS;
  for (int b = warp; b < B; b += GV_WARPS) norm_row_to_smem<XT>(x32 + b * ldx32, norm_w, xs + (long long)b * K, K, eps);
  __syncthreads();
  const int row = blockIdx.x * (GV_WARPS / KS) + ric;
  const bool live = row < N;
  const uint8_t* wrow = W + (size_t)(live ? row : 0) * row_bytes;
  for (int b0 = 0; b0 < B; b0 += NB) {
    float acc[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) acc[j] = 0.f;
    const int nb = min(NB, B - b0);
    if (live) row_partial<FMT, NB, KS, XT>(wrow, K, xs + (long long)b0 * K, K, nb, ks, acc);
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const float v0 = row_finish<KS>(acc[j], sm, ric, ks);
      if (live && j < nb && ks == 0 && (threadIdx.x & 31) == 0) {
        if (out_f32) reinterpret_cast<float*>(out)[(long long)(b0 + j) * ldo + row] = v0;
        else reinterpret_cast<XT*>(out)[(long long)(b0 + j) * ldo + row] = Cvt<XT>::from_f(v0);
      }
    }
  }
}

// Router of one token from its normalised activations in shared memory (rules of decode_route_kernel).  All threads
// of the block call it; the selection is left in esel / wsel (shared).
template <typename XT>
__device__ __forceinline__ void route_in_block(const XT* __restrict__ xs, const float* __restrict__ rw, const float* __restrict__ bias,
                                               int d, int ne, int top_k, float* __restrict__ lg, int* __restrict__ esel,
                                               float* __restrict__ wsel) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = warp; e < ne; e += GV_WARPS) {
    const float* wr = rw + (size_t)e * d;
    float s = 0.f;
    for (int i = lane * 2; i < d; i += 64) {
      const float2 xv = Cvt<XT>::unpack2(*reinterpret_cast<const uint32_t*>(xs + i));
      const float2 wv = *reinterpret_cast<const float2*>(wr + i);
      s += xv.x * wv.x + xv.y * wv.y;
    }
    s = warp_sum(s);
    if (lane == 0) lg[e] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mx = -INFINITY;
    for (int e = 0; e < ne; ++e) mx = fmaxf(mx, lg[e]);
    float sum = 0.f;
    for (int e = 0; e < ne; ++e) { lg[e] = __expf(lg[e] - mx); sum += lg[e]; }
    const float inv = 1.f / sum;
    unsigned long long taken = 0ull;
    float psel[8], psum = 0.f;
    for (int k = 0; k < top_k; ++k) {
      float bv = -INFINITY;
      int bi = 0;
      for (int e = 0; e < ne; ++e) {
        if (taken >> e & 1ull) continue;
        const float sc = lg[e] * inv + (bias ? bias[e] : 0.f);
        if (sc > bv) { bv = sc; bi = e; }
      }
      taken |= 1ull << bi;
      esel[k] = bi;
      psel[k] = lg[bi] * inv;
      psum += psel[k];
    }
    const float invs = psum > 1e-8f ? 1.f / psum : 0.f;
    for (int k = 0; k < top_k; ++k) wsel[k] = psel[k] * invs;
  }
  __syncthreads();
}

// Router of a token on its own: RMSNorm of the fp32 row + soft-max + bias-steered top-k; one block per token.  (Doing
// this inside every gate/up block was measured: thousands of blocks re-reading the router weights cost more than
// the launch it saved.)
template <typename XT>
__global__ void __launch_bounds__(GV_THREADS) route_norm_kernel(const float* __restrict__ x32, const float* __restrict__ norm_w,
                                                               float eps, const float* __restrict__ rw,
                                                               const float* __restrict__ bias, int d, int ne, int top_k,
                                                               int* __restrict__ idx_out, float* __restrict__ w_out) {
  pdl_wait();
  extern __shared__ __align__(16) uint8_t gv_dyn[];
  XT* xs = reinterpret_cast<XT*>(gv_dyn);
  __shared__ float lg[64];
  __shared__ int esel[8];
  __shared__ float wsel[8];
  const int b = blockIdx.x;
  if ((threadIdx.x >> 5) == 0) norm_row_to_smem<XT>(x32 + (long long)b * d, norm_w, xs, d, eps);
  __syncthreads();
  route_in_block<XT>(xs, rw, bias, d, ne, top_k, lg, esel, wsel);
  if (threadIdx.x < top_k) {
    idx_out[b * top_k + threadIdx.x] = esel[threadIdx.x];
    w_out[b * top_k + threadIdx.x] = wsel[threadIdx.x];
  }
}

// RMSNorm and router of a batch's tokens, one block per token: the 16-bit normed row, and the token's weight for every expert (zero where it
// is not chosen; 1 for the shared expert, the last).  ne == 0: the norm alone.  The norm's and the router's weights are asked for before the wait for
// the kernel ahead.  Up to 1024 columns and 8 experts everything stays in registers; more of either takes the loops behind.
// Bound by its chain of round trips: 32 tokens of width 768, 8 experts 3.2 us (norm, router, scan and sorted copy were 21).
template <typename XT>
__global__ void __launch_bounds__(GV_THREADS) norm_route_few_kernel(const float* __restrict__ x32, const float* __restrict__ norm_w, float eps,
                                                                    const float* __restrict__ rw, const float* __restrict__ bias, int d, int ne,
                                                                    int top_k, int shared, XT* __restrict__ x16, float* __restrict__ weights) {
  extern __shared__ __align__(16) uint8_t gv_dyn[];
  XT* xs = reinterpret_cast<XT*>(gv_dyn);                 // [d]
  __shared__ float lg[64], red[GV_WARPS];
  const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n4 = d / 4;
  constexpr int NR = 8;                                   // 16-byte loads of a router row per lane that are kept
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 r[NR], g = tid < n4 ? reinterpret_cast<const float4*>(norm_w)[tid] : zero;
#pragma unroll
  for (int k = 0; k < NR; ++k)
    r[k] = warp < ne && lane + 32 * k < n4 ? reinterpret_cast<const float4*>(rw + (size_t)warp * d)[lane + 32 * k] : zero;
  pdl_wait();
  const float4* xr = reinterpret_cast<const float4*>(x32 + (long long)b * d);
  const float4 x = tid < n4 ? xr[tid] : zero;
  float ss = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
  for (int i = tid + GV_THREADS; i < n4; i += GV_THREADS) { const float4 v = xr[i]; ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; }
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < GV_WARPS; ++i) tot += red[i];
  float inv = rsqrtf(tot / (float)d + eps);
  if (!isfinite(inv)) inv = 0.f;
  uint2* out = reinterpret_cast<uint2*>(x16 + (long long)b * d);
  auto put = [&](int i, const float4& v, const float4& w) {
    const uint2 q = make_uint2(Cvt<XT>::pack2(v.x * inv * w.x, v.y * inv * w.y), Cvt<XT>::pack2(v.z * inv * w.z, v.w * inv * w.w));
    reinterpret_cast<uint2*>(xs)[i] = q;
    out[i] = q;
  };
  if (tid < n4) put(tid, x, g);
  for (int i = tid + GV_THREADS; i < n4; i += GV_THREADS) put(i, xr[i], reinterpret_cast<const float4*>(norm_w)[i]);
  if (ne == 0) return;
  __syncthreads();
  for (int e = warp; e < ne; e += GV_WARPS) {
    const float4* wr = reinterpret_cast<const float4*>(rw + (size_t)e * d);
    float s = 0.f;
    auto dot = [&](int i, const float4& w) {
      const uint2 q = reinterpret_cast<const uint2*>(xs)[i];
      const float2 u = Cvt<XT>::unpack2(q.x), v = Cvt<XT>::unpack2(q.y);
      s += u.x * w.x + u.y * w.y + v.x * w.z + v.y * w.w;
    };
#pragma unroll
    for (int k = 0; k < NR; ++k)
      if (lane + 32 * k < n4) dot(lane + 32 * k, e == warp ? r[k] : wr[lane + 32 * k]);
    for (int i = lane + 32 * NR; i < n4; i += 32) dot(i, wr[i]);
    s = warp_sum(s);
    if (lane == 0) lg[e] = s;
  }
  __syncthreads();
  if (warp == 0) {
    int my_e;
    float my_w;
    warp_route(lane < ne ? lg[lane] : -INFINITY, lane + 32 < ne ? lg[lane + 32] : -INFINITY, bias, ne, top_k, my_e, my_w);
    float w0 = 0.f, w1 = 0.f;
    for (int k = 0; k < top_k; ++k) {
      const int e = __shfl_sync(0xffffffffu, my_e, k);
      const float w = __shfl_sync(0xffffffffu, my_w, k);
      if (e == lane) w0 = w;
      if (e == lane + 32) w1 = w;
    }
    float* dst = weights + (long long)b * (ne + (shared ? 1 : 0));
    if (lane < ne) dst[lane] = w0;
    if (lane + 32 < ne) dst[lane + 32] = w1;
    if (shared && lane == 0) dst[ne] = 1.f;
  }
}

// grid (ceil(E / rows per block), B * slots).  idx == nullptr: dense feed-forward (one "expert" 0).
template <int FMT, int KS, typename XT>
__global__ void __launch_bounds__(GV_THREADS) swiglu_norm_kernel(
    const uint8_t* __restrict__ Wg, const uint8_t* __restrict__ Wu, long long row_bytes, int ne, int E, int d,
    const float* __restrict__ x32, const float* __restrict__ norm_w, float eps, const int* __restrict__ idx, int top_k,
    int slots, XT* __restrict__ act) {
  pdl_wait();
  extern __shared__ __align__(16) uint8_t gv_dyn[];
  XT* xs = reinterpret_cast<XT*>(gv_dyn);                 // [d]
  __shared__ float sm[2 * GV_WARPS];
  const int warp = threadIdx.x >> 5, ric = warp / KS, ks = warp % KS;
  const int b = blockIdx.y / slots, slot = blockIdx.y % slots;
  if (warp == 0) norm_row_to_smem<XT>(x32 + (long long)b * d, norm_w, xs, d, eps);
  __syncthreads();
  const int e = idx ? (slot < top_k ? idx[b * top_k + slot] : ne) : 0;
  const int j = blockIdx.x * (GV_WARPS / KS) + ric;
  const bool live = j < E && e >= 0 && e <= ne;
  float g[1] = {0.f}, u[1] = {0.f};
  if (live) {
    const size_t r = (size_t)e * E + j;
    row_partial<FMT, 1, KS, XT>(Wg + r * row_bytes, d, xs, d, 1, ks, g);
    row_partial<FMT, 1, KS, XT>(Wu + r * row_bytes, d, xs, d, 1, ks, u);
  }
  const float gs = row_finish<KS>(g[0], sm, ric, ks);
  const float us = row_finish<KS>(u[0], sm + GV_WARPS, ric, ks);
  if (live && ks == 0 && (threadIdx.x & 31) == 0)
    act[((long long)b * slots + slot) * E + j] = Cvt<XT>::from_f(gs / (1.f + __expf(-gs)) * us);
}

// One warp per (sequence, head) over the q, k and v heads of the fused projection.  q heads: norm + rotation into
// `q_out`.  k heads: norm + rotation straight into the cache slot of the step.  v heads: copied into the cache.
template <typename T, int HD>
__global__ void qk_rope_append_kernel(const T* __restrict__ qkv, long long ld_in, T* __restrict__ q_out, long long ld_q,
                                      const float* __restrict__ qw, const float* __restrict__ kw, const float* __restrict__ cs,
                                      const int* __restrict__ pos, T* __restrict__ cK, T* __restrict__ cV,
                                      int* __restrict__ slot_pos, const gb_seq_state* __restrict__ st, int B, int H, int KV,
                                      int cap, int pinned, float eps, int rope_type) {
  pdl_wait();
  constexpr int PAIRS = HD / 2;
  constexpr int PPL = (PAIRS + 31) / 32;
  const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int heads = H + 2 * KV;
  if (gw >= B * heads) return;
  const int b = gw / heads, h = gw - b * heads;
  const gb_seq_state s = st[b];
  const int slot = s.cache_len < cap ? s.cache_len : pinned + s.ring_start;
  const long long kvd = (long long)KV * HD;
  const T* src = qkv + b * ld_in + (long long)h * HD;
  if (h >= H + KV) {                                         // v head: plain copy into the cache
    T* dv = cV + ((long long)b * cap + slot) * kvd + (long long)(h - H - KV) * HD;
    for (int i = lane * 2; i < HD; i += 64) *reinterpret_cast<uint32_t*>(dv + i) = *reinterpret_cast<const uint32_t*>(src + i);
    return;
  }
  T* dst = h < H ? q_out + b * ld_q + (long long)h * HD : cK + ((long long)b * cap + slot) * kvd + (long long)(h - H) * HD;
  if (h == H && lane == 0) slot_pos[(long long)b * cap + slot] = s.abs_pos;
  const float* w = (h < H) ? qw : kw;
  float a[PPL], c2[PPL];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < PPL; ++k) {
    const int p = lane + 32 * k;
    if (p < PAIRS) {
      const int i0 = rope_type == 0 ? 2 * p : p, i1 = rope_type == 0 ? 2 * p + 1 : p + PAIRS;
      a[k] = Cvt<T>::to_f(src[i0]);
      c2[k] = Cvt<T>::to_f(src[i1]);
      ss += a[k] * a[k] + c2[k] * c2[k];
    }
  }
  float inv = 1.f;
  if (w) {
    ss = warp_sum(ss);
    inv = rsqrtf(ss / (float)HD + eps);
    if (!isfinite(inv)) inv = 0.f;
  }
  const float* csr = cs + (size_t)pos[b] * HD;
#pragma unroll
  for (int k = 0; k < PPL; ++k) {
    const int p = lane + 32 * k;
    if (p < PAIRS) {
      const int i0 = rope_type == 0 ? 2 * p : p, i1 = rope_type == 0 ? 2 * p + 1 : p + PAIRS;
      float x0 = a[k], x1 = c2[k];
      if (w) { x0 *= inv * w[i0]; x1 *= inv * w[i1]; }
      const float c = csr[p], sn = csr[PAIRS + p];
      dst[i0] = Cvt<T>::from_f(x0 * c - x1 * sn);
      dst[i1] = Cvt<T>::from_f(x0 * sn + x1 * c);
    }
  }
}

}  // namespace gb

using namespace gb;

extern "C" long long gb_wfmt_row_bytes(int fmt, int K) {
  switch (fmt) {
    case GB_W_F16: case GB_W_BF16: return K % 8 ? -1 : 2LL * K;
    case GB_W_GGML_Q8_0: return K % 32 ? -1 : (K / 32) * 34LL;
    case GB_W_Q4_0: return K % 32 ? -1 : (K / 32) * 18LL;
    case GB_W_Q8_64: return K % 64 ? -1 : (K / 64) * 68LL;
    case GB_W_Q4_1: return K % 32 ? -1 : (K / 32) * 20LL;
  }
  return -1;
}

#define GB_FMT_SWITCH(fmt, CALL)                          \
  switch (fmt) {                                          \
    case GB_W_F16: { CALL(GB_W_F16); break; }             \
    case GB_W_BF16: { CALL(GB_W_BF16); break; }           \
    case GB_W_GGML_Q8_0: { CALL(GB_W_GGML_Q8_0); break; } \
    case GB_W_Q4_0: { CALL(GB_W_Q4_0); break; }           \
    case GB_W_Q8_64: { CALL(GB_W_Q8_64); break; }         \
    case GB_W_Q4_1: { CALL(GB_W_Q4_1); break; }           \
    default: return -1;                                   \
  }

extern "C" int gb_gemv(const void* W, int fmt, int N, int K, const void* x16, int ldx, int B, void* out, int ldo, int out_f32,
                       const float* addend, int ld_add, int is_bf16, cudaStream_t st) {
  const long long rb = gb_wfmt_row_bytes(fmt, K);
  if (!W || !x16 || !out || N <= 0 || B <= 0 || B > 32 || rb < 0 || (ldx % 8)) return -1;
  const bool split = N <= 8192;   // few rows: spread each over four warps (latency bound); many rows fill the GPU anyway
  const uint8_t* w = static_cast<const uint8_t*>(W);
#define GEMV_GO(F, NB, KS, XT)                                                                                     \
  GB_PDL_LAUNCH((gemv_kernel<F, NB, KS, XT>), dim3((N + GV_WARPS / KS - 1) / (GV_WARPS / KS)), dim3(GV_THREADS), st, \
                w, rb, N, K, (const XT*)x16, (long long)ldx, B, out, (long long)ldo, out_f32, addend, (long long)ld_add)
#define CALL(F)                                                                        \
  if (is_bf16) {                                                                       \
    if (B == 1 && split) GEMV_GO(F, 1, 4, __nv_bfloat16);                              \
    else if (B == 1) GEMV_GO(F, 1, 1, __nv_bfloat16);                                  \
    else GEMV_GO(F, 4, 1, __nv_bfloat16);                                              \
  } else {                                                                             \
    if (B == 1 && split) GEMV_GO(F, 1, 4, __half);                                     \
    else if (B == 1) GEMV_GO(F, 1, 1, __half);                                         \
    else GEMV_GO(F, 4, 1, __half);                                                     \
  }
  GB_FMT_SWITCH(fmt, CALL)
#undef CALL
#undef GEMV_GO
  return gb_launch_rc();
}

extern "C" int gb_gemv_expert_swiglu(const void* Wg, const void* Wu, int fmt, int ne, int E, int d, const void* x16, int B,
                                     const int* idx, int top_k, int shared, void* act16, int is_bf16, cudaStream_t st) {
  const long long rb = gb_wfmt_row_bytes(fmt, d);
  if (!Wg || !Wu || !x16 || !idx || !act16 || rb < 0 || B <= 0 || top_k <= 0) return -1;
  const int slots = top_k + (shared ? 1 : 0);
  const uint8_t *g = static_cast<const uint8_t*>(Wg), *u = static_cast<const uint8_t*>(Wu);
  const bool split = B * slots <= 64;
#define SW_GO(F, KS, XT)                                                                                              \
  GB_PDL_LAUNCH((expert_swiglu_kernel<F, KS, XT>), dim3((E + GV_WARPS / KS - 1) / (GV_WARPS / KS), B * slots),       \
                dim3(GV_THREADS), st, g, u, rb, ne, E, d, (const XT*)x16, idx, top_k, slots, (XT*)act16)
#define CALL(F)                                                                                   \
  if (is_bf16) { if (split) SW_GO(F, 4, __nv_bfloat16); else SW_GO(F, 1, __nv_bfloat16); }        \
  else { if (split) SW_GO(F, 4, __half); else SW_GO(F, 1, __half); }
  GB_FMT_SWITCH(fmt, CALL)
#undef CALL
  return gb_launch_rc();
}

extern "C" int gb_gemv_expert_down(const void* Wd, int fmt, int ne, int d, int E, const void* act16, int B, const int* idx,
                                   const float* w, int top_k, int shared, const float* resid, float* out, int is_bf16,
                                   cudaStream_t st) {
  const long long rb = gb_wfmt_row_bytes(fmt, E);
  if (!Wd || !act16 || !idx || !w || !resid || !out || rb < 0 || B <= 0 || top_k <= 0) return -1;
  const int slots = top_k + (shared ? 1 : 0);
  const uint8_t* wd = static_cast<const uint8_t*>(Wd);
  const bool split = B <= 16;
#define DN_GO(F, KS, XT)                                                                                    \
  GB_PDL_LAUNCH((expert_down_kernel<F, KS, XT>), dim3((d + GV_WARPS / KS - 1) / (GV_WARPS / KS), B), dim3(GV_THREADS), st, \
                wd, rb, ne, d, E, (const XT*)act16, idx, w, top_k, slots, resid, out)
#define CALL(F)                                                                                   \
  if (is_bf16) { if (split) DN_GO(F, 4, __nv_bfloat16); else DN_GO(F, 1, __nv_bfloat16); }        \
  else { if (split) DN_GO(F, 4, __half); else DN_GO(F, 1, __half); }
  GB_FMT_SWITCH(fmt, CALL)
#undef CALL
  return gb_launch_rc();
}

extern "C" int gb_decode_route(const void* x16, const float* router_w, const float* bias, int B, int d, int ne, int top_k,
                               int* idx, float* w, int is_bf16, cudaStream_t st) {
  if (!x16 || !router_w || !idx || !w || B <= 0 || ne <= 0 || ne > 64 || top_k <= 0 || top_k > 8 || top_k > ne || d % 2) return -1;
  if (is_bf16) GB_PDL_LAUNCH(decode_route_kernel<__nv_bfloat16>, dim3(B), dim3(256), st, (const __nv_bfloat16*)x16, router_w, bias, d, ne, top_k, idx, w);
  else GB_PDL_LAUNCH(decode_route_kernel<__half>, dim3(B), dim3(256), st, (const __half*)x16, router_w, bias, d, ne, top_k, idx, w);
  return gb_launch_rc();
}

extern "C" int gb_kv_append(const void* k16, long long ld_k, const void* v16, long long ld_v, void* cacheK, void* cacheV,
                            int* slot_pos, const gb_seq_state* state, int B, int cap, int pinned, int kv_dim, cudaStream_t st) {
  if (!k16 || !v16 || !cacheK || !cacheV || !slot_pos || !state || B <= 0 || cap <= pinned || kv_dim % 8 || ld_k % 8 || ld_v % 8)
    return -1;
  // 16-bit elements of either type are copied as raw bits
  GB_PDL_LAUNCH(kv_append_kernel<__half>, dim3(B), dim3(128), st, (const __half*)k16, ld_k, (const __half*)v16, ld_v, (__half*)cacheK,
                                              (__half*)cacheV, slot_pos, state, cap, pinned, kv_dim);
  return gb_launch_rc();
}

extern "C" int gb_kv_rows(const void* k, long long ld_k, const void* v, long long ld_v, void* cK, void* cV, int* slot_pos, const int* n,
                          int B, int T, int cap, int kv_dim, cudaStream_t st) {
  if (!k || !v || !cK || !cV || !slot_pos || !n || B <= 0 || T <= 0 || cap < T || kv_dim <= 0 || kv_dim % 8 || ld_k % 8 || ld_v % 8 ||
      ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(cK) | reinterpret_cast<uintptr_t>(cV)) & 15))
    return -1;
  const int rows = B * T;                       // copied as they are: one instantiation serves both 16-bit types
  kv_rows_kernel<__half><<<(rows + 7) / 8, 256, 0, st>>>((const __half*)k, ld_k, (const __half*)v, ld_v, (__half*)cK, (__half*)cV, slot_pos, n,
                                                         rows, T, cap, kv_dim);
  return gb_launch_rc();
}

extern "C" int gb_decode_advance(gb_seq_state* state, int* pos_out, int B, int cap, int pinned, cudaStream_t st) {
  if (!state || !pos_out || B <= 0) return -1;
  GB_PDL_LAUNCH(decode_advance_kernel, dim3((B + 63) / 64), dim3(64), st, state, pos_out, B, cap, pinned);
  return gb_launch_rc();
}

template <typename T, int HD>
static int launch_decode_attn(const void* q, long long ld_q, const void* cK, const void* cV, const int* slot_pos,
                              const gb_seq_state* state, void* out, long long ld_o, float* scratch, int splits, int B, int H,
                              int KV, int cap, int window, float scale, int early, int* ticket, cudaStream_t st) {
  const int G = H / KV;
  if (!ticket && splits > 2 * HD) return -4;      // the merge kernel reads at most two splits per thread
  // a cluster: no more than eight CTAs anywhere, and a slot's lanes hold its scores (heads of 32: up to four queries a key head).  Eight splits only
  // while all CTAs fit at once (four to an SM, two with more than four queries a key head): beyond that the plain kernel and its merge are faster (48 sequences,
  // 8 heads of 64 without groups, 4000 slots 65 us, the cluster 82; 96 sequences, 12/4 heads, 2000 slots 61 and 69)
  if (!ticket && splits <= 8 && (splits & (splits - 1)) == 0 && G <= HD / 8 && (splits < 8 || (long long)B * KV * splits <= (G <= 4 ? 592 : 296))) {
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = gb_pdl_config(dim3((unsigned)(B * KV * splits)), dim3(128), 0, st, &at[1]);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs += 1;
#define ATT(GG)                                                                                                                              \
  if constexpr (GG <= HD / 8)                                                                                                               \
    (void)cudaLaunchKernelEx(&cfg, decode_attn_cluster_kernel<T, HD, GG>, (const T*)q, ld_q, (const T*)cK, (const T*)cV, slot_pos, state, splits, \
                             H, KV, cap, window, scale, early, (T*)out, ld_o)
    switch (G) {
      case 1: ATT(1); break;
      case 2: ATT(2); break;
      case 3: ATT(3); break;
      case 4: ATT(4); break;
      case 6: ATT(6); break;
      case 8: ATT(8); break;
      default: return -3;
    }
#undef ATT
    return gb_launch_rc();
  }
  const dim3 grid(B * KV, splits);
#define ATT(GG)                                                                                                   \
  GB_PDL_LAUNCH((decode_attn_kernel<T, HD, GG>), grid, dim3(128), st, (const T*)q, ld_q, (const T*)cK, (const T*)cV, slot_pos, \
                state, scratch, splits, H, KV, cap, window, scale, ticket, (T*)out, ld_o)
  switch (G) {
    case 1: ATT(1); break;
    case 2: ATT(2); break;
    case 3: ATT(3); break;
    case 4: ATT(4); break;
    case 6: ATT(6); break;
    case 8: ATT(8); break;
    default: return -3;
  }
#undef ATT
  if (!ticket) GB_PDL_LAUNCH((decode_attn_merge_kernel<T, HD>), dim3(B * H), dim3(HD), st, (const float*)scratch, splits, (T*)out, ld_o, H);
  return gb_launch_rc();
}

static int decode_attn_any(const void* q16, long long ld_q, const void* cacheK, const void* cacheV, const int* slot_pos,
                           const gb_seq_state* state, void* out16, long long ld_o, float* scratch, int splits, int B, int H,
                           int KV, int hd, int cap, int window, float scale, int is_bf16, int early, int* ticket, cudaStream_t st) {
  if (!q16 || !cacheK || !cacheV || !slot_pos || !state || !out16 || !scratch || splits < 1 || B <= 0 || KV <= 0 || H % KV)
    return -1;
#define GO(T, HD) return launch_decode_attn<T, HD>(q16, ld_q, cacheK, cacheV, slot_pos, state, out16, ld_o, scratch, splits, B, H, KV, cap, window, scale, early, ticket, st)
  if (hd == 64) { if (is_bf16) GO(__nv_bfloat16, 64); else GO(__half, 64); }
  if (hd == 128) { if (is_bf16) GO(__nv_bfloat16, 128); else GO(__half, 128); }
  if (hd == 32) { if (is_bf16) GO(__nv_bfloat16, 32); else GO(__half, 32); }
#undef GO
  return -2;
}

extern "C" int gb_decode_attn(const void* q16, long long ld_q, const void* cacheK, const void* cacheV, const int* slot_pos,
                              const gb_seq_state* state, void* out16, long long ld_o, float* scratch, int splits, int B, int H,
                              int KV, int hd, int cap, int window, float scale, int is_bf16, int early, cudaStream_t st) {
  return decode_attn_any(q16, ld_q, cacheK, cacheV, slot_pos, state, out16, ld_o, scratch, splits, B, H, KV, hd, cap, window,
                         scale, is_bf16, early, nullptr, st);
}

// The same with the merge of the splits done by the last block to finish; `ticket` is B*KV ints, zero before the first call.
extern "C" int gb_decode_attn_fused(const void* q16, long long ld_q, const void* cacheK, const void* cacheV, const int* slot_pos,
                                    const gb_seq_state* state, void* out16, long long ld_o, float* scratch, int splits, int B,
                                    int H, int KV, int hd, int cap, int window, float scale, int is_bf16, int* ticket,
                                    cudaStream_t st) {
  if (!ticket) return -1;
  return decode_attn_any(q16, ld_q, cacheK, cacheV, slot_pos, state, out16, ld_o, scratch, splits, B, H, KV, hd, cap, window,
                         scale, is_bf16, 0, ticket, st);
}

// RMSNorm of x32 [B, K] (fp32) fused into out = W @ norm(x32).  Shared memory holds the normalised rows: B*K*2 bytes.
extern "C" int gb_gemv_norm(const void* W, int fmt, int N, int K, const float* x32, int ldx32, const float* norm_w, float eps,
                            int B, void* out, int ldo, int out_f32, int is_bf16, cudaStream_t st) {
  const long long rb = gb_wfmt_row_bytes(fmt, K);
  if (!W || !x32 || !norm_w || !out || N <= 0 || B <= 0 || B > 32 || rb < 0 || (K % 8) || (ldx32 % 4)) return -1;
  const size_t smem = (size_t)B * K * 2;
  if (smem > 40 * 1024) return -2;                          // the caller takes the two-kernel route
  const bool split = N <= 8192;
  const uint8_t* w = static_cast<const uint8_t*>(W);
#define GEMVN_GO(F, NB, KS, XT)                                                                                      \
  do {                                                                                                               \
    cudaLaunchAttribute gb_attr_;                                                                                    \
    cudaLaunchConfig_t gb_cfg_ = gb_pdl_config(dim3((N + GV_WARPS / KS - 1) / (GV_WARPS / KS)), dim3(GV_THREADS), smem, st, &gb_attr_); \
    (void)cudaLaunchKernelEx(&gb_cfg_, (gemv_norm_kernel<F, NB, KS, XT>), w, rb, N, K, x32, (long long)ldx32, norm_w, eps, B, \
                             out, (long long)ldo, out_f32);                                                          \
  } while (0)
#define CALL(F)                                                                         \
  if (is_bf16) {                                                                        \
    if (B == 1 && split) GEMVN_GO(F, 1, 4, __nv_bfloat16);                              \
    else if (B == 1) GEMVN_GO(F, 1, 1, __nv_bfloat16);                                  \
    else GEMVN_GO(F, 4, 1, __nv_bfloat16);                                              \
  } else {                                                                              \
    if (B == 1 && split) GEMVN_GO(F, 1, 4, __half);                                     \
    else if (B == 1) GEMVN_GO(F, 1, 1, __half);                                         \
    else GEMVN_GO(F, 4, 1, __half);                                                     \
  }
  GB_FMT_SWITCH(fmt, CALL)
#undef CALL
#undef GEMVN_GO
  return gb_launch_rc();
}

// RMSNorm + router of x32 [B, d]: idx_out / w_out [B, top_k].
extern "C" int gb_route_norm(const float* x32, const float* norm_w, float eps, const float* router_w, const float* bias, int B,
                             int d, int ne, int top_k, int* idx_out, float* w_out, int is_bf16, cudaStream_t st) {
  if (!x32 || !norm_w || !router_w || !idx_out || !w_out || B <= 0 || ne <= 0 || ne > 64 || top_k <= 0 || top_k > 8 ||
      top_k > ne || (d % 8))
    return -1;
  const size_t smem = (size_t)d * 2;
  if (smem > 40 * 1024) return -2;
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = gb_pdl_config(dim3(B), dim3(GV_THREADS), smem, st, &attr);
  if (is_bf16) (void)cudaLaunchKernelEx(&cfg, route_norm_kernel<__nv_bfloat16>, x32, norm_w, eps, router_w, bias, d, ne, top_k, idx_out, w_out);
  else (void)cudaLaunchKernelEx(&cfg, route_norm_kernel<__half>, x32, norm_w, eps, router_w, bias, d, ne, top_k, idx_out, w_out);
  return gb_launch_rc();
}

// RMSNorm of x32 [B, d] into x16 [B, d], and the weight of every token for every expert: weights [B, ne (+ 1 shared)] fp32 (ne == 0: the norm alone).  norm_w, router_w
// and bias are not what the launch ahead writes.
extern "C" int gb_norm_route_few(const float* x32, const float* norm_w, float eps, const float* router_w, const float* bias, int B, int d,
                                 int ne, int top_k, int shared, void* x16, float* weights, int is_bf16, cudaStream_t st) {
  if (!x32 || !norm_w || !x16 || B <= 0 || d <= 0 || d % 8) return -1;
  if (ne != 0 && (!router_w || !weights || ne < 0 || ne > 64 || top_k <= 0 || top_k > 8 || top_k > ne)) return -1;
  if ((reinterpret_cast<uintptr_t>(x32) | reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(router_w) | reinterpret_cast<uintptr_t>(x16)) & 15)
    return -1;
  const size_t smem = (size_t)d * 2;
  if (smem > 40 * 1024) return -2;
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = gb_pdl_config(dim3(B), dim3(GV_THREADS), smem, st, &attr);
  if (is_bf16) (void)cudaLaunchKernelEx(&cfg, norm_route_few_kernel<__nv_bfloat16>, x32, norm_w, eps, router_w, bias, d, ne, top_k, shared, (__nv_bfloat16*)x16, weights);
  else (void)cudaLaunchKernelEx(&cfg, norm_route_few_kernel<__half>, x32, norm_w, eps, router_w, bias, d, ne, top_k, shared, (__half*)x16, weights);
  return gb_launch_rc();
}

// RMSNorm + gate/up of the experts named by idx [B, top_k] (+ the shared one).  idx == nullptr: dense feed-forward.
extern "C" int gb_swiglu_norm(const void* Wg, const void* Wu, int fmt, int ne, int E, int d, const float* x32, const float* norm_w,
                              float eps, const int* idx, int B, int top_k, int shared, void* act16, int is_bf16,
                              cudaStream_t st) {
  const long long rb = gb_wfmt_row_bytes(fmt, d);
  if (!Wg || !Wu || !x32 || !norm_w || !act16 || rb < 0 || B <= 0 || top_k <= 0 || top_k > 8 || (d % 8)) return -1;
  const size_t smem = (size_t)d * 2;
  if (smem > 40 * 1024) return -2;
  const int slots = top_k + (shared ? 1 : 0);
  const uint8_t *g = static_cast<const uint8_t*>(Wg), *u = static_cast<const uint8_t*>(Wu);
  const bool split = B * slots <= 64;
#define SWN_GO(F, KS, XT)                                                                                            \
  do {                                                                                                               \
    cudaLaunchAttribute gb_attr_;                                                                                    \
    cudaLaunchConfig_t gb_cfg_ = gb_pdl_config(dim3((E + GV_WARPS / KS - 1) / (GV_WARPS / KS), B * slots), dim3(GV_THREADS), smem, st, &gb_attr_); \
    (void)cudaLaunchKernelEx(&gb_cfg_, (swiglu_norm_kernel<F, KS, XT>), g, u, rb, ne, E, d, x32, norm_w, eps, idx, top_k, slots, \
                             (XT*)act16);                                                                            \
  } while (0)
#define CALL(F)                                                                                     \
  if (is_bf16) { if (split) SWN_GO(F, 4, __nv_bfloat16); else SWN_GO(F, 1, __nv_bfloat16); }        \
  else { if (split) SWN_GO(F, 4, __half); else SWN_GO(F, 1, __half); }
  GB_FMT_SWITCH(fmt, CALL)
#undef CALL
#undef SWN_GO
  return gb_launch_rc();
}

extern "C" int gb_qk_rope_append(const void* qkv, long long ld_in, void* q_out, long long ld_q, const float* qw, const float* kw,
                                 const float* cos_sin, const int* pos, void* cacheK, void* cacheV, int* slot_pos,
                                 const gb_seq_state* state, int B, int H, int KV, int hd, int cap, int pinned, float eps,
                                 int rope_type, int is_bf16, cudaStream_t st) {
  if (!qkv || !q_out || !cos_sin || !pos || !cacheK || !cacheV || !slot_pos || !state || B <= 0 || H <= 0 || KV <= 0 ||
      cap <= pinned || (hd % 2) || (ld_in % 2))
    return -1;
  const int items = B * (H + 2 * KV);
  const int wpb = 8;
  const dim3 grid((items + wpb - 1) / wpb);
#define QKA(T, HD)                                                                                                       \
  GB_PDL_LAUNCH((qk_rope_append_kernel<T, HD>), grid, dim3(wpb * 32), st, (const T*)qkv, ld_in, (T*)q_out, ld_q, qw, kw, cos_sin, \
                pos, (T*)cacheK, (T*)cacheV, slot_pos, state, B, H, KV, cap, pinned, eps, rope_type)
  if (is_bf16) {
    switch (hd) { case 32: QKA(__nv_bfloat16, 32); break; case 64: QKA(__nv_bfloat16, 64); break; case 128: QKA(__nv_bfloat16, 128); break; default: return -2; }
  } else {
    switch (hd) { case 32: QKA(__half, 32); break; case 64: QKA(__half, 64); break; case 128: QKA(__half, 128); break; default: return -2; }
  }
#undef QKA
  return gb_launch_rc();
}
