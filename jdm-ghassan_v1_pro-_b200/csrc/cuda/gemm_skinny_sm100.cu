// GEMM of few rows for sm_100a: C[M, N] = A[M, K] * W[N, K]^T with M <= 128 (a batch of token steps, a short prompt).  Such a
// product is a stream of weights with one tile of rows, and in the persistent kernel (gemm_sm100.cu) a chain: 32 x 3840 by
// 1024 x 3840 has sixteen 64-column tiles, so sixteen SMs walk sixty k-blocks each while the others idle.  Here a cluster of S
// CTAs shares a 128 x 64 tile: each takes K / S of the reduction, keeps its part of the sum in its tensor memory, writes it to
// its shared memory, and every CTA adds and stores 1 / S of the tile, the parts in the order of K.
// us, the persistent kernel -> this one with early weights (floor by bytes at 6.5 TB/s): 32 x 3840 x 1024 16.7 -> 7.7 (1.2), 32 x 1024 x
// 2816 7.5 -> 6.0 (0.9), 32 x 768 x 1280 6.6 -> 4.5 (0.3), 8 x 6912 x 2560 26.9 -> 11.2 (5.5), 128 x 6912 x 2560 28.9 -> 14.3; 100 x 2816
// x 1024 14.2 -> 7.0 (15.0 with clusters of eight).  What is left is launch, the round trips of the first loads and the exchange.
//
// The kernel is launched with programmatic dependency: barriers, tensor memory and, where the caller says that W is not what
// the kernel before writes (weights), the first eight k-blocks of W are under way before griddepcontrol.wait.
//
// Shared memory of a stage holds only the rows of A that exist (a multiple of eight): the MMA reads 128 rows from there on, and
// what it reads behind them lands in accumulator rows that nothing stores.  Rows are independent, so that may be anything.
//
// Experts of few tokens.  A few dozen tokens visit nearly every expert, whose weights are then read once whatever the rows are: so all
// tokens go through all experts, without sorting them by expert.  Gate and up rows of 32 columns share a tile, whose
// epilogue makes silu(g) * u * (the token's weight for the expert, zero where the router has not chosen it); the down projection is
// one product whose K runs over all experts, each with a row block of its own in W.
// 32 tokens, 9 experts of 768, width 768 (32 MB of weights, 4.9 us at the copy rate): gate and up 7.3 us, down 8.7; sorted by expert 12.6, 9.1, and 14 for
// sorting and adding up.
#include "sm100_common.cuh"
#include "gb_api.h"

namespace gb {
namespace sk {

static constexpr int BN = 64, BK = 64, STAGES = 8, THREADS = 192;   // warps 0-3 accumulators, 4 TMA, 5 MMA
static constexpr int W_TMA = 4, W_MMA = 5;
static constexpr uint32_t W_BYTES = BN * BK * 2;
static constexpr int PITCH = BN + 4;                                // floats of a row of the partial sums: lanes hit all banks

struct Params {
  int M, N, K, fmt, split;      // split: CTAs of a cluster
  int a_rows;                   // rows of A per stage
  int w_early, relu2;
  void* out; int ldo;
  const float* addend; int ld_add;
  int* status;
  int k_group, w_group;         // K is cut into groups of k_group k-blocks (0: one), each with its own w_group rows of W
  const float* scale; int ld_scale, scale_cols;    // SwiGLU: factor of (row, column / scale_cols)
};

template <typename OutT, bool SWIGLU>
__global__ void __launch_bounds__(THREADS) gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                                                              const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int COLS = SWIGLU ? BN / 2 : BN;                        // columns of the result in a tile
  const int rank = (int)cluster_ctarank(), n0 = (int)cluster_id_x() * COLS;
  const uint32_t a_bytes = (uint32_t)p.a_rows * (BK * 2), stage_bytes = a_bytes + W_BYTES;
  const int blocks = (p.K + BK - 1) / BK;
  const int kb0 = rank * blocks / p.split, nkb = (rank + 1) * blocks / p.split - kb0;      // at least one: split <= blocks

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    abort_word = 0;
    fence_barrier_init();
  }
  if (warp == W_MMA) { tmem_alloc(&tmem_slot, BN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == W_TMA) {
    const uint32_t on = elect_one();
    auto stage = [&](int i) { return smem + (uint32_t)(i % STAGES) * stage_bytes; };
    auto load_w = [&](int i) {
      mbar_arrive_expect_tx_on(on, &full_bar[i % STAGES], stage_bytes);        // both operands' bytes
      if constexpr (SWIGLU) {        // stored in blocks of 64 gate rows and 64 up rows
        const int row = (n0 >> 6) * 128 + (n0 & 63);
        tma_load_2d_on(on, &tmW, &full_bar[i % STAGES], stage(i) + a_bytes, (kb0 + i) * BK, row);
        tma_load_2d_on(on, &tmW, &full_bar[i % STAGES], stage(i) + a_bytes + W_BYTES / 2, (kb0 + i) * BK, row + 64);
      } else {
        const int kb = kb0 + i, g = p.k_group ? kb / p.k_group : 0;
        tma_load_2d_on(on, &tmW, &full_bar[i % STAGES], stage(i) + a_bytes, (kb - g * p.k_group) * BK, g * p.w_group + n0);
      }
    };
    const int early = p.w_early ? min(nkb, STAGES) : 0;
    for (int i = 0; i < early; ++i) load_w(i);
    pdl_wait();
    for (int i = 0; i < nkb; ++i) {
      if (i >= STAGES) wait_or_leave(&empty_bar[i % STAGES], ((i / STAGES) & 1) ^ 1, p.status, ST_TIMEOUT_EMPTY, abort_flag);
      if (i >= early) load_w(i);
      tma_load_2d_on(on, &tmA, &full_bar[i % STAGES], stage(i), (kb0 + i) * BK, 0);
    }
    __syncwarp();
  } else if (warp == W_MMA) {
    const uint32_t on = elect_one();
    const uint32_t idesc = make_idesc_f16(p.fmt, 0, 0, 128, BN);
    for (int i = 0; i < nkb; ++i) {
      wait_or_report(&full_bar[i % STAGES], (i / STAGES) & 1, p.status, ST_TIMEOUT_FULL, abort_flag);
      tc_fence_after();
      const uint32_t sa = smem_u32(smem) + (uint32_t)(i % STAGES) * stage_bytes;
      const uint64_t da = make_smem_desc_sw128(sa, 16, 1024), dw = make_smem_desc_sw128(sa + a_bytes, 16, 1024);
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) umma_f16_on(on, tmem, da + kk * 2, dw + kk * 2, idesc, i > 0 || kk > 0 ? 1u : 0u);
      umma_commit_on(on, &empty_bar[i % STAGES]);
    }
    umma_commit_on(on, &done_bar);
    __syncwarp();
    pdl_wait();
  } else {
    pdl_wait();
    wait_or_report(&done_bar, 0, p.status, ST_TIMEOUT_TMEM_FULL, abort_flag);
    tc_fence_after();
    // every product is taken: the stages hold the partial sums now
    const int row = warp * 32 + lane;
    if (warp * 32 < p.M) {
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tmem + ((uint32_t)(warp * 32) << 16) + c * 32, r);
        tmem_ld_wait();
        if (row < p.M) {
          float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(smem) + row * PITCH + c * 32);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            dst[k] = make_float4(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]), __uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]));
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);    // copies still in flight get time to land
    __syncthreads();
  }
  cluster_sync_all();
  const int units = p.M * (COLS / 8), u0 = rank * units / p.split, u1 = (rank + 1) * units / p.split;
  for (int u = u0 + (int)threadIdx.x; u < u1; u += THREADS) {
    const int row = u / (COLS / 8), c = (u - row * (COLS / 8)) * 8, col = n0 + c;
    if (col >= p.N) continue;                          // N is a multiple of 8
    const uint32_t at = smem_u32(smem) + (uint32_t)(row * PITCH + c) * 4;
    float4 add[2];
    float scale = 1.f;
    if (p.addend) {
      const float4* src = reinterpret_cast<const float4*>(p.addend + (long long)row * p.ld_add + col);
      add[0] = src[0];
      add[1] = src[1];
    }
    if (SWIGLU && p.scale) scale = p.scale[(long long)row * p.ld_scale + col / p.scale_cols];
    auto total = [&](uint32_t from, float (&v)[8]) {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = 0.f;
#pragma unroll 4
      for (int g = 0; g < p.split; ++g) {
        const uint32_t src = mapa_shared(from, (uint32_t)g);
        float4 x, y;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(src) : "memory");
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w) : "r"(src + 16) : "memory");
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
      }
    };
    float v[8];
    total(at, v);
    if constexpr (SWIGLU) {
      float up[8];
      total(at + (BN / 2) * 4, up);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = scale == 0.f ? 0.f : v[k] / (1.f + __expf(-v[k])) * up[k] * scale;   // not chosen: zero, whatever the product is
    }
    if (p.addend) {
      v[0] += add[0].x; v[1] += add[0].y; v[2] += add[0].z; v[3] += add[0].w;
      v[4] += add[1].x; v[5] += add[1].y; v[6] += add[1].z; v[7] += add[1].w;
    }
    if (p.relu2) {
#pragma unroll
      for (int k = 0; k < 8; ++k) { v[k] = fmaxf(v[k], 0.f); v[k] *= v[k]; }
    }
    OutT* dst = reinterpret_cast<OutT*>(p.out) + (long long)row * p.ldo + col;
    if constexpr (sizeof(OutT) == 4) {
      reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
      uint4 q;
      q.x = Cvt<OutT>::pack2(v[0], v[1]);
      q.y = Cvt<OutT>::pack2(v[2], v[3]);
      q.z = Cvt<OutT>::pack2(v[4], v[5]);
      q.w = Cvt<OutT>::pack2(v[6], v[7]);
      *reinterpret_cast<uint4*>(dst) = q;
    }
  }
  cluster_sync_all();                                  // the other CTAs have read this one's shared memory
  if (warp == W_MMA) { tc_fence_after(); tmem_dealloc(tmem, BN); }
}

}  // namespace sk
}  // namespace gb

namespace {

template <typename OutT, bool SWIGLU = false>
int launch_skinny(const CUtensorMap& ta, const CUtensorMap& tw, const gb::sk::Params& p, cudaStream_t st) {
  namespace sk = gb::sk;
  auto kern = sk::gemm_skinny_kernel<OutT, SWIGLU>;
  // behind the last stage the MMA still reads up to 128 rows; the partial sums are smaller than eight stages
  const size_t smem = (size_t)sk::STAGES * (p.a_rows * 128 + sk::W_BYTES) + (128 - p.a_rows) * 128 + 1024;
  static_assert((size_t)sk::STAGES * (8 * 128 + sk::W_BYTES) >= 128 * sk::PITCH * 4, "partial sums fit the stages");
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, sk::STAGES * (128 * 128 + (int)sk::W_BYTES) + 1024) != cudaSuccess) return -10;
    attr = true;
  }
  constexpr int COLS = SWIGLU ? sk::BN / 2 : sk::BN;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = gb_pdl_config(dim3((unsigned)((p.N + COLS - 1) / COLS * p.split)), dim3(sk::THREADS), smem, st, &at[1]);
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.split; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs += 1;
  if (cudaLaunchKernelEx(&cfg, kern, ta, tw, p) != cudaSuccess) return -10;
  return gb_launch_rc();
}

}  // namespace

// gb_gemm with args->skinny: M <= 128, mode 0, K contiguous in both operands, N a multiple of 8, 16-byte aligned rows of out and addend.
// k_group > 0: K runs over groups of k_group values, group g against rows g * b_group_rows + (0 .. N - 1) of B.
// epilogue 1: SwiGLU over 2 N interleaved rows of B, column j times scale[row, j / scale_cols] where scale is given; 16-bit out.
extern "C" int gb_gemm_skinny(const gb_gemm_args* a, cudaStream_t st) {
  namespace sk = gb::sk;
  if (!a || a->M <= 0 || a->M > 128 || a->N <= 0 || a->N % 8 || a->K <= 0 || a->mode != 0 || a->a_mn_major || a->b_mn_major || !a->status) return -1;
  const bool swiglu = a->epilogue == 1;
  if (a->epilogue != 0 && a->epilogue != 4 && !swiglu) return -1;
  if (swiglu && (a->N % 64 || a->out_dtype == 2 || a->addend || a->k_group || (a->scale && (a->scale_cols <= 0 || a->scale_cols % 64)))) return -1;
  if (a->k_group < 0 || (a->k_group > 0 && (a->k_group % sk::BK || a->K % a->k_group || a->b_group_rows < a->N))) return -1;
  const int es = a->out_dtype == 2 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(a->out) & 15) || ((long long)a->ldo * es) % 16) return -1;
  if (a->addend && ((reinterpret_cast<uintptr_t>(a->addend) & 15) || a->ld_add % 4)) return -1;
  sk::Params p{};
  p.M = a->M; p.N = a->N; p.K = a->K; p.fmt = a->is_bf16;
  p.a_rows = (a->M + 7) / 8 * 8;
  p.w_early = a->b_static; p.relu2 = a->epilogue == 4;
  p.out = a->out; p.ldo = a->ldo; p.addend = a->addend; p.ld_add = a->ld_add; p.status = a->status;
  p.k_group = a->k_group / sk::BK; p.w_group = a->b_group_rows;
  p.scale = a->scale; p.ld_scale = a->ld_scale; p.scale_cols = a->scale_cols;
  // As many CTAs as the SMs hold at once: two per SM while their stages are small.  Fewer than two k-blocks per CTA do not
  // pay for the exchange.
  const int cols = swiglu ? sk::BN / 2 : sk::BN;
  const int tiles = (a->N + cols - 1) / cols, blocks = (a->K + sk::BK - 1) / sk::BK;
  const bool two = p.a_rows <= 32;
  const int room = 148 * (two ? 2 : 1), most = two ? 8 : 4;      // eight CTAs that need an SM each do not fit a GPC twice
  p.split = 1;
  while (p.split < most && tiles * p.split * 2 <= room && blocks >= p.split * 4) p.split *= 2;
  CUtensorMap ta, tw;
  int rc = gb_make_tmap_2d_16b(&ta, a->A, a->a_rows, a->a_cols, a->lda, p.a_rows, sk::BK, a->is_bf16);
  if (rc) return rc - 100;
  rc = gb_make_tmap_2d_16b(&tw, a->B, a->b_rows, a->b_cols, a->ldb, swiglu ? sk::BN / 2 : sk::BN, sk::BK, a->is_bf16);
  if (rc) return rc - 200;
  if (a->out_dtype == 2) return launch_skinny<float>(ta, tw, p, st);
  if (a->out_dtype == 1) return swiglu ? launch_skinny<__nv_bfloat16, true>(ta, tw, p, st) : launch_skinny<__nv_bfloat16>(ta, tw, p, st);
  return swiglu ? launch_skinny<__half, true>(ta, tw, p, st) : launch_skinny<__half>(ta, tw, p, st);
}
