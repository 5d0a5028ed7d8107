// GEMM of few rows for sm_100a: C[M, N] = A[M, K] * W[N, K]^T with M <= 128 (a batch of token steps, a short prompt).  Such a
// product is a stream of weights with one tile of rows, and in the persistent kernel (gemm_sm100.cu) a chain: 32 x 3840 by
// 1024 x 3840 has sixteen 64-column tiles, so sixteen SMs walk sixty k-blocks each while the others idle.  Here a cluster of S
// CTAs shares a 128 x 64 tile: each takes K / S of the reduction, keeps its part of the sum in its tensor memory and writes 1 / S of it
// into the shared memory of each of the others with a bulk copy; every CTA then adds and stores its share of the tile, the parts in the order of K.
// Row by row, in pieces of four columns, the same writes took 1 us; fetched from the others when all were there, another round trip and a second wait
// for the cluster so that nobody leaves early, 1 to 1.8 us more than now (from the last product to the last store 1.3 us).
// A CTA's own part of its share stays where it is.  us, the persistent kernel -> this one with early weights (floor by bytes at 6.5 TB/s): 32 x 3840 x 1024 16.7 -> 5.0
// (1.2), 32 x 1024 x 2816 7.5 -> 5.3 (0.9), 8 x 6912 x 2560 26.9 -> 10.3 (5.5), 128 x 6912 x 2560 28.9 -> 13.4.  With its own part copied, too, and
// four columns a thread whatever the rows: 128 x 2816 x 1024 7.4 instead of 6.2, 128 x 2560 x 6912 18.0 instead of 16.7.  What is left is launch, the round trips of the first loads and the exchange.
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
#include <atomic>

#include "sm100_common.cuh"
#include "gb_api.h"

namespace gb {
namespace sk {

static constexpr int BN = 64, BK = 64, STAGES = 8, THREADS = 192;   // warps 0-3 accumulators, 4 TMA, 5 MMA
static constexpr int W_TMA = 4, W_MMA = 5;
static constexpr uint32_t W_BYTES = BN * BK * 2;

struct Params {
  int M, N, K, fmt, split, lg;  // split: CTAs of a cluster, 2 to the power lg
  int stages;                   // at most STAGES
  int a_rows;                   // rows of A per stage
  int w_early, relu2;
  void* out; int ldo;
  const float* addend; int ld_add;
  int* status;
  int k_group, w_group;         // K is cut into groups of k_group k-blocks (0: one), each with its own w_group rows of W
  const float* scale; int ld_scale, scale_cols;    // SwiGLU: factor of (row, column / scale_cols)
  int n1; void* out2; int ldo2;                    // relu2: columns below n1 as they are into out, the others into out2
};

// Q: fours of columns that a thread takes at a time.  One while rows are few, so that all threads have some; two beyond 32 rows, in half as many turns with
// stores of 16 bytes.
template <typename OutT, bool SWIGLU, int Q>
__global__ void __launch_bounds__(THREADS) gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                                                              const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], done_bar, parts_bar;
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
  // Parts of this CTA's share of the tile: [source][row][BN / split columns and four more, so that lanes hit all banks].  They lie behind the stages, where
  // the MMAs read rows that nothing uses.
  const int width = BN >> p.lg, pitch = width + 4, share = p.M * pitch;
  float* parts = reinterpret_cast<float*>(smem + (uint32_t)p.stages * stage_bytes);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    mbar_init(&parts_bar, 1);
    abort_word = 0;
    fence_barrier_init();
    if (p.split > 1) mbar_arrive_expect_tx(&parts_bar, (uint32_t)((p.split - 1) * share) * 4);
  }
  if (warp == W_MMA) { tmem_alloc(&tmem_slot, BN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");       // waited for before the first write to another CTA
  // units of Q fours of columns; what a thread's first two are added to or scaled by is asked for before the sums are there
  constexpr int LG_ROW = (SWIGLU ? 3 : 4) - (Q - 1);
  const int per_row = 1 << (LG_ROW - p.lg), units = p.M * per_row;
  auto column = [&](int u) { return n0 + rank * (COLS >> p.lg) + (u & (per_row - 1)) * (4 * Q); };
  struct Add { float4 v[Q]; float scale; };
  auto add_of = [&](int u) {
    Add a;
    const int row = u >> (LG_ROW - p.lg), col = column(u);
    const bool in = u < units && col < p.N;
#pragma unroll
    for (int q = 0; q < Q; ++q)
      a.v[q] = p.addend && in ? reinterpret_cast<const float4*>(p.addend + (long long)row * p.ld_add + col)[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    a.scale = SWIGLU && p.scale && in ? p.scale[(long long)row * p.ld_scale + col / p.scale_cols] : 1.f;
    return a;
  };
  Add add0, add1;
  auto ahead = [&]() {
    add0 = add_of(threadIdx.x);
    add1 = add_of(threadIdx.x + THREADS);
  };

  if (warp == W_TMA) {
    const uint32_t on = elect_one();
    if (on) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    auto load_w = [&](int i, int slot) {
      uint8_t* dst = smem + (uint32_t)slot * stage_bytes + a_bytes;
      mbar_arrive_expect_tx_on(on, &full_bar[slot], stage_bytes);              // both operands' bytes
      if constexpr (SWIGLU) {        // stored in blocks of 64 gate rows and 64 up rows
        const int row = (n0 >> 6) * 128 + (n0 & 63);
        tma_load_2d_on(on, &tmW, &full_bar[slot], dst, (kb0 + i) * BK, row);
        tma_load_2d_on(on, &tmW, &full_bar[slot], dst + W_BYTES / 2, (kb0 + i) * BK, row + 64);
      } else {
        const int kb = kb0 + i, g = p.k_group ? kb / p.k_group : 0;
        tma_load_2d_on(on, &tmW, &full_bar[slot], dst, (kb - g * p.k_group) * BK, g * p.w_group + n0);
      }
    };
    const int early = p.w_early ? min(nkb, p.stages) : 0;
    for (int i = 0; i < early; ++i) load_w(i, i);
    pdl_wait();
    for (int i = 0, slot = 0, round = 0; i < nkb; ++i) {
      if (round > 0) wait_or_leave(&empty_bar[slot], (round & 1) ^ 1, p.status, ST_TIMEOUT_EMPTY, abort_flag);
      if (i >= early) load_w(i, slot);
      tma_load_2d_on(on, &tmA, &full_bar[slot], smem + (uint32_t)slot * stage_bytes, (kb0 + i) * BK, 0);
      if (++slot == p.stages) { slot = 0; ++round; }
    }
    __syncwarp();
    ahead();
  } else if (warp == W_MMA) {
    const uint32_t on = elect_one();
    const uint32_t idesc = make_idesc_f16(p.fmt, 0, 0, 128, BN);
    for (int i = 0, slot = 0, round = 0; i < nkb; ++i) {
      wait_or_report(&full_bar[slot], round & 1, p.status, ST_TIMEOUT_FULL, abort_flag);
      tc_fence_after();
      const uint32_t sa = smem_u32(smem) + (uint32_t)slot * stage_bytes;
      const uint64_t da = make_smem_desc_sw128(sa, 16, 1024), dw = make_smem_desc_sw128(sa + a_bytes, 16, 1024);
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) umma_f16_on(on, tmem, da + kk * 2, dw + kk * 2, idesc, i > 0 || kk > 0 ? 1u : 0u);
      umma_commit_on(on, &empty_bar[slot]);
      if (++slot == p.stages) { slot = 0; ++round; }
    }
    umma_commit_on(on, &done_bar);
    __syncwarp();
    pdl_wait();
    ahead();
  } else {
    pdl_wait();
    ahead();
    wait_or_report(&done_bar, 0, p.status, ST_TIMEOUT_TMEM_FULL, abort_flag);
    tc_fence_after();
    // every product is taken: the stages hold this CTA's part of the tile now, a share behind the other (SwiGLU: gate and up columns in one)
    const int row = warp * 32 + lane;
    if (warp * 32 < p.M) {
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tmem + ((uint32_t)(warp * 32) << 16) + c * 32, r);
        tmem_ld_wait();
        if (row < p.M) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int cg = c * 4 + k, own = SWIGLU ? k << p.lg >> 2 : cg << p.lg >> 3;
            const int at = SWIGLU ? c * (width >> 1) + ((k * 8) & ((width >> 1) - 1)) : (cg * 8) & (width - 1);
            uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<float*>(smem) + own * share + row * pitch + at);
            dst[0] = make_uint4(r[8 * k], r[8 * k + 1], r[8 * k + 2], r[8 * k + 3]);
            dst[1] = make_uint4(r[8 * k + 4], r[8 * k + 5], r[8 * k + 6], r[8 * k + 7]);
          }
        }
      }
    }
    tc_fence_before();
    fence_proxy_async();                               // read by the copies below
  }
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);    // copies still in flight get time to land
    __syncthreads();
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");          // the others have begun, their barriers are set up
  const float* mine = reinterpret_cast<const float*>(smem) + rank * share;      // this CTA's part of its own share stays where it is
  if (p.split > 1) {
    if (threadIdx.x == 0)
      for (int r = 1; r < p.split; ++r) {
        const uint32_t own = (uint32_t)((rank + r) & (p.split - 1));
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         mapa_shared(smem_u32(parts) + (uint32_t)(rank * share) * 4, own)),
                     "r"(smem_u32(smem) + own * (uint32_t)share * 4), "r"((uint32_t)share * 4), "r"(mapa_shared(smem_u32(&parts_bar), own))
                     : "memory");
      }
    wait_or_report(&parts_bar, 0, p.status, ST_TIMEOUT_AUX, abort_flag);
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // all copies into this CTA have landed
  }
  for (int u = (int)threadIdx.x; u < units; u += THREADS) {
    const int row = u >> (LG_ROW - p.lg), col = column(u);
    if (col >= p.N) continue;                          // N is a multiple of 8
    const int turn = u / THREADS, at = row * pitch + (u & (per_row - 1)) * (4 * Q);
    const Add add = turn == 0 ? add0 : turn == 1 ? add1 : add_of(u);
    auto total = [&](int from, float (&v)[4 * Q]) {
#pragma unroll
      for (int k = 0; k < 4 * Q; ++k) v[k] = 0.f;
#pragma unroll 4
      for (int g = 0; g < p.split; ++g) {
        const float4* src = reinterpret_cast<const float4*>((g == rank ? mine : parts + g * share) + from);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const float4 x = src[q];
          v[4 * q] += x.x; v[4 * q + 1] += x.y; v[4 * q + 2] += x.z; v[4 * q + 3] += x.w;
        }
      }
    };
    float v[4 * Q];
    total(at, v);
    if constexpr (SWIGLU) {
      float up[4 * Q];
      total(at + (width >> 1), up);
#pragma unroll
      for (int k = 0; k < 4 * Q; ++k) v[k] = add.scale == 0.f ? 0.f : v[k] / (1.f + __expf(-v[k])) * up[k] * add.scale;   // not chosen: zero, whatever the product is
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) { v[4 * q] += add.v[q].x; v[4 * q + 1] += add.v[q].y; v[4 * q + 2] += add.v[q].z; v[4 * q + 3] += add.v[q].w; }
    OutT* dst = reinterpret_cast<OutT*>(p.out) + (long long)row * p.ldo + col;
    if (p.relu2 && col >= p.n1) {
#pragma unroll
      for (int k = 0; k < 4 * Q; ++k) { v[k] = fmaxf(v[k], 0.f); v[k] *= v[k]; }
      if (p.out2) dst = reinterpret_cast<OutT*>(p.out2) + (long long)row * p.ldo2 + col - p.n1;
    }
    if constexpr (sizeof(OutT) == 4) {
#pragma unroll
      for (int q = 0; q < Q; ++q) reinterpret_cast<float4*>(dst)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else if constexpr (Q == 2) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(Cvt<OutT>::pack2(v[0], v[1]), Cvt<OutT>::pack2(v[2], v[3]), Cvt<OutT>::pack2(v[4], v[5]), Cvt<OutT>::pack2(v[6], v[7]));
    } else {
      *reinterpret_cast<uint2*>(dst) = make_uint2(Cvt<OutT>::pack2(v[0], v[1]), Cvt<OutT>::pack2(v[2], v[3]));
    }
  }
  if (warp == W_MMA) { tc_fence_after(); tmem_dealloc(tmem, BN); }
  __syncwarp();
  if (p.split > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");       // and all copies out of it
  if (*abort_flag)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);    // copies of a CTA whose waits ran out may still be on their way
}

}  // namespace sk
}  // namespace gb

namespace {

constexpr size_t MOST_SMEM = 226 * 1024, TWO_SMEM = 111 * 1024;       // of one CTA an SM, and of two (3 KB of each are static or the system's)

// Shared memory of a launch: stages, and behind them the larger of the parts (in the stages where a CTA has the whole reduction) and of the rows that the
// MMAs read past the last stage.
size_t skinny_smem(const gb::sk::Params& p) {
  namespace sk = gb::sk;
  const size_t parts = p.split > 1 ? (size_t)p.M * (sk::BN + 4 * p.split) * 4 : 0, tail = (size_t)(128 - p.a_rows) * 128;
  return (size_t)p.stages * (p.a_rows * 128 + sk::W_BYTES) + (parts > tail ? parts : tail) + 1024;
}

template <typename OutT, bool SWIGLU>
cudaLaunchConfig_t skinny_config(const gb::sk::Params& p, cudaStream_t st, cudaLaunchAttribute* at) {
  namespace sk = gb::sk;
  constexpr int COLS = SWIGLU ? sk::BN / 2 : sk::BN;
  cudaLaunchConfig_t cfg = gb_pdl_config(dim3((unsigned)((p.N + COLS - 1) / COLS * p.split)), dim3(sk::THREADS), skinny_smem(p), st, &at[1]);
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.split; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs += 1;
  return cfg;
}

template <typename OutT, bool SWIGLU, int Q>
int launch_skinny_q(const CUtensorMap& ta, const CUtensorMap& tw, gb::sk::Params p, cudaStream_t st) {
  namespace sk = gb::sk;
  auto kern = sk::gemm_skinny_kernel<OutT, SWIGLU, Q>;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST_SMEM) != cudaSuccess) { (void)cudaGetLastError(); return -10; }
    (void)cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    attr = true;
  }
  // CTAs of a tile: as many as leave all tiles resident at once (32 x 4352 x 1024, four CTAs a tile, had a few late clusters, 10.2 us; with two it has none, 6.0).
  // The driver is asked how many clusters fit with an SM for every CTA; up to 32 rows two CTAs share one, which its query does not see: counted as one they had
  // half as many CTAs, 8 x 2560 x 6912 15.0 us and 11.4, 8 x 6912 x 2560 12.0 and 10.3.  More CTAs than SMs pay for themselves from ten k-blocks a CTA
  // on (8 x 9472 x 768, six: 5.1 us with 148 CTAs, 6.2 with 296).  Fewer than two k-blocks per CTA do not pay for the exchange.
  constexpr int COLS = SWIGLU ? sk::BN / 2 : sk::BN, MOST = SWIGLU ? 4 : 8;
  const int tiles = (p.N + COLS - 1) / COLS, blocks = (p.K + sk::BK - 1) / sk::BK;
  static std::atomic<int> fits[4];                    // clusters of 2, 4, 8 CTAs that fit an SM each, plus one
  cudaLaunchAttribute at[2];
  p.split = 1;
  for (int lg = 1; (1 << lg) <= MOST && blocks >= (1 << lg) * 2; ++lg) {
    sk::Params q = p;
    q.split = 1 << lg;
    q.lg = lg;
    for (q.stages = sk::STAGES; skinny_smem(q) > MOST_SMEM;) --q.stages;
    int n = fits[lg].load(std::memory_order_relaxed);
    if (!n) {
      cudaLaunchConfig_t cfg = skinny_config<OutT, SWIGLU>(q, st, at);
      cfg.dynamicSmemBytes = MOST_SMEM;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
      fits[lg].store(++n, std::memory_order_relaxed);
    }
    const int an_sm = skinny_smem(q) <= TWO_SMEM && ((tiles << lg) <= 148 || blocks >> lg >= 10) ? 2 : 1;
    if (tiles > (n - 1) * an_sm) break;
    p.split = q.split;
    p.lg = lg;
  }
  for (p.stages = sk::STAGES; skinny_smem(p) > MOST_SMEM;) --p.stages;
  const cudaLaunchConfig_t cfg = skinny_config<OutT, SWIGLU>(p, st, at);
  if (cudaLaunchKernelEx(&cfg, kern, ta, tw, p) != cudaSuccess) return -10;
  return gb_launch_rc();
}

template <typename OutT, bool SWIGLU = false>
int launch_skinny(const CUtensorMap& ta, const CUtensorMap& tw, const gb::sk::Params& p, cudaStream_t st) {
  return p.M > 32 ? launch_skinny_q<OutT, SWIGLU, 2>(ta, tw, p, st) : launch_skinny_q<OutT, SWIGLU, 1>(ta, tw, p, st);
}

}  // namespace

// gb_gemm with args->skinny: M <= 128, mode 0, K contiguous in both operands, N a multiple of 8, 16-byte aligned rows of out and addend.
// k_group > 0: K runs over groups of k_group values, group g against rows g * b_group_rows + (0 .. N - 1) of B.
// epilogue 4 with n1: columns below n1 into out as they are, the others, squared where positive, into aux_out from its column 0.
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
  if (a->n1) {
    if (a->epilogue != 4 || a->n1 < 0 || a->n1 % 8 || a->n1 > a->N || !a->aux_out || (reinterpret_cast<uintptr_t>(a->aux_out) & 15) || ((long long)a->ld_aux * es) % 16)
      return -1;
    p.n1 = a->n1; p.out2 = a->aux_out; p.ldo2 = a->ld_aux;
  }
  CUtensorMap ta, tw;
  int rc = gb_make_tmap_2d_16b(&ta, a->A, a->a_rows, a->a_cols, a->lda, p.a_rows, sk::BK, a->is_bf16);
  if (rc) return rc - 100;
  rc = gb_make_tmap_2d_16b(&tw, a->B, a->b_rows, a->b_cols, a->ldb, swiglu ? sk::BN / 2 : sk::BN, sk::BK, a->is_bf16);
  if (rc) return rc - 200;
  if (a->out_dtype == 2) return launch_skinny<float>(ta, tw, p, st);
  if (a->out_dtype == 1) return swiglu ? launch_skinny<__nv_bfloat16, true>(ta, tw, p, st) : launch_skinny<__nv_bfloat16>(ta, tw, p, st);
  return swiglu ? launch_skinny<__half, true>(ta, tw, p, st) : launch_skinny<__half>(ta, tw, p, st);
}
