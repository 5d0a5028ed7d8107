// The whole token step of one sequence as ONE cooperative kernel: embedding row, every layer (RMSNorm + fused QKV
// projection, QK-norm + RoPE + cache append + split-KV attention, merge + output projection + residual, RMSNorm +
// router + gate/up + SwiGLU of the selected experts, down projection + residual), final norm and the vocabulary
// projection.  One CTA of 16 warps per SM.  The reference's decode loop (inference/generator.cpp:97-193,
// cuda/kernels.cu:876-1019) launches about fifteen kernels per layer.
//
// Exchange between CTAs.  A layer is a chain of six small vectors (x, q/k/v, partial attention, attention, x after attention,
// activations), each made by all CTAs and read by all or some of them.  Every number travels in one word together with the
// epoch of its layer (fp32 values: 64 bits, value and epoch; 16-bit values: 32 bits), written and read with single relaxed
// accesses, so no fence stands between a value and the news of it.  Readers look once a count of arrivals, bumped behind the
// stores without any ordering, says that the words are about to be there: polling the words themselves is right too, but a line that
// 148 SMs poll while sixteen CTAs write to it moves back and forth between the halves of L2.  768 fp32 values from all CTAs to all CTAs, a round: words
// polled 5.1 us, release and acquire around a count with the values read behind it 1.6, words behind a relaxed count 1.3 (the count alone 0.9).
// Why a word is not overwritten too early: who writes a vector of layer l + 1 has read x of layer l + 1 or something made from all
// of it, every CTA writes rows of x (d >= 256 > CTAs), and it does so after its last read of layer l.
//
// Work split.  Output rows of a projection are dealt to the CTAs round robin (row r belongs to CTA r mod grid); inside
// a CTA a row goes to one warp, or, when the CTA has fewer rows than warps, to KS warps that split the row's K range
// and meet in shared memory.  Rows are read in "super-units" of 256 stored values: a whole number of quantisation
// blocks in every format (512 B fp16/bf16, 272 B Q8_0, 144 B Q4_0, 272 B Q8_0(64), 160 B Q4_1) and a multiple of 16 bytes,
// so a run of super-units is one bulk copy and lane l expands values 8l..8l+7 of a super-unit from shared memory.  A warp starts the
// copies of the rows of its next piece of work as soon as it is done with the last one: weights do not depend on activations, so
// their DRAM round trip hides behind the exchange, and cache rows are asked of L2 a phase ahead.  (Asking L2 for experts before the
// router has chosen made a step slower: the requests stand in front of the copies that are needed.)
// The vocabulary projection, too many rows per CTA to stage, pulls its rows through a ring.
//
// What bounds it: the chain of dependent steps, six exchanges a layer of 1.2 to 1.5 us with what they wait for, and the instructions between them.  A step,
// us (five grid-wide barriers a layer, 360 bytes of spilled registers -> this form): 36 layers of 768, 12/4 heads, 5 of 9 experts of 1280, fp16,
// 1024 slots 1694 -> 930 (weights at the copy rate: 196); 26 layers, 3 of 9 experts of 768, 4 bits, 3001 slots 1061 -> 619 (36).  On the way: words and
// counts in place of barriers 1694 -> 1490, hardly anything spilled -> 1077, fewer instructions -> 966 (eager times, 36 layers).
//
// Every wait is bounded: a word that does not arrive within about two seconds writes status 401, a copy that
// never signals its mbarrier 402; the CTA then skips the rest of the step (the others follow when their own waits run
// out) and waits, again bounded, for its copies in flight before it leaves.  The launch is cooperative, so either all CTAs are
// resident or the launch fails.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "sm100_common.cuh"
#include "gb_decode.h"
#include "decode_fmt.cuh"

namespace gb {
namespace mg {

constexpr int WARPS = 16;
constexpr int THREADS = WARPS * 32;
constexpr int ROUTER_AREA = 32 * 1024;   // shared memory for a layer's router rows
constexpr int SU = 256;               // values per super-unit
constexpr int MAX_SLOTS = 9;          // top_k <= 8 routed experts plus the shared one
constexpr int MAX_HEADS = 128;
constexpr int ST_TIMEOUT_GRID = 401;
constexpr int ST_TIMEOUT_COPY = 402;      // a bulk copy of weight rows never signalled its barrier

template <int FMT> struct Fmt {
  static constexpr bool k16 = FMT == GB_W_F16 || FMT == GB_W_BF16;
  static constexpr int bytes = k16 ? 512 : FMT == GB_W_GGML_Q8_0 ? 272 : FMT == GB_W_Q4_0 ? 144 : FMT == GB_W_Q8_64 ? 272 : 160;
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// ------------------------------------------------------------------------------------------------ grid barrier, once a step
// Arrivals are counted in sync[0], which only ever grows; barrier k of a launch opens at base + k * grid, where base
// (sync[1]) is the count the previous launch left behind.
struct GridBar {
  unsigned* cnt;
  int* status;
  int* dead;          // shared memory: set once a wait of this CTA ran out
  unsigned next;      // count at which the next barrier opens
};

__device__ __forceinline__ bool grid_sync(GridBar& gb) {
  __syncthreads();
  if (threadIdx.x == 0 && !*gb.dead) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(gb.cnt), "r"(1u) : "memory");
    unsigned it = 0;
    unsigned long long t0 = 0;
    for (;;) {
      unsigned v;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(gb.cnt) : "memory");
      if ((int)(v - gb.next) >= 0) break;
      ++it;
      if (it == 2048) t0 = globaltimer_ns();
      if (it > 2048) {
        __nanosleep(64);
        if ((it & 1023) == 0 && globaltimer_ns() - t0 > 2000000000ull) {
          *gb.dead = 1;
          atomicCAS(gb.status, 0, ST_TIMEOUT_GRID);
          break;
        }
      }
    }
  }
  gb.next += gridDim.x;
  __syncthreads();
  return !*gb.dead;
}

// ------------------------------------------------------------------------------------------------ exchange words
// Relaxed loads at GPU scope: a word carries its own epoch, so nothing has to be ordered behind it, and an acquire would empty this SM's L1 every time.
__device__ __forceinline__ void put_f32(unsigned long long* p, float v, uint32_t epoch) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)epoch << 32 | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ unsigned long long peek_f32(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ ulonglong2 peek_f32x2(const unsigned long long* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool fresh(unsigned long long v, uint32_t epoch) { return (uint32_t)(v >> 32) == epoch; }
__device__ __forceinline__ float value(unsigned long long v) { return __uint_as_float((uint32_t)v); }
template <typename XT> __device__ __forceinline__ void put_16(uint32_t* p, XT v, uint32_t epoch) {
  unsigned short b;
  memcpy(&b, &v, 2);
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(epoch << 16 | b) : "memory");
}
__device__ __forceinline__ uint32_t peek_16(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint4 peek_16x4(const uint32_t* p) {       // four words, each whole in itself
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool fresh(uint32_t v, uint32_t epoch) { return (v >> 16) == (epoch & 0xffffu); }
__device__ __forceinline__ bool fresh(const uint4& v, uint32_t epoch) {
  return fresh(v.x, epoch) && fresh(v.y, epoch) && fresh(v.z, epoch) && fresh(v.w, epoch);
}
template <typename XT> __device__ __forceinline__ XT value16(uint32_t v) {
  const unsigned short b = (unsigned short)v;
  XT x;
  memcpy(&x, &b, 2);
  return x;
}

// Polls until `look` (which loads its words again and says whether all are fresh) succeeds.  Bounded: gives up after two seconds, or when
// another thread of the CTA has, and what was loaded last is then used for nothing that leaves the CTA's step.
template <class Look>
__device__ __forceinline__ void await(Look look, int* dead, int* status) {
  unsigned it = 0;
  unsigned long long t0 = 0;
  while (!look()) {
    if (++it < 4096) continue;
    if (it == 4096) t0 = globaltimer_ns();
    __nanosleep(64);
    if ((it & 255) == 0) {
      if (*reinterpret_cast<volatile int*>(dead)) return;
      if (globaltimer_ns() - t0 > 2000000000ull) {
        *reinterpret_cast<volatile int*>(dead) = 1;
        atomicCAS(status, 0, ST_TIMEOUT_GRID);
        return;
      }
    }
  }
}

// The counts of arrivals, a line each, ahead of the exchange words.  They only grow; a launch counts from what it found.
enum Vec { V_X, V_QKV, V_PART, V_ATT, V_MID, V_ACT, VECS };
constexpr int COUNT_WORDS = 16;       // 64-bit words of a line

struct Gate {
  unsigned long long* words;   // counts at words[v * COUNT_WORDS]
  unsigned* base;       // shared memory: the counts when the launch began
  unsigned* warps;      // shared memory: warps of this CTA that are done with a vector
  int* dead;
  int* status;
};
// This CTA's part of vector v is on its way: called by one thread.
__device__ __forceinline__ void arrive(const Gate& g, Vec v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(reinterpret_cast<unsigned*>(g.words + v * COUNT_WORDS)) : "memory");
}
// The same by every warp; the last one of the CTA arrives.
__device__ __forceinline__ void arrive_warp(const Gate& g, Vec v) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0 && atomicAdd(g.warps + v, 1u) == WARPS - 1) {
    g.warps[v] = 0;
    arrive(g, v);
  }
}
// Waits until `arrivals` more CTAs than at the launch's start have arrived, and for all warps of the CTA.
__device__ __forceinline__ void wait_for(const Gate& g, Vec v, unsigned arrivals) {
  if (threadIdx.x == THREADS - 32) {                  // a warp that has no rows where rows are few
    const unsigned* cnt = reinterpret_cast<const unsigned*>(g.words + v * COUNT_WORDS);
    const unsigned target = g.base[v] + arrivals;
    await([&] {
      unsigned c;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(cnt) : "memory");
      return (int)(c - target) >= 0;
    }, g.dead, g.status);
  }
  __syncthreads();
}

// The exchange words of a launch, in one buffer (gb_decode_mega_words counts them): offsets in 64-bit words.
struct Words {
  long long x, xmid, part, qkv, att, act, total;
};
__host__ __device__ inline Words words_of(const gb_mega_args& a) {
  const long long slots = a.ne > 0 ? a.top_k + (a.shared ? 1 : 0) : 1, qd = (long long)a.H * a.hd;
  Words w;
  w.x = VECS * COUNT_WORDS;
  w.xmid = w.x + a.d;
  w.part = w.xmid + a.d;                                                       // [H][max_splits][2 + hd]: max, sum, output
  w.qkv = w.part + (long long)a.H * a.max_splits * (a.hd + 2);
  w.att = w.qkv + (qd + 2LL * a.KV * a.hd) / 2;
  w.act = w.att + qd / 2;
  w.total = w.act + slots * a.E / 2;
  return w;
}

// ------------------------------------------------------------------------------------------------ rows of a phase
// One projection phase: every output is a sum over super-units.  They lie in stretches of nsu, super-unit su of stretch s of an output at
//   W + row_off(output) + off[s] + su * bytes
// (off absent: 0).  A plain row is one stretch, a gate/up pair two (two rows), the down projection of several experts one per slot.
struct Phase {
  const uint8_t* W;
  const long long* off;
  const float* wt;            // weights of the stretches, where stream_run is WEIGHTED
  int nsu;
};

// Which outputs of the CTA a warp computes: local output i = first + k * stride for k < n, super-units [pb, pe).
struct Plan {
  int rows;
  short n, first, stride, KS, pb, pe;      // a row's super-units are staged in shared memory, so there are few of any of these
  short s0, su0;      // pb as a stretch of nsu super-units and a place in it
};
__device__ __forceinline__ Plan make_plan(int N, int P, int nsu) {
  const int warp = threadIdx.x >> 5;
  const int grid = gridDim.x, cta = blockIdx.x;
  Plan pl;
  pl.rows = N > cta ? (N - cta + grid - 1) / grid : 0;
  pl.KS = 1; pl.first = (short)warp; pl.stride = WARPS; pl.pb = 0; pl.pe = P; pl.n = 0; pl.s0 = pl.su0 = 0;
  if (pl.rows == 0) return pl;
  const int ks = min(P, WARPS / pl.rows);
  if (ks >= 2) {
    pl.KS = ks;
    pl.first = warp / ks;
    const int k = warp - pl.first * ks;
    pl.pb = k * P / ks;
    pl.pe = (k + 1) * P / ks;
    pl.s0 = pl.pb / nsu;
    pl.su0 = pl.pb - pl.s0 * nsu;
    pl.n = pl.first < pl.rows ? 1 : 0;
  } else {
    pl.n = warp < pl.rows ? (pl.rows - warp + WARPS - 1) / WARPS : 0;
  }
  return pl;
}

// A byte of four small unsigned numbers as a float, plus 2^23: one permutation where a conversion takes two instructions, one of them slow.
__device__ __forceinline__ float byte_float(uint32_t four, int k) { return __uint_as_float(__byte_perm(four, 0x4B000000u, 0x7440 | k)); }

// Dot product of values 8 * lane .. of a super-unit with x: of the 16 bytes q that the lane holds of it (16-bit formats), or from `slot`.  A
// block's scale is one factor of the eight products.
template <int FMT>
__device__ __forceinline__ float su_dot(const uint4& q, const uint8_t* slot, const float (&x)[8]) {
  const int lane = threadIdx.x & 31;
  float s = 0.f;
  if constexpr (FMT == GB_W_F16) {
    const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); s += f.x * x[2 * i] + f.y * x[2 * i + 1]; }
  } else if constexpr (FMT == GB_W_BF16) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); s += f.x * x[2 * i] + f.y * x[2 * i + 1]; }
  } else if constexpr (FMT == GB_W_Q4_0) {             // blocks of 18 bytes; byte i: low nibble = value 2i
    const uint8_t* p = slot + (lane >> 2) * 18;
    const uint8_t* n = p + 2 + (lane & 3) * 4;
    const uint32_t v = (uint32_t)ld_u16(n) | ((uint32_t)ld_u16(n + 2) << 16), lo = v & 0x0F0F0F0Fu, hi = (v >> 4) & 0x0F0F0F0Fu;
#pragma unroll
    for (int i = 0; i < 4; ++i) s += (byte_float(lo, i) - 8388616.f) * x[2 * i] + (byte_float(hi, i) - 8388616.f) * x[2 * i + 1];
    s *= h2f(ld_u16(p));
  } else if constexpr (FMT == GB_W_GGML_Q8_0) {        // blocks of 34 bytes
    const uint8_t* p = slot + (lane >> 2) * 34;
    const uint8_t* n = p + 2 + (lane & 3) * 8;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t v = ((uint32_t)ld_u16(n + 4 * h) | ((uint32_t)ld_u16(n + 4 * h + 2) << 16)) ^ 0x80808080u;
#pragma unroll
      for (int i = 0; i < 4; ++i) s += (byte_float(v, i) - 8388736.f) * x[4 * h + i];
    }
    s *= h2f(ld_u16(p));
  } else {
    float w[8];
    load8<FMT>(slot, lane, w);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += w[i] * x[i];
  }
  return s;
}
template <typename XT>
__device__ __forceinline__ void x_of(const XT* x, float (&f)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(x + 8 * (threadIdx.x & 31));
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = Cvt<XT>::unpack2(u[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
template <int FMT> __device__ __forceinline__ uint4 su_word(const uint8_t* slot) {
  if constexpr (Fmt<FMT>::k16) return *reinterpret_cast<const uint4*>(slot + 16 * (threadIdx.x & 31));
  else return make_uint4(0u, 0u, 0u, 0u);
}

// ------------------------------------------------------------------------------------------------ row streaming
// The layer phases do not pull their rows through registers: lane 0 of a warp issues one bulk asynchronous copy per
// contiguous run of super-units of ALL the warp's work in the phase into the warp's own slice of shared memory (no
// other warp touches it), signalled on the warp's own mbarriers, and it does so right after the warp has finished the
// phase before: the weights of a phase are in flight while the previous phase's results are exchanged.
constexpr int MAXI = 4;               // outputs a warp stages at once (checked on the host)
constexpr int MAX_DYN = 220 * 1024;   // dynamic shared memory the kernel may ask for (227 KB per CTA, less than 7 KB static)

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}

struct Stage {
  uint8_t* base;        // this warp's slice
  uint64_t* bars;       // this warp's MAXI barriers
  uint32_t parity;      // bit k: parity that the next completion of bars[k] is waited with
  uint32_t pending;     // bit k: a copy onto bars[k] was issued and not yet waited for
  int* dead;
  int* status;
};

// Per-warp bytes of the staging slice for one phase: N outputs of P super-units each, dealt as make_plan does.
__host__ __device__ inline long long stage_need(long long N, int P, int grid, int su_bytes, int* items_out) {
  const long long rows = (N + grid - 1) / grid;
  long long items = 1, sus = P;
  if (rows == 0) { if (items_out) *items_out = 0; return 0; }
  const int ks = (int)(WARPS / rows) < P ? (int)(WARPS / rows) : P;
  if (ks >= 2) sus = (P + ks - 1) / ks;
  else items = (rows + WARPS - 1) / WARPS;
  if (items_out) *items_out = (int)items;
  return items * sus * su_bytes;
}

// One lane a run of super-units: `runs` is the most that an item has.  What was read from the slice was read in stream_run, which ends with the
// fence between those reads and these copies.  row_off(k, o): byte offset of the stored row of the warp's k-th output o.
template <int FMT, int RUNS, class RowOff>
__device__ __forceinline__ void stream_issue(const Phase& ph, const Plan& pl, int runs, Stage& st, RowOff row_off) {
  constexpr int SB = Fmt<FMT>::bytes;
  const int lane = threadIdx.x & 31, n = pl.n, pb = pl.pb, pe = pl.pe;
  if (RUNS) runs = RUNS;
  __syncwarp();                                  // every lane has finished reading the slice
  if (n == 0 || *st.dead) return;                // uniform over the warp
  st.pending |= (1u << n) - 1u;
  const int item_bytes = (pe - pb) * SB;
  if (lane < n) mbar_arrive_expect_tx(st.bars + lane, (uint32_t)item_bytes);
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < n * runs; i += 32) {
    const int k = i / runs, s = pl.s0 + i - k * runs;                    // stretch s of the warp's k-th output
    const int lo = max(pb, s * ph.nsu), hi = min(pe, (s + 1) * ph.nsu);
    if (lo >= hi) continue;
    const uint8_t* row = ph.W + row_off(k, (int)blockIdx.x + (pl.first + k * pl.stride) * (int)gridDim.x);
    bulk_g2s(smem_u32(st.base) + k * item_bytes + (lo - pb) * SB, row + (ph.off ? ph.off[s] : 0ll) + (long long)(lo - s * ph.nsu) * SB,
             (uint32_t)((hi - lo) * SB), smem_u32(st.bars + k));
  }
}

// epi(i, o, a0, a1): local output i (0 .. rows - 1 of the CTA), output o, by one thread per output.  Then the CTA has its part of `v` done.
// PAIR: two stretches that meet the same activations, each with a sum of its own (gate and up).  WEIGHTED: stretch s counts ph.wt[s] times.
template <int FMT, typename XT, bool PAIR, bool WEIGHTED, class Epi>
__device__ __forceinline__ void stream_run(const Phase& ph, const Plan& pl, const XT* xs, Stage& st, float (*red)[WARPS], const Gate& gate, Vec v_out,
                                           Epi epi) {
  constexpr int SB = Fmt<FMT>::bytes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grid = gridDim.x, cta = blockIdx.x, n = pl.n, pb = pl.pb, pe = pl.pe, KS = pl.KS;
  const int item_bytes = (pe - pb) * SB;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const bool got = mbar_wait(st.bars + k, (st.parity >> k) & 1u);
    if (!got) {                                  // bounded: the copy never landed
      if (lane == 0) { *st.dead = 1; atomicCAS(st.status, 0, ST_TIMEOUT_COPY); }
      break;
    }
    st.parity ^= 1u << k;
    st.pending &= ~(1u << k);
    const uint8_t* slot = st.base + (size_t)k * item_bytes;
    float a0 = 0.f, a1 = 0.f, x[8];
    if (PAIR && KS == 1) {                       // both stretches whole: one read of the activations
      const int half = ph.nsu * SB;
#pragma unroll 2
      for (int p = 0; p < ph.nsu; ++p, slot += SB) {
        x_of<XT>(xs + p * SU, x);
        a0 += su_dot<FMT>(su_word<FMT>(slot), slot, x);
        a1 += su_dot<FMT>(su_word<FMT>(slot + half), slot + half, x);
      }
    } else {
      int s = pl.s0, su = pl.su0;
#pragma unroll 2
      for (int p = pb; p < pe; ++p, slot += SB) {
        x_of<XT>(xs + (PAIR ? su : p) * SU, x);
        const float v = su_dot<FMT>(su_word<FMT>(slot), slot, x);
        if (PAIR && s == 1) a1 += v;
        else a0 += WEIGHTED ? ph.wt[s] * v : v;
        if ((PAIR || WEIGHTED) && ++su == ph.nsu) { su = 0; ++s; }
      }
    }
    a0 = warp_sum(a0);
    if (PAIR) a1 = warp_sum(a1);
    if (lane == 0) {
      const int i = pl.first + k * pl.stride;
      if (KS == 1) epi(i, cta + i * grid, a0, a1);
      else { red[0][warp] = a0; if (PAIR) red[1][warp] = a1; }
    }
  }
  fence_proxy_async();                           // the reads of the slice come before the copies that stream_issue starts next
  if (KS > 1) {                                  // uniform over the CTA
    __syncthreads();
    if (warp == 0) {                             // fewer rows than half the warps
      if (lane < pl.rows) {
        float a0 = 0.f, a1 = 0.f;
        for (int j = 0; j < KS; ++j) { a0 += red[0][lane * KS + j]; if (PAIR) a1 += red[1][lane * KS + j]; }
        epi(lane, cta + lane * grid, a0, a1);
      }
      __syncwarp();
      if (lane == 0) arrive(gate, v_out);
    }
  } else {
    arrive_warp(gate, v_out);
  }
}

// ------------------------------------------------------------------------------------------------ pieces
// RMSNorm of an fp32 vector into 16-bit shared memory, by the whole CTA.  The vector is polled from its exchange words, or read from
// `row` (the embedding).  The norm's weights come from DRAM: they are asked for before the wait.
template <typename XT>
__device__ __forceinline__ void block_norm(const Gate& gate, Vec v_in, unsigned arrivals, const unsigned long long* words, const float* row,
                                           uint32_t epoch, const float* __restrict__ w, XT* xs, int d, float eps, float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // d <= 8 * THREADS: at most four pairs per thread
  constexpr int NP = 4;
  float2 v[NP], g[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const int i = threadIdx.x + k * THREADS;
    v[k] = g[k] = make_float2(0.f, 0.f);
    if (k * THREADS >= d / 2) continue;            // uniform
    g[k] = i < d / 2 ? reinterpret_cast<const float2*>(w)[i] : make_float2(0.f, 0.f);
    if (row && i < d / 2) v[k] = reinterpret_cast<const float2*>(row)[i];
  }
  if (!row) {
    wait_for(gate, v_in, arrivals);
    await([&] {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        if (k * THREADS >= d / 2) break;
        const int i = threadIdx.x + k * THREADS;
        if (i < d / 2) {
          const ulonglong2 u = peek_f32x2(words + 2 * i);
          ok = ok && fresh(u.x, epoch) && fresh(u.y, epoch);
          v[k] = make_float2(value(u.x), value(u.y));
        }
      }
      return ok;
    }, gate.dead, gate.status);
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NP; ++k) ss += v[k].x * v[k].x + v[k].y * v[k].y;
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < WARPS; ++i) tot += red[i];
  float inv = rsqrtf(tot / (float)d + eps);
  if (!isfinite(inv)) inv = 0.f;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    if (k * THREADS >= d / 2) break;
    const int i = threadIdx.x + k * THREADS;
    if (i < d / 2) *reinterpret_cast<uint32_t*>(xs + 2 * i) = Cvt<XT>::pack2(v[k].x * inv * g[k].x, v[k].y * inv * g[k].y);
  }
  __syncthreads();
}

// QK-norm + rotation of one head by one warp (the arithmetic of qk_rope_append_kernel in decode.cu).  What does not depend on the step's
// vectors, the weights and angles of the lane's two pairs, is asked for ahead of the wait.
struct RopePair {
  float w0[2], w1[2], c[2], sn[2];
  __device__ __forceinline__ static int first(int p, int rope_type) { return rope_type == 0 ? 2 * p : p; }
  __device__ __forceinline__ static int second(int p, int rope_type, int pairs) { return rope_type == 0 ? 2 * p + 1 : p + pairs; }
  __device__ __forceinline__ void load(const float* __restrict__ w, const float* __restrict__ csr, int pairs, int rope_type) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int p = (threadIdx.x & 31) + 32 * k, pc = p < pairs ? p : 0;
      w0[k] = w ? w[first(pc, rope_type)] : 1.f;
      w1[k] = w ? w[second(pc, rope_type, pairs)] : 1.f;
      c[k] = csr[pc];
      sn[k] = csr[pairs + pc];
    }
  }
};
template <typename XT, class Store>
__device__ __forceinline__ void rope_head(const uint32_t* src, uint32_t epoch, const RopePair& r, bool norm, int hd, int rope_type, float eps,
                                          int* dead, int* status, Store st) {
  const int lane = threadIdx.x & 31, pairs = hd / 2;
  float a[2], b[2];
  await([&] {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int p = lane + 32 * k;
      a[k] = b[k] = 0.f;
      if (p < pairs) {
        const uint32_t u = peek_16(src + RopePair::first(p, rope_type)), v = peek_16(src + RopePair::second(p, rope_type, pairs));
        ok = ok && fresh(u, epoch) && fresh(v, epoch);
        a[k] = Cvt<XT>::to_f(value16<XT>(u));
        b[k] = Cvt<XT>::to_f(value16<XT>(v));
      }
    }
    return ok;
  }, dead, status);
  __syncwarp();
  float inv = 1.f;
  if (norm) {
    const float ss = warp_sum(a[0] * a[0] + b[0] * b[0] + a[1] * a[1] + b[1] * b[1]);
    inv = rsqrtf(ss / (float)hd + eps);
    if (!isfinite(inv)) inv = 0.f;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int p = lane + 32 * k;
    if (p < pairs) {
      float x0 = a[k], x1 = b[k];
      if (norm) { x0 *= inv * r.w0[k]; x1 *= inv * r.w1[k]; }
      st(RopePair::first(p, rope_type), x0 * r.c[k] - x1 * r.sn[k]);
      st(RopePair::second(p, rope_type, pairs), x0 * r.sn[k] + x1 * r.c[k]);
    }
  }
}

template <typename XT>
__device__ __forceinline__ void unpack8(const uint4& r, float (&f)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 v = Cvt<XT>::unpack2(w[i]); f[2 * i] = v.x; f[2 * i + 1] = v.y; }
}

struct Smem {          // static shared memory of the kernel
  float red[2][WARPS];
  float nred[WARPS];              // sums of squares of the norms
  unsigned base[VECS], warps[VECS];   // see Gate
  float lg[64];
  __align__(16) float q[4][128];
  __align__(16) uint16_t knew[128], vnew[128];   // the step's own key and value of this CTA's head
  float res[2][MAXI * WARPS];     // x (0) and x after attention (1) at the rows that this CTA owns
  gb_mega_layer layer[2];         // this layer's and the next one's pointers
  Plan plan[4][WARPS];            // what every warp computes in the projections A, C, D and E
  int d_row[MAXI * WARPS];
  unsigned char d_slot[MAXI * WARPS];               // D: row inside its expert, and slot, of the CTA's i-th output
  gb_seq_state seq;               // the sequence when the step began
  int pos, splits;
  unsigned long long *wx, *wmid, *wpart;            // exchange words
  uint32_t *wqkv, *watt, *wact;
  long long off_e[MAX_SLOTS];
  long long off_gu[2];
  float wsel[MAX_SLOTS];
  int esel[MAX_SLOTS];
  int dead;
};

// ------------------------------------------------------------------------------------------------ attention
// CTA `item` < KV * S serves key/value head item % KV over slots [lo, hi) of the cache (split item / KV): all query
// heads of the group in one walk.  The CTA whose range holds the step's own slot writes the new K (normalised,
// rotated) and V there.  Partial (max, sum, output) per (head, split) go out as exchange words.
// GC: query heads of a pass over the slots (the group's, or four at a time).  LPS: lanes of a slot, hd / 8, or 0 where they are not known here.
template <typename XT, int GC, int LPS>
__device__ __forceinline__ void attention_phase(const gb_mega_args& a, const gb_mega_layer& L, Smem& sm, float* amerge, uint32_t epoch,
                                                const Gate& gate, unsigned arrivals, unsigned long long*& prof) {
  const int item = blockIdx.x, S = sm.splits;
  const gb_seq_state s = sm.seq;
  const uint32_t* qkv = sm.wqkv;
  unsigned long long* part = sm.wpart;
  if (item >= a.KV * S) {
    if (prof) { const unsigned long long t = globaltimer_ns(); *prof++ = t; *prof++ = t; *prof++ = t; }
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hd = LPS ? 8 * LPS : a.hd, G = a.H / a.KV, lps = LPS ? LPS : hd / 8, spw = 32 / lps, grp = lane / lps, sub = lane - grp * lps;
  const int kvh = item % a.KV, split = item / a.KV;
  const int n_slots = min(a.cap, s.cache_len + 1);       // s: the sequence state, read once per step by the caller
  const int slot_new = s.cache_len < a.cap ? s.cache_len : a.pinned + s.ring_start;
  const int per = (n_slots + S - 1) / S;
  const int lo = split * per, hi = min(n_slots, lo + per);
  const bool owner = slot_new >= lo && slot_new < hi;
  const float* csr = a.cos_sin + (size_t)sm.pos * hd;
  float* am = amerge;                         // [WARPS][4]
  float* al = amerge + WARPS * 4;             // [WARPS][4]
  float* ao = amerge + WARPS * 8;             // [WARPS][4][hd]

#pragma unroll 1
  for (int g0 = 0; g0 < G; g0 += GC) {
    const int gc = GC < 4 ? GC : min(GC, G - g0);
    // hd / 8 lanes share a slot (one 16-byte load of its key, one of its value), so a warp works on 256 / hd slots side by side;
    // every group of lanes keeps its own soft-max, and the groups meet below.  The rows of the first trip do not depend on the
    // queries and are asked for before these are there; the step's own row comes from shared memory.
    auto live = [&](int j) {
      if (j >= hi) return false;
      if (a.window <= 0 || j == slot_new) return true;
      return s.abs_pos - __ldcg(a.slot_pos + j) < a.window;
    };
    bool ok;
    uint4 kr, vr;
    auto fetch = [&](int j) {
      ok = live(j);
      kr = vr = make_uint4(0u, 0u, 0u, 0u);
      if (ok && j != slot_new) {
        const size_t at = ((size_t)j * a.KV + kvh) * hd + sub * 8;
        kr = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const XT*>(L.cache_k) + at));
        vr = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const XT*>(L.cache_v) + at));
      }
    };
    fetch(lo + warp * spw + grp);
    const bool is_q = warp < gc, is_k = g0 == 0 && owner && warp == 4, is_v = g0 == 0 && owner && warp == 5;
    RopePair rp;
    if (is_q || is_k) rp.load(is_q ? L.q_norm : L.k_norm, csr, hd / 2, a.rope_type);
    if (g0 == 0) wait_for(gate, V_QKV, arrivals);
    if (is_q) {
      float* qd = sm.q[warp];
      const float scale = a.scale;
      rope_head<XT>(qkv + (size_t)(kvh * G + g0 + warp) * hd, epoch, rp, L.q_norm != nullptr, hd, a.rope_type, a.eps, &sm.dead, a.status,
                    [&](int i, float v) { qd[i] = Cvt<XT>::to_f(Cvt<XT>::from_f(v)) * scale; });
    } else if (is_k) {
      XT* dk = reinterpret_cast<XT*>(L.cache_k) + ((size_t)slot_new * a.KV + kvh) * hd;
      XT* sk = reinterpret_cast<XT*>(sm.knew);
      rope_head<XT>(qkv + (size_t)(a.H + kvh) * hd, epoch, rp, L.k_norm != nullptr, hd, a.rope_type, a.eps, &sm.dead, a.status,
                    [&](int i, float v) { dk[i] = sk[i] = Cvt<XT>::from_f(v); });
      if (kvh == 0 && lane == 0) a.slot_pos[slot_new] = s.abs_pos;
    } else if (is_v) {
      const uint32_t* src = qkv + (size_t)(a.H + a.KV + kvh) * hd;
      XT* dv = reinterpret_cast<XT*>(L.cache_v) + ((size_t)slot_new * a.KV + kvh) * hd;
      XT* sv = reinterpret_cast<XT*>(sm.vnew);
      for (int i = lane; i < hd; i += 32) {
        uint32_t v = 0;
        await([&] { v = peek_16(src + i); return fresh(v, epoch); }, &sm.dead, a.status);
        dv[i] = sv[i] = value16<XT>(v);
      }
    }
    __syncthreads();
    if (prof && g0 == 0) *prof++ = globaltimer_ns();          // queries rotated, the step's key and value stored

    float m[GC], l[GC], o[GC][8];
#pragma unroll
    for (int g = 0; g < GC; ++g) {
      m[g] = -INFINITY;
      l[g] = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[g][e] = 0.f;
    }
#pragma unroll 1
    for (int j0 = lo + warp * spw; j0 < hi; j0 += WARPS * spw) {             // the warp's first slot of the trip
      if (j0 != lo + warp * spw) fetch(j0 + grp);
      if (ok && j0 + grp == slot_new) {
        kr = *reinterpret_cast<const uint4*>(sm.knew + sub * 8);
        vr = *reinterpret_cast<const uint4*>(sm.vnew + sub * 8);
      }
      float f[8], d[GC];
      unpack8<XT>(kr, f);
#pragma unroll
      for (int g = 0; g < GC; ++g) {
        const float4* q = reinterpret_cast<const float4*>(&sm.q[g][sub * 8]);     // of heads past gc: old, finite, not used
        if (GC > 3) asm volatile("" ::: "memory");        // one head's queries in registers at a time: all four at once spill
        const float4 q0 = q[0], q1 = q[1];
        d[g] = q0.x * f[0] + q0.y * f[1] + q0.z * f[2] + q0.w * f[3] + q1.x * f[4] + q1.y * f[5] + q1.z * f[6] + q1.w * f[7];
      }
      for (int off = lps >> 1; off > 0; off >>= 1)
#pragma unroll
        for (int g = 0; g < GC; ++g) d[g] += __shfl_xor_sync(0xffffffffu, d[g], off);
      unpack8<XT>(vr, f);
      if (ok) {
#pragma unroll
        for (int g = 0; g < GC; ++g) {
          if (g < gc) {
            const float mn = fmaxf(m[g], d[g]);
            const float c = __expf(m[g] - mn), p = __expf(d[g] - mn);
            l[g] = l[g] * c + p;
#pragma unroll
            for (int e = 0; e < 8; ++e) o[g][e] = o[g][e] * c + p * f[e];
            m[g] = mn;
          }
        }
      }
    }
    for (int off = lps; off < 32; off <<= 1)
#pragma unroll
      for (int g = 0; g < GC; ++g) {
        const float mm = fmaxf(m[g], __shfl_xor_sync(0xffffffffu, m[g], off));
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
    if (prof && g0 == 0) *prof++ = globaltimer_ns();          // this warp's slots walked
    // the sixteen warps meet in shared memory, in warp order
#pragma unroll
    for (int g = 0; g < GC; ++g) {
      if (g < gc) {
        if (lane == 0) { am[warp * 4 + g] = m[g]; al[warp * 4 + g] = l[g]; }
        if (grp == 0) {
          float4* dst = reinterpret_cast<float4*>(ao + (size_t)(warp * 4 + g) * hd + sub * 8);
          dst[0] = make_float4(o[g][0], o[g][1], o[g][2], o[g][3]);
          dst[1] = make_float4(o[g][4], o[g][5], o[g][6], o[g][7]);
        }
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < gc * hd; t += THREADS) {
      const int g = t / hd, c = t - g * hd;
      float mm = -INFINITY;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, am[w * 4 + g]);
      float ll = 0.f, oo = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const float mw = am[w * 4 + g];
        const float f = mw == -INFINITY ? 0.f : __expf(mw - mm);
        ll += al[w * 4 + g] * f;
        oo += ao[(size_t)(w * 4 + g) * hd + c] * f;
      }
      unsigned long long* dst = part + ((size_t)(kvh * G + g0 + g) * S + split) * (hd + 2);
      put_f32(dst + 2 + c, oo, epoch);
      if (c == 0) { put_f32(dst, mm, epoch); put_f32(dst + 1, ll, epoch); }
    }
    __syncthreads();
    if (prof && g0 == 0) *prof++ = globaltimer_ns();          // partial results on their way
  }
  if (threadIdx.x == 0) arrive(gate, V_PART);
}

// Merge of the S partial results of all heads, dealt to the CTAs by output element (element c belongs to CTA c mod grid): a warp an
// element, its lanes over the splits, at most two each (S <= 64).  Every CTA merging everything for itself read S * H * (hd + 2) numbers on each SM.
template <typename XT>
__device__ __forceinline__ void merge_phase(const gb_mega_args& a, const Smem& sm, uint32_t epoch, const Gate& gate, unsigned arrivals) {
  wait_for(gate, V_PART, arrivals);
  const int S = sm.splits;
  const unsigned long long* part = sm.wpart;
  uint32_t* att = sm.watt;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hd = a.hd, st = hd + 2, qd = a.H * hd;
  for (int c = blockIdx.x + warp * (int)gridDim.x; c < qd; c += WARPS * (int)gridDim.x) {
    const int h = c / hd, cc = c - h * hd;
    const unsigned long long* base = part + (size_t)h * S * st;
    float m[2], l[2], o[2];
    await([&] {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int sp = lane + 32 * k;
        m[k] = -INFINITY;
        l[k] = o[k] = 0.f;
        if (sp < S) {
          const unsigned long long u = peek_f32(base + (size_t)sp * st), v = peek_f32(base + (size_t)sp * st + 1),
                                   w = peek_f32(base + (size_t)sp * st + 2 + cc);
          ok = ok && fresh(u, epoch) && fresh(v, epoch) && fresh(w, epoch);
          m[k] = value(u); l[k] = value(v); o[k] = value(w);
        }
      }
      return ok;
    }, gate.dead, gate.status);
    __syncwarp();
    const float M = warp_max(fmaxf(m[0], m[1]));
    const float f0 = m[0] == -INFINITY ? 0.f : __expf(m[0] - M), f1 = m[1] == -INFINITY ? 0.f : __expf(m[1] - M);
    const float ls = warp_sum(l[0] * f0 + l[1] * f1), os = warp_sum(o[0] * f0 + o[1] * f1);
    if (lane == 0) put_16<XT>(att + c, Cvt<XT>::from_f(ls > 0.f ? os / ls : 0.f), epoch);
  }
  arrive_warp(gate, V_ATT);
}

// n 16-bit values (a multiple of four) from their exchange words into shared memory, by the whole CTA.
template <typename XT, int NV>
__device__ __forceinline__ void gather16(const Gate& gate, Vec v_in, unsigned arrivals, const uint32_t* words, int n, uint32_t epoch, XT* xs) {
  wait_for(gate, v_in, arrivals);
#pragma unroll 1
  for (int i0 = threadIdx.x; i0 < n / 4; i0 += NV * THREADS) {
    uint4 v[NV];
    await([&] {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        if (NV > 1 && i0 - (int)threadIdx.x + k * THREADS >= n / 4) break;       // uniform
        if (i0 + k * THREADS < n / 4) {
          v[k] = peek_16x4(words + 4 * (i0 + k * THREADS));
          ok = ok && fresh(v[k], epoch);
        }
      }
      return ok;
    }, gate.dead, gate.status);
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (i0 + k * THREADS < n / 4) {
        uint2 o;
        o.x = (v[k].x & 0xffffu) | v[k].y << 16;
        o.y = (v[k].z & 0xffffu) | v[k].w << 16;
        reinterpret_cast<uint2*>(xs)[i0 + k * THREADS] = o;
      }
  }
  __syncthreads();
}

// Router of the normalised activations in shared memory (rules of route_in_block in decode.cu), then the tables the
// expert phases index by slot: expert, weight, byte offset of the expert's down-projection block.
template <typename XT, bool STAGED>
__device__ __forceinline__ void route_phase(const gb_mega_args& a, const gb_mega_layer& L, const XT* xs, Smem& sm, long long rb_E,
                                            const float* router_rows) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d = a.d, ne = a.ne, top_k = a.top_k;
  if (ne > 0) {
    // logits: up to eight experts take two warps each, over the halves of the row (d is a multiple of 256)
    const int split = 2 * ne <= WARPS ? 2 : 1;
    float* lg2 = sm.q[0];                                   // partial sums of the second halves (free in this phase)
    for (int t = warp; t < ne * split; t += WARPS) {
      const int e = split == 2 ? t >> 1 : t, hf = split == 2 ? t & 1 : 0;
      const int len = split == 2 ? d >> 1 : d;
      const float* wr = router_rows + e * d + hf * len;     // shared memory when STAGED, else the global rows
      const XT* xr = xs + hf * len;
      float s = 0.f;
#pragma unroll 4
      for (int c = lane * 4; c < len; c += 128) {
        float4 w;
        if constexpr (STAGED) {
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w) : "r"(smem_u32(wr + c)));
        } else {
          w = *reinterpret_cast<const float4*>(wr + c);
        }
        const uint2 xq = *reinterpret_cast<const uint2*>(xr + c);
        const float2 x0 = Cvt<XT>::unpack2(xq.x), x1 = Cvt<XT>::unpack2(xq.y);
        s += x0.x * w.x + x0.y * w.y + x1.x * w.z + x1.y * w.w;
      }
      s = warp_sum(s);
      if (lane == 0) { if (hf == 0) sm.lg[e] = s; else lg2[e] = s; }
    }
    __syncthreads();
    // softmax and the top_k picks by one warp, lane e holding experts e and e + 32 in registers (a single thread
    // walking the table in shared memory took most of this phase); ties go to the lower index, as in the serial rule
    if (warp == 0) {
      const float l0 = lane < ne ? sm.lg[lane] + (split == 2 ? lg2[lane] : 0.f) : -INFINITY;
      const float l1 = lane + 32 < ne ? sm.lg[lane + 32] + (split == 2 ? lg2[lane + 32] : 0.f) : -INFINITY;
      int my_e;
      float my_w;
      warp_route(l0, l1, L.bias, ne, top_k, my_e, my_w);
      if (lane < top_k) {
        sm.esel[lane] = my_e;
        sm.wsel[lane] = my_w;
        sm.off_e[lane] = (long long)my_e * d * rb_E;
        if (blockIdx.x == 0 && a.r_idx) { a.r_idx[lane] = my_e; a.r_w[lane] = my_w; }
      }
      if (a.shared && lane == top_k) { sm.esel[top_k] = ne; sm.wsel[top_k] = 1.f; sm.off_e[top_k] = (long long)ne * d * rb_E; }
    }
  } else if (threadIdx.x == 0) {
    sm.esel[0] = 0;
    sm.wsel[0] = 1.f;
    sm.off_e[0] = 0;
  }
  if (threadIdx.x == THREADS - 1) {      // byte offsets of the gate and the up block, for the projection that follows
    sm.off_gu[0] = 0;
    sm.off_gu[1] = reinterpret_cast<const uint8_t*>(L.wu) - reinterpret_cast<const uint8_t*>(L.wg);
  }
  __syncthreads();
}

// Vocabulary projection.  A warp has far more rows here than its staging slice holds, so the slice is a ring of
// `items` row slots (as many whole rows as fit, at most MAXI): row k lands in slot k % items, and the slot is refilled
// with row k + items as soon as the warp has read it.  head_issue before the last exchange starts the first rows.
// (Pulling the rows through registers one group ahead ran this phase at a fifth of the memory bandwidth.)  One row fits wherever the layers' rows do:
// 16 slices of a row of 4096 16-bit values beside the largest activations that MAXI rows a warp allow; gb_decode_mega_ok checks it.
template <int FMT>
__device__ __forceinline__ int head_items(const gb_mega_args& a) {
  const long long rb = (long long)(a.d / SU) * Fmt<FMT>::bytes;
  const long long fit = a.stage_bytes / rb;
  return (int)(fit < MAXI ? fit : MAXI);
}

// Rows k0 .. k1 - 1 of the warp into the slots from `slot` on.
template <int FMT>
__device__ __forceinline__ void head_issue(const gb_mega_args& a, const Plan& pl, Stage& st, int items, int k0, int k1, int slot = 0) {
  const uint32_t rb = (uint32_t)(a.d / SU) * Fmt<FMT>::bytes;
  k1 = min(k1, pl.n);
  if (k0 >= k1 || *st.dead) return;
  __syncwarp();                                  // every lane has finished reading the slots that are refilled
  st.pending |= ((1u << (k1 - k0)) - 1u) << slot;
  if ((threadIdx.x & 31) == 0) {
    for (int k = k0; k < k1; ++k, ++slot) {
      const long long o = (long long)blockIdx.x + (long long)(pl.first + k * pl.stride) * gridDim.x;
      mbar_arrive_expect_tx(st.bars + slot, rb);
      bulk_g2s(smem_u32(st.base + (size_t)slot * rb), reinterpret_cast<const uint8_t*>(a.head) + o * rb, rb,
               smem_u32(st.bars + slot));
    }
  }
}

template <int FMT, typename XT>
__device__ __forceinline__ void head_phase(const gb_mega_args& a, const XT* xs, Stage& st) {
  constexpr int SB = Fmt<FMT>::bytes;
  const int nsu = a.d / SU;
  const long long rb = (long long)nsu * SB;
  const Plan pl = make_plan(a.V, nsu, nsu);
  const int items = head_items<FMT>(a);
  const int lane = threadIdx.x & 31;
  constexpr int NX = 4;                          // activations of that many super-units stay in registers: a warp has a dozen rows
  float x[NX][8];
#pragma unroll
  for (int p = 0; p < NX; ++p)
    if (p < nsu) x_of<XT>(xs + p * SU, x[p]);
  int slot = 0;
#pragma unroll 1
  for (int k = 0; k < pl.n; ++k) {
    if (!mbar_wait(st.bars + slot, (st.parity >> slot) & 1u)) {
      if (lane == 0) { *st.dead = 1; atomicCAS(st.status, 0, ST_TIMEOUT_COPY); }
      break;
    }
    st.parity ^= 1u << slot;
    st.pending &= ~(1u << slot);
    const uint8_t* src = st.base + (size_t)slot * rb;
    float acc = 0.f;
#pragma unroll
    for (int p = 0; p < NX; ++p)
      if (p < nsu) acc += su_dot<FMT>(su_word<FMT>(src + (size_t)p * SB), src + (size_t)p * SB, x[p]);
    for (int p = NX; p < nsu; ++p) {
      float y[8];
      x_of<XT>(xs + p * SU, y);
      acc += su_dot<FMT>(su_word<FMT>(src + (size_t)p * SB), src + (size_t)p * SB, y);
    }
    fence_proxy_async();
    head_issue<FMT>(a, pl, st, items, k + items, k + items + 1, slot);
    acc = warp_sum(acc);
    if (lane == 0) a.logits[blockIdx.x + (pl.first + k * pl.stride) * (int)gridDim.x] = acc;
    if (++slot == items) slot = 0;
  }
}

// ------------------------------------------------------------------------------------------------ the kernel
// The L1 beside the staged rows holds a twentieth of 512 threads' local memory, so a register that is spilled comes back from L2, in
// the middle of a chain of dependent steps.  What is the same for a whole step is therefore kept in shared memory and read where it is used: a
// thread carries the layer, the epoch and the state of its copies from phase to phase, and nothing else.
template <int FMT, typename XT>
__global__ void __launch_bounds__(THREADS, 1) decode_mega_kernel(const __grid_constant__ gb_mega_args a) {
  extern __shared__ __align__(16) uint8_t dyn[];
  __shared__ Smem sm;
  __shared__ __align__(8) uint64_t bars[WARPS * MAXI];         // of the warps' staging slices
  // the router rows of a layer (ne x d fp32, the same for every token) are staged a phase and a half ahead too, into an area of their own
  __shared__ __align__(8) uint64_t rbar;
  const int warp_id = threadIdx.x >> 5;
  XT* xs = reinterpret_cast<XT*>(dyn);
  uint8_t* router_area = dyn + a.at_stage;
  float* amerge = reinterpret_cast<float*>(dyn + a.at_merge);
  Stage st{dyn + a.at_rows + (size_t)warp_id * a.stage_bytes, bars + warp_id * MAXI, 0u, 0u, &sm.dead, a.status};
  const Gate gate{a.words, sm.base, sm.warps, &sm.dead, a.status};
  unsigned long long* prof = (blockIdx.x == 0 && threadIdx.x == 0) ? a.prof : nullptr;    // thirteen points of a layer, the start and the end
  auto mark = [&]() { if (prof) *prof++ = globaltimer_ns(); };
  auto n_slots_of = [&]() { return a.ne > 0 ? a.top_k + (a.shared ? 1 : 0) : 1; };
  auto row_bytes = [](int values) { return (long long)(values / SU) * Fmt<FMT>::bytes; };
  uint32_t epoch, rparity = 0;
  bool rpending = false, ok;
  {
    const int d = a.d, qd = a.H * a.hd, E = a.E, slots = n_slots_of(), grid = gridDim.x;
    GridBar gb{a.sync, a.status, &sm.dead, a.sync[1] + gridDim.x};
    epoch = a.sync[3];                           // layer li of this launch exchanges words of epoch sync[3] + 1 + li
    mark();
    if (threadIdx.x == 0) {
      sm.dead = 0;
      mbar_init(&rbar, 1);
      const Words at = words_of(a);
      sm.wx = a.words + at.x;
      sm.wmid = a.words + at.xmid;
      sm.wpart = a.words + at.part;
      sm.wqkv = reinterpret_cast<uint32_t*>(a.words + at.qkv);
      sm.watt = reinterpret_cast<uint32_t*>(a.words + at.att);
      sm.wact = reinterpret_cast<uint32_t*>(a.words + at.act);
      sm.seq = a.state[0];
      sm.pos = a.pos[0];
      // number of cache splits: 64 slots per CTA (one trip: four a warp, side by side), more where the grid or the scratch holds no more CTAs.  The splits
      // are merged by all CTAs together, so more of them cost little: 3001 slots, 26 layers, 4 bits, 24 splits 665 us, 37 655
      const int n = min(a.cap, sm.seq.cache_len + 1);
      sm.splits = max(1, min(min(a.max_splits, grid / a.KV), (n + 63) / 64));
    }
    if (threadIdx.x < VECS) {                    // nothing arrives before the barrier below
      sm.base[threadIdx.x] = *reinterpret_cast<volatile unsigned*>(a.words + threadIdx.x * COUNT_WORDS);
      sm.warps[threadIdx.x] = 0;
    }
    if ((threadIdx.x & 31) == 0) {
      sm.plan[0][warp_id] = make_plan(qd + 2 * a.KV * a.hd, d / SU, d / SU);
      sm.plan[1][warp_id] = make_plan(d, qd / SU, qd / SU);
      sm.plan[2][warp_id] = make_plan(slots * E, 2 * (d / SU), d / SU);
      sm.plan[3][warp_id] = make_plan(d, slots * (E / SU), E / SU);
      for (int k = 0; k < MAXI; ++k) mbar_init(st.bars + k, 1);
      fence_barrier_init();
    }
    for (int i = threadIdx.x; i < MAXI * WARPS; i += THREADS) {
      const int o = blockIdx.x + i * grid;
      sm.d_slot[i] = (unsigned char)(o / E);
      sm.d_row[i] = o % E;
    }
    constexpr int LAYER_WORDS = sizeof(gb_mega_layer) / 8;
    if (threadIdx.x < LAYER_WORDS)
      reinterpret_cast<unsigned long long*>(&sm.layer[0])[threadIdx.x] = reinterpret_cast<const unsigned long long*>(a.layers)[threadIdx.x];
    __syncthreads();
    // rows of the first projection of the first layer: nothing to wait for
    Phase ph{reinterpret_cast<const uint8_t*>(sm.layer[0].wqkv), nullptr, nullptr, d / SU};
    stream_issue<FMT, 1>(ph, sm.plan[0][warp_id], 1, st, [&](int, int o) { return o * row_bytes(a.d); });
    int tok = a.cur_tok[0];
    if (tok < 0 || tok >= a.V) tok = 0;
    if ((int)threadIdx.x < sm.plan[1][0].rows) sm.res[0][threadIdx.x] = a.emb[(size_t)tok * d + blockIdx.x + threadIdx.x * grid];
    // Every CTA has read the sequence's state and the counts before one of them can move on.
    ok = grid_sync(gb);
  }
  for (int li = 0; li < a.n_layers && ok; ++li) {
    const gb_mega_layer& L = sm.layer[li & 1];
    const bool last = li + 1 == a.n_layers;
    // ---- A: RMSNorm + fused QKV projection; then this warp's rows of wo start to arrive
    {
      int tok = 0;
      if (li == 0) { tok = a.cur_tok[0]; if (tok < 0 || tok >= a.V) tok = 0; }
      block_norm<XT>(gate, V_X, li * gridDim.x, sm.wx, li == 0 ? a.emb + (size_t)tok * a.d : nullptr, epoch, L.attn_norm, xs, a.d, a.eps, sm.nred);
      if (sm.dead) { ok = false; break; }
      ++epoch;
      mark();
      constexpr int LAYER_WORDS = sizeof(gb_mega_layer) / 8;
      if (!last && threadIdx.x < LAYER_WORDS)      // the next layer's pointers; that half was last read a layer ago
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(reinterpret_cast<unsigned long long*>(&sm.layer[(li + 1) & 1]) + threadIdx.x)),
                     "l"(reinterpret_cast<const unsigned long long*>(a.layers + li + 1) + threadIdx.x)
                     : "memory");
      Phase ph{reinterpret_cast<const uint8_t*>(L.wqkv), nullptr, nullptr, a.d / SU};
      stream_run<FMT, XT, false, false>(ph, sm.plan[0][warp_id], xs, st, sm.red, gate, V_QKV, [&](int, int o, float v, float) { put_16<XT>(sm.wqkv + o, Cvt<XT>::from_f(v), epoch); });
      Phase phC{reinterpret_cast<const uint8_t*>(L.wo), nullptr, nullptr, a.H * a.hd / SU};
      stream_issue<FMT, 1>(phC, sm.plan[1][warp_id], 1, st, [&](int, int o) { return o * row_bytes(a.H * a.hd); });
      const int S = sm.splits;
      if ((int)blockIdx.x < a.KV * S) {
        // this CTA's slice of the cache is known before the queries are: ask L2 for its rows now (a cache row was last
        // touched a token ago, 1.2 GB of weights back, so it would otherwise come from DRAM inside the walk)
        const int kvh = blockIdx.x % a.KV, split = blockIdx.x / a.KV, hd = a.hd;
        const int n = min(a.cap, sm.seq.cache_len + 1), per = (n + S - 1) / S;
        const int lo = split * per, hi = min(n, lo + per);
        for (int j = lo + (int)threadIdx.x; j < hi; j += THREADS)
          for (int c = 0; c < hd; c += 64) {                   // one 128-byte line per 64 values
            const size_t at = ((size_t)j * a.KV + kvh) * hd + c;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const XT*>(L.cache_k) + at));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const XT*>(L.cache_v) + at));
          }
      }
      const uint32_t router_bytes = a.ne > 0 ? (uint32_t)a.ne * (uint32_t)a.d * 4u : 0u;
      if (router_bytes > 0 && router_bytes <= (uint32_t)ROUTER_AREA) {
        if (threadIdx.x == THREADS - 32) {       // every thread's reads of the previous layer's rows lie barriers back
          fence_proxy_async();
          mbar_arrive_expect_tx(&rbar, router_bytes);
          bulk_g2s(smem_u32(router_area), L.router, router_bytes, smem_u32(&rbar));
        }
        rpending = true;
      }
    }
    mark();
    // ---- B: attention over the cache, merge of its splits
    if (a.hd == 64) {
      switch (min(4, a.H / a.KV)) {
        case 1: attention_phase<XT, 1, 8>(a, L, sm, amerge, epoch, gate, (li + 1) * gridDim.x, prof); break;
        case 2: attention_phase<XT, 2, 8>(a, L, sm, amerge, epoch, gate, (li + 1) * gridDim.x, prof); break;
        case 3: attention_phase<XT, 3, 8>(a, L, sm, amerge, epoch, gate, (li + 1) * gridDim.x, prof); break;
        default: attention_phase<XT, 4, 8>(a, L, sm, amerge, epoch, gate, (li + 1) * gridDim.x, prof); break;
      }
    } else {
      attention_phase<XT, 4, 0>(a, L, sm, amerge, epoch, gate, (li + 1) * gridDim.x, prof);
    }
    merge_phase<XT>(a, sm, epoch, gate, (li + 1) * a.KV * sm.splits);
    mark();
    // ---- C: output projection + residual
    gather16<XT, 1>(gate, V_ATT, (li + 1) * gridDim.x, sm.watt, a.H * a.hd, epoch, xs);
    if (sm.dead) { ok = false; break; }
    mark();
    {
      Phase phC{reinterpret_cast<const uint8_t*>(L.wo), nullptr, nullptr, a.H * a.hd / SU};
      stream_run<FMT, XT, false, false>(phC, sm.plan[1][warp_id], xs, st, sm.red, gate, V_MID, [&](int i, int o, float v, float) {
        v += sm.res[0][i];
        sm.res[1][i] = v;
        put_f32(sm.wmid + o, v, epoch);
      });
    }
    mark();
    // ---- D: RMSNorm + router + gate/up of the chosen experts + SwiGLU; then the down-projection rows start to arrive
    {
      block_norm<XT>(gate, V_MID, (li + 1) * gridDim.x, sm.wmid, nullptr, epoch, L.ffn_norm, xs, a.d, a.eps, sm.nred);
      if (sm.dead) { ok = false; break; }
      mark();
      if (rpending) {
        if (!mbar_wait(&rbar, rparity)) {
          if (threadIdx.x == 0) { sm.dead = 1; atomicCAS(a.status, 0, ST_TIMEOUT_COPY); }
        }
        rparity ^= 1u;
      }
      if (rpending) route_phase<XT, true>(a, L, xs, sm, row_bytes(a.E), reinterpret_cast<const float*>(router_area));
      else route_phase<XT, false>(a, L, xs, sm, row_bytes(a.E), L.router);
      rpending = false;
      mark();
      Phase ph{reinterpret_cast<const uint8_t*>(L.wg), sm.off_gu, nullptr, a.d / SU};
      stream_issue<FMT, 2>(ph, sm.plan[2][warp_id], 2, st, [&](int k, int) {
        const int i = sm.plan[2][warp_id].first + k * sm.plan[2][warp_id].stride;
        return ((long long)sm.esel[sm.d_slot[i]] * a.E + sm.d_row[i]) * row_bytes(a.d);
      });
      stream_run<FMT, XT, true, false>(ph, sm.plan[2][warp_id], xs, st, sm.red, gate, V_ACT,
                          [&](int, int o, float g, float u) { put_16<XT>(sm.wact + o, Cvt<XT>::from_f(g / (1.f + __expf(-g)) * u), epoch); });
    }
    {
      const int slots = n_slots_of(), nsu_E = a.E / SU;
      Phase phE{reinterpret_cast<const uint8_t*>(L.wd), sm.off_e, sm.wsel, nsu_E};
      stream_issue<FMT, 0>(phE, sm.plan[3][warp_id], slots, st, [&](int, int o) { return o * row_bytes(a.E); });
      mark();
      asm volatile("cp.async.wait_all;" ::: "memory");         // the next layer's pointers, before the barriers of gather16
      // ---- E: down projection of the chosen experts, weighted, + residual; then the next layer's QKV rows
      gather16<XT, 4>(gate, V_ACT, (li + 1) * gridDim.x, sm.wact, slots * a.E, epoch, xs);
      if (sm.dead) { ok = false; break; }
      mark();
      stream_run<FMT, XT, false, true>(phE, sm.plan[3][warp_id], xs, st, sm.red, gate, V_X, [&](int i, int o, float v, float) {
        v += sm.res[1][i];
        sm.res[0][i] = v;
        put_f32(sm.wx + o, v, epoch);
      });
    }
    if (!last) {
      Phase ph{reinterpret_cast<const uint8_t*>(sm.layer[(li + 1) & 1].wqkv), nullptr, nullptr, a.d / SU};
      stream_issue<FMT, 1>(ph, sm.plan[0][warp_id], 1, st, [&](int, int o) { return o * row_bytes(a.d); });
    }
    mark();
  }
  if (ok) {
    // ---- final norm + vocabulary projection, whose first rows start to arrive
    {
      const Plan plH = make_plan(a.V, a.d / SU, a.d / SU);
      if (a.head_fmt == FMT) head_issue<FMT>(a, plH, st, head_items<FMT>(a), 0, head_items<FMT>(a));
      else if (a.head_fmt == GB_W_F16) head_issue<GB_W_F16>(a, plH, st, head_items<GB_W_F16>(a), 0, head_items<GB_W_F16>(a));
      else head_issue<GB_W_BF16>(a, plH, st, head_items<GB_W_BF16>(a), 0, head_items<GB_W_BF16>(a));
    }
    block_norm<XT>(gate, V_X, a.n_layers * gridDim.x, sm.wx, nullptr, epoch, a.final_norm, xs, a.d, a.eps, sm.nred);
    if (!sm.dead) {
      if (a.head_fmt == FMT) head_phase<FMT, XT>(a, xs, st);
      else if (a.head_fmt == GB_W_F16) head_phase<GB_W_F16, XT>(a, xs, st);
      else head_phase<GB_W_BF16, XT>(a, xs, st);
    }
  }
  // a step that was given up: the copies this warp still has in flight must land (or run out of time) before the
  // shared memory they target goes away
  for (int k = 0; k < MAXI; ++k)
    if (st.pending >> k & 1u) (void)mbar_wait(st.bars + k, (st.parity >> k) & 1u);
  if (rpending) (void)mbar_wait(&rbar, rparity);
  asm volatile("cp.async.wait_all;" ::: "memory");
  mark();
  // ---- bookkeeping: the last CTA out records where the counts stand; CTA 0 advances the sequence state
  __syncthreads();
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0 && ok && !sm.dead) {
      gb_seq_state s = a.state[0];
      if (s.cache_len < a.cap) s.cache_len += 1;
      else s.ring_start = (s.ring_start + 1) % max(1, a.cap - a.pinned);
      s.abs_pos += 1;
      a.state[0] = s;
      a.pos[0] = s.abs_pos;
    }
    __threadfence();
    const unsigned t = atomicAdd(&a.sync[2], 1u);
    if (t == gridDim.x - 1) {
      a.sync[1] = atomicAdd(&a.sync[0], 0u);
      a.sync[2] = 0u;
      a.sync[3] += (unsigned)a.n_layers;
      __threadfence();
    }
  }
}

// Dynamic shared memory: activations, router rows, merge of the warps' attention, staged rows.
static size_t dyn_bytes(gb_mega_args& a, long long stage_per_warp) {
  const int slots = a.ne > 0 ? a.top_k + (a.shared ? 1 : 0) : 1;
  const int xs_vals = std::max(std::max(a.d, a.H * a.hd), slots * a.E);
  a.at_stage = (int)(((size_t)xs_vals * 2 + 15) & ~(size_t)15);
  a.at_merge = a.at_stage + ROUTER_AREA;
  a.at_rows = a.at_merge + (WARPS * 8 + WARPS * 4 * a.hd) * 4;
  return (size_t)a.at_rows + (size_t)WARPS * (size_t)stage_per_warp;
}

static int su_bytes_of(int fmt) {
  switch (fmt) {
    case GB_W_F16: case GB_W_BF16: return 512;
    case GB_W_GGML_Q8_0: case GB_W_Q8_64: return 272;
    case GB_W_Q4_0: return 144;
    default: return 160;
  }
}

// Bytes of one warp's staging slice (the largest of the four layer phases and of the vocabulary ring), or -1 when a
// warp would have to stage more than MAXI outputs at once.
static long long stage_bytes_per_warp(gb_mega_args& a, int grid, int su_bytes) {
  const int slots = a.ne > 0 ? a.top_k + (a.shared ? 1 : 0) : 1;
  const int nsu_d = a.d / SU, nsu_q = a.H * a.hd / SU, nsu_E = a.E / SU;
  const long long n[4] = {(long long)(a.H + 2 * a.KV) * a.hd, a.d, (long long)slots * a.E, a.d};
  const int P[4] = {nsu_d, nsu_q, 2 * nsu_d, slots * nsu_E};
  long long need = 16;
  for (int i = 0; i < 4; ++i) {
    int items = 0;
    need = std::max(need, stage_need(n[i], P[i], grid, su_bytes, &items));
    if (items > MAXI) return -1;
  }
  need = (need + 15) & ~15ll;
  // room for a ring of up to MAXI rows of the vocabulary projection, as far as the shared memory allows
  const long long head_row = (long long)nsu_d * su_bytes_of(a.head_fmt);
  const long long head_rows = ((long long)a.V + (long long)grid * WARPS - 1) / ((long long)grid * WARPS);
  for (long long r = std::min<long long>(MAXI, head_rows); r >= 1; --r)
    if (dyn_bytes(a, std::max(need, r * head_row)) <= (size_t)MAX_DYN) { need = std::max(need, r * head_row); break; }
  return need;
}

}  // namespace mg
}  // namespace gb

using namespace gb;

extern "C" int gb_decode_mega_ok(const gb_mega_args* a) {
  if (!a || a->n_layers <= 0) return -1;
  if (a->d % mg::SU || (a->H * a->hd) % mg::SU || a->E % mg::SU) return -2;          // whole super-units per stored row
  if (a->hd != 32 && a->hd != 64 && a->hd != 128) return -3;
  if (a->KV <= 0 || a->H % a->KV || a->H > mg::MAX_HEADS) return -3;
  if (a->ne > 64 || a->ne < 0 || (a->ne > 0 && (a->top_k < 1 || a->top_k > 8 || a->top_k > a->ne))) return -4;
  if (a->fmt < GB_W_F16 || a->fmt > GB_W_Q4_1) return -5;
  if (a->head_fmt != a->fmt && a->head_fmt != GB_W_F16 && a->head_fmt != GB_W_BF16) return -5;
  if (a->d > 8 * mg::THREADS || a->max_splits > 64) return -6;
  if (a->max_splits < 1 || a->cap < 1 || a->pinned < 0 || a->pinned >= a->cap) return -6;
  const int grid = gb_decode_mega_grid();
  if (grid <= 0 || grid < a->KV || a->d < grid) return -9;           // a.d < grid: a CTA without rows would not be waited for
  gb_mega_args b = *a;
  const long long per_warp = mg::stage_bytes_per_warp(b, grid, mg::su_bytes_of(a->fmt));
  if (per_warp < 0 || per_warp < (long long)(a->d / mg::SU) * mg::su_bytes_of(a->head_fmt) || mg::dyn_bytes(b, per_warp) > mg::MAX_DYN) return -7;
  return 0;
}

// Number of CTAs of the launch: one per SM (a cooperative launch needs all of them resident at once).
extern "C" int gb_decode_mega_grid() {
  static const int n = []() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
  }();
  return n;
}

template <int FMT, typename XT>
static int launch_mega(const gb_mega_args& a_in, cudaStream_t st) {
  auto kern = mg::decode_mega_kernel<FMT, XT>;
  const int grid = gb_decode_mega_grid();
  if (grid <= 0 || grid < a_in.KV) return -9;
  gb_mega_args a = a_in;
  a.stage_bytes = (int)mg::stage_bytes_per_warp(a, grid, mg::Fmt<FMT>::bytes);
  const size_t smem = mg::dyn_bytes(a, a.stage_bytes);
  static bool attr_done = false;                 // one process drives one device
  if (!attr_done) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, mg::MAX_DYN) != cudaSuccess) { (void)cudaGetLastError(); return -8; }
    attr_done = true;
  }
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(mg::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return -(1000 + (int)e); }
  return 0;
}

extern "C" long long gb_decode_mega_words(const gb_mega_args* a) { return mg::words_of(*a).total; }

extern "C" int gb_decode_mega(const gb_mega_args* a, cudaStream_t st) {
  const int rc = gb_decode_mega_ok(a);
  if (rc) return rc;
#define GB_MEGA_CASE(F)                                                    \
  case F:                                                                  \
    return a->is_bf16 ? launch_mega<F, __nv_bfloat16>(*a, st) : launch_mega<F, __half>(*a, st);
  switch (a->fmt) {
    GB_MEGA_CASE(GB_W_F16)
    GB_MEGA_CASE(GB_W_BF16)
    GB_MEGA_CASE(GB_W_GGML_Q8_0)
    GB_MEGA_CASE(GB_W_Q4_0)
    GB_MEGA_CASE(GB_W_Q8_64)
    GB_MEGA_CASE(GB_W_Q4_1)
  }
#undef GB_MEGA_CASE
  return -5;
}
