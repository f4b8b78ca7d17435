// Paged GQA prefill / chunked-prefill attention and multi-head latent attention prefill on tcgen05 + TMEM, fed by TMA
// (head_dim 128, 16-bit).  The reference's `prefill_attention` call (v1/attention/backends/kunlun_attn.py:805-947) and the
// compute-friendly prefill form of latent attention (v1/attention/backends/mla/common.py:1782-1843).
//
// A persistent CTA works on two 128-row query tiles ("streams") that read the same K / V tiles: two query heads of one
// key / value head over the same rows, or, where heads do not share keys, 256 consecutive rows of one head.  Per
// 128-key tile and stream:
//     S[128 rows, 128 keys]  = Q . K_tile^T                 (Q, K in shared memory)
//     O[128 rows, 128 dims] += P[128 rows, 128 keys] . V    (P in TMEM, over the columns of S; V in shared memory)
// TMEM holds S0, S1, O0, O1 (4 x 128 columns).  Each stream has four softmax warps (thread = row) that read S, write P
// back in 16 bits over it and hand it over in two halves of 64 keys; the tensor core works on one stream while the
// other one is in its softmax.  A stream's products are issued in the order P.V(i), S(i + 1), so the arrival of
// S(i + 1) also says that O holds P.V(i): the (rare, lazy) rescale of O needs no barrier of its own.
// What bounds it: per tile the tensor core needs 1024 cycles (2 x 128^3 products), the special-function units 1024 (128 x
// 128 exponentials at 16 a cycle); with two streams both are shared by two tiles.  P goes through TMEM because a
// product with both operands in shared memory reads 64 KB for 512 cycles, all that shared memory delivers.
// 384 threads: warp 0 TMA producer, warp 1 MMA issuer, warps 4-7 / 8-11 softmax and epilogue of stream 0 / 1.  The grid has a CTA per
// work item, in descending order of row blocks, and a CTA that is done cancels the launch of the next pending one and takes its
// item (cluster launch control): items of one call differ a hundredfold where prompts or their contexts do, which a fixed
// distribution cannot balance.  us with items dealt out in turn, and now: 37 requests of 16 heads, one of 4096 tokens, the others
// 16: 1031 and 130 (425 with one tile a CTA); 512 tokens each, one behind 16000: 919 and 297 (386); 11 ragged prompts 40 and 31; 4 x
// 2048 tokens 173 and 170.  TMA loads carry no cluster multicast.  Every wait is bounded; on time-out
// the status word is set and the CTA unwinds.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include "../api.h"
#include "../common/launch.cuh"
#include "../common/ptx.cuh"
#include "../gemm/gemm_common.cuh"

namespace b200 {
namespace pair {

constexpr int kThreads = 3 * 128;
// Registers a thread of the first warpgroup (TMA, MMA, two idle warps) keeps and one of the softmax warpgroups gets: the
// launch brings 168 x 384 = 64512, and the split takes 128 x (104 + 200 + 200) = 64512.
constexpr int kRegsIssue = 104, kRegsSoft = 200;
constexpr int kTile = 128, kPage = 64, kD = 128;
constexpr int kBlockBytes = kTile * 128;       // one 64-dim block of a 128-row operand tile
constexpr int kVBytes = kPage * 2 * 128;       // V of one 64-key page: [2 dim blocks][64 keys][128 B]
constexpr int kTmemCols = 512;
constexpr float kMaxSlack = 8.f;
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

template <bool kMla> struct Cfg {
  static constexpr int kQBlocks = kMla ? 3 : 2;                 // 64-dim blocks of q / k
  static constexpr int kKBytes = kQBlocks * kBlockBytes;        // one Q tile or one K stage
  static constexpr int kKStages = kMla ? 2 : 3;
  static constexpr int kVStages = kMla ? 2 : 4;                 // in pages of 64 keys
  static constexpr size_t kSmem = 1024 + (size_t)(2 + kKStages) * kKBytes + (size_t)kVStages * kVBytes + 512;
};

struct Params {
  void* out;                // [T, Hq, 128]
  float* lse;               // [T, Hq] natural-log sum-exp (optional)
  const int* block_tables;  // [B, max_blocks]
  const int* seq_lens;
  const int* qsl;
  const int* kv_starts;     // latent form: first key row of each request in the contiguous K / V tensors
  const float* sinks;       // [Hq] or null
  const void* gate;         // [T, >= Hq] in the output's type, or null
  int64_t gate_stride;
  int* status;
  int Hq, Hkv, block_size, max_blocks, window, causal;
  int units;                // head pairs (by_heads) or heads
  int by_heads;             // streams are two heads over the same rows, otherwise two row tiles of one head
  int single;               // one stream only: as many CTAs as there are tiles
  int row_blocks, B;
  int take;                // CTAs may be pending: whoever is done takes their items
  int64_t num_blocks;
  float scale_log2;
};

__device__ __forceinline__ void tmem_ld_x32_p(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_x32_p(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_x16_p(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; issued by ONE thread.  A: lane = row, two 16-bit elements of K per column.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// two fp32 values in one 64-bit register: a fused multiply-add or an add of both is one instruction
__device__ __forceinline__ uint64_t f2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unf2(uint64_t r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// 2^x on the special-function unit (-inf -> 0)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T> struct FmtOf;
template <> struct FmtOf<__nv_bfloat16> { static constexpr uint32_t v = 1; };
template <> struct FmtOf<__half> { static constexpr uint32_t v = 0; };
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// One work item: what the two streams of a CTA share and their own rows.
struct Item {
  int req, qs, q_len, ctx, seq_len, kv_begin;
  int head[2], row0[2], rows[2], n[2];   // per stream: head, first row within the request, valid rows, key tiles
  int n_max;
};

// Item `idx` of the call.  Items are ordered by descending row block, so by descending number of key tiles for prompts of one length.
template <bool kMla>
__device__ __forceinline__ void get_item(const Params& p, int idx, Item& it) {
  const int per = p.B * p.units, rb = p.row_blocks - 1 - idx / per, rem = idx % per;
  it.req = rem / p.units;
  const int u = rem % p.units;
  it.qs = p.qsl[it.req];
  it.q_len = p.qsl[it.req + 1] - it.qs;
  it.seq_len = p.seq_lens[it.req];
  // not causal: every row sees all of the request's keys - as if it sat far behind them
  it.ctx = (kMla && !p.causal) ? (1 << 29) : it.seq_len - it.q_len;
  const int step = (p.by_heads || p.single) ? kTile : 2 * kTile;
  it.n_max = 0;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    it.head[s] = p.by_heads ? 2 * u + s : u;
    it.row0[s] = rb * step + (p.by_heads ? 0 : s * kTile);
    it.rows[s] = (s == 1 && p.single) ? 0 : max(0, min(kTile, it.q_len - it.row0[s]));
  }
  // a window hides everything in front of the first row's first visible key (whole tiles of it)
  it.kv_begin = p.window > 0 ? max(0, it.ctx + it.row0[0] - p.window + 1) / kTile * kTile : 0;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    // keys visible to the tile end with the position of its last row
    const int kv_end = it.rows[s] > 0 ? min(it.seq_len, it.ctx + it.row0[s] + it.rows[s]) : 0;
    it.n[s] = max(0, (kv_end - it.kv_begin + kTile - 1) / kTile);
    it.n_max = max(it.n_max, it.n[s]);
  }
}

// Asks for the index of a CTA of this grid that has not been started, which then never will be: 16 bytes at `dst`, complete_tx on `bar`.
__device__ __forceinline__ void ask_for_cta(uint32_t dst, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(dst),
               "r"(smem_u32(bar)) : "memory");
}
// The answer: a CTA's index, or -1 when all have been started or taken (then no further question may be asked).
__device__ __forceinline__ int taken_cta(uint32_t src) {
  uint32_t ok, x = 0;
  asm volatile(
      "{\n\t.reg .b128 r;\n\t.reg .b64 lo, hi;\n\t.reg .pred p;\n\t"
      "ld.shared.v2.b64 {lo, hi}, [%2];\n\t"
      "mov.b128 r, {lo, hi};\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
      : "=r"(ok), "=r"(x) : "r"(src) : "memory");
  return ok ? (int)x : -1;
}

template <typename T, bool kMla>
__global__ void __launch_bounds__(kThreads, 1)
prefill_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                    const __grid_constant__ CUtensorMap tmKpe, const __grid_constant__ Params p) {
  using C = Cfg<kMla>;
  constexpr int kQBlocks = C::kQBlocks, kKBytes = C::kKBytes, kKStages = C::kKStages, kVStages = C::kVStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                  // [2 streams][kQBlocks dim blocks][128 rows][128 B]
  uint8_t* sK = sQ + 2 * kKBytes;                      // [kKStages][kQBlocks dim blocks][128 keys][128 B]
  uint8_t* sV = sK + kKStages * kKBytes;               // [kVStages][2 dim blocks][64 keys][128 B]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kVStages * kVBytes);
  uint64_t* q_full = bars;              // one phase per item
  uint64_t* q_empty = bars + 1;         // the item's last S has been computed
  uint64_t* k_full = bars + 2;          // [3]
  uint64_t* k_empty = bars + 5;         // [3] both streams' S of the tile have been computed
  uint64_t* v_full = bars + 8;          // [4]
  uint64_t* v_empty = bars + 12;        // [4]
  uint64_t* s_full = bars + 16;         // [2 streams]
  uint64_t* p_ready = bars + 18;        // [2 streams][2 halves] one arrival per softmax warp
  uint64_t* o_final = bars + 22;        // [2 streams] one phase per item with work for the stream
  // answers about the next item: question k uses slot k & 1
  uint64_t* next_full = bars + 24;      // [2]
  uint64_t* next_empty = bars + 26;     // [2] read by the MMA thread and the eight softmax warps
  const uint32_t next_at = smem_u32(bars + 28);   // [2] x 16 bytes
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 32);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Abort ab{p.status, abort_flag};
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int b = 0; b < kKStages; ++b) { mbar_init(&k_full[b], 1); mbar_init(&k_empty[b], 1); }
    for (int b = 0; b < kVStages; ++b) { mbar_init(&v_full[b], 1); mbar_init(&v_empty[b], 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&o_final[s], 1);
      for (int h = 0; h < 2; ++h) mbar_init(&p_ready[s * 2 + h], 4);
      mbar_init(&next_full[s], 1);
      mbar_init(&next_empty[s], 9);
    }
    mbar_fence_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmKV);
    if (kMla) prefetch_tmap(&tmKpe);
    griddep_launch();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  griddep_wait();   // q, the lengths and this step's cache rows come from the preceding kernels
  Item it;
  // MMA thread, softmax warps: answer k.  -1: there is no further item, or a wait gave up (then `ok` is false as well).
  auto next_item = [&](int k, bool whole_warp, bool& ok) {
    if (!p.take) return -1;
    ok = wait_or_abort(&next_full[k & 1], (k >> 1) & 1, ab, 829);
    if (whole_warp) ok = !__any_sync(0xffffffffu, !ok);
    if (!ok) return -1;
    const int idx = taken_cta(next_at + 16 * (k & 1));
    fence_proxy_async_smem();           // read before the next answer is written here
    if (whole_warp) __syncwarp();
    if (!whole_warp || lane == 0) mbar_arrive(&next_empty[k & 1]);
    return idx;
  };

  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int kc = 0, vc = 0, qc = 0, asked = 0;    // K tiles, V pages and items issued, questions asked so far
      bool ok = true;
      // asked when the item's last loads are due: late enough that a CTA does not hold an item it cannot start, early enough that the
      // answer is there before the last tiles have been worked on
      auto ask = [&]() {
        const int b = asked & 1;
        if (asked >= 2 && !wait_or_abort(&next_empty[b], ((asked >> 1) - 1) & 1, ab, 830)) return false;
        mbar_expect_tx(&next_full[b], 16);
        ask_for_cta(next_at + 16 * b, &next_full[b]);
        ++asked;
        return true;
      };
      for (int idx = blockIdx.x; ok && idx >= 0;) {
        get_item<kMla>(p, idx, it);
        const int n_max = it.n_max;
        if (n_max > 0) {
          if (qc > 0 && !wait_or_abort(q_empty, (qc - 1) & 1, ab, 820)) { ok = false; break; }
          mbar_expect_tx(q_full, kKBytes * ((it.n[0] > 0) + (it.n[1] > 0)));
#pragma unroll
          for (int s = 0; s < 2; ++s)
            if (it.n[s] > 0) {
#pragma unroll
              for (int h = 0; h < kQBlocks; ++h)
                tma_load_2d(sQ + s * kKBytes + h * kBlockBytes, &tmQ, q_full, it.head[s] * (kQBlocks * 64) + h * 64,
                            it.qs + it.row0[s]);
            }
          ++qc;
          const int* bt = kMla ? nullptr : p.block_tables + (int64_t)it.req * p.max_blocks;
          const int kvh = it.head[0] / (p.Hq / p.Hkv), kv_row0 = kMla ? p.kv_starts[it.req] : 0;
          const int key_end = min(it.seq_len, it.kv_begin + n_max * kTile);
          // cache row of a key's page (paged form): masked keys read any initialised page
          auto page_row = [&](int key) -> int64_t {
            const int bi = key / p.block_size;
            int64_t blk = (key < key_end && bi < p.max_blocks) ? bt[bi] : 0;
            if (blk < 0 || blk >= p.num_blocks) blk = 0;
            return ((blk * 2) * p.Hkv + kvh) * p.block_size + (key % p.block_size);
          };
          for (int j = 0; ok && j <= n_max; ++j) {      // K(0), K(1), V(0), K(2), V(1), ...
            if (j == n_max - 1 && p.take && !ask()) { ok = false; break; }
            if (j < n_max) {
              const int st = kc % kKStages, use = kc / kKStages;
              if (use > 0 && !wait_or_abort(&k_empty[st], (use - 1) & 1, ab, 821)) { ok = false; break; }
              mbar_expect_tx(&k_full[st], kKBytes);
#pragma unroll
              for (int pg = 0; pg < kTile / kPage; ++pg) {
                const int key = it.kv_begin + j * kTile + pg * kPage;
                uint8_t* dst = sK + st * kKBytes + pg * (kPage * 128);
                if constexpr (kMla) {
                  // rows past the request's keys belong to the next request or lie outside the tensor (zero fill): masked
#pragma unroll
                  for (int h = 0; h < 2; ++h)
                    tma_load_2d(dst + h * kBlockBytes, &tmKV, &k_full[st], it.head[0] * 256 + h * 64, kv_row0 + key);
                  tma_load_2d(dst + 2 * kBlockBytes, &tmKpe, &k_full[st], 0, kv_row0 + key);
                } else {
                  const int64_t row = page_row(key);
#pragma unroll
                  for (int h = 0; h < 2; ++h) tma_load_2d(dst + h * kBlockBytes, &tmKV, &k_full[st], h * 64, (int)row);
                }
              }
              ++kc;
            }
            if (j >= 1) {
#pragma unroll
              for (int pg = 0; pg < kTile / kPage; ++pg) {
                const int st = vc % kVStages, use = vc / kVStages;
                if (use > 0 && !wait_or_abort(&v_empty[st], (use - 1) & 1, ab, 822)) { ok = false; break; }
                mbar_expect_tx(&v_full[st], kVBytes);
                const int key = it.kv_begin + (j - 1) * kTile + pg * kPage;
                uint8_t* dst = sV + st * kVBytes;
                if constexpr (kMla) {
#pragma unroll
                  for (int h = 0; h < 2; ++h)
                    tma_load_2d(dst + h * (kVBytes / 2), &tmKV, &v_full[st], it.head[0] * 256 + 128 + h * 64, kv_row0 + key);
                } else {
                  const int64_t row = page_row(key) + (int64_t)p.Hkv * p.block_size;
#pragma unroll
                  for (int h = 0; h < 2; ++h) tma_load_2d(dst + h * (kVBytes / 2), &tmKV, &v_full[st], h * 64, (int)row);
                }
                ++vc;
              }
            }
          }
        } else if (p.take) {
          ok = ask();
        }
        if (!p.take) break;
        if (!ok || !wait_or_abort(&next_full[(asked - 1) & 1], ((asked - 1) >> 1) & 1, ab, 829)) { ok = false; break; }
        idx = taken_cta(next_at + 16 * ((asked - 1) & 1));
        fence_proxy_async_smem();
      }
      if (!ok) {   // let the copies in flight land before the CTA's shared memory goes away (bounded)
        auto drain = [](uint64_t* bar, uint32_t parity) {
          for (uint32_t q = 0; q < (1u << 16); ++q)
            if (mbar_try_wait(bar, parity)) break;
        };
        if (qc > 0) drain(q_full, (qc - 1) & 1);
        for (int i = max(0, kc - kKStages); i < kc; ++i) drain(&k_full[i % kKStages], (i / kKStages) & 1);
        for (int i = max(0, vc - kVStages); i < vc; ++i) drain(&v_full[i % kVStages], (i / kVStages) & 1);
        if (asked > 0) drain(&next_full[(asked - 1) & 1], ((asked - 1) >> 1) & 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t fmt = FmtOf<T>::v;
      const uint32_t idesc_s = umma_idesc(kTile, kTile, fmt, fmt, 0, 0);   // A = Q, B = K tile, both K-major
      const uint32_t idesc_o = umma_idesc(kTile, kD, fmt, fmt, 0, 1);      // A = P (TMEM), B = V tile (MN-major)
      int kc = 0, vc = 0, qc = 0, tc[2] = {0, 0};   // consumed so far; tc: tiles of each stream whose P has been awaited
      bool ok = true;
      for (int idx = blockIdx.x, round = 0; idx >= 0; idx = ok ? next_item(round++, false, ok) : -1) {
        get_item<kMla>(p, idx, it);
        if (it.n_max == 0) continue;
        const int n_max = it.n_max;
        // S of tile j of the item; the last reader of a K stage (of Q) gives it back
        auto issue_s = [&](int s, int j) {
          const uint32_t q_addr = smem_u32(sQ + s * kKBytes), k_addr = smem_u32(sK + ((kc + j) % kKStages) * kKBytes);
#pragma unroll
          for (int k = 0; k < kQBlocks * 4; ++k)
            umma_f16(tmem_base + s * kTile, umma_desc_k_sw128(q_addr + (k / 4) * kBlockBytes + (k % 4) * 32),
                     umma_desc_k_sw128(k_addr + (k / 4) * kBlockBytes + (k % 4) * 32), idesc_s, k > 0 ? 1u : 0u);
          umma_commit(&s_full[s]);
          const bool last = s == 1 || j >= it.n[1];
          if (last) {
            umma_commit(&k_empty[(kc + j) % kKStages]);
            if (j == n_max - 1) umma_commit(q_empty);
          }
        };
        ok = wait_or_abort(q_full, qc & 1, ab, 823) && wait_or_abort(&k_full[kc % kKStages], (kc / kKStages) & 1, ab, 824);
        if (!ok) break;
        ++qc;
        tc_fence_after_sync();
        if (it.n[0] > 0) issue_s(0, 0);
        if (it.n[1] > 0) issue_s(1, 0);
        for (int i = 0; ok && i < n_max; ++i) {
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            if (!ok || i >= it.n[s]) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int v = vc + 2 * i + h;
              ok = ok && wait_or_abort(&v_full[v % kVStages], (v / kVStages) & 1, ab, 825) &&
                   wait_or_abort(&p_ready[s * 2 + h], tc[s] & 1, ab, 826);
              if (!ok) break;
              tc_fence_after_sync();
              const uint32_t v_addr = smem_u32(sV + (v % kVStages) * kVBytes);
#pragma unroll
              for (int k = 0; k < kPage / 16; ++k)
                umma_f16_ts(tmem_base + (2 + s) * kTile, tmem_base + s * kTile + h * 32 + k * 8,
                            umma_desc_mn_sw128(v_addr + k * 2048, kVBytes / 2, 1024), idesc_o,
                            (i > 0 || h > 0 || k > 0) ? 1u : 0u);
              if (s == 1 || i >= it.n[1]) umma_commit(&v_empty[v % kVStages]);
            }
            if (!ok) break;
            ++tc[s];
            if (i == it.n[s] - 1) {
              umma_commit(&o_final[s]);
            } else {
              const int k = kc + i + 1;
              if (!wait_or_abort(&k_full[k % kKStages], (k / kKStages) & 1, ab, 824)) { ok = false; break; }
              tc_fence_after_sync();
              issue_s(s, i + 1);
            }
          }
        }
        kc += n_max;
        vc += 2 * n_max;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax + epilogue: thread = query row
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoft));
    const int s = (warp >> 2) - 1, quarter = warp & 3;
    const int r = quarter * 32 + lane;                 // row of the tile = TMEM lane
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem_base + s * kTile + lane_off, tO = tmem_base + (2 + s) * kTile + lane_off;
    const float sc = p.scale_log2;
    int tc = 0, oc = 0;    // tiles and items of this stream so far
    bool fail = false;
    bool ok = true;
    for (int idx = blockIdx.x, round = 0; idx >= 0; idx = next_item(round++, true, ok)) {
      get_item<kMla>(p, idx, it);
      const int n = s ? it.n[1] : it.n[0];
      if (n == 0) continue;
      const int head = s ? it.head[1] : it.head[0], row0 = s ? it.row0[1] : it.row0[0], rows = s ? it.rows[1] : it.rows[0];
      const bool row_ok = r < rows;
      const int pos_first = it.ctx + row0, pos_last = pos_first + rows - 1, pos = pos_first + r;
      float m_used = -INFINITY, l_sum = 0.f;
      for (int i = 0; i < n; ++i, ++tc) {
        if (__any_sync(0xffffffffu, !wait_or_abort(&s_full[s], tc & 1, ab, 827))) { fail = true; break; }
        tc_fence_after_sync();
        const int key0 = it.kv_begin + i * kTile;
        uint32_t v[kTile];
#pragma unroll
        for (int c = 0; c < kTile; c += 32) tmem_ld_x32_p(tS + c, v + c);
        tmem_ld_wait();
        // a tile that every row of this stream sees in full needs no mask
        const bool full_tile = key0 + kTile - 1 <= pos_first && key0 + kTile <= it.seq_len &&
                               (p.window <= 0 || key0 > pos_last - p.window);
        if (!full_tile) {
          const int hi = min(pos, it.seq_len - 1) - key0, lo = p.window > 0 ? pos - p.window + 1 - key0 : 0;
#pragma unroll
          for (int e = 0; e < kTile; ++e) v[e] = (e <= hi && e >= lo) ? v[e] : 0xff800000u;   // -inf
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < kTile; e += 8) {
#pragma unroll
          for (int u = 0; u < 4; ++u) mx[u] = fmaxf(fmaxf(mx[u], __uint_as_float(v[e + u])), __uint_as_float(v[e + u + 4]));
        }
        float tmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc;   // scale > 0: max commutes
        if (!row_ok) tmax = -INFINITY;
        // ---- lazy running maximum (it moves when a tile exceeds it by more than 8 in log2 units); the rescale of O is
        // warp-collective (TMEM access), so the warp decides together.  S(i) has arrived, so P.V(i - 1) is in O.
        const bool bump = tmax > m_used + kMaxSlack;
        const float alpha = bump ? exp2f(m_used - tmax) : 1.f;
        if (bump) { m_used = tmax; l_sum *= alpha; }
        if (__any_sync(0xffffffffu, bump) && i > 0) {
#pragma unroll 1
          for (int c = 0; c < kD; c += 32) {   // rare path: 32 columns at a time keeps the register count down
            uint32_t o[32];
            tmem_ld_x32_p(tO + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st_x32_p(tO + c, o);
          }
        }
        const float neg_m = (m_used == -INFINITY || !row_ok) ? -INFINITY : -m_used;   // invalid rows: P = 0
        const uint64_t sc2 = f2(sc, sc), neg2 = f2(neg_m, neg_m);
        uint64_t ls[4] = {0, 0, 0, 0};
#pragma unroll
        for (int c = 0; c < kTile; c += 32) {
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            float a, b;
            unf2(fma2(f2(__uint_as_float(v[c + e]), __uint_as_float(v[c + e + 1])), sc2, neg2), a, b);
            a = ex2_approx(a);
            b = ex2_approx(b);
            ls[(e >> 1) & 3] = add2(ls[(e >> 1) & 3], f2(a, b));
            pk[e / 2] = pack2<T>(a, b);
          }
          tmem_st_x16_p(tS + c / 2, pk);
          if (c == 32 || c == 96) {   // 64 keys of P are on their way: hand them over
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[s * 2 + c / 64]);
          }
        }
        float a0, a1, b0, b1;
        unf2(add2(ls[0], ls[1]), a0, a1);
        unf2(add2(ls[2], ls[3]), b0, b1);
        l_sum += (a0 + a1) + (b0 + b1);
      }
      if (fail) break;
      // ---- epilogue
      if (__any_sync(0xffffffffu, !wait_or_abort(&o_final[s], oc & 1, ab, 828))) { fail = true; break; }
      ++oc;
      tc_fence_after_sync();
      const int64_t tok = it.qs + row0 + r, orow = tok * p.Hq + head;
      float den = l_sum;
      const float ms = (m_used == -INFINITY) ? 0.f : m_used;
      if (p.sinks != nullptr) den += exp2f(p.sinks[head] * kLog2e - ms);
      float inv = den > 0.f ? 1.f / den : 0.f;
      if (p.gate != nullptr && row_ok) {
        const float g = to_float(reinterpret_cast<const T*>(p.gate)[tok * p.gate_stride + head]);
        inv = inv / (1.f + __expf(-g));
      }
      T* dst = reinterpret_cast<T*>(p.out) + orow * kD;
#pragma unroll
      for (int c = 0; c < kD; c += 64) {
        uint32_t o[64];
        tmem_ld_x32_p(tO + c, o);          // warp-collective: every lane loads
        tmem_ld_x32_p(tO + c + 32, o + 32);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              w[u] = pack2<T>(__uint_as_float(o[q * 8 + 2 * u]) * inv, __uint_as_float(o[q * 8 + 2 * u + 1]) * inv);
            *reinterpret_cast<uint4*>(dst + c + q * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      if (row_ok && p.lse != nullptr) p.lse[orow] = den > 0.f ? (ms + log2f(den)) * kLn2 : -INFINITY;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <typename T, bool kMla>
static int launch(Params& p, const CUtensorMap& tmQ, const CUtensorMap& tmKV, const CUtensorMap& tmKpe, int max_query_len,
                  int num_sms, cudaStream_t st) {
  auto kern = prefill_pair_kernel<T, kMla>;
  cudaError_t e = ensure_dynamic_smem((const void*)kern, (int)Cfg<kMla>::kSmem);
  if (e != cudaSuccess) return (int)e;
  const int64_t tiles = (int64_t)p.B * p.Hq * ((max_query_len + kTile - 1) / kTile);
  p.by_heads = !kMla && (p.Hq / p.Hkv) % 2 == 0;
  p.single = 0;
  if (tiles <= num_sms) { p.single = 1; p.by_heads = 0; }
  p.units = p.by_heads ? p.Hq / 2 : p.Hq;
  const int step = (p.by_heads || p.single) ? kTile : 2 * kTile;
  p.row_blocks = (max_query_len + step - 1) / step;
  const int64_t items = (int64_t)p.B * p.units * p.row_blocks;
  if (items > (1 << 30)) return 3;
  p.take = items > num_sms;
  return (int)launch_pdl(kern, dim3((unsigned)items), dim3(kThreads), Cfg<kMla>::kSmem, st, tmQ,
                         tmKV, tmKpe, p);
}

}  // namespace pair
}  // namespace b200

// Paged GQA prefill attention (head_dim 128, block_size a multiple of 64).  `tmQ`: q as a 2-D [T, Hq * 128] 16-bit tensor
// with 64-column x 128-row boxes; `tmKV`: the cache as [rows, 128] with 64 x 64 boxes; both with 128-byte swizzle.
// `gate` [T][>= Hq] (or null): raw output gates.  Returns 3 for shapes it does not serve.
extern "C" int b200_prefill_attention_pair(void* out, float* lse, const void* tmQ, const void* tmKV, const int* block_tables,
                                           const int* seq_lens, const int* qsl, const float* sinks, int* status, int B,
                                           int Hq, int Hkv, int D, int block_size, int max_blocks, int64_t num_blocks,
                                           int max_query_len, int window, float scale, const void* gate,
                                           int64_t gate_stride, int dtype, int num_sms, cudaStream_t st) {
  using namespace b200;
  if (B == 0 || max_query_len <= 0) return 0;
  if (D != 128 || Hq % Hkv || block_size % pair::kPage || B > 65535 || Hq > 65535 || num_sms < 1) return 3;
  pair::Params p = {};
  p.out = out; p.lse = lse; p.block_tables = block_tables; p.seq_lens = seq_lens; p.qsl = qsl; p.sinks = sinks;
  p.status = status; p.Hq = Hq; p.Hkv = Hkv; p.block_size = block_size; p.max_blocks = max_blocks; p.window = window;
  p.num_blocks = num_blocks; p.scale_log2 = scale * pair::kLog2e; p.causal = 1; p.gate = gate; p.gate_stride = gate_stride;
  p.B = B;
  const CUtensorMap& q = *reinterpret_cast<const CUtensorMap*>(tmQ);
  const CUtensorMap& kv = *reinterpret_cast<const CUtensorMap*>(tmKV);
  if (dtype == 1) return pair::launch<__nv_bfloat16, false>(p, q, kv, kv, max_query_len, num_sms, st);
  if (dtype == 2) return pair::launch<__half, false>(p, q, kv, kv, max_query_len, num_sms, st);
  return 3;
}

// Multi-head latent attention prefill in the compute-friendly form (192-dim q / k, 128-dim v).  `tmQ`: q as [T, Hq * 192]
// with 64-column x 128-row boxes; `tmKV`: the up-projected keys / values as [rows, Hq * 256] (k_nope | v per head) with 64
// x 64 boxes; `tmKpe`: the rotary keys as [rows, 64] with 64 x 64 boxes; all 16-bit with 128-byte swizzle and row
// extents equal to the number of valid rows.  Request r owns key rows kv_starts[r] .. kv_starts[r] + kv_lens[r] and
// query rows qsl[r] .. qsl[r + 1]; causal: its queries are its last keys.  Rows of requests with no key are not
// written (the caller presets out = 0, lse = -inf).
extern "C" int b200_mla_prefill_pair(void* out, float* lse, const void* tmQ, const void* tmKV, const void* tmKpe,
                                     const int* kv_starts, const int* kv_lens, const int* qsl, const float* sinks,
                                     const void* gate, int64_t gate_stride, int* status, int B, int Hq, int max_query_len,
                                     int causal, int window, float scale, int dtype, int num_sms, cudaStream_t st) {
  using namespace b200;
  if (B == 0 || max_query_len <= 0) return 0;
  if (B > 65535 || Hq > 65535 || num_sms < 1) return 3;
  if (window < 0 || (window > 0 && !causal)) return 2;
  pair::Params p = {};
  p.out = out; p.lse = lse; p.seq_lens = kv_lens; p.qsl = qsl; p.kv_starts = kv_starts; p.sinks = sinks; p.gate = gate;
  p.gate_stride = gate_stride; p.status = status; p.Hq = Hq; p.Hkv = Hq; p.block_size = pair::kPage; p.window = window;
  p.causal = causal ? 1 : 0; p.scale_log2 = scale * pair::kLog2e; p.B = B;
  const CUtensorMap& q = *reinterpret_cast<const CUtensorMap*>(tmQ);
  const CUtensorMap& kv = *reinterpret_cast<const CUtensorMap*>(tmKV);
  const CUtensorMap& kpe = *reinterpret_cast<const CUtensorMap*>(tmKpe);
  if (dtype == 1) return pair::launch<__nv_bfloat16, true>(p, q, kv, kpe, max_query_len, num_sms, st);
  if (dtype == 2) return pair::launch<__half, true>(p, q, kv, kpe, max_query_len, num_sms, st);
  return 3;
}
