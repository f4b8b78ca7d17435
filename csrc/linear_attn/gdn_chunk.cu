// Gated delta rule of prompts, 64 tokens at a time on tcgen05 (bf16 q / k / v, key and value heads of 128, L2-normalised
// q and k).  The same recurrence as gdn_recurrent_kernel (gdn.cu); the reference's chunked form is ops/fla/chunk.py:23-140.
//
// With c_i the summed gates up to token i of the chunk, S [dv, dk] the state in front of it, k and q normalised:
//     A_ij = beta_i (k_i . k_j) exp(c_i - c_j)  (j < i)        T = (1 + A)^-1
//     R_j  = beta_j (v_j - exp(c_j) S k_j)                      U_i = sum_j T_ij R_j
//     o_i  = exp(c_i) S q_i + sum_{j <= i} (q_i . k_j) exp(c_i - c_j) U_j
//     S'   = exp(c_63) S + sum_j exp(c_63 - c_j) U_j k_j^T
// One CTA walks through one (request, value head); all products have the 128 rows dv as lanes.  The norms of q and k, the
// gates and beta are applied to fp32 columns, so q and k enter the tensor core as they are in memory; every fp32 operand
// (S, R, T, U, P) is cut into three bf16 pieces that add up to all its 24 bits, and of a product of two such
// operands six pairs are summed.  Pieces are cut and not rounded, so the pairs left out are below 2^-22 of the leading one; against 64
// bits states are off by 1.3e-7, the scan's by 1.3e-7 to 1.4e-6.  Sums of gates are kept as
// pairs of floats (from doubles), because a difference of two sums is what is raised to a power.
//
// Warps 0-3: A, T and P of the chunk ahead; warps 4-11: the chain S -> R -> U -> S, a thread = one row x half of the
// columns, S in registers; warp 12: MMA issue; warps 13 to 15: loads, norms and gates, up to two chunks ahead.  What bounds it is that chain: three dependent products
// (24, 24 and 12 MMA steps) with a pass through registers between them, 64 tokens a turn; the outputs and the
// next chunk's T are computed beside it.  6 us a chunk and CTA, of which 2.9 are products (4 x 2048 tokens, 32 heads:
// 214 us, 3308 us as a scan; 1 x 4096 tokens, 16 heads: 392 us, 1910 us as a scan).  Waits and loops are kept small (70 KB of
// code in all): unrolled throughout, the roles evicted one another's instructions and a chunk took 13 us.  Every wait is bounded; a CTA that gives up sets the status word and runs out.
// Zeros hide later keys, and zero times a NaN or an infinity is not zero: a chunk ends in front of a token with such a value in k,
// v, its gate or beta, which is the first token of the next one.  So it reaches its own and later tokens only, as in the scan
// (one in q stays in its own row of every product).  Looking for them costs 8 of 214 us (4 x 2048 tokens): the loads are on
// the way to the next chunk's T.  Finite inputs whose squares or products overflow are taken for such values or not found.
#include <cuda.h>
#include <cuda_bf16.h>
#include <limits.h>

#include "../api.h"
#include "../common/ptx.cuh"
#include "../common/launch.cuh"
#include "../common/utils.cuh"
#include "../gemm/gemm_common.cuh"

namespace b200 {
namespace gdnc {

constexpr int kC = 64;                          // tokens of a chunk
constexpr int kPrep = 128, kChain = 256, kThreads = kPrep + kChain + 128;
// registers a thread: 512 x 128 at launch, then 128 x (104 + 168 + 168 + 72) = 65536
constexpr int kRegsChain = 168, kRegsPrep = 104, kRegsIssue = 72;
constexpr int kHalf = 128 * 128;                // one 64-dim half of the [64 K rows | 64 Q rows] operand tile
constexpr int kStage = 2 * kHalf;
constexpr int kVStage = kC * 128 * 2;
constexpr int kPiece = kC * 128;                // one bf16 piece of a 64 x 64 operand
constexpr int kPitch = 68;                      // floats of a row of the fp32 64 x 64 scratch (16-byte aligned, no bank conflicts)

struct Scalars {                                // per token of a chunk
  float beta[kC], gh[kC], gl[kC], rk[kC], rq[kC];   // gate sums in log2 units, high and low part; inverse norms (rq with scale)
  float c1[kC], c2[kC], c3[kC];                 // beta exp(c) rk;  exp(c_63 - c) rk;  exp(c) rq
  float decay;                                  // exp(c_63)
  int n, pad[2];                                // tokens of the chunk
};

struct Smem {
  uint8_t kq[2][kStage];                        // [stage][dim half][K rows, Q rows][128 B], 128-byte swizzle
  uint8_t v[2][kVStage];                        // [stage][token][128]
  uint8_t p[2][3][kPiece];                      // [buffer][piece][row][64], 128-byte swizzle
  uint8_t t[3][kPiece];
  float a[kC][kPitch];
  float f[kC][kPitch];                          // T in fp32
  float m[32][32];
  Scalars sc[2];
  float ones[8];
  uint64_t raw[2], full[2], d0, d0_read, t_ready, s_ready, x1, x2, r_ready, u_full, ut_ready, uo_ready, d3, y[2], o_read, end;   // y: one per buffer of P
  uint32_t tmem;
  int abort_flag;
  int cut;                                      // tokens of a chunk that ends in front of a value that is not finite
  int n_prep;                                   // tokens of the chunk, one copy for the four warps of the first role
};
constexpr int kSmemBytes = (int)sizeof(Smem) + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

// TMEM columns.  X1 and U lie where D3 (the state's update) comes afterwards; the pieces of U for the update and D0
// (the next chunk's products of keys) lie over the pieces of S, which are spent by then; U's pieces for the output over R's.
constexpr int kX1 = 0, kU = 64, kD3 = 0, kSp = 128, kUt = 128, kD0 = 256, kX2 = 320, kRp = 384, kUo = 384, kTmemCols = 512;

struct Params {
  __nv_bfloat16* out;
  const float *g, *beta;
  float* states;
  const int *cu, *slots;
  InitFlags has_init;
  int* status;
  int64_t o_stride;
  int Hk, Hv, min_len;
  float scale;
};

__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// two fp32 values in one 64-bit register: a * b + c for both in one instruction
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
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// acc + 0 * v on pairs of bf16: acc stays zero while everything is finite, and is a NaN from then on
__device__ __forceinline__ uint32_t times_zero(uint32_t v, uint32_t acc) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(v), "r"(0u), "r"(acc));
  return d;
}
// squares of two bf16 in fp32 added to a pair
__device__ __forceinline__ uint64_t square2(uint32_t v, uint64_t acc) {
  const uint64_t x = f2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
  return fma2(x, x, acc);
}
// three bf16 pairs that add up to (a, b): the leading 8 bits of each, of what is left, and the rest
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint64_t minus = f2(-1.f, -1.f);
  const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
  hi = __byte_perm(ua, ub, 0x7632);
  unf2(fma2(f2(__uint_as_float(ua & 0xffff0000u), __uint_as_float(ub & 0xffff0000u)), minus, f2(a, b)), a, b);
  const uint32_t va = __float_as_uint(a), vb = __float_as_uint(b);
  mid = __byte_perm(va, vb, 0x7632);
  unf2(fma2(f2(__uint_as_float(va & 0xffff0000u), __uint_as_float(vb & 0xffff0000u)), minus, f2(a, b)), a, b);
  lo = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
// 32 values of this thread's row as the columns [0, 16) of three TMEM pieces `step` columns apart
__device__ __forceinline__ void store_pieces(uint32_t taddr, int step, const float* v) {
  uint32_t hi[16], mid[16], lo[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) split3(v[2 * e], v[2 * e + 1], hi[e], mid[e], lo[e]);
  tmem_st_x16(taddr, hi);
  tmem_st_x16(taddr + step, mid);
  tmem_st_x16(taddr + 2 * step, lo);
}
// 8 values as one 16-byte piece of row `row`, columns 8 c .. 8 c + 7, of three swizzled shared-memory pieces
__device__ __forceinline__ void store_pieces_smem(uint8_t* base, int row, int c, const float* v) {
  uint32_t hi[4], mid[4], lo[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) split3(v[2 * e], v[2 * e + 1], hi[e], mid[e], lo[e]);
  const int off = row * 128 + ((c ^ (row & 7)) << 4);
  *reinterpret_cast<uint4*>(base + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(base + kPiece + off) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
  *reinterpret_cast<uint4*>(base + 2 * kPiece + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}
// Tokens of a chunk that its loader has published; `left` of the request are not in a chunk yet.  At least one and none too many
// whatever was read (after a wait that gave up): every role ends, and writes stay within the request.
__device__ __forceinline__ int take_chunk(int n, int& left) {
  n = min(max(n, 1), min(kC, left));
  left -= n;
  return n;
}
// a barrier of n threads that tells all of them whether `any` holds for one
__device__ __forceinline__ bool bar_any(int id, int n, bool any) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred q, p;\n\tsetp.ne.u32 q, %3, 0;\n\tbar.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(r) : "r"(id), "r"(n), "r"((uint32_t)any) : "memory");
  return r != 0;
}
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

__device__ __forceinline__ void load8(float (&v)[8], const float* src) {
  *reinterpret_cast<float4*>(&v[0]) = *reinterpret_cast<const float4*>(src);
  *reinterpret_cast<float4*>(&v[4]) = *reinterpret_cast<const float4*>(src + 4);
}
// Inverses of diagonal blocks of 2 B rows from those of B rows: T21 = -T22 A21 T11 for 32 / B pairs of blocks side by side.  A
// warp takes a quarter of the rows of every pair, a lane two columns of half of these rows.  Called by the four warps of
// the first warpgroup.
template <int B>
__device__ __forceinline__ void join_blocks(Smem& sm, int warp, int lane) {
  constexpr int R = B / 8;                       // rows of a thread
  const int wide = (lane & 15) * 2;              // first of this lane's two columns, over all pairs
  const int at = wide / B * 2 * B, col = wide % B, r0 = warp * (B / 4) + (lane >> 4) * R;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float* left = h == 0 ? &sm.a[at + B + r0][at] : &sm.f[at + B + r0][at + B];
    const float* right = h == 0 ? &sm.f[at][at + col] : &sm.m[0][wide];
    const int pitch = h == 0 ? kPitch : 32;
    uint64_t acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0;
#pragma unroll
    for (int l = 0; l < B; l += 4) {
      float2 t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) t[u] = *reinterpret_cast<const float2*>(right + (l + u) * pitch);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(left + i * kPitch + l);
        acc[i] = fma2(f2(a.x, a.x), f2(t[0].x, t[0].y), acc[i]);
        acc[i] = fma2(f2(a.y, a.y), f2(t[1].x, t[1].y), acc[i]);
        acc[i] = fma2(f2(a.z, a.z), f2(t[2].x, t[2].y), acc[i]);
        acc[i] = fma2(f2(a.w, a.w), f2(t[3].x, t[3].y), acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float2 v;
      unf2(acc[i], v.x, v.y);
      if (h == 0) *reinterpret_cast<float2*>(&sm.m[r0 + i][wide]) = make_float2(-v.x, -v.y);
      else *reinterpret_cast<float2*>(&sm.f[at + B + r0 + i][at + col]) = v;
    }
    bar_sync(2, kPrep);
  }
}

__global__ void __launch_bounds__(kThreads, 1) gdn_chunk_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ Params p) {
  const int hv = blockIdx.x, r = blockIdx.y;
  const int s0 = p.cu[r], L = p.cu[r + 1] - s0, slot = p.slots[r];
  if (L < p.min_len || slot < 0) return;
  extern __shared__ uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  Abort ab{p.status, &sm.abort_flag};
  if (tid == 0) {
    sm.abort_flag = 0;
    for (int i = 0; i < 8; ++i) sm.ones[i] = 1.f;
    for (int i = 0; i < 2; ++i) { mbar_init(&sm.raw[i], 1); mbar_init(&sm.full[i], 64); }
    mbar_init(&sm.d0, 1); mbar_init(&sm.x1, 1); mbar_init(&sm.x2, 1); mbar_init(&sm.u_full, 1);
    mbar_init(&sm.d3, 1); mbar_init(&sm.y[0], 1); mbar_init(&sm.y[1], 1); mbar_init(&sm.end, 1);
    mbar_init(&sm.d0_read, 4); mbar_init(&sm.t_ready, kPrep);
    mbar_init(&sm.s_ready, 8); mbar_init(&sm.r_ready, 8); mbar_init(&sm.ut_ready, 8); mbar_init(&sm.uo_ready, 8);
    mbar_init(&sm.o_read, 8);
    mbar_fence_init();
  }
  if (tid < kPrep) {
    // T and P are zero above their diagonal blocks, A is not read there
    for (int i = tid; i < kC * kPitch; i += kPrep) sm.f[i / kPitch][i % kPitch] = 0.f;
    for (int i = tid; i < (int)sizeof(sm.p) / 16; i += kPrep) reinterpret_cast<uint4*>(sm.p)[i] = make_uint4(0, 0, 0, 0);
  }
  if (warp == 12) {
    tmem_alloc(&sm.tmem, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = sm.tmem;
  int failed = 0;   // once a wait has given up nothing waits any more: every role runs its loop to the end
  auto wait_one = [&](uint64_t* bar, int phase, int code) {
    if (failed) return;
#pragma unroll 1
    for (uint32_t i = 0; !mbar_try_wait(bar, phase & 1); ++i)
      if (i == (1u << 20) || ((i & 255) == 255 && *ab.flag != 0)) {
        *ab.flag = failed = code;
        return;
      }
  };
  auto wait = [&](uint64_t* bar, int phase, int code) {   // one lane polls for its warp
    if (lane == 0) wait_one(bar, phase, code);
    __syncwarp();
  };

  if (warp < 4) {
    // ------------------------------------------------------------------ the chunk ahead: A, T, P
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsPrep));
    const bool is_q = warp >= 2;                 // warps 2, 3: P (lanes 64-127 of D0); 0, 1: A
    int left = L;
    for (int n = 0;; ++n) {
      const Scalars& sc = sm.sc[n & 1];
      wait(&sm.full[n & 1], n >> 1, 901);
      if (tid == 0) sm.n_prep = sc.n;
      wait(&sm.d0, n, 902);
      tc_fence_after_sync();
      const int row = (warp & 1) * 32 + lane;
      const uint32_t td = tm + kD0 + ((uint32_t)(warp * 32) << 16);
      const float gh = sc.gh[row], gl = sc.gl[row], fac = is_q ? sc.rq[row] : sc.beta[row] * sc.rk[row];
      // The output of chunk n - 2 has been computed from this buffer of P.  A barrier per buffer: its next phase needs the P that is
      // written here, so it cannot complete before this wait has looked (the output of chunk n - 1, in the other buffer, can).
      if (is_q && n >= 2) wait(&sm.y[n & 1], (n - 2) >> 1, 903);
      const int last = is_q ? row : row - 1;           // last column that is kept
      // what lies above the diagonal of a warp's 32 rows is zero and was set at the start
#pragma unroll 1
      for (int hb = 0; hb <= (warp & 1); ++hb) {
        uint32_t d[32];
        tmem_ld_x32(td + 32 * hb, d);
        tmem_ld_wait();
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          const int c = 4 * hb + cc;
          float v[8], jh[8], jl[8], jr[8];
          load8(jh, &sc.gh[8 * c]);
          load8(jl, &sc.gl[8 * c]);
          load8(jr, &sc.rk[8 * c]);
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const uint64_t h = fma2(f2(jh[e], jh[e + 1]), f2(-1.f, -1.f), f2(gh, gh));
            const uint64_t l = fma2(f2(jl[e], jl[e + 1]), f2(-1.f, -1.f), f2(gl, gl));
            unf2(fma2(h, f2(1.f, 1.f), l), v[e], v[e + 1]);
            const uint64_t w = fma2(f2(ex2(v[e]), ex2(v[e + 1])), fma2(f2(fac, fac), f2(jr[e], jr[e + 1]), 0), 0);
            unf2(fma2(w, f2(__uint_as_float(d[8 * cc + e]), __uint_as_float(d[8 * cc + e + 1])), 0), v[e], v[e + 1]);
            v[e] = 8 * c + e <= last ? v[e] : 0.f;
            v[e + 1] = 8 * c + e + 1 <= last ? v[e + 1] : 0.f;
          }
          if (is_q) {
            store_pieces_smem(sm.p[n & 1][0], row, c, v);
          } else {
            *reinterpret_cast<float4*>(&sm.a[row][8 * c]) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(&sm.a[row][8 * c + 4]) = make_float4(v[4], v[5], v[6], v[7]);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.d0_read);
      if (!is_q) {
        // inverses of the eight 8 x 8 diagonal blocks, a thread = one column of one
        bar_sync(1, 64);
        const int b0 = (tid >> 3) * 8, col = tid & 7;
        float a[8][8], t[8];
#pragma unroll
        for (int i = 1; i < 8; ++i) load8(a[i], &sm.a[b0 + i][b0]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          t[i] = i == col ? 1.f : 0.f;
#pragma unroll
          for (int l = 0; l < i; ++l) t[i] -= a[i][l] * t[l];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) sm.f[b0 + i][b0 + col] = t[i];
      }
      bar_sync(2, kPrep);
      take_chunk(sm.n_prep, left);                     // the same for all four: they meet at barriers, after a failure too
      join_blocks<8>(sm, warp, lane);
      join_blocks<16>(sm, warp, lane);
      join_blocks<32>(sm, warp, lane);
      if (n >= 1) wait(&sm.u_full, n - 1, 905);        // the previous chunk's T has been used
      const int trow = tid >> 1, half = tid & 1;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float v[8];
        load8(v, &sm.f[trow][half * 32 + c * 8]);
        store_pieces_smem(sm.t[0], trow, half * 4 + c, v);
      }
      fence_proxy_async_smem();
      mbar_arrive(&sm.t_ready);
      bar_sync(2, kPrep);                              // sm.f and sm.a are written again for the next chunk
      if (left == 0) break;
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ the chain
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsChain));
    const int wg = (warp >> 2) - 1, quarter = warp & 3, dv = quarter * 32 + lane;
    const uint32_t tl = tm + ((uint32_t)(quarter * 32) << 16);
    float* sp = p.states + (((int64_t)slot * p.Hv + hv) * 128 + dv) * 128 + wg * 64;
    float S[64];
    if (p.has_init[r]) {
#pragma unroll
      for (int j = 0; j < 64; j += 4) *reinterpret_cast<float4*>(&S[j]) = *reinterpret_cast<const float4*>(sp + j);
    } else {
#pragma unroll
      for (int j = 0; j < 64; ++j) S[j] = 0.f;
    }
    auto arrive = [&](uint64_t* bar) {
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto wait_tc = [&](uint64_t* bar, int phase, int code) {
      wait(bar, phase, code);
      tc_fence_after_sync();
    };
    int n = 0, left = L;                               // tokens of the chunk; of the request behind it
    __nv_bfloat16* dst = p.out + (s0 + wg * 32) * p.o_stride + hv * 128 + dv;
    auto write_out = [&](int c, int tokens) {          // outputs of chunk c, this thread: one dv, 32 tokens
      wait_tc(&sm.y[c & 1], c >> 1, 910);
      uint32_t o[32];
      tmem_ld_x32(tl + kX2 + wg * 32, o);
      tmem_ld_wait();
      arrive(&sm.o_read);
      __nv_bfloat16* at = dst;
#pragma unroll
      for (int j = 0; j < 32; ++j, at += p.o_stride)
        if (wg * 32 + j < tokens) *at = __float2bfloat16(__uint_as_float(o[j]));
      dst += tokens * p.o_stride;
    };
    for (int c = 0;; ++c) {
      const int st = c & 1;
      const Scalars& sc = sm.sc[st];
      if (left > 0) {
        wait_tc(&sm.d0_read, c, 911);                  // D0 lies over the pieces of S
        store_pieces(tl + kSp + wg * 32, 64, S);
        store_pieces(tl + kSp + wg * 32 + 16, 64, S + 32);
        arrive(&sm.s_ready);
      }
      if (c > 0) write_out(c - 1, n);
      if (left == 0) break;
      wait(&sm.full[st], c >> 1, 912);
      n = take_chunk(__shfl_sync(0xffffffffu, sc.n, 0), left);   // one value for the warp, after a failure too
      wait_tc(&sm.x1, c, 913);
      uint32_t x[32];
      float w[32];
      tmem_ld_x32(tl + kX1 + wg * 32, x);
      tmem_ld_wait();
      const __nv_bfloat16* vs = reinterpret_cast<const __nv_bfloat16*>(sm.v[st]) + wg * 32 * 128 + dv;
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 b4 = *reinterpret_cast<const float4*>(&sc.beta[wg * 32 + j]);
        const float4 c4 = *reinterpret_cast<const float4*>(&sc.c1[wg * 32 + j]);
        w[j] = b4.x * to_f(vs[j * 128]) - c4.x * __uint_as_float(x[j]);
        w[j + 1] = b4.y * to_f(vs[(j + 1) * 128]) - c4.y * __uint_as_float(x[j + 1]);
        w[j + 2] = b4.z * to_f(vs[(j + 2) * 128]) - c4.z * __uint_as_float(x[j + 2]);
        w[j + 3] = b4.w * to_f(vs[(j + 3) * 128]) - c4.w * __uint_as_float(x[j + 3]);
      }
      store_pieces(tl + kRp + wg * 16, 32, w);
      arrive(&sm.r_ready);
      // exp(c_i) S q_i: scaled in place, the product with U is added to it
      wait_tc(&sm.x2, c, 914);
      tmem_ld_x32(tl + kX2 + wg * 32, x);
      tmem_ld_wait();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t y[16];
#pragma unroll
        for (int j = 0; j < 16; j += 8) {
          float f[8];
          load8(f, &sc.c3[wg * 32 + h * 16 + j]);
#pragma unroll
          for (int e = 0; e < 8; ++e) y[j + e] = __float_as_uint(__uint_as_float(x[h * 16 + j + e]) * f[e]);
        }
        tmem_st_x16(tl + kX2 + wg * 32 + h * 16, y);
      }
      const float decay = sc.decay;                    // the scalars' stage is given back with D3
      wait_tc(&sm.u_full, c, 915);
      tmem_ld_x32(tl + kU + wg * 32, x);
      tmem_ld_wait();
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {                    // for the state's update, then for the outputs
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          float f[8];
          load8(f, h == 0 ? &sc.c2[wg * 32 + j] : &sm.ones[0]);
#pragma unroll
          for (int e = 0; e < 8; ++e) w[j + e] = __uint_as_float(x[j + e]) * f[e];
        }
        store_pieces(tl + (h == 0 ? kUt : kUo) + wg * 16, 32, w);
        arrive(h == 0 ? &sm.ut_ready : &sm.uo_ready);
      }
      wait_tc(&sm.d3, c, 916);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        tmem_ld_x32(tl + kD3 + wg * 64 + h * 32, x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) S[h * 32 + j] = S[h * 32 + j] * decay + __uint_as_float(x[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 64; j += 4) *reinterpret_cast<float4*>(sp + j) = *reinterpret_cast<const float4*>(&S[j]);
  } else {
    // ------------------------------------------------------------------ MMA issue, loads
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp >= 13) {
      // ------------------------------------------------------------------ loads, norms and gates (13, 14), what is not finite in v (15)
      const int lt = tid - 13 * 32;              // 0 .. 63, a token of the chunk
      const int hk = hv / (p.Hv / p.Hk);
      int issued = 0;
      for (int c = 0, pos = 0; pos < L; ++c) {
        const int st = c & 1;
        const int64_t tok0 = s0 + (int64_t)pos;
        Scalars& sc = sm.sc[st];
        int n = min(kC, L - pos);
        float beta = lt < n ? p.beta[(tok0 + lt) * p.Hv + hv] : 0.f;
        bool bad = !(fabsf(beta) < INFINITY) && lt > 0;   // a value that is not finite behind the chunk's first token
        double first = 0., sum = 0.;             // gate sums up to tokens 2 lane and 2 lane + 1 (warp 13)
        if (warp == 13) {
          const float g0 = 2 * lane < n ? p.g[(tok0 + 2 * lane) * p.Hv + hv] : 0.f;
          const float g1 = 2 * lane + 1 < n ? p.g[(tok0 + 2 * lane + 1) * p.Hv + hv] : 0.f;
          bad |= (!(g0 < INFINITY) && lane > 0) || !(g1 < INFINITY);
          // a gate below -128 is a factor of zero in fp32 either way; clamped, the sums stay finite (a NaN stays one)
          const double a = (g0 < -128.f ? -128.f : g0) * 1.4426950408889634, b = (g1 < -128.f ? -128.f : g1) * 1.4426950408889634;
          sum = a + b;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
          }
          first = __shfl_up_sync(0xffffffffu, sum, 1);   // not sum - b: b may be a NaN
          first = lane == 0 ? a : first + a;
        }
        if (c >= 2) wait(&sm.d3, c - 2, 904);    // the last reader of this stage
        if (lt == 0 && !failed) {
          mbar_expect_tx(&sm.raw[st], kStage + kVStage);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            tma_load_2d(sm.kq[st] + h * kHalf, &tmK, &sm.raw[st], hk * 128 + h * 64, (int)tok0);
            tma_load_2d(sm.kq[st] + h * kHalf + kC * 128, &tmQ, &sm.raw[st], hk * 128 + h * 64, (int)tok0);
          }
          tma_load_2d(sm.v[st], &tmV, &sm.raw[st], hv * 256, (int)tok0);
          ++issued;
        }
        if (warp == 13) {
          sc.gh[2 * lane] = (float)first;
          sc.gl[2 * lane] = (float)(first - (double)(float)first);
          sc.gh[2 * lane + 1] = (float)sum;
          sc.gl[2 * lane + 1] = (float)(sum - (double)(float)sum);
        }
        wait(&sm.raw[st], c >> 1, 906);
        float k2 = 0.f, q2 = 0.f;
        if (warp == 15) {                        // (rows behind the request's end, too: they are told apart below)
          uint32_t acc[4] = {0, 0, 0, 0};
#pragma unroll 8
          for (int i = 0; i < 32; ++i) {
            const uint4 a = *reinterpret_cast<const uint4*>(sm.v[st] + i * 512 + lane * 16);
            acc[0] = times_zero(a.x, acc[0]);
            acc[1] = times_zero(a.y, acc[1]);
            acc[2] = times_zero(a.z, acc[2]);
            acc[3] = times_zero(a.w, acc[3]);
          }
          bad = ((acc[0] | acc[1] | acc[2] | acc[3]) & 0x7fff7fffu) != 0;
        } else if (lt < n) {                     // a thread = one row of K and Q
          uint64_t k4[2] = {0, 0}, q4[2] = {0, 0};
#pragma unroll 4
          for (int i = 0; i < 16; ++i) {
            const uint8_t* src = sm.kq[st] + (i >> 3) * kHalf + lt * 128 + (((i & 7) ^ (lt & 7)) << 4);
            const uint4 kv = *reinterpret_cast<const uint4*>(src), qv = *reinterpret_cast<const uint4*>(src + kC * 128);
            k4[0] = square2(kv.x, k4[0]); q4[0] = square2(qv.x, q4[0]);
            k4[1] = square2(kv.y, k4[1]); q4[1] = square2(qv.y, q4[1]);
            k4[0] = square2(kv.z, k4[0]); q4[0] = square2(qv.z, q4[0]);
            k4[1] = square2(kv.w, k4[1]); q4[1] = square2(qv.w, q4[1]);
          }
          float a, b;
          unf2(fma2(k4[0], f2(1.f, 1.f), k4[1]), a, b);
          k2 = a + b;
          unf2(fma2(q4[0], f2(1.f, 1.f), q4[1]), a, b);
          q2 = a + b;
          bad |= !(k2 < INFINITY) && lt > 0;
        }
        if (bar_any(3, 96, bad)) {               // rare: end the chunk in front of such a token
          if (warp == 15) {
            int first_bad = n;
#pragma unroll 1
            for (int row = n - 1; row > 0; --row) {
              const uint2 v = *reinterpret_cast<const uint2*>(sm.v[st] + row * 256 + lane * 8);
              const uint2 k = *reinterpret_cast<const uint2*>(sm.kq[st] + (lane >> 4) * kHalf + row * 128 + (lane & 15) * 8);
              const uint32_t z = times_zero(v.x, times_zero(v.y, times_zero(k.x, times_zero(k.y, 0))));
              const int64_t at = (tok0 + row) * p.Hv + hv;
              if (__any_sync(0xffffffffu, (z & 0x7fff7fffu) != 0 || !(fabsf(p.beta[at]) < INFINITY) || !(p.g[at] < INFINITY))) first_bad = row;
            }
            if (lane == 0) sm.cut = first_bad;
          }
          bar_sync(3, 96);
          n = sm.cut;
          if (lt >= n && lt < kC) {              // no gates behind the end: the sums stay what they are there
            sc.gh[lt] = sc.gh[n - 1];
            sc.gl[lt] = sc.gl[n - 1];
          }
          bar_sync(3, 96);
        }
        if (lt >= n && warp < 15) {              // rows behind the chunk's end are the next one's or another request's: zeros
          beta = k2 = q2 = 0.f;
#pragma unroll 2
          for (int i = 0; i < 16; ++i) {
            uint8_t* dst = sm.kq[st] + (i >> 3) * kHalf + lt * 128 + ((i & 7) << 4);
            *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(dst + kC * 128) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(sm.v[st] + lt * 256 + i * 16) = make_uint4(0, 0, 0, 0);
          }
        }
        pos += n;
        if (warp < 15) {
          const float rk = rsqrtf(k2 + 1e-6f), rq = p.scale * rsqrtf(q2 + 1e-6f), e = ex2(sc.gh[lt] + sc.gl[lt]);
          sc.beta[lt] = beta;
          sc.rk[lt] = rk;
          sc.rq[lt] = rq;
          sc.c1[lt] = beta * e * rk;
          sc.c2[lt] = ex2((sc.gh[kC - 1] - sc.gh[lt]) + (sc.gl[kC - 1] - sc.gl[lt])) * rk;
          sc.c3[lt] = e * rq;
          if (lt == kC - 1) sc.decay = e;
          if (lt == 0) sc.n = n;
          fence_proxy_async_smem();
          mbar_arrive(&sm.full[st]);
        }
        bar_sync(3, 96);                         // the next chunk's sums and cuts are written
      }
      if (lt == 0 && failed)                     // copies in flight land before the shared memory goes away (bounded)
        for (int c = max(0, issued - 2); c < issued; ++c)
          for (uint32_t i = 0; i < (1u << 16); ++i)
            if (mbar_try_wait(&sm.raw[c & 1], (c >> 1) & 1)) break;
    } else if (warp == 12 && elect_one()) {
    const uint32_t id64 = umma_idesc(128, 64, 1, 1), id128mn = umma_idesc(128, 128, 1, 1, 0, 1);
    const uint32_t kq_addr = smem_u32(sm.kq[0]), t_addr = smem_u32(sm.t[0]), p_addr = smem_u32(sm.p[0][0]);
    auto products = [&](int c) {                       // D0 = [K; Q] K^T of chunk c
      const uint64_t kq = umma_desc_k_sw128(kq_addr + (c & 1) * kStage);
#pragma unroll 1
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t a = kq + ((h * kHalf + k * 32) >> 4);
          umma_f16(tm + kD0, a, a, id64, h > 0 || k > 0);
        }
      umma_commit(&sm.d0);
    };
    auto state_times = [&](int d, uint32_t b) {        // D = S [128 rows at b]^T, least pieces first
      const uint64_t desc = umma_desc_k_sw128(b);
#pragma unroll 1
      for (int i = 5; i >= 0; --i)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ts(tm + d, tm + kSp + i * 32 + k * 8, desc + (((i & 1) * kHalf + k * 32) >> 4), id64, i < 5 || k > 0);
    };
    auto tokens_times = [&](int d, int a, uint32_t b, uint32_t first) {   // D (+)= A [64 x 64 at b]^T, both in three pieces
      const uint64_t desc = umma_desc_k_sw128(b);
      uint32_t acc = first;
#pragma unroll 1
      for (int s = 2; s >= 0; --s)
#pragma unroll 1
        for (int pa = 0; pa <= s; ++pa)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_ts(tm + d, tm + a + pa * 32 + k * 8, desc + (((s - pa) * kPiece + k * 32) >> 4), id64, acc);
            acc = 1;
          }
    };
    wait_one(&sm.full[0], 0, 920);
    tc_fence_after_sync();
    products(0);
    int left = L;
    for (int c = 0; left > 0; ++c) {
      const uint32_t kq = kq_addr + (c & 1) * kStage;
      take_chunk(sm.sc[c & 1].n, left);
      wait_one(&sm.s_ready, c, 921);
      tc_fence_after_sync();
      state_times(kX1, kq);
      umma_commit(&sm.x1);
      if (c > 0) { wait_one(&sm.o_read, c - 1, 922); tc_fence_after_sync(); }
      state_times(kX2, kq + kC * 128);
      umma_commit(&sm.x2);
      // the next chunk's products of keys as early as its loads allow, but not in the way of this chunk's chain
      bool ahead = left == 0;
      for (int turn = 0; turn < 2; ++turn) {
        if (!ahead && (turn == 1 || mbar_try_wait(&sm.full[(c + 1) & 1], ((c + 1) >> 1) & 1))) {
          wait_one(&sm.full[(c + 1) & 1], (c + 1) >> 1, 925);
          tc_fence_after_sync();
          products(c + 1);
          ahead = true;
        }
        if (turn == 0) {
          wait_one(&sm.t_ready, c, 923);
          wait_one(&sm.r_ready, c, 924);
          tc_fence_after_sync();
          tokens_times(kU, kRp, t_addr, 0);
          umma_commit(&sm.u_full);
        }
      }
      wait_one(&sm.ut_ready, c, 926);
      tc_fence_after_sync();
      const uint64_t kt = umma_desc_mn_sw128(kq, kHalf, 1024);
#pragma unroll 1
      for (int pc = 2; pc >= 0; --pc)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ts(tm + kD3, tm + kUt + pc * 32 + k * 8, kt + ((k * 2048) >> 4), id128mn, pc < 2 || k > 0);
      umma_commit(&sm.d3);
      wait_one(&sm.uo_ready, c, 927);
      tc_fence_after_sync();
      tokens_times(kX2, kUo, p_addr + (c & 1) * 3 * kPiece, 1);
      umma_commit(&sm.y[c & 1]);
    }
    umma_commit(&sm.end);
    for (uint32_t i = 0; i < (1u << 16); ++i)          // nothing is in flight when TMEM is given back (bounded)
      if (mbar_try_wait(&sm.end, 0)) break;
    }
  }
  if (failed) ab.raise(failed);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 12) {
    tc_fence_after_sync();
    tmem_dealloc(tm, kTmemCols);
  }
}

}  // namespace gdnc

// Requests of at least `min_len` of the T tokens; the others are left as they are.  Dk = Dv = 128, bf16, L2-normalised q and
// k.  Returns -1, with nothing launched, when q, k or v cannot be read by tensor maps (alignment, strides).
int gdn_chunk(void* out, int64_t o_stride, const void* q, const void* k, int64_t qk_stride, const void* v, int64_t v_stride,
              const float* g, const float* beta, float* states, const int* cu, const int* slots, InitFlags has_init,
              int64_t T, int R, int Hk, int Hv, float scale, int min_len, int* status, cudaStream_t st) {
  CUtensorMap tm[3];
  if (T > INT_MAX || R > 65535 || qk_stride < Hk * 128 || v_stride < Hv * 128) return -1;
  if (b200_encode_tmap_2d(&tm[0], q, T, Hk * 128, qk_stride * 2, gdnc::kC, 64, 2) != 0 ||
      b200_encode_tmap_2d(&tm[1], k, T, Hk * 128, qk_stride * 2, gdnc::kC, 64, 2) != 0 ||
      b200_encode_tmap_2d_raw(&tm[2], v, T, Hv * 256, v_stride * 2, gdnc::kC, 256) != 0)
    return -1;
  gdnc::Params p = {};
  p.out = (__nv_bfloat16*)out; p.g = g; p.beta = beta; p.states = states; p.cu = cu; p.slots = slots; p.has_init = has_init;
  p.status = status; p.o_stride = o_stride; p.Hk = Hk; p.Hv = Hv; p.min_len = min_len; p.scale = scale;
  cudaError_t e = ensure_dynamic_smem((const void*)gdnc::gdn_chunk_kernel, gdnc::kSmemBytes);
  if (e != cudaSuccess) return (int)e;
  gdnc::gdn_chunk_kernel<<<dim3(Hv, R), gdnc::kThreads, gdnc::kSmemBytes, st>>>(tm[0], tm[1], tm[2], p);
  return cudaGetLastError() != cudaSuccess;
}

}  // namespace b200
