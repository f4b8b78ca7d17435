// fp8 (e4m3) GEMM with 128 x 128 weight scales and 1 x 128 activation scales, grouped by expert or dense, for more than a
// few rows a group:  out[r, n] = sum_kb as[kb][r] ws[e][n / 128][kb] sum_{k in kb} x[r, k] W[e(r), n, k].
// (gemm_grouped.cu keeps the narrow tiles of decode batches and the 16-bit forms.)
//
// Here the rows of x are the UMMA M side (128 a tile, one per TMEM lane) and 256 weight rows its N side, so that the scale of
// a k-block is one number per thread and 128 columns: with the weights on the lanes every column has a scale of its own, and
// reading these from shared memory, whose bandwidth the operands take, cost three times the product.
// The tensor core leaves the product of every 128-wide k-block in one of two TMEM slots; eight epilogue warps (thread = a
// row of x, two warpgroups with 64 columns of either block of 128 weight rows) multiply it by the scales into fp32 registers.
// What bounds it: a k-block is 512 tensor-core cycles; the two epilogue warps of a scheduler need 2 x (64 packed
// multiply-adds + 4 TMEM loads), somewhat less.  Warp 2 brings the scales, several k-blocks ahead: loaded one k-block ahead by
// the epilogue itself, a k-block took as long as that load (1300 cycles).
// Measured, us (before: weights on the lanes, four epilogue warps, 128 columns a tile, activation and quantiser in a kernel
// of their own): 4096 x 4096 x 6144 dense with the quantiser in front 148 (354); experts of 4096 tokens, 8 of 128, 2048 -> 2 x 768
// -> 2048, with routing and permutation 430 (1031).
//
// Fused form: the two blocks are 128 gate and the 128 up rows of the same columns; the epilogue rounds both to the model's
// type, applies the activation and writes e4m3 with 1 x 128 scales, as act_mul_quant_fp8_kernel (moe.cu) would.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "../api.h"
#include "../common/launch.cuh"
#include "../common/ptx.cuh"
#include "gemm_common.cuh"

namespace b200 {
namespace gf8 {

constexpr int kM = 128, kN = 256, kBK = 128, kBox = 64;
constexpr int kThreads = 384;
// a thread's registers: 384 x 168 = 64512 at launch, then 128 x (104 + 200 + 200) = 64512
constexpr int kRegsIssue = 104, kRegsEpi = 200;
constexpr int kMaxExperts = 512;
constexpr int kAhead = 4;                                       // k-blocks between the load of a scale and its use
constexpr int kSlots = 2, kStages = 4;                          // TMEM slots of 256 columns, shared-memory stages
constexpr int kBytesA = kM * kBK, kBytesB = kN * kBK, kStage = kBytesA + kBytesB;
constexpr size_t kSmem = 1024 + (size_t)kStages * kStage + (2 * kM + kSlots * (kM + 4)) * 4 + (kMaxExperts + 1) * 4 + 512;

struct Params {
  void* out;            // [M, ldo]
  const void* bias;     // [E, N] or null
  const int* lod;       // [E + 1] or null (one group)
  const float* a_scale; // [K/128, a_stride]
  const float* w_scale; // [E, ceil(N/128), ceil(K/128)]
  int* status;
  // fused form: out is e4m3 [M, N / 2], its scales [N / 256, out_stride]
  float* out_scale;
  int M, N, K, E, ldo, a_stride, out_stride, act;
};

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
template <typename OutT> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
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

template <bool kFused, typename OutT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_grouped_fp8_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  float* amax_smem = reinterpret_cast<float*>(smem + kStages * kStage);   // [2 warpgroups][128 rows]
  float* sc_smem = amax_smem + 2 * kM;                                    // [kSlots][128 rows, 2 weight blocks]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sc_smem + kSlots * (kM + 4));
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  uint64_t* tmem_full = bars + 2 * kStages;       // [kSlots] the product and the scales of a k-block
  uint64_t* tmem_empty = tmem_full + kSlots;      // [kSlots]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + kSlots);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* tile_start = reinterpret_cast<int*>(tmem_slot + 4);                // [E + 1]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb = (p.K + kBK - 1) / kBK, n_blocks = (p.N + 127) / 128;    // blocks of 128 weight rows
  const int n_tiles = (n_blocks + 1) / 2;
  const int E = p.lod ? p.E : 1;
  Abort ab{p.status, abort_flag};
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < kSlots; ++b) { mbar_init(&tmem_full[b], 2); mbar_init(&tmem_empty[b], 8); }
    mbar_fence_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
    griddep_launch();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  griddep_wait();   // lod, x and its scales come from the preceding kernels
  if (warp == 2) {  // exclusive prefix of tiles per expert
    int run = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      int cnt = 0;
      if (e < E) {
        const int rows = p.lod ? (p.lod[e + 1] - p.lod[e]) : p.M;
        cnt = ((rows + kM - 1) / kM) * n_tiles;
      }
      int inc = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffff, inc, o);
        if (lane >= o) inc += v;
      }
      if (e < E) tile_start[e] = run + inc - cnt;
      run += __shfl_sync(0xffffffff, inc, 31);
    }
    if (lane == 0) tile_start[E] = run;
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int total_tiles = tile_start[E];

  // tile -> expert, its two blocks of 128 weight rows (the second one may lie behind the matrix), first row and end of the
  // rows; a role meets its tiles in ascending order
  struct Tile { int e, b0, b1, row0, row_end; };
  auto locate = [&](int tile, Tile& t) {
    while (tile >= tile_start[t.e + 1]) ++t.e;
    const int local = tile - tile_start[t.e], base = p.lod ? p.lod[t.e] : 0, rows = p.lod ? (p.lod[t.e + 1] - base) : p.M;
    const int mt = (rows + kM - 1) / kM, nt = local / mt;
    t.b0 = kFused ? nt : 2 * nt;
    t.b1 = kFused ? nt + n_tiles : 2 * nt + 1;
    t.row0 = base + (local - nt * mt) * kM;
    t.row_end = base + rows;
  };
  Tile t;
  t.e = 0;

  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        locate(tile, t);
        const int boxes = t.row_end - t.row0 > kBox ? 2 : 1;
        const bool two = t.b1 < n_blocks;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!wait_or_abort(&empty_bar[stage], phase ^ 1, ab, 131)) { ok = false; break; }
          uint8_t* sa = smem + stage * kStage;
          mbar_expect_tx(&full_bar[stage], boxes * (kBox * kBK) + (two ? 2 : 1) * (128 * kBK));
          // rows behind the group's are the next group's or outside the tensor (zero fill): they are not written
          for (int b = 0; b < boxes; ++b) tma_load_2d(sa + b * (kBox * kBK), &tmX, &full_bar[stage], kb * kBK, t.row0 + b * kBox);
          tma_load_2d(sa + kBytesA, &tmW, &full_bar[stage], kb * kBK, t.e * p.N + t.b0 * 128);
          if (two) tma_load_2d(sa + kBytesA + 128 * kBK, &tmW, &full_bar[stage], kb * kBK, t.e * p.N + t.b1 * 128);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {   // let the copies in flight land before the CTA's shared memory goes away (bounded)
        for (int s = 0; s < kStages; ++s)
          for (uint32_t q = 0; q < (1u << 14); ++q)
            if (mbar_try_wait(&full_bar[s], phase) || mbar_try_wait(&full_bar[s], phase ^ 1)) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0, it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        locate(tile, t);
        const uint32_t idesc = umma_idesc(kM, t.b1 < n_blocks ? kN : kN / 2, 0, 0);
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int buf = it % kSlots;
          if (!wait_or_abort(&tmem_empty[buf], ((it / kSlots) & 1) ^ 1, ab, 132) ||
              !wait_or_abort(&full_bar[stage], phase, ab, 133)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * kStage);
          const uint64_t da = umma_desc_k_sw128(sa), db = umma_desc_k_sw128(sa + kBytesA);
#pragma unroll
          for (int k = 0; k < kBK / 32; ++k) umma_f8(tmem_base + buf * kN, da + k * 2, db + k * 2, idesc, k > 0 ? 1u : 0u);
          umma_commit(&empty_bar[stage]);
          umma_commit(&tmem_full[buf]);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ scales, loaded kAhead k-blocks before their use
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      locate(tile, t);
      const float* ws = p.w_scale + ((size_t)t.e * n_blocks + ((lane & 1) && t.b1 < n_blocks ? t.b1 : t.b0)) * nkb;
      float a[kAhead][4], w[kAhead];
      auto fetch = [&](int u, int kb) {
        if (kb >= nkb) return;
        w[u] = ws[kb];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = t.row0 + lane + 32 * i;
          a[u][i] = r < t.row_end ? p.a_scale[(size_t)kb * p.a_stride + r] : 0.f;
        }
      };
#pragma unroll
      for (int u = 0; u < kAhead; ++u) fetch(u, u);
      for (int kb0 = 0; kb0 < nkb; kb0 += kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (kb0 + u < nkb && ok) {
            const int buf = it % kSlots;
            ok = !__any_sync(0xffffffffu, !wait_or_abort(&tmem_empty[buf], ((it / kSlots) & 1) ^ 1, ab, 134));
            float* dst = sc_smem + buf * (kM + 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[lane + 32 * i] = a[u][i];
            if (lane < 2) dst[kM + lane] = w[u];
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_full[buf]);
            fetch(u, kb0 + u + kAhead);
            ++it;
          }
        }
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue: thread = row of x
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpi));
    const int half = (warp >> 2) - 1, lane_row = (warp & 3) * 32 + lane;
    const uint32_t tl = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + half * 64;
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
      locate(tile, t);
      __syncwarp();
      const int row = t.row0 + lane_row;
      const bool row_ok = row < t.row_end;
      uint64_t acc[2][32];                             // [block][pair of columns]
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[b][j] = 0;
      for (int kb = 0; kb < nkb && ok; ++kb, ++it) {
        const int buf = it % kSlots;
        if (__any_sync(0xffffffffu, !wait_or_abort(&tmem_full[buf], (it / kSlots) & 1, ab, 135))) { ok = false; break; }
        const float* sc = sc_smem + buf * (kM + 4);
        const float s0 = sc[lane_row] * sc[kM], s1 = sc[lane_row] * sc[kM + 1];
        tc_fence_after_sync();
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const uint64_t s = b == 0 ? f2(s0, s0) : f2(s1, s1);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld_x32(tl + buf * kN + b * 128 + h * 32, r);
            tmem_ld_wait();
            if (b == 1 && h == 1) {                    // the slot has been read
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&tmem_empty[buf]);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
              acc[b][h * 16 + j] = fma2(f2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), s, acc[b][h * 16 + j]);
          }
        }
      }
      const OutT* bias = reinterpret_cast<const OutT*>(p.bias);
      if (bias != nullptr) {
        bias += (size_t)t.e * p.N + half * 64;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int n = (b == 0 ? t.b0 : t.b1) * 128 + 2 * j, limit = p.N - half * 64;
            float v0, v1;
            unf2(acc[b][j], v0, v1);
            acc[b][j] = f2(v0 + (n < limit ? to_float<OutT>(bias[n]) : 0.f), v1 + (n + 1 < limit ? to_float<OutT>(bias[n + 1]) : 0.f));
          }
      }
      if (kFused) {
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float v[2], g[2], u[2];
          unf2(acc[0][j], g[0], g[1]);
          unf2(acc[1][j], u[0], u[1]);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            // rounded where the separate kernels would hand over
            const float gf = to_float<OutT>(from_float<OutT>(g[i])), uf = to_float<OutT>(from_float<OutT>(u[i]));
            float a;
            if (p.act == 0) a = gf / (1.f + __expf(-gf));
            else a = gf / (1.f + __expf(-1.5957691216f * (gf + 0.044715f * gf * gf * gf)));
            v[i] = to_float<OutT>(from_float<OutT>(a * uf));
            amax = fmaxf(amax, fabsf(v[i]));
          }
          acc[0][j] = f2(v[0], v[1]);
        }
        amax_smem[half * kM + lane_row] = amax;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        amax = fmaxf(fmaxf(amax_smem[lane_row], amax_smem[kM + lane_row]), 1e-10f);
        asm volatile("bar.sync 1, 256;" ::: "memory");   // read before the next tile writes it
        const float scale = amax / 448.f, inv = 1.f / scale;
        if (half == 0 && ok && row_ok) p.out_scale[(size_t)t.b0 * p.out_stride + row] = scale;
        uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + (size_t)row * p.ldo + t.b0 * 128 + half * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float v0, v1, v2, v3;
            unf2(acc[0][c * 8 + i * 2], v0, v1);
            unf2(acc[0][c * 8 + i * 2 + 1], v2, v3);
            w[i] = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v0 * inv, v1 * inv), __NV_SATFINITE, __NV_E4M3) |
                   (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v2 * inv, v3 * inv), __NV_SATFINITE, __NV_E4M3) << 16;
          }
          if (ok && row_ok) *reinterpret_cast<uint4*>(dst + c * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      } else if (ok && row_ok) {
        // 16-byte stores where every row of the output allows them
        const bool wide = (p.ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int n0 = (b == 0 ? t.b0 : t.b1) * 128 + half * 64;
          OutT* dst = reinterpret_cast<OutT*>(p.out) + (size_t)row * p.ldo + n0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float v0, v1;
              unf2(acc[b][c * 4 + i], v0, v1);
              w[i] = pack2<OutT>(v0, v1);
            }
            if (wide && n0 + c * 8 + 8 <= p.N) {
              *reinterpret_cast<uint4*>(dst + c * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (n0 + c * 8 + i < p.N) reinterpret_cast<unsigned short*>(dst)[c * 8 + i] = (unsigned short)(w[i / 2] >> (16 * (i & 1)));
            }
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <bool kFused, typename OutT>
static int launch(const GroupedGemmArgs& a, const CUtensorMap& tmW, const CUtensorMap& tmX, cudaStream_t st) {
  auto kern = gemm_grouped_fp8_kernel<kFused, OutT>;
  cudaError_t e = ensure_dynamic_smem((const void*)kern, (int)kSmem);
  if (e != cudaSuccess) return (int)e;
  Params p = {};
  p.out = a.out; p.bias = a.bias; p.lod = a.lod; p.a_scale = a.a_scale; p.w_scale = a.w_scale; p.status = a.status;
  p.M = a.M; p.N = a.N; p.K = a.K; p.E = a.E; p.ldo = a.ldo; p.a_stride = a.a_stride; p.out_scale = a.out_scale;
  p.out_stride = a.out_stride; p.act = a.fused_act;
  return (int)launch_pdl(kern, dim3(a.grid), dim3(kThreads), kSmem, st, tmW, tmX, p);
}

}  // namespace gf8

// `tmX`: x with boxes of 64 rows; `tmW`: boxes of 128.  One CTA an SM (a.grid).
int grouped_fp8_launch(const GroupedGemmArgs& a, const CUtensorMap& tmW, const CUtensorMap& tmX, cudaStream_t st) {
  if (a.E > gf8::kMaxExperts) return 2;
  if (a.out_scale != nullptr) {
    if (a.N % 256 || a.ldo % 16) return 2;
    return a.out_fmt == 1 ? gf8::launch<true, __nv_bfloat16>(a, tmW, tmX, st) : gf8::launch<true, __half>(a, tmW, tmX, st);
  }
  return a.out_fmt == 1 ? gf8::launch<false, __nv_bfloat16>(a, tmW, tmX, st) : gf8::launch<false, __half>(a, tmW, tmX, st);
}

}  // namespace b200
