// Gated DeltaNet (Qwen3-Next linear-attention layers) device ops: varlen causal conv1d with a state
// cache, single-token conv update, gating, and the gated delta rule as a sequential scan that keeps the
// [Dv, Dk] state of one head in registers.
//
// Reference entry points: kunlun_ops.causal_conv1d_fn / causal_conv1d_update
// (vllm_kunlun/ops/mamba/causal_conv1d.py:15-74,118-225), fused_gdn_gating (models/qwen3_next.py:262-781),
// fused_recurrent_gated_delta_rule (ops/fla/fused_recurrent.py:52-155) and the chunked form
// (ops/fla/chunk.py:23-140), which is numerically the same recurrence.
#include "../api.h"
#include "../common/launch.cuh"
#include "../common/utils.cuh"

#include <limits.h>

namespace b200 {
// gdn_chunk.cu
int gdn_chunk(void* out, int64_t o_stride, const void* q, const void* k, int64_t qk_stride, const void* v, int64_t v_stride,
              const float* g, const float* beta, float* states, const int* cu, const int* slots, InitFlags has_init,
              int64_t T, int R, int Hk, int Hv, float scale, int min_len, int* status, cudaStream_t st);

namespace {

// fp32 tensors keep full fp32 accuracy (this file is compiled without fast-math); 16-bit outputs use the fast forms
template <typename T> __device__ __forceinline__ float silu(float v) { return __fdividef(v, 1.f + __expf(-v)); }
template <> __device__ __forceinline__ float silu<float>(float v) { return v / (1.f + expf(-v)); }

__device__ __forceinline__ int find_seq(const int* __restrict__ cu, int R, int t) {
  int lo = 0, hi = R;  // largest r with cu[r] <= t
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (cu[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// y[t, c] = act(bias[c] + sum_j w[c, j] * in[t - (W-1) + j, c]); positions before the sequence start read
// the cached state (rows W-1+p.. of the previous inputs) or zero.
// One thread = one 16-byte channel vector x kTok consecutive tokens, with a sliding window of the last W-1 input rows in
// registers, so every input row is loaded once per thread; the loads of kBatch rows are in flight together.  A request's first row
// in a thread costs a chain of loads (offsets, slot, history), one request after the other, so many short requests want few
// tokens a thread, and long ones many, for the taps and the window's first rows.
template <typename T, int W, int kTok, int kBatch>
__global__ void __launch_bounds__(128) conv1d_fwd_kernel(T* __restrict__ out, int64_t out_stride, const T* __restrict__ x,
                                                         int64_t x_stride, const T* __restrict__ w, const T* __restrict__ bias,
                                                         const int* __restrict__ cu, int R, const T* __restrict__ states,
                                                         const int* __restrict__ slots, InitFlags has_init,
                                                         int C, int act, int64_t Ttot) {
  constexpr int V = Vec16<T>::N;
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  const int64_t t0 = (int64_t)blockIdx.y * kTok;
  if (c0 >= C || t0 >= Ttot) return;
  float wv[W][V], bv[V];
  const T* wc = w + (int64_t)c0 * W;              // the V channels' taps are V * W consecutive numbers
  if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const Vec16<T> a = ld_vec(wc + i * V);
#pragma unroll
      for (int e = 0; e < V; ++e) wv[(i * V + e) % W][(i * V + e) / W] = to_f(a.v[e]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < W * V; ++i) wv[i % W][i / W] = to_f(wc[i]);
  }
#pragma unroll
  for (int e = 0; e < V; ++e) bv[e] = bias ? to_f(bias[c0 + e]) : 0.f;
  float win[W][V];  // win[j] = input row at (current token) - (W-1) + j
  int r = find_seq(cu, R, (int)t0);
  int seq_start = cu[r], seq_end = cu[r + 1];
  auto load_hist = [&](int64_t t) {  // fill win[0 .. W-2] with the W-1 rows in front of token t
    const int p = (int)t - seq_start;
    const int slot = slots[r];
    const bool init = has_init[r] && slot >= 0;
#pragma unroll
    for (int j = 0; j < W - 1; ++j) {
      const int q = p - (W - 1) + j;
      if (q >= 0) {
        Vec16<T> v = ld_vec(x + (t - (W - 1) + j) * x_stride + c0);
#pragma unroll
        for (int e = 0; e < V; ++e) win[j][e] = to_f(v.v[e]);
      } else if (init) {
        Vec16<T> v = ld_vec(states + ((int64_t)slot * (W - 1) + (W - 1 + q)) * C + c0);
#pragma unroll
        for (int e = 0; e < V; ++e) win[j][e] = to_f(v.v[e]);
      } else {
#pragma unroll
        for (int e = 0; e < V; ++e) win[j][e] = 0.f;
      }
    }
  };
  load_hist(t0);
#pragma unroll 1
  for (int i0 = 0; i0 < kTok; i0 += kBatch) {
    Vec16<T> rows[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
      if (t0 + i0 + i < Ttot) rows[i] = ld_vec(x + (t0 + i0 + i) * x_stride + c0);
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int64_t t = t0 + i0 + i;
      if (t >= Ttot) return;
      if (t >= seq_end) {  // crossed into the next (non-empty) sequence: its history comes from its own state
        while (t >= seq_end) { ++r; seq_start = cu[r]; seq_end = cu[r + 1]; }
        load_hist(t);
      }
      Vec16<T> o;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        win[W - 1][e] = to_f(rows[i].v[e]);
        float acc = bv[e];
#pragma unroll
        for (int j = 0; j < W; ++j) acc += wv[j][e] * win[j][e];
        o.v[e] = from_f<T>(act ? silu<T>(acc) : acc);
      }
      st_vec(out + t * out_stride + c0, o);
#pragma unroll
      for (int j = 0; j < W - 1; ++j) {
#pragma unroll
        for (int e = 0; e < V; ++e) win[j][e] = win[j + 1][e];
      }
    }
  }
}

// Any number of taps: one thread per (token, channel), every input row read from memory.
template <typename T>
__global__ void conv1d_fwd_generic_kernel(T* __restrict__ out, int64_t out_stride, const T* __restrict__ x, int64_t x_stride,
                                          const T* __restrict__ w, const T* __restrict__ bias, const int* __restrict__ cu,
                                          int R, const T* __restrict__ states, const int* __restrict__ slots,
                                          InitFlags has_init, int C, int W, int act, int64_t Ttot) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t = blockIdx.y;
  if (c >= C || t >= Ttot) return;
  const int r = find_seq(cu, R, (int)t);
  const int p = (int)t - cu[r], slot = slots[r];
  const bool init = has_init[r] && slot >= 0;
  float acc = bias ? to_f(bias[c]) : 0.f;
  for (int j = 0; j < W; ++j) {
    const int q = p - (W - 1) + j;
    float v = 0.f;
    if (q >= 0) v = to_f(x[(t - (W - 1) + j) * x_stride + c]);
    else if (init) v = to_f(states[((int64_t)slot * (W - 1) + (W - 1 + q)) * C + c]);
    acc += to_f(w[(int64_t)c * W + j]) * v;
  }
  out[t * out_stride + c] = from_f<T>(act ? silu<T>(acc) : acc);
}

// states[slot] <- last W-1 rows of (old state ++ x[seq]); one thread owns a channel column.  Row j takes old row
// j + L (or an input row): ascending j never reads a row it has already overwritten.
template <typename T>
__global__ void conv1d_state_kernel(T* __restrict__ states, const T* __restrict__ x, int64_t x_stride,
                                    const int* __restrict__ cu, const int* __restrict__ slots,
                                    InitFlags has_init, int C, int W) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (c >= C) return;
  const int s = cu[r], L = cu[r + 1] - s, slot = slots[r];
  if (L == 0 || slot < 0) return;
  const bool init = has_init[r];
  T* st = states + (int64_t)slot * (W - 1) * C + c;
  for (int j = 0; j < W - 1; ++j) {
    const int q = L - (W - 1) + j;
    T v = from_f<T>(0.f);
    if (q >= 0) v = x[(int64_t)(s + q) * x_stride + c];
    else if (init) v = st[(int64_t)(j + L) * C];
    st[(int64_t)j * C] = v;
  }
}

// One token per sequence.  `has_init` (optional): a row whose flag is 0 starts from zeros, whatever its slot holds.
template <typename T>
__global__ void conv1d_update_kernel(T* out, int64_t out_stride, const T* x, int64_t x_stride,
                                     T* states, const T* w, const T* bias,
                                     const int* slots, const int* has_init, int C, int W, int act) {
  griddep_launch();
  griddep_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (c >= C) return;
  const int slot = slots[b];
  if (slot < 0) { out[(int64_t)b * out_stride + c] = from_f<T>(0.f); return; }
  const bool init = has_init == nullptr || has_init[b] != 0;
  T* st = states + (int64_t)slot * (W - 1) * C + c;
  float acc = bias ? to_f(bias[c]) : 0.f;
  float cur = to_f(x[(int64_t)b * x_stride + c]);
  for (int j = 0; j < W - 1; ++j) {
    float v = init ? to_f(st[(int64_t)j * C]) : 0.f;
    acc += to_f(w[(int64_t)c * W + j]) * v;
    if (j > 0) st[(int64_t)(j - 1) * C] = from_f<T>(v);
  }
  acc += to_f(w[(int64_t)c * W + W - 1]) * cur;
  if (W > 1) st[(int64_t)(W - 2) * C] = from_f<T>(cur);
  out[(int64_t)b * out_stride + c] = from_f<T>(act ? silu<T>(acc) : acc);
}

// g = -exp(A_log) * softplus(a + dt_bias), beta = sigmoid(b)
template <typename T>
__global__ void gdn_gating_kernel(float* __restrict__ g, float* __restrict__ beta, const T* __restrict__ a, int64_t a_stride,
                                  const T* __restrict__ b, int64_t b_stride, const float* __restrict__ A_log,
                                  const float* __restrict__ dt_bias, int H, int64_t T_) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= T_ * H) return;
  int64_t t = i / H;
  int h = (int)(i % H);
  float xa = to_f(a[t * a_stride + h]) + dt_bias[h];
  float sp = xa > 20.f ? xa : log1pf(__expf(xa));
  g[i] = -__expf(A_log[h]) * sp;
  beta[i] = __fdividef(1.f, 1.f + __expf(-to_f(b[t * b_stride + h])));
}

// Sequential gated delta rule.  Block = 128 threads = 32 state rows (of Dv) x 4 quarters of Dk; grid
// (Dv/32, Hv, sequences).  Per token: S *= exp(g); pred = S k; S += beta (v - pred) k^T; o = S q.
// Tokens are staged through shared memory in chunks of kGdnChunk: while the block works through one chunk
// (no block-wide barrier inside: a row's four quarter-threads are adjacent lanes), every thread already holds its
// share of the next chunk's q / k / v / g / beta in registers, so global-memory latency never sits on the
// recurrence and the block synchronises twice per chunk instead of once per token.
constexpr int kGdnChunk = 16;
// New tokens of a request from which gdn_chunk.cu takes it.  While every head has an SM of its own the scan costs 10 us + 0.5 us a
// token and 64 tokens in chunk form 21 us (one request of 24 / 48 / 64 tokens, 32 heads: scan 18.0 / 27.5 / 35.7 us); with more
// heads than SMs the scan's blocks share them (8 requests of 24 tokens: scan 62.6 us, chunk form 44).
constexpr int kGdnChunkMin = 40, kGdnChunkMinMany = 16;
// Most rows of a request for which gdn_step_kernel is launched when the lengths are known.  With SMs to spare the row counts: one
// request, 32 heads, 2 / 4 / 8 / 16 rows: scan 11 / 12 / 14 / 18 us, step 9 / 12 / 16 / 26.  From half as many heads as SMs the
// states' traffic does: 4 requests scan 17 / 21 / 27 / 36, step 12 / 14 / 20 / 29; 64 requests scan 117 / 146 / 197 / 283, step
// 53 / 72 / 117 / 211.
constexpr int kGdnStepMax = 4, kGdnStepMaxMany = 16;

template <typename T, int DK>
__global__ void __launch_bounds__(128) gdn_recurrent_kernel(
    T* __restrict__ out, int64_t o_stride, const T* __restrict__ q, const T* __restrict__ k, int64_t qk_stride,
    const T* __restrict__ v, int64_t v_stride, const float* __restrict__ g, const float* __restrict__ beta,
    float* __restrict__ states /*[slots, Hv, Dv, DK]*/, const int* __restrict__ cu, const int* __restrict__ slots,
    InitFlags has_init, int Hk, int Hv, int Dv, float scale, int l2norm, int chunk_min) {
  static_assert(DK % 16 == 0 && DK <= 128, "DK");
  constexpr int QW = DK / 4;                      // state columns per thread
  constexpr int CH = kGdnChunk;
  constexpr int QK_PER = CH * DK / 128;           // q (and k) elements of a chunk per thread
  constexpr int V_PER = CH * 32 / 128;            // v elements of a chunk per thread
  __shared__ __align__(16) float sk[CH][DK];
  __shared__ __align__(16) float sq[CH][DK];
  __shared__ float sv[CH][32];
  __shared__ float sg[CH], sb[CH], srk[CH], srq[CH];
  const int tid = threadIdx.x, rl = tid >> 2, qd = tid & 3, warp = tid >> 5, lane = tid & 31;
  const int hv = blockIdx.y, r = blockIdx.z, hk = hv / (Hv / Hk);
  const int row0 = blockIdx.x * 32, row = row0 + rl;
  const int s = cu[r], L = cu[r + 1] - s, slot = slots[r];
  if (L == 0 || L >= chunk_min || slot < 0) return;
  // Column ownership is interleaved in 16-byte pieces: registers S[4i .. 4i+3] of quarter qd hold columns
  // 16 i + 4 qd .. + 3, so that the four quarter-lanes of a row read four consecutive float4 of the shared k / q row
  // (distinct banks) instead of four addresses 128 bytes apart (one bank, a 4-way conflict on every load).
  float* sp = states + (((int64_t)slot * Hv + hv) * Dv + row) * DK + qd * 4;
  float S[QW];
  if (has_init[r]) {
#pragma unroll
    for (int j = 0; j < QW; j += 4) *reinterpret_cast<float4*>(&S[j]) = *reinterpret_cast<const float4*>(sp + j * 4);
  } else {
#pragma unroll
    for (int j = 0; j < QW; ++j) S[j] = 0.f;
  }
  // register staging of one chunk: element e of the flattened [CH, DK] (resp. [CH, 32]) tile, e = i * 128 + tid
  float rk_[QK_PER], rq_[QK_PER], rv_[V_PER], rg = 0.f, rb = 0.f;
  auto fetch = [&](int c0) {
#pragma unroll
    for (int i = 0; i < QK_PER; ++i) {
      const int e = i * 128 + tid, t = e / DK, d = e % DK;
      const bool ok = c0 + t < L;
      const int64_t tok = s + c0 + t;
      rk_[i] = ok ? to_f(k[tok * qk_stride + hk * DK + d]) : 0.f;
      rq_[i] = ok ? to_f(q[tok * qk_stride + hk * DK + d]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < V_PER; ++i) {
      const int e = i * 128 + tid, t = e / 32, d = e % 32;
      rv_[i] = (c0 + t < L) ? to_f(v[(int64_t)(s + c0 + t) * v_stride + hv * Dv + row0 + d]) : 0.f;
    }
    if (tid < CH && c0 + tid < L) {
      rg = g[(int64_t)(s + c0 + tid) * Hv + hv];
      rb = beta[(int64_t)(s + c0 + tid) * Hv + hv];
    }
  };
  fetch(0);
  for (int c0 = 0; c0 < L; c0 += CH) {
    __syncthreads();  // the previous chunk has been consumed
#pragma unroll
    for (int i = 0; i < QK_PER; ++i) {
      const int e = i * 128 + tid;
      sk[e / DK][e % DK] = rk_[i];
      sq[e / DK][e % DK] = rq_[i];
    }
#pragma unroll
    for (int i = 0; i < V_PER; ++i) {
      const int e = i * 128 + tid;
      sv[e / 32][e % 32] = rv_[i];
    }
    if (tid < CH) { sg[tid] = __expf(rg); sb[tid] = rb; }
    __syncthreads();
    // squared norms: warp w handles tokens w, w + 4, ...
    for (int t = warp; t < CH; t += 4) {
      float k2 = 0.f, q2 = 0.f;
      for (int d = lane; d < DK; d += 32) { k2 += sk[t][d] * sk[t][d]; q2 += sq[t][d] * sq[t][d]; }
      k2 = warp_sum(k2);
      q2 = warp_sum(q2);
      if (lane == 0) {
        srk[t] = l2norm ? rsqrtf(k2 + 1e-6f) : 1.f;
        srq[t] = l2norm ? scale * rsqrtf(q2 + 1e-6f) : scale;
      }
    }
    if (c0 + CH < L) fetch(c0 + CH);  // next chunk's global loads fly while this one is processed
    __syncthreads();
    const int n = min(CH, L - c0);
    for (int t = 0; t < n; ++t) {
      const float gt = sg[t], bt = sb[t], vt = sv[t][rl], rk = srk[t], rq = srq[t];
      const float* kk = &sk[t][qd * 4];
      const float* qq = &sq[t][qd * 4];
      float pred = 0.f, pred2 = 0.f;
#pragma unroll
      for (int j = 0; j < QW; j += 4) {
        float4 k4 = *reinterpret_cast<const float4*>(kk + j * 4);
        S[j] *= gt; S[j + 1] *= gt; S[j + 2] *= gt; S[j + 3] *= gt;
        pred += S[j] * k4.x + S[j + 1] * k4.y;
        pred2 += S[j + 2] * k4.z + S[j + 3] * k4.w;
      }
      pred += pred2;
      pred += __shfl_xor_sync(0xffffffff, pred, 1);
      pred += __shfl_xor_sync(0xffffffff, pred, 2);
      const float delta = (vt - pred * rk) * bt * rk;
      float o = 0.f, o2 = 0.f;
#pragma unroll
      for (int j = 0; j < QW; j += 4) {
        float4 k4 = *reinterpret_cast<const float4*>(kk + j * 4);
        float4 q4 = *reinterpret_cast<const float4*>(qq + j * 4);
        S[j] += delta * k4.x; S[j + 1] += delta * k4.y; S[j + 2] += delta * k4.z; S[j + 3] += delta * k4.w;
        o += S[j] * q4.x + S[j + 1] * q4.y;
        o2 += S[j + 2] * q4.z + S[j + 3] * q4.w;
      }
      o += o2;
      o += __shfl_xor_sync(0xffffffff, o, 1);
      o += __shfl_xor_sync(0xffffffff, o, 2);
      if (qd == 0) out[(int64_t)(s + c0 + t) * o_stride + hv * Dv + row] = from_f<T>(o * rq);
    }
  }
#pragma unroll
  for (int j = 0; j < QW; j += 4) *reinterpret_cast<float4*>(sp + j * 4) = *reinterpret_cast<const float4*>(&S[j]);
}

// The same for a few tokens a request (decode, verification): bound by reading and writing the states, 128 KB a head and
// request.  A warp owns eight rows of a 128-wide state, a lane four columns of each; all eight are in flight at once, q and k
// come straight from memory, and eight row sums are folded together (9 exchanges instead of 40).  No shared memory and no barrier:
// 64 requests, 32 heads (268 MB) 39 us, 96 in the scan above.  Some 11 us a further row there, which the exchanges and sums take: q,
// k and v a row ahead are worth it in 32 bits only (64 requests, four rows each: 71 us, 82 without; in bf16 79, 72 without).
__device__ __forceinline__ float sum_of_8(float (&v)[8], int lane) {   // lane l returns the sum over the warp of v[l / 4]
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {
    const bool up = lane & (4 * h);
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffff, give, 4 * h);
    }
  }
  float s = v[0];
  s += __shfl_xor_sync(0xffffffff, s, 2);
  return s + __shfl_xor_sync(0xffffffff, s, 1);
}
template <typename T> struct alignas(4 * sizeof(T)) Four { T v[4]; };
template <typename T> __device__ __forceinline__ Four<T> ld4(const T* p) { return *reinterpret_cast<const Four<T>*>(p); }
template <typename T> __device__ __forceinline__ float4 to_f4(const Four<T>& a) {
  return make_float4(to_f(a.v[0]), to_f(a.v[1]), to_f(a.v[2]), to_f(a.v[3]));
}

template <typename T>
__global__ void __launch_bounds__(128) gdn_step_kernel(
    T* __restrict__ out, int64_t o_stride, const T* __restrict__ q, const T* __restrict__ k, int64_t qk_stride,
    const T* __restrict__ v, int64_t v_stride, const float* __restrict__ g, const float* __restrict__ beta,
    float* __restrict__ states /*[slots, Hv, Dv, 128]*/, const int* __restrict__ cu, const int* __restrict__ slots,
    InitFlags has_init, int Hk, int Hv, int Dv, float scale, int l2norm, int limit) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hv = blockIdx.y, r = blockIdx.z, hk = hv / (Hv / Hk), row0 = blockIdx.x * 32 + warp * 8;
  const int s = cu[r], L = cu[r + 1] - s, slot = slots[r];
  if (L == 0 || L >= limit || slot < 0) return;
  float4* sp = reinterpret_cast<float4*>(states + (((int64_t)slot * Hv + hv) * Dv + row0) * 128) + lane;
  float4 S[8];
  const bool init = has_init[r];
#pragma unroll
  for (int i = 0; i < 8; ++i) S[i] = init ? sp[i * 32] : make_float4(0.f, 0.f, 0.f, 0.f);
  struct Token { Four<T> k, q; T v; float g, beta; } next;   // as they are in memory: a conversion would wait for the load
  auto fetch = [&](int t) {
    next.k = ld4(k + t * qk_stride + hk * 128 + lane * 4);
    next.q = ld4(q + t * qk_stride + hk * 128 + lane * 4);
    next.v = v[t * v_stride + hv * Dv + row0 + (lane >> 2)];   // of the row whose sum this lane gets
    next.g = g[(int64_t)t * Hv + hv];
    next.beta = beta[(int64_t)t * Hv + hv];
  };
  constexpr bool kAhead = sizeof(T) == 4;
  if (kAhead) fetch(s);
  for (int t = s; t < s + L; ++t) {
    if (!kAhead) fetch(t);
    const float4 kk = to_f4(next.k), qq = to_f4(next.q);
    const float gt = __expf(next.g), bt = next.beta, vt = to_f(next.v);
    if (kAhead && t + 1 < s + L) fetch(t + 1);
    float rk = 1.f, rq = scale;
    if (l2norm) {
      rk = rsqrtf(warp_sum(kk.x * kk.x + kk.y * kk.y + kk.z * kk.z + kk.w * kk.w) + 1e-6f);
      rq = scale * rsqrtf(warp_sum(qq.x * qq.x + qq.y * qq.y + qq.z * qq.z + qq.w * qq.w) + 1e-6f);
    }
    float part[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      S[i].x *= gt; S[i].y *= gt; S[i].z *= gt; S[i].w *= gt;
      part[i] = (S[i].x * kk.x + S[i].y * kk.y) + (S[i].z * kk.z + S[i].w * kk.w);
    }
    const float delta = (vt - sum_of_8(part, lane) * rk) * bt * rk;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float d = __shfl_sync(0xffffffff, delta, i * 4);
      S[i].x += d * kk.x; S[i].y += d * kk.y; S[i].z += d * kk.z; S[i].w += d * kk.w;
      part[i] = (S[i].x * qq.x + S[i].y * qq.y) + (S[i].z * qq.z + S[i].w * qq.w);
    }
    const float o = sum_of_8(part, lane);
    if ((lane & 3) == 0) out[(int64_t)t * o_stride + hv * Dv + row0 + (lane >> 2)] = from_f<T>(o * rq);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) sp[i * 32] = S[i];
}

// MTP input glue: out[t] = [rmsnorm(embed[t]) * (pos != 0), rmsnorm(hidden[t])]  (deepseek_mtp.py:79-87)
template <typename T>
__global__ void mtp_concat_norm_kernel(T* __restrict__ out, const T* __restrict__ embed, const T* __restrict__ hidden,
                                       const T* __restrict__ we, const T* __restrict__ wh, const int64_t* __restrict__ pos,
                                       int H, float eps) {
  __shared__ float red[32];
  const int64_t t = blockIdx.x;
  const bool zero = pos && pos[t] == 0;
  float se = 0.f, sh = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float e = zero ? 0.f : to_f(embed[t * H + i]), h = to_f(hidden[t * H + i]);
    se += e * e;
    sh += h * h;
  }
  se = block_sum(se, red);
  sh = block_sum(sh, red);
  const float re = rsqrtf(se / H + eps), rh = rsqrtf(sh / H + eps);
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float e = zero ? 0.f : to_f(embed[t * H + i]), h = to_f(hidden[t * H + i]);
    out[t * 2 * H + i] = from_f<T>(e * re * to_f(we[i]));
    out[t * 2 * H + H + i] = from_f<T>(h * rh * to_f(wh[i]));
  }
}

// out[t, i] = o[t, i] * sigmoid(gate[t, i]) with a strided gate (column slice of a fused projection)
template <typename T>
__global__ void sigmoid_gate_mul_kernel(T* __restrict__ out, const T* __restrict__ o, const T* __restrict__ gate,
                                        int64_t gate_stride, int D, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t t = i / D;
  int c = (int)(i % D);
  float gv = to_f(gate[t * gate_stride + c]);
  out[i] = from_f<T>(__fdividef(to_f(o[i]), 1.f + __expf(-gv)));
}

}  // namespace
}  // namespace b200

namespace b200 {
namespace {
template <typename T>
int launch_conv_fwd(void* out, int64_t out_stride, const void* x, int64_t x_stride, const void* w, const void* bias,
                    const int* cu, int R, void* states, const int* slots, InitFlags has_init, int C, int W, int act,
                    int64_t T_, cudaStream_t st) {
  constexpr int V = Vec16<T>::N;
  if (C % V != 0 || (x_stride % V) != 0 || (out_stride % V) != 0) return 3;
  dim3 g2((C + 255) / 256, R);
  const bool fits = T_ <= 8 * 65535;   // as blocks of eight tokens into a grid
#define B200_CONV(WW, TOK, BATCH)                                                                                            \
  conv1d_fwd_kernel<T, WW, TOK, BATCH><<<dim3((C / V + 127) / 128, (unsigned)((T_ + TOK - 1) / TOK)), 128, 0, st>>>(            \
      (T*)out, out_stride, (const T*)x, x_stride, (const T*)w, (const T*)bias, cu, R, (const T*)states, slots, has_init, C, act, T_)
  // Up to four taps: eight tokens a thread, four rows in flight (eight of 32-bit numbers, which are half as many).  us with 8 and with
  // 16 tokens, bf16, 8192 channels, four taps: 4 x 2048 tokens 97 and 97, 64 x 1 20 and 29, 63 x 1 + 2048 42 and 52; fp32 124 and 137.
#define B200_CONV_FEW(WW) \
  if (fits) B200_CONV(WW, 8, (sizeof(T) == 4 ? 8 : 4)); else B200_CONV(WW, 16, 8)
  // More: the window's first rows weigh more, so sixteen, but where requests are short and few tokens in all hide the chain.  4096
  // channels, eight taps: 4 x 2048 tokens 125 and 95, 63 x 1 + 2048 52 and 83, 255 x 1 + 8192 165 and 132.
#define B200_CONV_MANY(WW) \
  if (fits && T_ < 64 * (int64_t)R && T_ * (C / V) < (2 << 20)) B200_CONV(WW, 8, 8); else B200_CONV(WW, 16, 8)
  switch (W) {
    case 1: B200_CONV_FEW(1); break;
    case 2: B200_CONV_FEW(2); break;
    case 3: B200_CONV_FEW(3); break;
    case 4: B200_CONV_FEW(4); break;
    case 5: B200_CONV_MANY(5); break;
    case 6: B200_CONV_MANY(6); break;
    case 7: B200_CONV_MANY(7); break;
    case 8: B200_CONV_MANY(8); break;
    default:
      if (T_ > 65535) return 3;
      conv1d_fwd_generic_kernel<T><<<dim3((C + 127) / 128, (unsigned)T_), 128, 0, st>>>(
          (T*)out, out_stride, (const T*)x, x_stride, (const T*)w, (const T*)bias, cu, R, (const T*)states, slots, has_init, C,
          W, act, T_);
  }
#undef B200_CONV_MANY
#undef B200_CONV_FEW
#undef B200_CONV
  if (W == 1) return cudaGetLastError() != cudaSuccess;  // no history to keep
  conv1d_state_kernel<T><<<g2, 256, 0, st>>>((T*)states, (const T*)x, x_stride, cu, slots, has_init, C, W);
  return cudaGetLastError() != cudaSuccess;
}
}  // namespace
}  // namespace b200

extern "C" int b200_causal_conv1d_fwd(void* out, int64_t out_stride, const void* x, int64_t x_stride, const void* w,
                                      const void* bias, const int* cu, int R, void* states, const int* slots,
                                      const void* has_init, int init_wide, int C, int W, int act, int64_t T_, int dtype, cudaStream_t st) {
  if (W < 1) return 3;
  if (T_ == 0) return 0;
  B200_DISPATCH_DTYPE(dtype, return (b200::launch_conv_fwd<T>(out, out_stride, x, x_stride, w, bias, cu, R, states, slots,
                                                              b200::InitFlags{has_init, init_wide}, C, W, act, T_, st)));
  return 1;
}

extern "C" int b200_causal_conv1d_update(void* out, int64_t out_stride, const void* x, int64_t x_stride, void* states,
                                         const void* w, const void* bias, const int* slots, const int* has_init,
                                         int64_t B, int C, int W, int act, int dtype, cudaStream_t st) {
  if (W < 1) return 3;
  if (B == 0) return 0;
  dim3 g((C + 255) / 256, (unsigned)B);
  B200_DISPATCH_DTYPE(dtype, (b200::launch_pdl(b200::conv1d_update_kernel<T>, g, dim3(256), 0, st, (T*)out, out_stride,
                                               (const T*)x, x_stride, (T*)states, (const T*)w, (const T*)bias, slots, has_init,
                                               C, W, act)));
  return cudaGetLastError() != cudaSuccess;
}

extern "C" int b200_gdn_gating(float* g, float* beta, const void* a, int64_t a_stride, const void* b, int64_t b_stride,
                               const float* A_log, const float* dt_bias, int H, int64_t T_, int dtype, cudaStream_t st) {
  if (T_ == 0) return 0;
  unsigned blocks = (unsigned)((T_ * H + 255) / 256);
  B200_DISPATCH_DTYPE(dtype, (b200::gdn_gating_kernel<T><<<blocks, 256, 0, st>>>(g, beta, (const T*)a, a_stride, (const T*)b,
                                                                                 b_stride, A_log, dt_bias, H, T_)));
  return cudaGetLastError() != cudaSuccess;
}

// Which kernels a call of the rule takes.  `lens`: rows of every request as the host knows them, or null.  Returns the rows of a
// request from which gdn_chunk.cu takes it (INT_MAX: none), and in `step` whether the others go through gdn_step_kernel or the scan.
// These are choices of speed only: the kernels go by the lengths on the device, and every length has one that serves it.
//  - Chunks where a request is long enough.  Without `lens` the longest may have T - (R - 1) rows, each of the others one; at two
//    rows a request or less on average all are taken for decoding or verification.
//  - The step kernel where none of the other requests has more rows than kGdnStepMax.  63 decoding requests beside one of 2048 tokens,
//    32 heads: 314 us with the scan for the 63, 267 with the step kernel; 64 verified requests of 2 rows 130 (an empty launch of the
//    chunk kernel and the scan) and 53.
extern "C" int b200_gdn_route(int64_t T_, int R, int Hv, int num_sms, int chunkable, const int* lens, int* step) {
  const int min_len = (int64_t)R * Hv > num_sms ? b200::kGdnChunkMinMany : b200::kGdnChunkMin;
  const int step_max = (int64_t)R * Hv > num_sms / 2 ? b200::kGdnStepMaxMany : b200::kGdnStepMax;
  int64_t longest = T_ <= 2 * (int64_t)R ? 0 : T_ - (R - 1);
  if (lens != nullptr) {
    longest = 0;
    for (int r = 0; r < R; ++r) longest = lens[r] > longest ? lens[r] : longest;
  }
  const bool chunk = chunkable && longest >= min_len;
  const int chunk_min = !chunk ? INT_MAX : R == 1 ? 1 : min_len;   // a lone request needs no second launch
  *step = lens != nullptr || longest == 0;
  if (lens != nullptr)
    for (int r = 0; r < R; ++r) *step &= lens[r] <= step_max || lens[r] >= chunk_min;
  return chunk_min;
}

extern "C" int b200_gdn_recurrent(void* out, int64_t o_stride, const void* q, const void* k, int64_t qk_stride, const void* v,
                                  int64_t v_stride, const float* g, const float* beta, float* states, const int* cu,
                                  const int* slots, const void* has_init, int init_wide, int R, int Hk, int Hv, int Dk, int Dv, float scale,
                                  int l2norm, int dtype, int64_t T_, const int* lens, int num_sms, int* status, cudaStream_t st) {
  if (R == 0) return 0;
  if (Dv % 32 != 0 || Hv % Hk != 0) return 3;
  const b200::InitFlags flags{has_init, init_wide};
  int step, chunk_min = b200_gdn_route(T_, R, Hv, num_sms, status != nullptr, lens, &step);
  if (chunk_min != INT_MAX) {
    const int rc = b200::gdn_chunk(out, o_stride, q, k, qk_stride, v, v_stride, g, beta, states, cu, slots, flags, T_, R, Hk,
                                   Hv, scale, chunk_min, status, st);
    if (rc > 0) return rc;
    if (rc == 0 && R == 1) return 0;
    if (rc < 0) chunk_min = b200_gdn_route(T_, R, Hv, num_sms, 0, lens, &step);
  }
  dim3 grid(Dv / 32, Hv, R);
  const size_t esz = dtype == b200::kF32 ? 4 : 2, vec = 4 * esz;
  auto aligned = [&](const void* x) { return reinterpret_cast<uintptr_t>(x) % vec == 0; };
  if (step && Dk == 128 && qk_stride % 4 == 0 && aligned(q) && aligned(k)) {
    B200_DISPATCH_DTYPE(dtype, (b200::gdn_step_kernel<T><<<grid, 128, 0, st>>>(
                                   (T*)out, o_stride, (const T*)q, (const T*)k, qk_stride, (const T*)v, v_stride, g, beta,
                                   states, cu, slots, flags, Hk, Hv, Dv, scale, l2norm, chunk_min)));
    return cudaGetLastError() != cudaSuccess;
  }
#define B200_GDN_LAUNCH(DK)                                                                                          \
  B200_DISPATCH_DTYPE(dtype, (b200::gdn_recurrent_kernel<T, DK><<<grid, 128, 0, st>>>(                                  \
                                 (T*)out, o_stride, (const T*)q, (const T*)k, qk_stride, (const T*)v, v_stride, g, beta, \
                                 states, cu, slots, flags, Hk, Hv, Dv, scale, l2norm, chunk_min)))
  if (Dk == 128) { B200_GDN_LAUNCH(128); }
  else if (Dk == 64) { B200_GDN_LAUNCH(64); }
  else if (Dk == 32) { B200_GDN_LAUNCH(32); }
  else if (Dk == 16) { B200_GDN_LAUNCH(16); }
  else return 3;
#undef B200_GDN_LAUNCH
  return cudaGetLastError() != cudaSuccess;
}

extern "C" int b200_mtp_concat_norm(void* out, const void* embed, const void* hidden, const void* we, const void* wh,
                                    const int64_t* pos, int64_t T_, int H, float eps, int dtype, cudaStream_t st) {
  if (T_ == 0) return 0;
  B200_DISPATCH_DTYPE(dtype, (b200::mtp_concat_norm_kernel<T><<<(unsigned)T_, 512, 0, st>>>(
                                 (T*)out, (const T*)embed, (const T*)hidden, (const T*)we, (const T*)wh, pos, H, eps)));
  return cudaGetLastError() != cudaSuccess;
}

extern "C" int b200_sigmoid_gate_mul(void* out, const void* o, const void* gate, int64_t gate_stride, int D, int64_t T_,
                                     int dtype, cudaStream_t st) {
  if (T_ == 0) return 0;
  int64_t n = T_ * D;
  B200_DISPATCH_DTYPE(dtype, (b200::sigmoid_gate_mul_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
                                 (T*)out, (const T*)o, (const T*)gate, gate_stride, D, n)));
  return cudaGetLastError() != cudaSuccess;
}
