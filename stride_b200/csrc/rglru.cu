// The recurrent block with a real-gated linear recurrent unit (RG-LRU), the pieces between its projections:
//
//   u_t = conv(x)_t          a causal convolution per channel over the last `taps` inputs x = W_x h + b_x (zeros before the sequence)
//   r_t = sigmoid(A_b u_t,b + a_b), i_t = sigmoid(I_b u_t,b + i_b)      per block b of channels (the products are made by the caller)
//   a_t = exp(-8 r_t softplus(lam)),  S_t = a_t S_(t-1) + sqrt(1 - a_t^2) (i_t u_t),  out_t = S_t * gelu_tanh(W_y h + b_y)_t
//
// Per request the state record [taps][C] float32 holds the last taps - 1 inputs of the convolution (rows 0 .. taps - 2, oldest
// first) and S (row taps - 1); a request that starts at position 0 starts from zeros whatever the record holds. Everything is
// 32-bit. Three steps: `rglru_conv_kernel` (earlier inputs come from the step's own rows or from the record), `rglru_gates_kernel`
// and its form for few tokens (the blocks' products in true float32, then a, the driven input and the gelu
// branch), and `rglru_scan_kernel` (a thread per request and channel walks the tokens in order, one fused multiply-add a token,
// and writes the record back). A token's result has the same bits however the sequence was cut into steps.
#include "common.cuh"
#include "step_ops.h"

SB_DEFINE_LAST_ERROR()

namespace {

using bf16 = __nv_bfloat16;
constexpr int kInFlight = 8;
constexpr int kMaxTaps = 16;

__device__ __forceinline__ float folded(const float* p, int n_partials, int64_t stride) {
  float part[kInFlight];
#pragma unroll
  for (int s = 0; s < kInFlight; ++s)
    if (s < n_partials) part[s] = p[s * stride];
  float sum = part[0];
#pragma unroll
  for (int s = 1; s < kInFlight; ++s)
    if (s < n_partials) sum += part[s];
  for (int s = kInFlight; s < n_partials; ++s) sum += p[s * stride];
  return sum;
}

__device__ __forceinline__ float gelu_tanh(float z) {
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

struct Proj {
  const float* p;            // [P][n][2 C]: columns y | x
  int n_partials;
  int64_t stride;
};

template <int VE>
__device__ __forceinline__ void load_row(float (&v)[VE], const float* at) {
  if constexpr (VE == 4) {
    const float4 x = *reinterpret_cast<const float4*>(at);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  } else {
    v[0] = *at;
  }
}
// The projection's partial sums at VE neighbouring elements, ascending.
template <int VE>
__device__ __forceinline__ void load_folded(float (&v)[VE], const Proj& proj, int64_t at) {
  constexpr int kTogether = VE == 4 ? 4 : kInFlight;
  float part[kTogether][VE];
#pragma unroll
  for (int s = 0; s < kTogether; ++s)
    if (s < proj.n_partials) load_row<VE>(part[s], proj.p + at + s * proj.stride);
#pragma unroll
  for (int e = 0; e < VE; ++e) v[e] = part[0][e];
#pragma unroll
  for (int s = 1; s < kTogether; ++s)
    if (s < proj.n_partials) {
#pragma unroll
      for (int e = 0; e < VE; ++e) v[e] += part[s][e];
    }
  for (int s = kTogether; s < proj.n_partials; ++s) {
    float more[VE];
    load_row<VE>(more, proj.p + at + s * proj.stride);
#pragma unroll
    for (int e = 0; e < VE; ++e) v[e] += more[e];
  }
}

// u[r, c] = conv_b[c] + sum_j taps[c, j] * x[position - (K - 1 - j)]
// A thread owns VE neighbouring channels (16-byte accesses with 4) and ROWS rows one after the other, so that the taps are read once for
// them. The order of a sum is the same in every form. 1,250 rows of 2,048 channels, four taps and one buffer: 22 us, 28 with one row and
// 44 us with one channel of one row a thread.
// HELD: taps kept in registers and read before the wait.
template <class TW, int VE, int ROWS, int HELD>
__global__ void __launch_bounds__(128, HELD == 0 ? 16 : 0) rglru_conv_kernel(Proj proj, const TW* __restrict__ x_bias, const TW* __restrict__ taps, const TW* __restrict__ conv_bias,
                                  const int32_t* __restrict__ positions, const int32_t* __restrict__ slots, const float* __restrict__ state,
                                  float* __restrict__ u, int n, int C, int K) {
  constexpr int kHeld = HELD;
  sb::grid_launch_dependents();
  const int first = blockIdx.x * ROWS, c = (blockIdx.y * blockDim.x + threadIdx.x) * VE;
  if (c >= C) return;
  float xb[VE], cb[VE], held[kHeld ? kHeld : 1][VE];
#pragma unroll
  for (int e = 0; e < VE; ++e) {
    xb[e] = sb::widen(x_bias[c + e]), cb[e] = sb::widen(conv_bias[c + e]);
#pragma unroll
    for (int j = 0; j < kHeld; ++j)
      if (j < K) held[j][e] = sb::widen(taps[(c + e) * K + j]);
  }
  // how many tokens in front of each row the step itself brings (rows of a request are contiguous and ascending)
  int mine[ROWS], pos[ROWS], slot[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int row = min(first + i, n - 1);
    pos[i] = positions[row], slot[i] = slots[row], mine[i] = 0;
    while (mine[i] < K - 1 && row - mine[i] - 1 >= 0 && slots[row - mine[i] - 1] == slot[i]) ++mine[i];
  }
  sb::grid_dependency_wait();
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int row = first + i;
    if (row >= n) break;
    float sum[VE];
#pragma unroll
    for (int e = 0; e < VE; ++e) sum[e] = cb[e];
    auto tap = [&](int j, auto weight) {              // oldest first
      const int back = K - 1 - j;
      float x[VE];
#pragma unroll
      for (int e = 0; e < VE; ++e) x[e] = 0.0f;
      if (back <= mine[i]) {
        load_folded<VE>(x, proj, static_cast<int64_t>(row - back) * 2 * C + C + c);
#pragma unroll
        for (int e = 0; e < VE; ++e) x[e] += xb[e];
      } else if (pos[i] - back >= 0) {
        // the record's row j holds the input at position first - (K - 1) + j, first = pos - mine being the step's first position
        load_row<VE>(x, state + (static_cast<int64_t>(slot[i]) * K + (j + mine[i])) * C + c);
      }
#pragma unroll
      for (int e = 0; e < VE; ++e) sum[e] = fmaf(weight(e), x[e], sum[e]);
    };
#pragma unroll
    for (int j = 0; j < kHeld; ++j)
      if (j < K) tap(j, [&](int e) { return held[j][e]; });
    for (int j = kHeld; j < K; ++j) tap(j, [&](int e) { return sb::widen(taps[(c + e) * K + j]); });
    float* to = u + static_cast<int64_t>(row) * C + c;
    if constexpr (VE == 4) *reinterpret_cast<float4*>(to) = make_float4(sum[0], sum[1], sum[2], sum[3]);
    else to[0] = sum[0];
  }
}

// The gates. For channel j of a block of bw channels: r's and i's sums over the block's inputs k of gate_w[b][k][j] u[t][k] and
// gate_w[b][k][bw + j] u[t][k], the inputs cut into four quarters (a function of the block's size alone), each one chain of fused
// multiply-adds in ascending k, the quarters added in ascending order; then a, the driven input d = sqrt(1 - a^2) i u and
// y = gelu(W_y h + b_y). Nothing of that depends on the step: the same bits from either of the two kernels below.
constexpr int kQuarters = 4;

struct GateParams {
  const float *r_bias, *i_bias, *lam, *y_bias, *u;
  Proj proj;
  float *a, *d, *y;
  int n, C, bw;
};

struct GateValues {
  float a, d, y;
};
// z: the y projection's sum (no bias yet)
__device__ __forceinline__ GateValues gate_values(float sr, float si, float ut, float z, float rb, float ib, float softplus, float yb) {
  const float rg = 1.0f / (1.0f + expf(-(sr + rb)));
  const float ig = 1.0f / (1.0f + expf(-(si + ib)));
  const float log_a = -8.0f * rg * softplus;
  return {expf(log_a), sqrtf(-expm1f(2.0f * log_a)) * (ig * ut), gelu_tanh(z + yb)};
}
__device__ __forceinline__ float softplus_of(float l) { return l > 20.0f ? l : log1pf(expf(l)); }

// Few tokens: a CTA is (TOKENS tokens, block of channels, 32 of its channels), a thread one gate of one channel over one quarter of the inputs;
// its weights are requested 32 (16) at a time, the first ones before the kernels in front are waited for. 8 tokens of 16 blocks of 128: 5.5 us
// for what two gates a thread and eight weights at a time behind the wait took 21.
constexpr int kFewOutputs = 32;
template <class TG, int TOKENS>
__global__ void __launch_bounds__(kQuarters * 2 * kFewOutputs, TOKENS == 16 ? 4 : 0) rglru_gates_few_kernel(const TG* __restrict__ gate_w, GateParams p) {
  extern __shared__ __align__(16) float us[];         // [bw][TOKENS]
  __shared__ float red[kQuarters][2][TOKENS][kFewOutputs];
  sb::grid_launch_dependents();
  const int bw = p.bw, t0 = blockIdx.x * TOKENS, b = blockIdx.y, nt = min(TOKENS, p.n - t0);
  const int lane = threadIdx.x & 31, gate = (threadIdx.x >> 5) & 1, quarter = threadIdx.x >> 6, j = blockIdx.z * kFewOutputs + lane;
  const int per = (bw + kQuarters - 1) / kQuarters, k_begin = min(bw, quarter * per), k_end = min(bw, k_begin + per);
  constexpr int kAhead = TOKENS == 16 ? 16 : 32;
  const TG* w = gate_w + static_cast<int64_t>(b) * bw * 2 * bw + gate * bw + min(j, bw - 1);
  TG ahead[kAhead];
  auto request = [&](int k0) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (k0 + i < k_end) ahead[i] = w[static_cast<int64_t>(k0 + i) * 2 * bw];
  };
  request(k_begin);
  const int c = b * bw + min(j, bw - 1);      // (the epilogue's channel)
  const float rb = p.r_bias[c], ib = p.i_bias[c], softplus = softplus_of(p.lam[c]), yb = p.y_bias[c];
  sb::grid_dependency_wait();
  for (int i = threadIdx.x; i < TOKENS * bw; i += blockDim.x) {
    const int t = i / bw, k = i - t * bw;
    us[k * TOKENS + t] = t < nt ? p.u[static_cast<int64_t>(t0 + t) * p.C + b * bw + k] : 0.0f;
  }
  __syncthreads();
  float acc[TOKENS];
#pragma unroll
  for (int t = 0; t < TOKENS; ++t) acc[t] = 0.0f;
  for (int k0 = k_begin; k0 < k_end; k0 += kAhead) {
    if (k0 != k_begin) request(k0);
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (k0 + i < k_end) {
        const float wk = sb::widen(ahead[i]);
        const float4* x4 = reinterpret_cast<const float4*>(us + (k0 + i) * TOKENS);
#pragma unroll
        for (int t = 0; t < TOKENS / 4; ++t) {
          const float4 x = x4[t];
          acc[4 * t] = fmaf(wk, x.x, acc[4 * t]);
          acc[4 * t + 1] = fmaf(wk, x.y, acc[4 * t + 1]);
          acc[4 * t + 2] = fmaf(wk, x.z, acc[4 * t + 2]);
          acc[4 * t + 3] = fmaf(wk, x.w, acc[4 * t + 3]);
        }
      }
  }
#pragma unroll
  for (int t = 0; t < TOKENS; ++t) red[quarter][gate][t][lane] = acc[t];
  __syncthreads();
  if (j >= bw) return;
#pragma unroll
  for (int ct = threadIdx.x >> 5; ct < TOKENS; ct += 2 * kQuarters) {      // a token a warp
    if (ct >= nt) break;
    float sr = red[0][0][ct][lane], si = red[0][1][ct][lane];
#pragma unroll
    for (int q = 1; q < kQuarters; ++q) sr += red[q][0][ct][lane], si += red[q][1][ct][lane];
    const float z = folded(p.proj.p + static_cast<int64_t>(t0 + ct) * 2 * p.C + c, p.proj.n_partials, p.proj.stride);
    const GateValues v = gate_values(sr, si, us[j * TOKENS + ct], z, rb, ib, softplus, yb);
    const int64_t i = static_cast<int64_t>(t0 + ct) * p.C + c;
    p.a[i] = v.a, p.d[i] = v.d, p.y[i] = v.y;
  }
}

// More tokens: a CTA is (TOKENS tokens, block of channels, 64 of its channels), a warp four tokens, a lane two channels with both gates: 16
// sums a thread for one read of the tokens' inputs and two of the weights a k, both staged in shared memory 32 inputs at a time, the next
// tile's on their way in registers meanwhile. A thread has whole sums (quarter after quarter) and so makes its outputs without an exchange,
// its inputs requested together in front of them. KN: weights a request (16 bytes for blocks of a multiple of 16 channels, four for
// multiples of four, else one); EVEN: 16-byte requests of the tokens' inputs and 8-byte outputs (blocks of a multiple of 16 channels).
// 1,250 tokens of 16 blocks of 128: 59 us; 167 us as one channel of 16 tokens a thread with its weights from global memory, 131 us as
// here but with single-element requests that nothing overlapped.
constexpr int kManyOutputs = 64, kManyInputs = 32;
template <int BYTES>
struct RawOf;
template <>
struct RawOf<16> { using type = uint4; };
template <>
struct RawOf<8> { using type = uint2; };
template <>
struct RawOf<4> { using type = uint32_t; };
template <>
struct RawOf<2> { using type = uint16_t; };
template <class TG, int KN, bool EVEN, int TOKENS>
__global__ void __launch_bounds__(TOKENS * 8, TOKENS == 16 && KN == 8 ? 4 : 0) rglru_gates_kernel(const TG* __restrict__ gate_w, GateParams p) {
  constexpr int kThreads = TOKENS * 8;
  __shared__ __align__(16) float ws[kManyInputs][2][kManyOutputs];
  __shared__ __align__(16) float us[kManyInputs][TOKENS + 4];          // (rows of 16-byte pieces that start at different banks)
  sb::grid_launch_dependents();
  const int bw = p.bw, t0 = blockIdx.x * TOKENS, b = blockIdx.y, j0 = blockIdx.z * kManyOutputs;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tg = warp * 4;
  const int per = (bw + kQuarters - 1) / kQuarters;
  const TG* w = gate_w + static_cast<int64_t>(b) * bw * 2 * bw;
  const float* u = p.u + b * bw;
  constexpr int kW = kManyInputs * 2 * kManyOutputs / KN / kThreads;   // requests a thread and tile
  using Raw = typename RawOf<KN * sizeof(TG)>::type;
  Raw wr[kW];
  float ur[4];
  const int st = threadIdx.x / 8, sk = threadIdx.x % 8 * 4;            // the token and the first of the four inputs that a thread stages
  auto request = [&](int k0, int nk) {
#pragma unroll
    for (int i = 0; i < kW; ++i) {
      const int at = (threadIdx.x + kThreads * i) * KN, k = at / (2 * kManyOutputs), g = at / kManyOutputs % 2, o = at % kManyOutputs;
      wr[i] = k < nk && j0 + o < bw ? *reinterpret_cast<const Raw*>(w + static_cast<int64_t>(k0 + k) * 2 * bw + g * bw + j0 + o) : Raw{};
    }
    const float* at = u + static_cast<int64_t>(t0 + st) * p.C + k0 + sk;
    if constexpr (EVEN) {
      const float4 x = t0 + st < p.n && sk < nk ? *reinterpret_cast<const float4*>(at) : make_float4(0, 0, 0, 0);
      ur[0] = x.x, ur[1] = x.y, ur[2] = x.z, ur[3] = x.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) ur[e] = t0 + st < p.n && sk + e < nk ? at[e] : 0.0f;
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int i = 0; i < kW; ++i) {
      float* to = &ws[0][0][0] + (threadIdx.x + kThreads * i) * KN;
      const TG* v = reinterpret_cast<const TG*>(&wr[i]);
      if constexpr (KN >= 4) {
#pragma unroll
        for (int e = 0; e < KN; e += 4)
          *reinterpret_cast<float4*>(to + e) = make_float4(sb::widen(v[e]), sb::widen(v[e + 1]), sb::widen(v[e + 2]), sb::widen(v[e + 3]));
      } else {
        to[0] = sb::widen(v[0]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) us[sk + e][st] = ur[e];
  };
  sb::grid_dependency_wait();
  request(0, min(kManyInputs, min(bw, per)));
  float sum[2][4][2], acc[2][4][2];                    // gate, token, channel
  for (int q = 0; q < kQuarters; ++q) {
    const int k_begin = min(bw, q * per), k_end = min(bw, k_begin + per);
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int t = 0; t < 4; ++t) acc[g][t][0] = acc[g][t][1] = 0.0f;
    for (int k0 = k_begin; k0 < k_end; k0 += kManyInputs) {
      const int nk = min(kManyInputs, k_end - k0);
      __syncthreads();
      stage();
      __syncthreads();
      const bool same = k0 + kManyInputs < k_end;      // the next tile, of this quarter or of the next one (only the last ones may be empty)
      const int next = same ? k0 + kManyInputs : k_end, end = same ? k_end : min(bw, k_end + per);
      if (next < end) request(next, min(kManyInputs, end - next));
      auto one = [&](int k) {
        const float4 x = *reinterpret_cast<const float4*>(&us[k][tg]);
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const float2 v = *reinterpret_cast<const float2*>(&ws[k][g][2 * lane]);
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[g][t][0] = fmaf(v.x, xs[t], acc[g][t][0]), acc[g][t][1] = fmaf(v.y, xs[t], acc[g][t][1]);
        }
      };
      if (nk == kManyInputs) {
#pragma unroll 8
        for (int k = 0; k < kManyInputs; ++k) one(k);
      } else {
        for (int k = 0; k < nk; ++k) one(k);
      }
    }
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int o = 0; o < 2; ++o) sum[g][t][o] = q == 0 ? acc[g][t][o] : sum[g][t][o] + acc[g][t][o];
  }
  const int j = j0 + 2 * lane, c = b * bw + j;
  if (j >= bw) return;
  const bool two = j + 1 < bw;
  float rb[2], ib[2], softplus[2], yb[2], ut[4][2], z[4][2];
#pragma unroll
  for (int o = 0; o < 2; ++o)
    if (o == 0 || two) rb[o] = p.r_bias[c + o], ib[o] = p.i_bias[c + o], softplus[o] = softplus_of(p.lam[c + o]), yb[o] = p.y_bias[c + o];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int row = t0 + tg + t;
    if (row >= p.n) break;
    const float* zs = p.proj.p + static_cast<int64_t>(row) * 2 * p.C + c;
    if constexpr (EVEN) {
      const float2 x = *reinterpret_cast<const float2*>(p.u + static_cast<int64_t>(row) * p.C + c);
      ut[t][0] = x.x, ut[t][1] = x.y;
      float2 f = *reinterpret_cast<const float2*>(zs);
      for (int k = 1; k < p.proj.n_partials; ++k) {
        const float2 more = *reinterpret_cast<const float2*>(zs + k * p.proj.stride);
        f.x += more.x, f.y += more.y;
      }
      z[t][0] = f.x, z[t][1] = f.y;
    } else {
#pragma unroll
      for (int o = 0; o < 2; ++o)
        if (o == 0 || two) ut[t][o] = p.u[static_cast<int64_t>(row) * p.C + c + o], z[t][o] = folded(zs + o, p.proj.n_partials, p.proj.stride);
    }
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int row = t0 + tg + t;
    if (row >= p.n) break;
    GateValues v[2];
#pragma unroll
    for (int o = 0; o < 2; ++o)
      if (o == 0 || two) v[o] = gate_values(sum[0][t][o], sum[1][t][o], ut[t][o], z[t][o], rb[o], ib[o], softplus[o], yb[o]);
    const int64_t i = static_cast<int64_t>(row) * p.C + c;
    if constexpr (EVEN) {
      *reinterpret_cast<float2*>(p.a + i) = make_float2(v[0].a, v[1].a);
      *reinterpret_cast<float2*>(p.d + i) = make_float2(v[0].d, v[1].d);
      *reinterpret_cast<float2*>(p.y + i) = make_float2(v[0].y, v[1].y);
    } else {
#pragma unroll
      for (int o = 0; o < 2; ++o)
        if (o == 0 || two) p.a[i + o] = v[o].a, p.d[i + o] = v[o].d, p.y[i + o] = v[o].y;
    }
  }
}

// A thread owns a channel of one entry and walks its tokens. The tokens' a, d and y reach shared memory in chunks of kScanChunk tokens
// by asynchronous copies, a chunk ahead of the one being walked, so that what a step of the walk waits for is one fused
// multiply-add and a read of shared memory.
constexpr int kScanChannels = 64, kScanChunk = 32;

__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

template <class TW, class TO>
__global__ void __launch_bounds__(kScanChannels) rglru_scan_kernel(const float* __restrict__ a, const float* __restrict__ d, const float* __restrict__ y,
                                                                    Proj proj, const TW* __restrict__ x_bias, const int32_t* __restrict__ meta,
                                                                    int meta_stride, float* __restrict__ state, TO* __restrict__ out, int C, int K) {
  __shared__ float stage[2][3][kScanChunk][kScanChannels];
  sb::grid_launch_dependents();
  const int e = blockIdx.x, c = blockIdx.y * kScanChannels + threadIdx.x;
  const int slot = meta[e], row0 = meta[meta_stride + e], len = meta[2 * meta_stride + e], pos0 = meta[3 * meta_stride + e];
  const bool live = c < C;
  sb::grid_dependency_wait();
  float* rec = state + static_cast<int64_t>(slot) * K * C + c;
  float S = (live && pos0 > 0) ? rec[static_cast<int64_t>(K - 1) * C] : 0.0f;
  const int64_t base = static_cast<int64_t>(row0) * C + c;
  // a thread copies its own channel's values, so no other thread waits for them
  auto request = [&](int chunk) {
    const int buf = chunk & 1, nt = min(kScanChunk, len - chunk * kScanChunk);
    if (live)
      for (int t = 0; t < nt; ++t) {
        const int64_t i = base + static_cast<int64_t>(chunk * kScanChunk + t) * C;
        copy_async4(&stage[buf][0][t][threadIdx.x], a + i);
        copy_async4(&stage[buf][1][t][threadIdx.x], d + i);
        copy_async4(&stage[buf][2][t][threadIdx.x], y + i);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int chunks = (len + kScanChunk - 1) / kScanChunk;
  request(0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    if (chunk + 1 < chunks) {
      request(chunk + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    const int buf = chunk & 1, nt = min(kScanChunk, len - chunk * kScanChunk);
    if (live) {
#pragma unroll 8
      for (int t = 0; t < nt; ++t) {
        S = fmaf(stage[buf][0][t][threadIdx.x], S, stage[buf][1][t][threadIdx.x]);
        out[base + static_cast<int64_t>(chunk * kScanChunk + t) * C] = sb::narrow<TO>(S * stage[buf][2][t][threadIdx.x]);
      }
    }
  }
  if (!live) return;
  // the record for the step behind this one: the inputs at positions end - (K - 1) .. end - 1 and S
  float hist[kMaxTaps];
  const float xb = sb::widen(x_bias[c]);
  for (int j = 0; j < K - 1; ++j) {
    const int back = K - 1 - j;                       // the input `back` tokens before the next one
    float x = 0.0f;
    if (back <= len) x = folded(proj.p + static_cast<int64_t>(row0 + len - back) * 2 * C + C + c, proj.n_partials, proj.stride) + xb;
    else if (pos0 + len - back >= 0) x = rec[static_cast<int64_t>(j + len) * C];      // (only if pos0 > 0: the record is then valid)
    hist[j] = x;
  }
  for (int j = 0; j < K - 1; ++j) rec[static_cast<int64_t>(j) * C] = hist[j];
  rec[static_cast<int64_t>(K - 1) * C] = S;
}

}  // namespace

SB_EXPORT int sb_rglru_conv(const float* proj, int n_partials, int64_t partial_stride, const void* x_bias, const void* taps, const void* conv_bias,
                            int w_dtype, const int32_t* positions, const int32_t* slots, const float* state, float* u, int n, int C, int K,
                            cudaStream_t stream) {
  if (n <= 0) return 0;
  if (K < 1 || K > kMaxTaps) return sb::fail("sb_rglru_conv: %d taps (1 to %d)", K, kMaxTaps);
  if (n_partials < 1) return sb::fail("sb_rglru_conv: n_partials must be >= 1");
  const Proj pr{proj, n_partials, partial_stride};
  // Four channels a thread have four partial sums on their way and the taps' weights in registers up to four: more of either are round trips
  // one after the other, which only very many elements hide (64 rows of 2,048 behind nine buffers 4.0 us, 5.1 with four channels; with eight
  // taps and one buffer, 256 rows 19.6 and 19.8, 1,250 rows 84 and 74). Four rows a thread once those threads fill the SMs: 700 rows of 2,048
  // 14.7 us, 17.3 with one; 256 rows 6.1 and 6.3; 128 rows 5.4 and 3.8.
  const bool aligned = C % 4 == 0 && partial_stride % 4 == 0 &&
                       ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(u)) & 15) == 0;
  // Single channels: the taps in registers while the threads are few (8 rows of 2,050 2.1 us, 3.0 without), else more of them an SM without.
  const int64_t elements = static_cast<int64_t>(n) * C;
  const bool vec = aligned && n_partials <= 4 && (K <= 4 || elements >= 1 << 21), rows4 = vec && elements >= 1 << 19;
#define SB_CONV(TW, VE, ROWS, HELD)                                                                                                                    \
  sb::launch_pdl(rglru_conv_kernel<TW, VE, ROWS, HELD>, dim3((n + ROWS - 1) / ROWS, (C / VE + 127) / 128), dim3(128), 0, stream, pr,                   \
                 static_cast<const TW*>(x_bias), static_cast<const TW*>(taps), static_cast<const TW*>(conv_bias), positions, slots, state, u, n, C, K)
#define SB_CONV_T(TW)                              \
  do {                                             \
    if (rows4) SB_CONV(TW, 4, 4, 4);               \
    else if (vec) SB_CONV(TW, 4, 1, 4);            \
    else if (elements <= 3 << 16) SB_CONV(TW, 1, 1, 4); \
    else SB_CONV(TW, 1, 1, 0);                     \
  } while (0)
  if (w_dtype == 0) SB_CONV_T(float);
  else if (w_dtype == 1) SB_CONV_T(bf16);
  else return sb::fail("sb_rglru_conv: unsupported dtype %d", w_dtype);
#undef SB_CONV
#undef SB_CONV_T
  return sb::check_launch("sb_rglru_conv");
}

// gate_w [blocks][bw][2 bw] (float32 or bfloat16): per block the matrices of r and i side by side, transposed ([input][output]).
SB_EXPORT int sb_rglru_gates(const void* gate_w, int gate_dtype, const void* r_bias, const void* i_bias, const void* lam, const void* y_bias, int w_dtype,
                             const float* u, const float* proj, int n_partials, int64_t partial_stride, float* a, float* d, float* y, int n, int C,
                             int blocks, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (blocks <= 0 || C % blocks != 0) return sb::fail("sb_rglru_gates: %d channels do not divide into %d blocks", C, blocks);
  const int bw = C / blocks;
  if (bw > 2048) return sb::fail("sb_rglru_gates: blocks of %d channels (at most 2048)", bw);
  if (w_dtype != 0) return sb::fail("sb_rglru_gates: biases and lam are float32");
  const GateParams p{static_cast<const float*>(r_bias), static_cast<const float*>(i_bias), static_cast<const float*>(lam), static_cast<const float*>(y_bias),
                     u, Proj{proj, n_partials, partial_stride}, a, d, y, n, C, bw};
  // 0, 1: 8 and 16 tokens a CTA with its weights from memory; 2, 3: 16 and 32 tokens that share staged ones. Microseconds with bfloat16 weights,
  // 16 blocks of 128: 32 tokens 6.0, 9.3, 9.6, 12; 64 tokens 11.6, 13, 13, 12; 128 tokens 22, 14, 17, 18; 200 tokens 33, 23, 17, 21; 400 tokens
  // 63, 40, 28, 21. Wide blocks leave few CTAs to share the weights' way (one of 2,048, 24 tokens: 76, 88, 67, 103); where every weight is a
  // request of its own (odd blocks), staging pays later (8 of 33, 700 tokens: 20, 12, 16, 14; 2,048 tokens 54, 33, 28, 26).
  const int form = bw >= 1024 ? (n < 8 ? 0 : n < 320 ? 2 : 3) : n <= 64 ? 0 : bw % 4 != 0 ? (n <= 128 ? 0 : n <= 1400 ? 1 : 3) : n <= 144 ? 1 : n < 320 ? 2 : 3;
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const bool quads = bw % 4 == 0 && aligned(gate_w);
  const bool even = bw % 16 == 0 && partial_stride % 4 == 0 && aligned(gate_w) && aligned(u) && aligned(proj) && aligned(a) && aligned(d) && aligned(y);
#define SB_GATES_FEW(TG, TOKENS)                                                                                                              \
  do {                                                                                                                                        \
    const size_t smem = sizeof(float) * TOKENS * bw;                                                                                          \
    if (smem > 16 * 1024) cudaFuncSetAttribute(rglru_gates_few_kernel<TG, TOKENS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    sb::launch_pdl(rglru_gates_few_kernel<TG, TOKENS>, dim3((n + TOKENS - 1) / TOKENS, blocks, (bw + kFewOutputs - 1) / kFewOutputs),         \
                   dim3(kQuarters * 2 * kFewOutputs), smem, stream, static_cast<const TG*>(gate_w), p);                                       \
  } while (0)
#define SB_GATES_MANY(TG, KN, EVEN, TOKENS)                                                                                                   \
  sb::launch_pdl(rglru_gates_kernel<TG, KN, EVEN, TOKENS>, dim3((n + TOKENS - 1) / TOKENS, blocks, (bw + kManyOutputs - 1) / kManyOutputs),   \
                 dim3(TOKENS * 8), 0, stream, static_cast<const TG*>(gate_w), p)
#define SB_GATES(TG)                                                               \
  do {                                                                             \
    if (form == 0) SB_GATES_FEW(TG, 8);                                            \
    else if (form == 1) SB_GATES_FEW(TG, 16);                                      \
    else if (even && form == 2) SB_GATES_MANY(TG, 16 / (int)sizeof(TG), true, 16); \
    else if (even) SB_GATES_MANY(TG, 16 / (int)sizeof(TG), true, 32);              \
    else if (quads && form == 2) SB_GATES_MANY(TG, 4, false, 16);                  \
    else if (quads) SB_GATES_MANY(TG, 4, false, 32);                               \
    else if (form == 2) SB_GATES_MANY(TG, 1, false, 16);                           \
    else SB_GATES_MANY(TG, 1, false, 32);                                          \
  } while (0)
  if (gate_dtype == 0) SB_GATES(float);
  else if (gate_dtype == 1) SB_GATES(bf16);
  else return sb::fail("sb_rglru_gates: unsupported dtype %d", gate_dtype);
#undef SB_GATES
#undef SB_GATES_FEW
#undef SB_GATES_MANY
  return sb::check_launch("sb_rglru_gates");
}

SB_EXPORT int sb_rglru_scan(const float* a, const float* d, const float* y, const float* proj, int n_partials, int64_t partial_stride,
                            const void* x_bias, int w_dtype, const int32_t* meta, int meta_stride, int entries, float* state, void* out,
                            int out_dtype, int C, int K, cudaStream_t stream) {
  if (entries <= 0) return 0;
  if (K < 1 || K > kMaxTaps) return sb::fail("sb_rglru_scan: %d taps (1 to %d)", K, kMaxTaps);
  const Proj pr{proj, n_partials, partial_stride};
  const dim3 grid(entries, (C + kScanChannels - 1) / kScanChannels);
#define SB_SCAN(TW, TO) sb::launch_pdl(rglru_scan_kernel<TW, TO>, grid, dim3(kScanChannels), 0, stream, a, d, y, pr, static_cast<const TW*>(x_bias), meta, meta_stride, state, static_cast<TO*>(out), C, K)
  if (w_dtype == 0 && out_dtype == 0) SB_SCAN(float, float);
  else if (w_dtype == 0 && out_dtype == 1) SB_SCAN(float, bf16);
  else if (w_dtype == 1 && out_dtype == 0) SB_SCAN(bf16, float);
  else if (w_dtype == 1 && out_dtype == 1) SB_SCAN(bf16, bf16);
  else return sb::fail("sb_rglru_scan: unsupported dtypes weights=%d out=%d", w_dtype, out_dtype);
#undef SB_SCAN
  return sb::check_launch("sb_rglru_scan");
}

// ------------------------------------------------------------------ operations of the native step program (step_ops.h)
// i: 0 projection partial sums (flat), 1 K ranges S, 2 most tokens with a buffer per range, 3 x bias, 4 taps, 5 conv bias, 6 their dtype, 7 state,
//    8 u, 9 C, 10 K
SB_EXPORT int sb_op_rglru_conv(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int C = (int)op->i[9];
  return sb_rglru_conv(ptr<const float>(op->i[0]), partial_count(op->i[1], op->i[2], s->n), static_cast<int64_t>(s->n) * 2 * C, ptr<const void>(op->i[3]),
                       ptr<const void>(op->i[4]), ptr<const void>(op->i[5]), (int)op->i[6], positions(s), slots(s), ptr<const float>(op->i[7]),
                       ptr<float>(op->i[8]), s->n, C, (int)op->i[10], static_cast<cudaStream_t>(stream));
}

// i: 0 gate weights, 1 their dtype, 2 r bias, 3 i bias, 4 lam, 5 y bias, 6 their dtype, 7 u, 8 projection partial sums, 9 K ranges S,
//    10 most tokens with a buffer per range, 11 a, 12 d, 13 y, 14 C, 15 blocks
SB_EXPORT int sb_op_rglru_gates(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int C = (int)op->i[14];
  return sb_rglru_gates(ptr<const void>(op->i[0]), (int)op->i[1], ptr<const void>(op->i[2]), ptr<const void>(op->i[3]), ptr<const void>(op->i[4]),
                        ptr<const void>(op->i[5]), (int)op->i[6], ptr<const float>(op->i[7]), ptr<const float>(op->i[8]),
                        partial_count(op->i[9], op->i[10], s->n), static_cast<int64_t>(s->n) * 2 * C, ptr<float>(op->i[11]), ptr<float>(op->i[12]),
                        ptr<float>(op->i[13]), s->n, C, (int)op->i[15], static_cast<cudaStream_t>(stream));
}

// i: 0 a, 1 d, 2 y, 3 projection partial sums, 4 K ranges S, 5 most tokens with a buffer per range, 6 x bias, 7 its dtype, 8 state, 9 out, 10 out dtype,
//    11 C, 12 K
SB_EXPORT int sb_op_rglru_scan(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int C = (int)op->i[11];
  return sb_rglru_scan(ptr<const float>(op->i[0]), ptr<const float>(op->i[1]), ptr<const float>(op->i[2]), ptr<const float>(op->i[3]),
                       partial_count(op->i[4], op->i[5], s->n), static_cast<int64_t>(s->n) * 2 * C, ptr<const void>(op->i[6]), (int)op->i[7],
                       entry_meta(s), s->max_rows, s->entries, ptr<float>(op->i[8]), ptr<void>(op->i[9]), (int)op->i[10], C, (int)op->i[12],
                       static_cast<cudaStream_t>(stream));
}
