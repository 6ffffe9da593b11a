// Linear attention with a decay per head ("lightning attention"), as a recurrence over a state kept per request (linear_scan.cuh):
//
//   S_t = decay_h * S_(t-1) + k_t v_t^T        S: [D, V] float32 per head
//   o_t = S_t^T q_t
//
// with q, k, v = silu of the projections. Everything here is 32-bit: the activations, the decay, the state and the sums. A step in which
// an entry brings several tokens applies the activation once for all of them and then walks them (sbscan::scan_kernel); steps of single
// tokens fold, activate and take their token in one kernel. A token's output has the same bits either way.
//
// What follows the recurrence: an RMS norm over all heads' outputs of a token, times a gain, times sigmoid of the gate projection.
#include <type_traits>

#include "common.cuh"
#include "linear_scan.cuh"
#include "step_ops.h"

SB_DEFINE_LAST_ERROR()

namespace {

using bf16 = __nv_bfloat16;

constexpr int kInFlight = 4;     // partial sums requested at once

__device__ __forceinline__ float silu(float a) { return a / (1.0f + expf(-a)); }

// Sum of the projection's partial buffers at one element, ascending.
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

// The same over four neighbouring elements (p and the stride 16-byte aligned).
template <bool ONE>
__device__ __forceinline__ float4 folded4(const float* p, int n_partials, int64_t stride) {
  if constexpr (ONE) return *reinterpret_cast<const float4*>(p);      // (without the registers for more, more blocks live on an SM)
  float4 part[kInFlight];
#pragma unroll
  for (int s = 0; s < kInFlight; ++s)
    if (s < n_partials) part[s] = *reinterpret_cast<const float4*>(p + s * stride);
  float4 sum = part[0];
  auto add = [&](float4 a) { sum.x += a.x, sum.y += a.y, sum.z += a.z, sum.w += a.w; };
#pragma unroll
  for (int s = 1; s < kInFlight; ++s)
    if (s < n_partials) add(part[s]);
  for (int s = kInFlight; s < n_partials; ++s) add(*reinterpret_cast<const float4*>(p + s * stride));
  return sum;
}

// Steps in which every entry brings one token (decoding): the partial sums folded (and activated) inside.
template <int DL>
__global__ void __launch_bounds__(DL * 64, DL == 2 ? 7 : 1024 / (DL * 64)) lightning_step_kernel(const sbscan::Params p, int n_partials, int64_t partial_stride, int activated) {
  extern __shared__ __align__(16) float smem[];
  sb::grid_launch_dependents();
  const int e = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * 32;
  const int slot = p.meta[e], row0 = p.meta[p.meta_stride + e], len = p.meta[2 * p.meta_stride + e], pos0 = p.meta[3 * p.meta_stride + e];
  sb::grid_dependency_wait();
  sbscan::step_core<DL, false>(p, smem, slot, row0, len, pos0, [&](float* to, int Ds, int row) {
    const float* src = p.rows + static_cast<int64_t>(row) * p.width;
#pragma unroll 1
    for (int j = threadIdx.x; j < 2 * Ds + 32; j += blockDim.x) {
      const int d = j >= Ds ? j - Ds : j;
      const float* at = nullptr;
      if (j < 2 * Ds) {
        if (d < p.D) at = src + (j >= Ds ? p.k_off : p.q_off) + h * p.D + d;
      } else if (c0 + j - 2 * Ds < p.V) {
        at = src + p.v_off + h * p.V + c0 + j - 2 * Ds;
      }
      float v = 0.0f;
      if (at != nullptr) {
        v = folded(at, n_partials, partial_stride);
        if (!activated) v = silu(v);
      }
      to[j] = v;
    }
  });
}

// act[r, j] = silu(sum of the partial buffers at [r, j]) for the first `cols` columns of every row: what the recurrence
// reads, made once for all of a long step's tokens instead of by every CTA that needs a token's keys and queries.
// VE: 4 where the columns and buffers allow 16-byte accesses, else 1. grid: (rows, pieces of a row). Bound by memory: 2,048 rows of 6,144
// columns (101 MB) 17 us, 48 us with one element and a 64-bit division a thread and round.
template <int VE, bool ONE>
__global__ void __launch_bounds__(256) lightning_activate_kernel(const float* __restrict__ proj, int n_partials, int64_t partial_stride, int width,
                                                                 float* __restrict__ act, int cols) {
  sb::grid_launch_dependents();
  sb::grid_dependency_wait();
  const float* src = proj + static_cast<int64_t>(blockIdx.x) * width;
  float* dst = act + static_cast<int64_t>(blockIdx.x) * cols;
  for (int i = (blockIdx.y * blockDim.x + threadIdx.x) * VE; i < cols; i += gridDim.y * blockDim.x * VE) {
    if constexpr (VE == 4) {
      const float4 v = folded4<ONE>(src + i, n_partials, partial_stride);
      *reinterpret_cast<float4*>(dst + i) = make_float4(silu(v.x), silu(v.y), silu(v.z), silu(v.w));
    } else {
      dst[i] = silu(folded(src + i, n_partials, partial_stride));
    }
  }
}

// out[r, j] = o[r, j] / sqrt(mean_j(o[r, :]^2) + eps) * gain[j] * sigmoid(gate[r, j]); the gate is a column range of the
// projection's partial sums. One block per row. VE: 4 where the width and every buffer allow 16-byte accesses, else 1; which one depends on
// the width and the buffers alone, never on the rows. A thread keeps up to kKeep pieces of o and of the gate in registers, requested before
// the block's sum; of what lies beyond, o waits in shared memory and the gate is read behind it. 2,048 rows of 2,048: 11.6 us, 24 us with single elements and the gate behind the sum.
template <class TW, class TO, int VE, bool ONE>
__global__ void __launch_bounds__(1024) gated_rmsnorm_kernel(const float* __restrict__ o, const float* __restrict__ proj, int n_partials,
                                                              int64_t partial_stride, int width, int g_off,
                                                              const TW* __restrict__ gain, TO* __restrict__ out, int W, float eps) {
  using V = typename std::conditional<VE == 4, float4, float>::type;
  constexpr int kKeep = 2;
  extern __shared__ __align__(16) float beyond_raw[];
  __shared__ float red[32];
  sb::grid_launch_dependents();
  sb::grid_dependency_wait();
  const int64_t r = blockIdx.x;
  const int units = W / VE, kept = kKeep * blockDim.x;
  V* rest = reinterpret_cast<V*>(beyond_raw);
  const V* src = reinterpret_cast<const V*>(o + r * W);
  const float* gate = proj + r * width + g_off;
  auto gate_at = [&](int i) {
    if constexpr (VE == 4) return folded4<ONE>(gate + 4 * i, n_partials, partial_stride);
    else return folded(gate + i, n_partials, partial_stride);
  };
  V v[kKeep], g[kKeep];
#pragma unroll
  for (int j = 0; j < kKeep; ++j) {
    const int i = threadIdx.x + j * blockDim.x;
    if (i < units) v[j] = src[i], g[j] = gate_at(i);
  }
  float ss = 0.0f;
  auto square = [&](V a) {
    if constexpr (VE == 4) ss = fmaf(a.x, a.x, ss), ss = fmaf(a.y, a.y, ss), ss = fmaf(a.z, a.z, ss), ss = fmaf(a.w, a.w, ss);
    else ss = fmaf(a, a, ss);
  };
#pragma unroll
  for (int j = 0; j < kKeep; ++j)
    if (threadIdx.x + j * blockDim.x < units) square(v[j]);
  for (int i = threadIdx.x + kept; i < units; i += blockDim.x) square(rest[i - kept] = src[i]);
  const float scale = 1.0f / sqrtf(sb::block_sum(ss, red) / static_cast<float>(W) + eps);
  auto one = [&](float a, float b, float w) { return a * scale * w * (1.0f / (1.0f + expf(-b))); };
  auto write = [&](int i, V a, V b) {
    const TW* w = gain + i * VE;
    TO* to = out + r * W + i * VE;
    if constexpr (VE == 4) {
      const float x = one(a.x, b.x, sb::widen(w[0])), y = one(a.y, b.y, sb::widen(w[1])), z = one(a.z, b.z, sb::widen(w[2])), u = one(a.w, b.w, sb::widen(w[3]));
      if constexpr (sizeof(TO) == 2) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(x, y), hi = __floats2bfloat162_rn(z, u);
        uint2 packed;
        packed.x = *reinterpret_cast<const uint32_t*>(&lo);
        packed.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(to) = packed;
      } else {
        *reinterpret_cast<float4*>(to) = make_float4(x, y, z, u);
      }
    } else {
      to[0] = sb::narrow<TO>(one(a, b, sb::widen(w[0])));
    }
  };
#pragma unroll
  for (int j = 0; j < kKeep; ++j) {
    const int i = threadIdx.x + j * blockDim.x;
    if (i < units) write(i, v[j], g[j]);
  }
  for (int i = threadIdx.x + kept; i < units; i += blockDim.x) write(i, rest[i - kept], gate_at(i));
}

}  // namespace

// The recurrence for every entry of a step. proj: the projection's partial sums [n_partials][n][width] (float32) with
// q at column q_off (H D), k at k_off (H D), v at v_off (H V); meta: the step's entry records [4][meta_stride]
// on the device; state [slots][H][D][V] float32; out [n][H V] float32.
// act: scratch [n][q, k, v columns] float32. Steps in which an entry brings several tokens apply the activation in a kernel
// of its own first; steps of single tokens apply it inside theirs (the same function on the same sums: the same bits).
// `ready` = 1: `proj` already holds q, k and v as the recurrence takes them (another design's activation, made by a kernel in front), and
// nothing is applied here.
SB_EXPORT int sb_lightning_scan_ex(const float* proj, int n_partials, int64_t partial_stride, int width, int q_off, int k_off, int v_off,
                                   const int32_t* meta, int meta_stride, int entries, int n, const float* decay, float* state, float* out,
                                   float* act, int H, int D, int V, int ready, cudaStream_t stream) {
  if (entries <= 0 || n <= 0) return 0;
  if (H <= 0 || D <= 0 || V <= 0 || D > 256) return sb::fail("sb_lightning_scan: heads %d, key size %d (at most 256), value size %d", H, D, V);
  if (n_partials < 1) return sb::fail("sb_lightning_scan: n_partials must be >= 1");
  sbscan::Params p{proj, width, q_off, k_off, v_off, 0, meta, meta_stride, decay, state, out, H, D, V};
  if (n == entries) {     // one token an entry (decoding): small CTAs, many of them, nothing staged ahead
    const auto kernel = sbscan::lane_elements(D) == 2 ? lightning_step_kernel<2> : sbscan::lane_elements(D) == 4 ? lightning_step_kernel<4> : lightning_step_kernel<8>;
    sb::launch_pdl(kernel, dim3(entries, H, (V + 31) / 32), dim3(sbscan::step_threads(D)), sbscan::step_smem(D, false), stream, p, n_partials, partial_stride, ready);
    return sb::check_launch("sb_lightning_scan");
  }
  // steps with longer entries: the activation once for all tokens, then the recurrence
  if (ready) {
    if (n_partials != 1) return sb::fail("sb_lightning_scan: ready-made q, k, v come as one buffer");
    return sbscan::launch_scan<false>(p, entries, n, "sb_lightning_scan", stream);
  }
  if (act == nullptr) return sb::fail("sb_lightning_scan: a step with an entry of several tokens needs the scratch for the activated sums");
  const int cols = max(max(q_off + H * D, k_off + H * D), v_off + H * V);
  const bool vec = cols % 4 == 0 && width % 4 == 0 && partial_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(act)) & 15) == 0;
  const dim3 vgrid(n, (cols / 4 + 255) / 256);
  if (vec && n_partials == 1) sb::launch_pdl(lightning_activate_kernel<4, true>, vgrid, dim3(256), 0, stream, proj, n_partials, partial_stride, width, act, cols);
  else if (vec) sb::launch_pdl(lightning_activate_kernel<4, false>, vgrid, dim3(256), 0, stream, proj, n_partials, partial_stride, width, act, cols);
  else sb::launch_pdl(lightning_activate_kernel<1, false>, dim3(n, (cols + 1023) / 1024), dim3(256), 0, stream, proj, n_partials, partial_stride, width, act, cols);
  p.rows = act;
  p.width = cols;
  return sbscan::launch_scan<false>(p, entries, n, "sb_lightning_scan", stream);
}

SB_EXPORT int sb_lightning_scan(const float* proj, int n_partials, int64_t partial_stride, int width, int q_off, int k_off, int v_off,
                                const int32_t* meta, int meta_stride, int entries, int n, const float* decay, float* state, float* out,
                                float* act, int H, int D, int V, cudaStream_t stream) {
  return sb_lightning_scan_ex(proj, n_partials, partial_stride, width, q_off, k_off, v_off, meta, meta_stride, entries, n, decay, state, out, act,
                              H, D, V, 0, stream);
}

// out [n][W] (float32 or bfloat16) = rmsnorm(o [n][W] float32) * gain * sigmoid(gate), the gate being columns g_off.. of `proj`.
SB_EXPORT int sb_gated_rmsnorm(const float* o, const float* proj, int n_partials, int64_t partial_stride, int width, int g_off,
                               const void* gain, int gain_dtype, void* out, int out_dtype, int n, int W, float eps, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n_partials < 1) return sb::fail("sb_gated_rmsnorm: n_partials must be >= 1");
  if (W > 50 * 1024) return sb::fail("sb_gated_rmsnorm: width %d (at most 51200)", W);
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const bool vec = W % 4 == 0 && width % 4 == 0 && g_off % 4 == 0 && partial_stride % 4 == 0 && aligned(o) && aligned(proj) && aligned(gain) && aligned(out);
  const int units = vec ? W / 4 : W;      // (single elements: several a thread, so that an SM holds more than one row)
  const int threads = vec ? (units > 1024 ? 1024 : units > 512 ? 512 : units > 256 ? 256 : 128) : W >= 4096 ? 1024 : W >= 2048 ? 512 : W >= 512 ? 256 : 128;
  const size_t smem = units > 2 * threads ? static_cast<size_t>(units - 2 * threads) * (vec ? 16 : 4) : 0;      // (kKeep pieces a thread are in registers)
#define SB_GN_V(TW, TO, VE, ONE)                                                                                                      \
  do {                                                                                                                                \
    if (smem > 40 * 1024) cudaFuncSetAttribute(gated_rmsnorm_kernel<TW, TO, VE, ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    sb::launch_pdl(gated_rmsnorm_kernel<TW, TO, VE, ONE>, n, threads, smem, stream, o, proj, n_partials, partial_stride, width, g_off, \
                   static_cast<const TW*>(gain), static_cast<TO*>(out), W, eps);                                                      \
  } while (0)
#define SB_GN(TW, TO)                                     \
  do {                                                    \
    if (vec && n_partials == 1) SB_GN_V(TW, TO, 4, true); \
    else if (vec) SB_GN_V(TW, TO, 4, false);              \
    else SB_GN_V(TW, TO, 1, false);                       \
  } while (0)
  if (gain_dtype == 0 && out_dtype == 0) SB_GN(float, float);
  else if (gain_dtype == 0 && out_dtype == 1) SB_GN(float, bf16);
  else if (gain_dtype == 1 && out_dtype == 0) SB_GN(bf16, float);
  else if (gain_dtype == 1 && out_dtype == 1) SB_GN(bf16, bf16);
  else return sb::fail("sb_gated_rmsnorm: unsupported dtypes gain=%d out=%d", gain_dtype, out_dtype);
#undef SB_GN
#undef SB_GN_V
  return sb::check_launch("sb_gated_rmsnorm");
}

// ------------------------------------------------------------------ operations of the native step program (step_ops.h)
// i: 0 projection partial sums (flat), 1 their width, 2 K ranges S, 3 most tokens with a buffer per range, 4 q_off, 5 k_off,
//    6 v_off, 7 decay (float32 [H]), 8 state, 9 out (float32 [n, H V]), 10 H, 11 D, 12 V, 13 scratch for the activated sums,
//    14 q, k, v are ready-made (one buffer, nothing applied)
SB_EXPORT int sb_op_lightning_scan(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int P = partial_count(op->i[2], op->i[3], s->n);
  return sb_lightning_scan_ex(ptr<const float>(op->i[0]), P, static_cast<int64_t>(s->n) * op->i[1], (int)op->i[1], (int)op->i[4], (int)op->i[5],
                              (int)op->i[6], entry_meta(s), s->max_rows, s->entries, s->n, ptr<const float>(op->i[7]), ptr<float>(op->i[8]),
                              ptr<float>(op->i[9]), ptr<float>(op->i[13]), (int)op->i[10], (int)op->i[11], (int)op->i[12], (int)op->i[14],
                              static_cast<cudaStream_t>(stream));
}

// i: 0 o (float32 [n, W]), 1 projection partial sums (flat), 2 their width, 3 K ranges S, 4 most tokens with a buffer per range,
//    5 g_off, 6 gain, 7 gain dtype, 8 out, 9 out dtype, 10 W
// f: 0 eps
SB_EXPORT int sb_op_gated_rmsnorm(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int P = partial_count(op->i[3], op->i[4], s->n);
  return sb_gated_rmsnorm(ptr<const float>(op->i[0]), ptr<const float>(op->i[1]), P, static_cast<int64_t>(s->n) * op->i[2], (int)op->i[2],
                          (int)op->i[5], ptr<const void>(op->i[6]), (int)op->i[7], ptr<void>(op->i[8]), (int)op->i[9], s->n, (int)op->i[10],
                          static_cast<float>(op->f[0]), static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------------------------------------------------
// Retention: the same recurrence with rotated, not activated, queries and keys, and what other linear-attention designs put behind it.
//
// `rotate_qk_kernel`: out[r] = [q | k | v] in 32-bit from the projection's partial sums: the first `rot` elements of every q and k head
// turned by the token's position (pairs (i, i + rot / 2), or (2i, 2i + 1) when interleaved), k times a constant behind the rotation, v
// as it is. The recurrence then takes the buffer as ready-made.
//
// `group_norm_gate_kernel`: every head's result divided by its root mean square, times a gain of the head's size shared by all heads
// (or none), times silu or sigmoid of the gate, a column range of some projection's partial sums. A warp per (token, head).
namespace {

struct RotateParams {
  const float* proj;
  int n_partials;
  int64_t partial_stride;
  int width, q_off, k_off, v_off;
  const int32_t* positions;
  const float* cos_sin;      // [positions][rot / 2][2]
  int rot, interleaved;
  float k_scale;
  float* out;                // [n][2 H D + H V]
  int H, D, V;
};

__global__ void __launch_bounds__(256) rotate_qk_kernel(RotateParams p) {
  sb::grid_launch_dependents();
  const int row = blockIdx.x, nqk = 2 * p.H * p.D, cols = nqk + p.H * p.V, rh = p.rot / 2;
  const int pos = p.positions[row];
  sb::grid_dependency_wait();
  const float* src = p.proj + static_cast<int64_t>(row) * p.width;
  float* dst = p.out + static_cast<int64_t>(row) * cols;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < cols; i += gridDim.y * blockDim.x) {
    if (i >= nqk) {
      dst[i] = folded(src + p.v_off + (i - nqk), p.n_partials, p.partial_stride);
      continue;
    }
    const bool is_k = i >= p.H * p.D;
    const int e = is_k ? i - p.H * p.D : i, d = e % p.D;
    const float* at = src + (is_k ? p.k_off : p.q_off) + e;
    float v = folded(at, p.n_partials, p.partial_stride);
    if (d < p.rot) {
      int pair, other;
      bool low;
      if (p.interleaved) pair = d >> 1, low = (d & 1) == 0, other = low ? 1 : -1;
      else low = d < rh, pair = low ? d : d - rh, other = low ? rh : -rh;
      const float b = folded(at + other, p.n_partials, p.partial_stride);
      const float2 cs = *reinterpret_cast<const float2*>(p.cos_sin + (static_cast<int64_t>(pos) * rh + pair) * 2);
      v = low ? __fsub_rn(__fmul_rn(v, cs.x), __fmul_rn(b, cs.y)) : __fadd_rn(__fmul_rn(v, cs.x), __fmul_rn(b, cs.y));
    }
    dst[i] = is_k ? __fmul_rn(v, p.k_scale) : v;
  }
}

struct GroupGateParams {
  const float* o;            // [n][H V]
  const float* proj;         // the gate's partial sums [P][n][width], columns g_off ..
  int n_partials;
  int64_t partial_stride;
  int width, g_off;
  const void* gain;          // [V] or null
  int gain_bf16;
  void* out;
  int n, H, V, silu_gate;
  float eps;
};

template <class TO>
__global__ void __launch_bounds__(128) group_norm_gate_kernel(GroupGateParams p) {
  sb::grid_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t unit = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  sb::grid_dependency_wait();
  if (unit >= static_cast<int64_t>(p.n) * p.H) return;
  const int64_t row = unit / p.H;
  const int h = static_cast<int>(unit % p.H);
  const float* o = p.o + unit * p.V;
  const float* gate = p.proj + row * p.width + p.g_off + h * p.V;
  float ss = 0.0f;
  for (int d = lane; d < p.V; d += 32) ss = fmaf(o[d], o[d], ss);
  for (int k = 16; k > 0; k >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, k);
  const float r = 1.0f / sqrtf(ss / static_cast<float>(p.V) + p.eps);
  TO* out = static_cast<TO*>(p.out) + unit * p.V;
  for (int d = lane; d < p.V; d += 32) {
    float v = __fmul_rn(o[d], r);
    if (p.gain != nullptr) v = __fmul_rn(v, p.gain_bf16 ? __bfloat162float(static_cast<const bf16*>(p.gain)[d]) : static_cast<const float*>(p.gain)[d]);
    const float g = folded(gate + d, p.n_partials, p.partial_stride);
    const float sg = 1.0f / (1.0f + expf(-g));
    out[d] = sb::narrow<TO>(__fmul_rn(v, p.silu_gate ? g * sg : sg));
  }
}

}  // namespace

// i: 0 projection partial sums (flat), 1 their width, 2 K ranges S, 3 most tokens with a buffer per range, 4 q_off, 5 k_off, 6 v_off, 7 cos_sin,
//    8 rot, 9 interleaved pairs, 10 out (float32 [n][2 H D + H V]), 11 H, 12 D, 13 V      f: 0 the constant on k
SB_EXPORT int sb_op_rotate_qk(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int width = (int)op->i[1], rot = (int)op->i[8], H = (int)op->i[11], D = (int)op->i[12], V = (int)op->i[13];
  if (rot < 0 || rot % 2 != 0 || rot > D) return sb::fail("sb_op_rotate_qk: %d rotated elements of %d", rot, D), SB_OP_FAILED;
  RotateParams p{ptr<const float>(op->i[0]), partial_count(op->i[2], op->i[3], s->n), static_cast<int64_t>(s->n) * width, width, (int)op->i[4],
                 (int)op->i[5], (int)op->i[6], positions(s), ptr<const float>(op->i[7]), rot, (int)op->i[9], (float)op->f[0], ptr<float>(op->i[10]),
                 H, D, V};
  const int cols = 2 * H * D + H * V;
  sb::launch_pdl(rotate_qk_kernel, dim3(s->n, (cols + 1023) / 1024), dim3(256), 0, static_cast<cudaStream_t>(stream), p);
  return sb::check_launch("sb_op_rotate_qk");
}

// i: 0 o (float32 [n, H V]), 1 the gate's partial sums (flat), 2 their width, 3 K ranges S, 4 most tokens with a buffer per range, 5 g_off,
//    6 gain ([V], or 0), 7 gain dtype, 8 out, 9 out dtype, 10 H, 11 V, 12 the gate's activation (0 sigmoid, 1 silu)      f: 0 eps
SB_EXPORT int sb_op_group_norm_gate(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int width = (int)op->i[2];
  GroupGateParams p{ptr<const float>(op->i[0]), ptr<const float>(op->i[1]), partial_count(op->i[3], op->i[4], s->n), static_cast<int64_t>(s->n) * width,
                    width, (int)op->i[5], ptr<const void>(op->i[6]), (int)(op->i[7] == 1), ptr<void>(op->i[8]), s->n, (int)op->i[10], (int)op->i[11],
                    (int)op->i[12], (float)op->f[0]};
  const int64_t units = static_cast<int64_t>(p.n) * p.H;
  const dim3 grid(static_cast<unsigned>((units + 3) / 4));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (op->i[9] == 0) sb::launch_pdl(group_norm_gate_kernel<float>, grid, dim3(128), 0, st, p);
  else if (op->i[9] == 1) sb::launch_pdl(group_norm_gate_kernel<bf16>, grid, dim3(128), 0, st, p);
  else return sb::fail("sb_op_group_norm_gate: unsupported dtype %d", (int)op->i[9]), SB_OP_FAILED;
  return sb::check_launch("sb_op_group_norm_gate");
}
