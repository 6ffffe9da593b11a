// Linear attention with a gate per key channel and token, as a recurrence over a state kept per request:
//
//   S_t = diag(g_t) S_(t-1) + k_t v_t^T        S: [D, V] float32 per head, g_t and k_t: [D]
//   o_t = S_t^T q_t
//
// The kernel takes q, g, k, v as columns of one float32 row per token, so whatever makes them is a kernel in front.
// HGRN2 is one such maker (`hgrn2_activate_kernel`): q = silu(W_q x), g = l + (1 - l) sigmoid(W_f x + b) with a lower
// bound l per channel, k = 1 - g (the gate's complement is the key: what a channel does not keep, it takes in), v = W_v x.
// Everything here is 32-bit; the recurrence is linear_scan.cuh's, whose outputs have the same bits in a prompt, in a portion and decoded alone.
//
// `group_rmsnorm_kernel` is what follows: every head's output RMS-normed on its own with one gain vector for all heads.
#include "common.cuh"
#include "linear_scan.cuh"
#include "step_ops.h"

SB_DEFINE_LAST_ERROR()

namespace {

using bf16 = __nv_bfloat16;
constexpr int kInFlight = 8;

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

template <bool ONE>
__device__ __forceinline__ float4 folded4(const float* p, int n_partials, int64_t stride) {      // four neighbouring elements, 16-byte aligned
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

// proj [P][n][2 HD + HV]: columns q | f | v. act [n][3 HD + HV]: columns q | g | k | v. grid: (rows, pieces of a row). VE = 4: four elements
// an access where the sizes and buffers allow it. PIECES: single elements of a row a thread, requested together (four where the rows are many:
// blocks of one are then too short-lived). Bound by memory: 1,250 rows of 16 heads of 128 | 128 15.5 us, 37 us with one element and a 64-bit
// division a thread and round.
template <class TW, int VE, bool ONE, int PIECES>
__global__ void __launch_bounds__(128) hgrn2_activate_kernel(const float* __restrict__ proj, int n_partials, int64_t partial_stride,
                                                             const TW* __restrict__ f_bias, const TW* __restrict__ lower, float* __restrict__ act, int HD, int HV) {
  sb::grid_launch_dependents();
  const int in_w = 2 * HD + HV, j0 = (blockIdx.y * PIECES * blockDim.x + threadIdx.x) * VE;
  if (j0 >= in_w) return;
  float l[PIECES][VE], fb[PIECES][VE], z[PIECES][VE];
#pragma unroll
  for (int k = 0; k < PIECES; ++k) {
    const int j = j0 + k * blockDim.x * VE;
    if (j >= HD && j < 2 * HD) {
#pragma unroll
      for (int i = 0; i < VE; ++i) l[k][i] = sb::widen(lower[j - HD + i]), fb[k][i] = sb::widen(f_bias[j - HD + i]);
    }
  }
  sb::grid_dependency_wait();
  const float* src = proj + static_cast<int64_t>(blockIdx.x) * in_w;
#pragma unroll
  for (int k = 0; k < PIECES; ++k) {
    const int j = j0 + k * blockDim.x * VE;
    if constexpr (VE == 4) {
      const float4 v = folded4<ONE>(src + j, n_partials, partial_stride);
      z[k][0] = v.x, z[k][1] = v.y, z[k][2] = v.z, z[k][3] = v.w;
    } else if (PIECES == 1 || j < in_w) {
      z[k][0] = folded(src + j, n_partials, partial_stride);
    }
  }
  auto store = [&](float* to, const float (&v)[VE]) {
    if constexpr (VE == 4) *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
    else to[0] = v[0];
  };
  float* row = act + static_cast<int64_t>(blockIdx.x) * (3 * HD + HV);
#pragma unroll
  for (int k = 0; k < PIECES; ++k) {
    const int j = j0 + k * blockDim.x * VE;
    if (PIECES > 1 && j >= in_w) break;
    if (j >= HD && j < 2 * HD) {
      float g[VE];
#pragma unroll
      for (int i = 0; i < VE; ++i) {
        const float s = 1.0f / (1.0f + expf(-(z[k][i] + fb[k][i])));
        g[i] = fmaf(1.0f - l[k][i], s, l[k][i]);
        z[k][i] = 1.0f - g[i];
      }
      store(row + j, g);
      store(row + HD + j, z[k]);
      continue;
    }
    if (j < HD) {
#pragma unroll
      for (int i = 0; i < VE; ++i) z[k][i] = z[k][i] / (1.0f + expf(-z[k][i]));
    }
    store(row + (j < HD ? j : HD + j), z[k]);
  }
}

// Steps in which every entry brings one token.
template <int DL>
__global__ void __launch_bounds__(DL * 64, 1024 / (DL * 64)) gated_step_kernel(const sbscan::Params p) {
  extern __shared__ __align__(16) float smem[];
  sb::grid_launch_dependents();
  const int e = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * 32;
  const int slot = p.meta[e], row0 = p.meta[p.meta_stride + e], len = p.meta[2 * p.meta_stride + e], pos0 = p.meta[3 * p.meta_stride + e];
  sb::grid_dependency_wait();
  sbscan::step_core<DL, true>(p, smem, slot, row0, len, pos0, [&](float* to, int Ds, int row) {
    // up to three values a thread, requested together (2 Ds threads, 3 Ds + 32 values, Ds >= 16)
    const float* src = p.rows + static_cast<int64_t>(row) * p.width;
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int j = threadIdx.x + k * blockDim.x;
      v[k] = 0.0f;
      if (j < 3 * Ds) {
        const int which = j / Ds, d = j - which * Ds;          // q, k, g
        if (d < p.D) v[k] = src[(which == 0 ? p.q_off : which == 1 ? p.k_off : p.g_off) + h * p.D + d];
      } else if (j < 3 * Ds + 32 && c0 + j - 3 * Ds < p.V) {
        v[k] = src[p.v_off + h * p.V + c0 + j - 3 * Ds];
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (threadIdx.x + k * blockDim.x < 3 * Ds + 32) to[threadIdx.x + k * blockDim.x] = v[k];
  });
}

// out[r, h V + j] = o[r, h V + j] / sqrt(mean_j(o[r, h V + :]^2) + eps) * gain[j]: a warp per (row, head).
template <class TW, class TO>
__global__ void group_rmsnorm_kernel(const float* __restrict__ o, const TW* __restrict__ gain, TO* __restrict__ out, int64_t groups, int V, float eps) {
  sb::grid_launch_dependents();
  sb::grid_dependency_wait();
  const int64_t gidx = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gidx >= groups) return;
  const float* src = o + gidx * V;
  float ss = 0.0f;
  for (int j = lane; j < V; j += 32) ss = fmaf(src[j], src[j], ss);
  for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
  const float scale = 1.0f / sqrtf(ss / static_cast<float>(V) + eps);
  for (int j = lane; j < V; j += 32) out[gidx * V + j] = sb::narrow<TO>(src[j] * scale * sb::widen(gain[j]));
}

}  // namespace

SB_EXPORT int sb_hgrn2_activate(const float* proj, int n_partials, int64_t partial_stride, const void* f_bias, const void* lower, int w_dtype,
                                float* act, int n, int HD, int HV, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n_partials < 1) return sb::fail("sb_hgrn2_activate: n_partials must be >= 1");
  const bool vec = HD % 4 == 0 && HV % 4 == 0 && partial_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(act)) & 15) == 0;
  const bool many = !vec && n > 1024;
  const dim3 grid(n, (2 * HD + HV + (vec || many ? 511 : 127)) / (vec || many ? 512 : 128));
#define SB_ACT(TW, VE, ONE, PIECES) \
  sb::launch_pdl(hgrn2_activate_kernel<TW, VE, ONE, PIECES>, grid, dim3(128), 0, stream, proj, n_partials, partial_stride, static_cast<const TW*>(f_bias), \
                 static_cast<const TW*>(lower), act, HD, HV)
#define SB_ACT_T(TW)                                          \
  do {                                                        \
    if (vec && n_partials == 1) SB_ACT(TW, 4, true, 1);       \
    else if (vec) SB_ACT(TW, 4, false, 1);                    \
    else if (many) SB_ACT(TW, 1, false, 4);                   \
    else SB_ACT(TW, 1, false, 1);                             \
  } while (0)
  if (w_dtype == 0) SB_ACT_T(float);
  else if (w_dtype == 1) SB_ACT_T(bf16);
  else return sb::fail("sb_hgrn2_activate: unsupported dtype %d", w_dtype);
#undef SB_ACT_T
#undef SB_ACT
  return sb::check_launch("sb_hgrn2_activate");
}

// n: the step's tokens
SB_EXPORT int sb_gated_scan(const float* act, int width, int q_off, int g_off, int k_off, int v_off, const int32_t* meta, int meta_stride,
                            int entries, int n, float* state, float* out, int H, int D, int V, cudaStream_t stream) {
  if (entries <= 0) return 0;
  if (H <= 0 || D <= 0 || V <= 0 || D > 256) return sb::fail("sb_gated_scan: heads %d, key size %d (at most 256), value size %d", H, D, V);
  sbscan::Params p{act, width, q_off, k_off, v_off, g_off, meta, meta_stride, nullptr, state, out, H, D, V};
  if (n == entries) {
    const auto kernel = sbscan::lane_elements(D) == 2 ? gated_step_kernel<2> : sbscan::lane_elements(D) == 4 ? gated_step_kernel<4> : gated_step_kernel<8>;
    sb::launch_pdl(kernel, dim3(entries, H, (V + 31) / 32), dim3(sbscan::step_threads(D)), sbscan::step_smem(D, true), stream, p);
    return sb::check_launch("sb_gated_scan");
  }
  return sbscan::launch_scan<true>(p, entries, n, "sb_gated_scan", stream);
}

SB_EXPORT int sb_group_rmsnorm(const float* o, const void* gain, int gain_dtype, void* out, int out_dtype, int n, int H, int V, float eps,
                               cudaStream_t stream) {
  if (n <= 0) return 0;
  const int64_t groups = static_cast<int64_t>(n) * H;
  const dim3 grid(static_cast<unsigned>((groups + 7) / 8));
#define SB_GN(TW, TO) sb::launch_pdl(group_rmsnorm_kernel<TW, TO>, grid, dim3(256), 0, stream, o, static_cast<const TW*>(gain), static_cast<TO*>(out), groups, V, eps)
  if (gain_dtype == 0 && out_dtype == 0) SB_GN(float, float);
  else if (gain_dtype == 0 && out_dtype == 1) SB_GN(float, bf16);
  else if (gain_dtype == 1 && out_dtype == 0) SB_GN(bf16, float);
  else if (gain_dtype == 1 && out_dtype == 1) SB_GN(bf16, bf16);
  else return sb::fail("sb_group_rmsnorm: unsupported dtypes gain=%d out=%d", gain_dtype, out_dtype);
#undef SB_GN
  return sb::check_launch("sb_group_rmsnorm");
}

// ------------------------------------------------------------------ operations of the native step program (step_ops.h)
// i: 0 projection partial sums (flat), 1 K ranges S, 2 most tokens with a buffer per range, 3 f bias, 4 lower bound, 5 their dtype, 6 act, 7 HD, 8 HV
SB_EXPORT int sb_op_hgrn2_activate(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  const int HD = (int)op->i[7], HV = (int)op->i[8];
  return sb_hgrn2_activate(ptr<const float>(op->i[0]), partial_count(op->i[1], op->i[2], s->n), static_cast<int64_t>(s->n) * (2 * HD + HV),
                           ptr<const void>(op->i[3]), ptr<const void>(op->i[4]), (int)op->i[5], ptr<float>(op->i[6]), s->n, HD, HV,
                           static_cast<cudaStream_t>(stream));
}

// i: 0 act, 1 width, 2 q_off, 3 g_off, 4 k_off, 5 v_off, 6 state, 7 out, 8 H, 9 D, 10 V
SB_EXPORT int sb_op_gated_scan(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  return sb_gated_scan(ptr<const float>(op->i[0]), (int)op->i[1], (int)op->i[2], (int)op->i[3], (int)op->i[4], (int)op->i[5], entry_meta(s),
                       s->max_rows, s->entries, s->n, ptr<float>(op->i[6]), ptr<float>(op->i[7]), (int)op->i[8], (int)op->i[9], (int)op->i[10],
                       static_cast<cudaStream_t>(stream));
}

// i: 0 o, 1 gain, 2 gain dtype, 3 out, 4 out dtype, 5 H, 6 V      f: 0 eps
SB_EXPORT int sb_op_group_rmsnorm(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  if (s->n <= 0) return SB_OP_SKIPPED;
  return sb_group_rmsnorm(ptr<const float>(op->i[0]), ptr<const void>(op->i[1]), (int)op->i[2], ptr<void>(op->i[3]), (int)op->i[4], s->n,
                          (int)op->i[5], (int)op->i[6], (float)op->f[0], static_cast<cudaStream_t>(stream));
}
