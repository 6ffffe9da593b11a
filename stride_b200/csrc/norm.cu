// RMSNorm, fused with the reduction of split-K partial sums into the residual. All arithmetic is
// 32-bit; only the gain and the normed values may be bfloat16.
//
// Counterpart in arhaamatiq/stride: RmsNorm (src/kernels.cu:119-200).
#include "common.cuh"
#include "step_ops.h"

SB_DEFINE_LAST_ERROR()

namespace {

using bf16 = __nv_bfloat16;

// ------------------------------------------------------------------ rmsnorm
// One block per row. The row is h + (partial_0 + partial_1 + ...), the partials summed left to
// right first (as the tensor-core kernel adds its K ranges when it does so itself) and then added
// to h; when partials are given the sum is written back to h. Then
// r = 1/sqrt(sum(x^2)/H + eps) and out = w * (x * r). VEC = 4 reads float4 (H % 4 == 0);
// FLIGHT partials are fetched together so that their loads overlap.
template <int VEC>
struct VecF;
template <>
struct VecF<4> { using type = float4; };
template <>
struct VecF<1> { using type = float; };

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float add4(float a, float b) { return a + b; }

// FLIGHT: the partial sums requested together. 12 while all rows run at once: every one is a round trip to L2. With more rows 6, twice the
// blocks an SM (256 rows of 2,048 behind nine buffers 5.4 us, 7.1 with 12; 256 rows of 1,024, which run at once with 12, 3.7 and 3.0).
// The additions are the same: equal bits. BLOCKS: the blocks an SM that the registers are cut for (0: left to the compiler); two in the
// single-element form (2,048 rows of 2,050 behind one buffer: 30 us, 43 with one).
template <class TW, class TO, int VEC, int MAXT, int FLIGHT, int BLOCKS>     // MAXT: the most threads of a block
__global__ void __launch_bounds__(MAXT, BLOCKS) rmsnorm_kernel(float* __restrict__ h, const float* __restrict__ partials, int n_partials,
                               int64_t partial_stride, const TW* __restrict__ weight, TO* __restrict__ out,
                               int H, float eps) {
  using V = typename VecF<VEC>::type;
  extern __shared__ __align__(16) float row[];
  __shared__ float red[32];
  sb::grid_launch_dependents();
  const int r = blockIdx.x;
  const int units = H / VEC;
  // The gain does not depend on the kernels before this one: fetch this thread's first piece of it before waiting.
  float w_first[VEC];
  if (threadIdx.x < units) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) w_first[e] = sb::widen(weight[threadIdx.x * VEC + e]);
  }
  sb::grid_dependency_wait();
  V* hr = reinterpret_cast<V*>(h + static_cast<int64_t>(r) * H);
  float ss = 0.0f;
  for (int i = threadIdx.x; i < units; i += blockDim.x) {
    V v = hr[i];
    if (n_partials > 0) {
      constexpr int kInFlight = FLIGHT;
      const V* p = reinterpret_cast<const V*>(partials + static_cast<int64_t>(r) * H) + i;
      const int64_t ps = partial_stride / VEC;
      V part[kInFlight];
#pragma unroll
      for (int s = 0; s < kInFlight; ++s)
        if (s < n_partials) part[s] = p[s * ps];
      V sum = part[0];
#pragma unroll
      for (int s = 1; s < kInFlight; ++s)
        if (s < n_partials) sum = add4(sum, part[s]);
      for (int s = kInFlight; s < n_partials; ++s) sum = add4(sum, p[s * ps]);
      v = add4(v, sum);
      hr[i] = v;
    }
    reinterpret_cast<V*>(row)[i] = v;
    if constexpr (VEC == 4) {
      ss = fmaf(v.x, v.x, ss);
      ss = fmaf(v.y, v.y, ss);
      ss = fmaf(v.z, v.z, ss);
      ss = fmaf(v.w, v.w, ss);
    } else {
      ss = fmaf(v, v, ss);
    }
  }
  const float total = sb::block_sum(ss, red);
  const float scale = 1.0f / sqrtf(total / static_cast<float>(H) + eps);
  TO* o = out + static_cast<int64_t>(r) * H;
  for (int i = threadIdx.x; i < units; i += blockDim.x) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const float w = i == static_cast<int>(threadIdx.x) ? w_first[e] : sb::widen(weight[i * VEC + e]);
      o[i * VEC + e] = sb::narrow<TO>(w * (row[i * VEC + e] * scale));
    }
  }
}

// Four gains from element i of a bfloat16 or float32 vector (the widening is exact).
__device__ __forceinline__ float4 load_gain4(const void* w, bool is_bf16, int i) {
  if (is_bf16) {
    const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const bf16*>(w) + i);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
  }
  return *reinterpret_cast<const float4*>(static_cast<const float*>(w) + i);
}
template <class TO>
__device__ __forceinline__ void store_normed4(TO* o, float4 v, float4 w, float scale) {
  if constexpr (sizeof(TO) == 2) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(w.x * (v.x * scale), w.y * (v.y * scale));
    __nv_bfloat162 hi = __floats2bfloat162_rn(w.z * (v.z * scale), w.w * (v.w * scale));
    uint2 packed;
    packed.x = *reinterpret_cast<uint32_t*>(&lo);
    packed.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(o) = packed;
  } else {
    *reinterpret_cast<float4*>(o) = make_float4(w.x * (v.x * scale), w.y * (v.y * scale), w.z * (v.z * scale), w.w * (v.w * scale));
  }
}

// Few rows behind several partial buffers (decoding): a row's ten reads of 8 KB are more than one SM takes in during a round trip to L2, so a
// row is a cluster of four blocks, each with a quarter of rmsnorm_kernel's threads and their shares; the warps' sums of squares go to all four
// blocks' shared memory and are added in rmsnorm_kernel's order: equal bits. One to 64 rows of 2,048 behind nine buffers, within a decode
// step: 3.4 to 4.1 us, 4.1 to 4.5 as a block a row.
__device__ __forceinline__ void cluster_store(const float* p, uint32_t rank, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(sb::cluster_peer_address(p, rank)), "f"(v) : "memory");
}
constexpr int kRowBlocks = 4;
template <class TW, class TO>
__global__ void __launch_bounds__(256) rmsnorm_cluster_kernel(float* __restrict__ h, const float* __restrict__ partials, int n_partials,
                                                              int64_t partial_stride, const TW* __restrict__ weight, TO* __restrict__ out, int H, float eps) {
  __shared__ float red[32];
  sb::grid_launch_dependents();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // (all four blocks have begun: waited for below)
  const int64_t r = blockIdx.x / kRowBlocks;
  const int rank = blockIdx.x % kRowBlocks, units = H / 4, threads = kRowBlocks * blockDim.x, t = rank * blockDim.x + threadIdx.x;
  float4 w_first = make_float4(0, 0, 0, 0);
  if (t < units) w_first = load_gain4(weight, sizeof(TW) == 2, 4 * t);
  sb::grid_dependency_wait();
  float4* hr = reinterpret_cast<float4*>(h + r * H);
  const int64_t ps = partial_stride / 4;
  float4 first = make_float4(0, 0, 0, 0);
  float ss = 0.0f;
  for (int i = t; i < units; i += threads) {
    constexpr int kInFlight = 12;
    const float4* p = reinterpret_cast<const float4*>(partials + r * H) + i;
    float4 v = hr[i], part[kInFlight];
#pragma unroll
    for (int s = 0; s < kInFlight; ++s)
      if (s < n_partials) part[s] = p[s * ps];
    float4 sum = part[0];
#pragma unroll
    for (int s = 1; s < kInFlight; ++s)
      if (s < n_partials) sum = add4(sum, part[s]);
    for (int s = kInFlight; s < n_partials; ++s) sum = add4(sum, p[s * ps]);
    v = add4(v, sum);
    hr[i] = v;
    if (i == t) first = v;
    ss = fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, ss))));
  }
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  const int lane = threadIdx.x & 31;
  if (lane < kRowBlocks) cluster_store(&red[t >> 5], lane, ss);
  __syncwarp();
  sb::cluster_sync();
  float total = red[0];
  for (int i = 1; i < threads >> 5; ++i) total += red[i];
  const float scale = 1.0f / sqrtf(total / static_cast<float>(H) + eps);
  TO* o = out + r * H;
  if (t < units) store_normed4<TO>(o + 4 * t, first, w_first, scale);
  for (int i = t + threads; i < units; i += threads) store_normed4<TO>(o + 4 * i, hr[i], load_gain4(weight, sizeof(TW) == 2, 4 * i), scale);
}

// At most one partial buffer (prompts, whose projections fold their K ranges themselves; the 32-bit path): half as many threads as
// rmsnorm_kernel has for the width, each with the shares of two of its threads, t and t + blockDim.x, so that twice as much is in flight a
// thread and no register is kept for partial buffers that do not exist. The squares are added in rmsnorm_kernel's order (a warp stands for
// two of its warps): equal bits. 2,048 rows of 2,048: 11.8 us; 17 us as a warp a row, 19 with rmsnorm_kernel's threads.
template <class TW, class TO>
__global__ void __launch_bounds__(512) rmsnorm_pairs_kernel(float* __restrict__ h, const float* __restrict__ partial, const TW* __restrict__ weight,
                                                            TO* __restrict__ out, int H, float eps) {
  __shared__ float red[32];
  sb::grid_launch_dependents();
  sb::grid_dependency_wait();
  const int64_t r = blockIdx.x;
  const int units = H / 4, half = blockDim.x, warps = half >> 5;
  float4* hr = reinterpret_cast<float4*>(h + r * H);
  const float4* pr = reinterpret_cast<const float4*>(partial + r * H);
  auto square = [](float4 v, float ss) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, ss)))); };
  float4 keep[2], add[2];
  float ss[2] = {0.0f, 0.0f};
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = threadIdx.x + j * half;
    if (i < units) {
      keep[j] = hr[i];
      if (partial != nullptr) add[j] = pr[i];
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = threadIdx.x + j * half;
    if (i < units) {
      if (partial != nullptr) hr[i] = keep[j] = add4(keep[j], add[j]);
      ss[j] = square(keep[j], 0.0f);
    }
    for (int k = i + 2 * half; k < units; k += 2 * half) {      // wider rows are read again behind the sum
      float4 v = hr[k];
      if (partial != nullptr) hr[k] = v = add4(v, pr[k]);
      ss[j] = square(v, ss[j]);
    }
    float c = ss[j];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) red[j * warps + (threadIdx.x >> 5)] = c;
  }
  __syncthreads();
  float total = red[0];
  for (int i = 1; i < 2 * warps; ++i) total += red[i];
  const float scale = 1.0f / sqrtf(total / static_cast<float>(H) + eps);
  TO* o = out + r * H;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = threadIdx.x + j * half;
    if (i < units) store_normed4<TO>(o + 4 * i, keep[j], load_gain4(weight, sizeof(TW) == 2, 4 * i), scale);
    for (int k = i + 2 * half; k < units; k += 2 * half) store_normed4<TO>(o + 4 * k, hr[k], load_gain4(weight, sizeof(TW) == 2, 4 * k), scale);
  }
}

// ------------------------------------------------------------------ layer norm
// One block per row: x = h + (partial_0 + partial_1 + ...) as in rmsnorm_kernel (written back to h when partials are given);
// mean = sum(x) / H; var = sum((x - mean)^2) / H; out = (x - mean) / sqrt(var + eps) * w + b. Both sums in the order of sb::block_sum.
// VEC = 4: four elements an access where the width and every buffer allow it; which form runs depends on the width and the buffers alone,
// never on the rows, so a row's result does not either. A thread keeps its first kKeep pieces in registers through both sums, those beyond in
// shared memory. Bound by memory: 2,048 rows of 2,048 with one partial buffer 10.5 us (22 with the registers for eight partial buffers,
// hence FLIGHT), single elements in shared memory 24 us.
//
// layernorm_blocks: the blocks an SM that its registers are cut for (0: left to the compiler).
constexpr int layernorm_blocks(int VEC, int MAXT, int FLIGHT, size_t bytes) {
  if (VEC == 1) return 2048 / MAXT;
  if (FLIGHT == 1) return bytes == 4 ? 4 : 3;      // (of 512 threads: 32 registers a thread where gain and output are bfloat16, else 40)
  return FLIGHT == 4 ? 1024 / MAXT : 0;
}
template <class TW, class TO, int VEC, int MAXT, int FLIGHT>     // MAXT: the most threads of a block, FLIGHT: the partial sums requested together
__global__ void __launch_bounds__(MAXT, layernorm_blocks(VEC, MAXT, FLIGHT, sizeof(TW) + sizeof(TO))) layernorm_kernel(
    float* __restrict__ h, const float* __restrict__ partials, int n_partials, int64_t partial_stride, const TW* __restrict__ weight,
    const TW* __restrict__ bias, TO* __restrict__ out, int H, float eps) {
  using V = typename VecF<VEC>::type;
  constexpr int kKeep = VEC == 4 ? 2 : 1;
  constexpr bool kBeyond = VEC == 1 || MAXT > 512 || FLIGHT == 8;      // (512 threads and fewer keep all of a
  // row; with eight partial sums the kernel is the faster one with these loops compiled in: 4.4 us, 5.6 without, 256 rows of 2,048 behind nine)
  extern __shared__ __align__(16) float beyond_raw[];
  __shared__ float red[32];
  sb::grid_launch_dependents();
  sb::grid_dependency_wait();
  const int64_t r = blockIdx.x;
  const int units = H / VEC;
  V* hr = reinterpret_cast<V*>(h + r * H);
  auto fetch = [&](int i) {
    V v = hr[i];
    if (n_partials > 0) {
      constexpr int kInFlight = FLIGHT;
      const V* p = reinterpret_cast<const V*>(partials + r * H) + i;
      const int64_t ps = partial_stride / VEC;
      V part[kInFlight];
#pragma unroll
      for (int s = 0; s < kInFlight; ++s)
        if (s < n_partials) part[s] = p[s * ps];
      V sum = part[0];
#pragma unroll
      for (int s = 1; s < kInFlight; ++s)
        if (s < n_partials) sum = add4(sum, part[s]);
      if constexpr (FLIGHT > 1)      // (1: there is no more than one)
        for (int s = kInFlight; s < n_partials; ++s) sum = add4(sum, p[s * ps]);
      v = add4(v, sum);
      hr[i] = v;
    }
    return v;
  };
  auto total = [](V v) {
    if constexpr (VEC == 4) return ((v.x + v.y) + v.z) + v.w;
    else return v;
  };
  auto apart = [](V v, float mean, float sq) {
    if constexpr (VEC == 4) {
      const float x = v.x - mean, y = v.y - mean, z = v.z - mean, w = v.w - mean;
      return fmaf(w, w, fmaf(z, z, fmaf(y, y, fmaf(x, x, sq))));
    } else {
      return fmaf(v - mean, v - mean, sq);
    }
  };
  const int kept = kKeep * blockDim.x, beyond = kept + threadIdx.x;
  V* rest = reinterpret_cast<V*>(beyond_raw);
  V keep[kKeep];
  float sum = 0.0f;
#pragma unroll
  for (int j = 0; j < kKeep; ++j)
    if (threadIdx.x + j * blockDim.x < units) sum += total(keep[j] = fetch(threadIdx.x + j * blockDim.x));
  for (int i = beyond; kBeyond && i < units; i += blockDim.x) sum += total(rest[i - kept] = fetch(i));
  const float mean = sb::block_sum(sum, red) / static_cast<float>(H);
  float sq = 0.0f;
#pragma unroll
  for (int j = 0; j < kKeep; ++j)
    if (threadIdx.x + j * blockDim.x < units) sq = apart(keep[j], mean, sq);
  for (int i = beyond; kBeyond && i < units; i += blockDim.x) sq = apart(rest[i - kept], mean, sq);
  const float scale = 1.0f / sqrtf(sb::block_sum(sq, red) / static_cast<float>(H) + eps);
  auto write = [&](int i, V v) {
    if constexpr (VEC == 4) {
      const float4 w = load_gain4(weight, sizeof(TW) == 2, 4 * i), b = bias != nullptr ? load_gain4(bias, sizeof(TW) == 2, 4 * i) : make_float4(0, 0, 0, 0);
      const float4 o = make_float4(fmaf((v.x - mean) * scale, w.x, b.x), fmaf((v.y - mean) * scale, w.y, b.y), fmaf((v.z - mean) * scale, w.z, b.z),
                                   fmaf((v.w - mean) * scale, w.w, b.w));
      store_normed4<TO>(out + r * H + 4 * i, o, make_float4(1, 1, 1, 1), 1.0f);
    } else {
      out[r * H + i] = sb::narrow<TO>(fmaf((v - mean) * scale, sb::widen(weight[i]), bias != nullptr ? sb::widen(bias[i]) : 0.0f));
    }
  };
#pragma unroll
  for (int j = 0; j < kKeep; ++j)
    if (threadIdx.x + j * blockDim.x < units) write(threadIdx.x + j * blockDim.x, keep[j]);
  for (int i = beyond; kBeyond && i < units; i += blockDim.x) write(i, rest[i - kept]);
}

}  // namespace

// Layer norm with gain and bias over rows of H; arguments as sb_rmsnorm, plus the bias (of the gain's dtype; null: none).
SB_EXPORT int sb_layernorm(float* h, const float* partials, int n_partials, int64_t partial_stride, const void* weight,
                           const void* bias, int weight_dtype, void* out, int out_dtype, int n, int H, float eps, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (H > 50 * 1024) return sb::fail("sb_layernorm: width %d (at most 51200)", H);
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool vec = H % 4 == 0 && aligned(h) && aligned(partials) && aligned(weight) && aligned(bias) && aligned(out) && partial_stride % 4 == 0;
  // Single elements: several a thread, so that an SM holds more than one row (2,048 rows of 2,050: 17 us, 44 with 1,024 threads).
  const int units = vec ? H / 4 : H;
  const int threads = vec ? (units > 1024 ? 1024 : units > 512 ? 512 : units > 256 ? 256 : 128) : H >= 4096 ? 1024 : H >= 2048 ? 512 : H >= 512 ? 256 : 128;
  const int kept = (vec ? 2 : 1) * threads;      // (kKeep pieces a thread are in registers)
  const size_t smem = units > kept ? static_cast<size_t>(units - kept) * (vec ? 16 : 4) : 0;
  const bool at_once = n <= sb::sm_count() * (512 / threads);
  // (with eight partial sums requested together an SM holds 512 threads; more rows take four together, twice the threads: 2,048 rows of 3,072
  // behind nine buffers 66 us, 95 with eight)
#define SB_LN_V(TW, TO, VEC, MAXT, FLIGHT)                                                                                       \
  do {                                                                                                                        \
    if (smem > 40 * 1024)                                                                                                     \
      cudaFuncSetAttribute(layernorm_kernel<TW, TO, VEC, MAXT, FLIGHT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    sb::launch_pdl(layernorm_kernel<TW, TO, VEC, MAXT, FLIGHT>, n, threads, smem, stream, h, partials, n_partials, partial_stride, \
                   static_cast<const TW*>(weight), static_cast<const TW*>(bias), static_cast<TO*>(out), H, eps);              \
  } while (0)
#define SB_LN(TW, TO)                                                                \
  do {                                                                               \
    if (vec && threads <= 512 && n_partials <= 1) SB_LN_V(TW, TO, 4, 512, 1);        \
    else if (vec && threads <= 512 && at_once) SB_LN_V(TW, TO, 4, 512, 8);           \
    else if (vec && threads <= 512) SB_LN_V(TW, TO, 4, 512, 4);                      \
    else if (vec) SB_LN_V(TW, TO, 4, 1024, 4);                                       \
    else SB_LN_V(TW, TO, 1, 1024, 8);                                                \
  } while (0)
  if (weight_dtype == 0 && out_dtype == 0) SB_LN(float, float);
  else if (weight_dtype == 0 && out_dtype == 1) SB_LN(float, bf16);
  else if (weight_dtype == 1 && out_dtype == 0) SB_LN(bf16, float);
  else if (weight_dtype == 1 && out_dtype == 1) SB_LN(bf16, bf16);
  else return sb::fail("sb_layernorm: unsupported dtypes weight=%d out=%d", weight_dtype, out_dtype);
#undef SB_LN
#undef SB_LN_V
  return sb::check_launch("sb_layernorm");
}

// dtype codes shared with the Python side: 0 = float32, 1 = bfloat16.
SB_EXPORT int sb_rmsnorm(float* h, const float* partials, int n_partials, int64_t partial_stride, const void* weight,
                         int weight_dtype, void* out, int out_dtype, int n, int H, float eps, cudaStream_t stream) {
  if (n <= 0) return 0;
  const size_t smem = static_cast<size_t>(H) * sizeof(float);
  if (smem > 200 * 1024) return sb::fail("sb_rmsnorm: width %d (at most 51200)", H);      // (rmsnorm_kernel's row; one limit for every form)
  const bool vec = H % 4 == 0 && partial_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(partials)) & 15) == 0;
  const int units = vec ? H / 4 : H;
  const int threads = units >= 1024 ? 1024 : units >= 512 ? 512 : units >= 256 ? 256 : 128;
  const bool at_once = n <= sb::sm_count() * (640 / threads);      // (102 registers a thread: one block of 512 an SM, two of 256, five of 128)
#define SB_NORM_V(TW, TO, VEC, MAXT, FLIGHT, BLOCKS)                                                                     \
  do {                                                                                                           \
    if (smem > 48 * 1024)                                                                                        \
      cudaFuncSetAttribute(rmsnorm_kernel<TW, TO, VEC, MAXT, FLIGHT, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    sb::launch_pdl(rmsnorm_kernel<TW, TO, VEC, MAXT, FLIGHT, BLOCKS>, n, threads, smem, stream, h, partials, n_partials, partial_stride, \
                   static_cast<const TW*>(weight), static_cast<TO*>(out), H, eps);                               \
  } while (0)
  // Clusters: 32 rows behind nine buffers, width 2,048 3.0 us, 3.1 as a block a row (one row 2.3 and 2.8), 8,192 4.5 and 6.5; 64 rows 3.2 and 3.1,
  // 4.7 and 6.6. Narrower rows are one round trip of a block either way (1,024: one row 2.2, 64 rows 2.9).
#define SB_NORM(TW, TO)                                                                                                         \
  do {                                                                                                                          \
    if (vec && n_partials <= 1 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(weight)) & 15) == 0)         \
      sb::launch_pdl(rmsnorm_pairs_kernel<TW, TO>, dim3(n), dim3(threads / 2), 0, stream, h, n_partials == 1 ? partials : nullptr, \
                     static_cast<const TW*>(weight), static_cast<TO*>(out), H, eps);                                            \
    else if (vec && n <= 64 && threads >= 512 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(weight)) & 15) == 0) \
      sb::launch_pdl_cluster(rmsnorm_cluster_kernel<TW, TO>, dim3(n * kRowBlocks), dim3(threads / kRowBlocks), 0, stream, dim3(kRowBlocks), h, partials, \
                             n_partials, partial_stride, static_cast<const TW*>(weight), static_cast<TO*>(out), H, eps);        \
    else if (vec && threads > 512) SB_NORM_V(TW, TO, 4, 1024, 8, 1);                                                            \
    else if (vec && !at_once) SB_NORM_V(TW, TO, 4, 512, 6, 2);                                                                  \
    else if (vec) SB_NORM_V(TW, TO, 4, 512, 12, 0);                                                                             \
    else if (threads > 512 && n > sb::sm_count()) SB_NORM_V(TW, TO, 1, 1024, 8, 0);                                             \
    else if (threads > 512) SB_NORM_V(TW, TO, 1, 1024, 8, 1);                                                                   \
    else SB_NORM_V(TW, TO, 1, 512, 12, 0);                                                                                      \
  } while (0)
  if (weight_dtype == 0 && out_dtype == 0) SB_NORM(float, float);
  else if (weight_dtype == 0 && out_dtype == 1) SB_NORM(float, bf16);
  else if (weight_dtype == 1 && out_dtype == 0) SB_NORM(bf16, float);
  else if (weight_dtype == 1 && out_dtype == 1) SB_NORM(bf16, bf16);
  else return sb::fail("sb_rmsnorm: unsupported dtypes weight=%d out=%d", weight_dtype, out_dtype);
#undef SB_NORM
#undef SB_NORM_V
  return sb::check_launch("sb_rmsnorm");
}

// ------------------------------------------------------------------ operation of the native step program (step_ops.h)
// i: 0 h, 1 pending partial sums (flat; 0: none), 2 K ranges S, 3 most tokens with a buffer per range, 4 weight,
//    5 weight dtype, 6 out, 7 out dtype, 8 H, 9 rows: 0 = the step's tokens, 1 = the rows whose logits are wanted
// f: 0 eps
SB_EXPORT int sb_op_rmsnorm(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  const int n = op->i[9] ? s->wanted : s->n;
  if (n <= 0) return SB_OP_SKIPPED;
  const float* partials = ptr<const float>(op->i[1]);
  const int P = partials ? partial_count(op->i[2], op->i[3], n) : 0;
  return sb_rmsnorm(ptr<float>(op->i[0]), partials, P, static_cast<int64_t>(n) * op->i[8], ptr<const void>(op->i[4]), (int)op->i[5],
                    ptr<void>(op->i[6]), (int)op->i[7], n, (int)op->i[8], static_cast<float>(op->f[0]), static_cast<cudaStream_t>(stream));
}

// i: as sb_op_rmsnorm, and 10 the bias (or 0)
SB_EXPORT int sb_op_layernorm(const SbOp* op, const SbStep* s, void* stream) {
  using namespace sbstep;
  const int n = op->i[9] ? s->wanted : s->n;
  if (n <= 0) return SB_OP_SKIPPED;
  const float* partials = ptr<const float>(op->i[1]);
  const int P = partials ? partial_count(op->i[2], op->i[3], n) : 0;
  return sb_layernorm(ptr<float>(op->i[0]), partials, P, static_cast<int64_t>(n) * op->i[8], ptr<const void>(op->i[4]), ptr<const void>(op->i[10]),
                      (int)op->i[5], ptr<void>(op->i[6]), (int)op->i[7], n, (int)op->i[8], static_cast<float>(op->f[0]),
                      static_cast<cudaStream_t>(stream));
}
