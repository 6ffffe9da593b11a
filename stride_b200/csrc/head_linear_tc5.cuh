// A matrix per head on tcgen05, for many tokens: out[r, h, :] = W_h^T in[r, h, :], W [H][K][N] with n contiguous, optionally times the
// sigmoid of a gate. One CTA per (128 rows, head, up to 256 columns): K in pieces of 64 through a ring of stages by TMA, the rows [128][64]
// as the K-major A operand, the weights [64 k][64 n] pieces as the MN-major B operand; the accumulator's lane is the row, so that a thread of
// the epilogue has a row's gates in a line of memory. The result is rounded, staged in shared memory and stored by TMA, which leaves rows
// beyond the step's tokens out. A sum runs over k in steps of 16 from zero: the bits of head_linear_tc_kernel (mma.sync).
#pragma once

#include "tc5.cuh"

namespace sb {
namespace heads5 {

using namespace sb::tc5;
using bf16 = __nv_bfloat16;

constexpr int kRows = 128, kThreads = 192, kMaxStages = 4;
constexpr int kABytes = kRows * 128, kPieceBytes = 64 * 128;
constexpr int kSmemBudget = 96 * 1024;      // two CTAs an SM: one's loads run under the other's epilogue

struct Params {
  int n, K, N, cols, stages;         // cols: columns of a CTA, a multiple of 64 that divides N
  const float* gate;                 // [n][gate_width], or null
  int gate_width;
  int* status;
};

template <bool GATED>
__global__ void __launch_bounds__(kThreads, 2)
head_linear_tc5_kernel(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_out,
                       const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], accum_bar;
  __shared__ uint32_t tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int r0 = blockIdx.x * kRows, h = blockIdx.y, n0 = blockIdx.z * p.cols;
  const int stage_bytes = kABytes + p.cols * 128, iters = p.K / 64, pieces = p.cols / 64;
  uint32_t tmem_cols = 64;
  while (tmem_cols < static_cast<uint32_t>(p.cols)) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_in);
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_out);
    for (int s = 0; s < p.stages; ++s) mbar_init(smem_u32(&full_bar[s]), 1), mbar_init(smem_u32(&empty_bar[s]), 1);
    mbar_init(smem_u32(&accum_bar), 1);
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_base_s), tmem_cols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  sb::grid_launch_dependents();

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- loads; the first ring of weights before the wait for the kernels in front
      auto load_w = [&](int i, int s) {
        mbar_expect_tx(smem_u32(&full_bar[s]), stage_bytes);
        for (int j = 0; j < pieces; ++j)
          tma_load_2d(smem0 + s * stage_bytes + kABytes + j * kPieceBytes, &map_w, smem_u32(&full_bar[s]), n0 + 64 * j, h * p.K + 64 * i);
      };
      const int ahead = min(iters, p.stages);
      for (int i = 0; i < ahead; ++i) load_w(i, i);
      sb::grid_dependency_wait();
      uint32_t s = 0, par = 1;
      for (int i = 0; i < iters; ++i) {
        if (i >= ahead) {
          mbar_wait(smem_u32(&empty_bar[s]), par, p.status, 1);
          load_w(i, s);
        }
        tma_load_3d(smem0 + s * stage_bytes, &map_in, smem_u32(&full_bar[s]), 64 * i, h, r0);
        if (++s == static_cast<uint32_t>(p.stages)) s = 0, par ^= 1;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- products
      const uint32_t idesc = instr_desc(kRows, p.cols, true);
      const uint64_t fixed = smem_desc_sw128(0), da0 = fixed + (smem0 >> 4);
      const uint64_t db0 = (fixed | (static_cast<uint64_t>(kPieceBytes >> 4) << 16)) + ((smem0 + kABytes) >> 4);
      uint32_t s = 0, par = 0;
      for (int i = 0; i < iters; ++i) {
        mbar_wait(smem_u32(&full_bar[s]), par, p.status, 2);
        fence_after_sync();
        const uint64_t da = da0 + s * (stage_bytes >> 4), db = db0 + s * (stage_bytes >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem_base, da + 2 * k, db + k * (2048 >> 4), idesc, (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(smem_u32(&empty_bar[s]));
        if (++s == static_cast<uint32_t>(p.stages)) s = 0, par ^= 1;
      }
      umma_commit(smem_u32(&accum_bar));
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: warps 2..5, thread = row of the tile
    const int quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    uint8_t* staged = smem_raw + (smem0 - smem_u32(smem_raw));
    sb::grid_dependency_wait();
    const bool ok = mbar_wait(smem_u32(&accum_bar), 0, p.status, 3);       // (and with it the ring is free)
    fence_after_sync();
    const bool live = r0 + r < p.n;
    const float* gate = GATED && live ? p.gate + static_cast<int64_t>(r0 + r) * p.gate_width + h * p.N + n0 : nullptr;
    for (int c0 = 0; c0 < p.cols; c0 += 32) {
      float v[32], g[32];
      if (GATED && live) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 x = *reinterpret_cast<const float4*>(gate + c0 + i);
          g[i] = x.x, g[i + 1] = x.y, g[i + 2] = x.z, g[i + 3] = x.w;
        }
      }
      tmem_load32(acc + c0, v);
      if (GATED && live) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] *= 1.0f / (1.0f + expf(-g[i]));
      }
      uint8_t* row = staged + (c0 >> 6) * kABytes + r * 128;
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(v[i + 2 * k], v[i + 2 * k + 1]);
          w[k] = *reinterpret_cast<const uint32_t*>(&b);
        }
        *reinterpret_cast<uint4*>(row + (((((c0 & 63) + i) >> 3) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    fence_async_smem();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (threadIdx.x == 64 && ok) {
      for (int j = 0; j < pieces; ++j) tma_store_3d(&map_out, smem0 + j * kABytes, n0 + 64 * j, h, r0);
      tma_store_wait();
    }
    fence_before_sync();
  }
  __syncthreads();
  if (warp == 1) {
    fence_after_sync();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

}  // namespace heads5
}  // namespace sb
