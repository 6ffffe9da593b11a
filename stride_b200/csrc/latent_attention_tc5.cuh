// Attention over latent rows of 512 elements whose values are the rows themselves, for prompts and for steps of few entries (launch_latent has the
// lines): the tile kernel of masked_attention.cu on tcgen05, in the same arithmetic and the same bits.
//
// One CTA per (tile of 128 query rows of an entry and key/value head, half of the 512 value columns). A row is a (position, head), the heads
// of the group side by side: 128 / (H / G) positions. The CTA walks the tiles of 64 keys, cut by absolute position, that any row sees:
//
//   loading warp   Q once (eight pieces of 128 rows x 64 elements) and the tiles' rows as pieces of 64 keys x 64 elements in the 128-byte
//                  swizzle, by TMA through the block table, in a ring of three groups of four pieces. A piece is the B operand of the scores
//                  (K-major) and, in the CTA's half, of the value product (MN-major): the group of the other half goes back once the scores
//                  are made, the group of the own half once the values are added.
//   issuing warp   scores: four sums side by side, each over every fourth step of 16 elements, in four accumulators of 64 columns;
//                  values: O += hi V, then lo V, step of 16 keys by step, onto the accumulator (256 columns) that the softmax warps rescale.
//   softmax warps  two threads a row (TMEM lane = row; a thread has 32 keys of a tile and 128 of the 256 columns): the four sums joined,
//                  scaled, masked, the running maximum, the weights in 32-bit, split into two bfloat16 parts that go to tensor memory as
//                  the A operand of the value product, over the fourth sum's columns. While they work, the first three sums of the next
//                  tile are made; the fourth follows the value product that reads the weights.
//
// Every sum has the order of masked_attention_tile_kernel (16 partial row sums of the weights among them), so a row has the bits of that
// kernel: a token may come in a prompt, in a portion or alone. The tensor cores' two instructions accumulate alike (attention_math.cuh).
//
// A key that a row does not see has weight 0, and what lies in its row must not meet the row even if it is an infinity. Keys that no row
// of the tile sees are zeroed in shared memory; a key that some rows see and others do not, with a value that is not finite, is zeroed too
// and added by ordinary multiply-adds to the rows that see it.
//
// Measured (16 heads, window 1,024, a sink; within a step): prompts of 333, 584 and 1,025 tokens 282 us a layer on mma.sync, 103 here; one of 2,048
// tokens 176 (alone behind a flush of L2 604 and 182). Of the 5,650 cycles a tile takes (by the clock, in a block that walks many), the products take
// about 3,700 from issue to completion (scores 2,400: operands from shared memory; both halves' CTAs make all scores, since 512 columns of values
// and the scores do not fit one SM's tensor memory), of which the tensor pipe works 2,100 (counters: 29% of a launch's active cycles); the rest is the wait for
// the pieces whose place the tile in front leaves last, and the softmax warps' 2,870 cycles where the products do not cover them.
#pragma once

#include "tc5.cuh"

namespace sb {
namespace latent5 {

using namespace sb::tc5;
using bf16 = __nv_bfloat16;

constexpr int kRows = 128, kKeys = 64, kDim = 512;
constexpr int kPieces = kDim / 64, kHalfPieces = kPieces / 2, kHalfDim = kDim / 2;
constexpr int kQPieceBytes = kRows * 128, kPieceBytes = kKeys * 128, kGroupBytes = kHalfPieces * kPieceBytes, kGroups = 3;
constexpr int kSoftmaxThreads = 256, kThreads = kSoftmaxThreads + 64;
constexpr int kSmemBytes = kPieces * kQPieceBytes + kGroups * kGroupBytes;      // Q | ring: 224 KB
constexpr int kOutBytes = kHalfDim * 2 + 16;                                    // a staged row of the result, apart from the next one's banks
constexpr uint32_t kTmemP = 192, kTmemO = 256;                                  // S [0, 256), the weights over its last 64 columns, O [256, 512)

struct Params {
  bf16* out;                 // [n][H 512]
  const int32_t* block_table;
  int max_pages, page_shift, page_size;
  int rows_per_page, rows_head;      // distances in rows of 512 elements
  int box_rows;                      // rows one TMA box brings: min(page_size, 64)
  const int32_t* meta;               // [4][meta_stride]: slot, first row, length, first position of every entry
  int meta_stride, entries;
  const float* sinks;                // [H] or null
  int H, G, window;
  float scale;
  int* status;
};

// all softmax threads; and the two warps that share their rows (the warps' quarter of the tensor memory's lanes)
__device__ __forceinline__ void softmax_barrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ void rows_barrier(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory"); }
__device__ __forceinline__ bool not_finite(uint32_t pair) { return (pair & 0x7F80u) == 0x7F80u || (pair & 0x7F800000u) == 0x7F800000u; }

__global__ void __launch_bounds__(kThreads, 1)
latent_attention_tc5_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full, full_bar[kGroups], empty_bar[kGroups], s_full, s_free, p_full, o_full;
  __shared__ uint32_t tmem_base_s, odd_keys[2];       // odd_keys: keys of an edge tile that are not finite and not seen by all rows
  __shared__ float xch[2][kRows];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int Hg = p.H / p.G, ppt = kRows / Hg, g = blockIdx.y, half = blockIdx.x & 1;
  // the blocks that start first take the last tiles: those see the most keys
  int e = 0, tile = (static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x)) >> 1, len = 0;
  for (; e < p.entries; ++e) {
    len = p.meta[2 * p.meta_stride + e];
    const int tiles = (len + ppt - 1) / ppt;
    if (tile < tiles) break;
    tile -= tiles;
  }
  if (e >= p.entries) return;
  const int slot = p.meta[e], row0 = p.meta[p.meta_stride + e] + tile * ppt, first_pos = p.meta[3 * p.meta_stride + e] + tile * ppt;
  const int npos = min(ppt, len - tile * ppt), last_pos = first_pos + npos - 1;
  const int first_key = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
  const int kt0 = first_key / kKeys, T = last_pos / kKeys - kt0 + 1;

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem0 - smem_u32(smem_raw));
  const uint32_t ring = smem0 + kPieces * kQPieceBytes;
  // Group 2 t of the ring holds the pieces of tile t outside the CTA's half, group 2 t + 1 those of its half.
  auto group_of = [](int group) { return static_cast<uint32_t>(group % kGroups); };

  if (tid == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    mbar_init(smem_u32(&q_full), 1);
    for (int i = 0; i < kGroups; ++i) mbar_init(smem_u32(&full_bar[i]), 1), mbar_init(smem_u32(&empty_bar[i]), 1);
    mbar_init(smem_u32(&s_full), 1);
    mbar_init(smem_u32(&s_free), kSoftmaxThreads);
    mbar_init(smem_u32(&p_full), kSoftmaxThreads);
    mbar_init(smem_u32(&o_full), 1);
    mbar_init_fence();
    odd_keys[0] = odd_keys[1] = 0;
  }
  if (warp == 8) tmem_alloc(smem_u32(&tmem_base_s), 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;

  sb::grid_launch_dependents();
  sb::grid_dependency_wait();

  if (warp == 8) {
    if (lane == 0) {
      // ------------------------------------------------ loads
      const int32_t* table = p.block_table + static_cast<int64_t>(slot) * p.max_pages;
      mbar_expect_tx(smem_u32(&q_full), kPieces * ppt * Hg * 128);
      for (int b = 0; b < kPieces; ++b) tma_load_3d(smem0 + b * kQPieceBytes, &map_q, smem_u32(&q_full), 64 * b, g * Hg, row0);
      for (int group = 0; group < 2 * T; ++group) {
        const uint32_t at = group_of(group);
        mbar_wait(smem_u32(&empty_bar[at]), ((group / kGroups) & 1) ^ 1, p.status, 1);
        mbar_expect_tx(smem_u32(&full_bar[at]), kGroupBytes);
        const int b0 = (group & 1) == half ? kHalfPieces : 0;      // (odd groups: the pieces of the own half)
        for (int sub = 0; sub < kKeys / p.box_rows; ++sub) {
          const int key = (kt0 + (group >> 1)) * kKeys + sub * p.box_rows;
          // (keys in front of the first or behind the last that a row sees: a page of the request that is held; nobody uses what comes)
          const int page = table[min(max(key, first_key), last_pos) >> p.page_shift];
          const int row = page * p.rows_per_page + g * p.rows_head + (p.page_size > p.box_rows ? (key & (p.page_size - 1)) : 0);
          for (int b = 0; b < kHalfPieces; ++b)
            tma_load_2d(ring + at * kGroupBytes + b * kPieceBytes + sub * p.box_rows * 128, &map_k, smem_u32(&full_bar[at]), 64 * (b0 + b), row);
        }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    if (lane == 0) {
      // ------------------------------------------------ products
      const uint32_t idesc_qk = instr_desc(kRows, kKeys, false), idesc_pv = instr_desc(kRows, kHalfDim, true);
      const uint64_t dQ = smem_desc_sw128(smem0), dRing = smem_desc_sw128(ring);
      // the 64-element pieces of the value columns lie a piece apart
      const uint64_t dV = dRing | (static_cast<uint64_t>(kPieceBytes >> 4) << 16);
      auto scores = [&](int t, int from, int to) {       // the sums [from, to) of tile t
        for (int b = 0; b < kPieces; ++b) {
          const int group = 2 * t + (b / kHalfPieces == half ? 1 : 0);
          const uint64_t dk = dRing + ((group_of(group) * kGroupBytes + (b % kHalfPieces) * kPieceBytes) >> 4);
          const uint64_t dq = dQ + (static_cast<uint32_t>(b * kQPieceBytes) >> 4);
          for (int c = from; c < to; ++c) umma_bf16(tmem_base + c * kKeys, dq + 2 * c, dk + 2 * c, idesc_qk, b > 0 ? 1u : 0u);
        }
      };
      auto wait_tile = [&](int t) {
        for (int group = 2 * t; group < 2 * t + 2; ++group) mbar_wait(smem_u32(&full_bar[group_of(group)]), (group / kGroups) & 1, p.status, 2);
      };
      auto scores_done = [&](int t) {
        umma_commit(smem_u32(&s_full));
        umma_commit(smem_u32(&empty_bar[group_of(2 * t)]));
      };
      mbar_wait(smem_u32(&q_full), 0, p.status, 3);
      wait_tile(0);
      fence_after_sync();
      scores(0, 0, 4);
      scores_done(0);
      for (int t = 0; t < T; ++t) {
        if (t + 1 < T) {
          wait_tile(t + 1);
          mbar_wait(smem_u32(&s_free), t & 1, p.status, 4);
          fence_after_sync();
          scores(t + 1, 0, 3);
        }
        mbar_wait(smem_u32(&p_full), t & 1, p.status, 5);
        fence_after_sync();
        const uint64_t dv = dV + ((group_of(2 * t + 1) * kGroupBytes) >> 4);
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k) {
          umma_ts_bf16(tmem_base + kTmemO, tmem_base + kTmemP + 8 * k, dv + k * (2048 >> 4), idesc_pv, 1u);
          umma_ts_bf16(tmem_base + kTmemO, tmem_base + kTmemP + 32 + 8 * k, dv + k * (2048 >> 4), idesc_pv, 1u);
        }
        umma_commit(smem_u32(&o_full));
        umma_commit(smem_u32(&empty_bar[group_of(2 * t + 1)]));
        if (t + 1 < T) {
          mbar_wait(smem_u32(&o_full), t & 1, p.status, 6);       // the weights have been read: the fourth sum may take their place
          fence_after_sync();
          scores(t + 1, 3, 4);
          scores_done(t + 1);
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ softmax: thread `part` of a row has keys [32 part, 32 part + 32) of every tile and the
    // columns [128 part, 128 part + 128) of the CTA's half
    const int r = tid & (kRows - 1), part = tid >> 7;
    const int pi = r / Hg;
    const bool valid = pi < npos;
    const int row_pos = valid ? first_pos + pi : -1;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t o_addr = lane_addr + kTmemO + part * 128;
    float m = -INFINITY, l[2][4];         // l: the row's sum in the tile kernel's order: per 16 keys, per pair of keys modulo 8
#pragma unroll
    for (int i = 0; i < 8; ++i) l[i >> 2][i & 3] = 0.0f;
    {
      uint32_t zero[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) zero[i] = 0;
#pragma unroll
      for (int c = 0; c < 128; c += 16) tmem_store16(o_addr + c, zero);
      tmem_store_wait();
    }
    for (int t = 0; t < T; ++t) {
      const int key0 = (kt0 + t) * kKeys;
      const bool edge = key0 + kKeys - 1 > first_pos || (p.window > 0 && key0 <= last_pos - p.window) || npos < ppt;
      float s[32];
      {
        uint32_t a[32], b[32];
        mbar_wait(smem_u32(&s_full), t & 1, p.status, 7);
        fence_after_sync();
        tmem_load32_nowait(lane_addr + part * 32, a);
        tmem_load32_nowait(lane_addr + kKeys + part * 32, b);
        tmem_load_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = __fadd_rn(__uint_as_float(a[j]), __uint_as_float(b[j]));
        tmem_load32_nowait(lane_addr + 2 * kKeys + part * 32, a);
        tmem_load32_nowait(lane_addr + 3 * kKeys + part * 32, b);
        tmem_load_wait();
        fence_before_sync();
        mbar_arrive(smem_u32(&s_free));
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = __fmul_rn(__fadd_rn(s[j], __fadd_rn(__uint_as_float(a[j]), __uint_as_float(b[j]))), p.scale);
      }
      auto seen = [&](int j) { return j <= row_pos && (p.window <= 0 || row_pos - j < p.window); };
      if (edge) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (!seen(key0 + part * 32 + j)) s[j] = -INFINITY;
      }
      float top = s[0];
#pragma unroll
      for (int j = 1; j < 32; ++j) top = fmaxf(top, s[j]);
      xch[part][r] = top;        // (read by all before any thread hands its weights over, written again behind the next tile's scores)
      rows_barrier(warp & 3);
      top = fmaxf(m, fmaxf(top, xch[part ^ 1][r]));
      const float f = top == m ? 1.0f : __expf(m - top);
      m = top;
      uint32_t hi[16], lo[16];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float add = 0.0f;
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            const int j = i * 16 + n * 8 + q * 2;
            const float w0 = s[j] == -INFINITY ? 0.0f : __expf(s[j] - m), w1 = s[j + 1] == -INFINITY ? 0.0f : __expf(s[j + 1] - m);
            add += w0 + w1;
            const __nv_bfloat162 h = __floats2bfloat162_rn(w0, w1);
            const __nv_bfloat162 d = __floats2bfloat162_rn(w0 - __low2float(h), w1 - __high2float(h));
            hi[j >> 1] = *reinterpret_cast<const uint32_t*>(&h);
            lo[j >> 1] = *reinterpret_cast<const uint32_t*>(&d);
          }
          l[i][q] = fmaf(l[i][q], f, add);
        }
      }
      // the value product of the tile before has ended: the accumulator is this thread's, and so are the weights' columns
      if (t > 0) mbar_wait(smem_u32(&o_full), (t - 1) & 1, p.status, 8);
      fence_after_sync();
      if (__any_sync(0xffffffffu, f != 1.0f)) {
#pragma unroll
        for (int c = 0; c < 128; c += 64) {
          uint32_t v[64];
          tmem_load32_nowait(o_addr + c, v);
          tmem_load32_nowait(o_addr + c + 32, v + 32);
          tmem_load_wait();
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
#pragma unroll
          for (int i = 0; i < 64; i += 16) tmem_store16(o_addr + c + i, v + i);
        }
        tmem_store_wait();
      }
      if (edge) {
        mbar_wait(smem_u32(&full_bar[group_of(2 * t + 1)]), ((2 * t + 1) / kGroups) & 1, p.status, 10);       // (long over: the scores needed it)
        uint8_t* values = smem + kPieces * kQPieceBytes + group_of(2 * t + 1) * kGroupBytes;
        auto clear = [&](int j) {          // row j of the value pieces, by the lanes of a warp
          *reinterpret_cast<uint4*>(values + (lane >> 3) * kPieceBytes + j * 128 + (lane & 7) * 16) = make_uint4(0, 0, 0, 0);
        };
        for (int j = warp; j < kKeys; j += 8) {
          const int key = key0 + j;
          if (key > last_pos || key < first_key) {
            clear(j);
          } else if (key > first_pos || (p.window > 0 && key <= last_pos - p.window)) {
            const uint4 v = *reinterpret_cast<const uint4*>(values + (lane >> 3) * kPieceBytes + j * 128 + (lane & 7) * 16);
            if (__any_sync(0xffffffffu, not_finite(v.x) || not_finite(v.y) || not_finite(v.z) || not_finite(v.w)) && lane == 0)
              atomicOr(&odd_keys[j >> 5], 1u << (j & 31));
          }
        }
        softmax_barrier();
        const uint32_t odd[2] = {odd_keys[0], odd_keys[1]};
        if (odd[0] | odd[1]) {
          for (int j = 0; j < kKeys; ++j) {
            if (!((odd[j >> 5] >> (j & 31)) & 1)) continue;
            if (part == j >> 5) {
              float w = 0.0f;
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (i == (j & 31)) w = s[i] == -INFINITY ? 0.0f : __expf(s[i] - m);
              xch[0][r] = w;
            }
            softmax_barrier();
            const float w = xch[0][r];
#pragma unroll 1
            for (int c = 0; c < 128; c += 16) {
              uint32_t v[16];
              tmem_load16_nowait(o_addr + c, v);
              tmem_load_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const int col = part * 128 + c + i, in = col & 63;
                const bf16 x = *reinterpret_cast<const bf16*>(values + (col >> 6) * kPieceBytes + j * 128 + (((in >> 3) ^ (j & 7)) << 4) + (in & 7) * 2);
                if (seen(key0 + j)) v[i] = __float_as_uint(fmaf(w, __bfloat162float(x), __uint_as_float(v[i])));
              }
              tmem_store16(o_addr + c, v);
            }
            tmem_store_wait();
            softmax_barrier();
            if (warp == 0) clear(j);
          }
          softmax_barrier();
          if (tid == 0) odd_keys[0] = odd_keys[1] = 0;
        }
        fence_async_smem();
      }
      tmem_store16(lane_addr + kTmemP + part * 16, hi);
      tmem_store16(lane_addr + kTmemP + 32 + part * 16, lo);
      tmem_store_wait();
      fence_before_sync();
      mbar_arrive(smem_u32(&p_full));
    }
    // the row's sum: pairs, 16 keys by 16 keys; then the sink
    mbar_wait(smem_u32(&o_full), (T - 1) & 1, p.status, 9);
    fence_after_sync();
    rows_barrier(warp & 3);
    const float sum0 = (l[0][0] + l[0][1]) + (l[0][2] + l[0][3]), sum1 = (l[1][0] + l[1][1]) + (l[1][2] + l[1][3]);
    if (part == 0) xch[0][r] = sum0 + sum1;
    rows_barrier(warp & 3);
    if (part == 1) xch[1][r] = (xch[0][r] + sum0) + sum1;
    rows_barrier(warp & 3);
    float total = xch[1][r];
    const int head = g * Hg + r % Hg;
    if (p.sinks != nullptr) total += __expf(p.sinks[head] - m);
    const float inv = 1.0f / total;
    // A row's half is staged in shared memory, over the queries that no product reads any more, and stored by a warp as a line of 512 bytes.
    // (Stored from the thread that has it, 16 bytes a lane to 32 rows, a tile with all rows took 1 us longer: four entries of 16 tokens of 16 heads
    // behind 20 tokens 11.2 us, 10.0 so; the tile kernel 10.4.)
    uint8_t* staged = smem + r * kOutBytes + part * 256;
#pragma unroll
    for (int c = 0; c < 128; c += 32) {
      float v[32];
      tmem_load32(o_addr + c, v);
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(v[i + 2 * k] * inv, v[i + 2 * k + 1] * inv);
          w[k] = *reinterpret_cast<const uint32_t*>(&b);
        }
        *reinterpret_cast<uint4*>(staged + (c + i) * 2) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    rows_barrier(warp & 3);
    const int shift = 31 - __clz(Hg), rows = min(npos * Hg, (warp & 3) * 32 + part * 16 + 16);      // (Hg divides 128)
#pragma unroll 4
    for (int i = (warp & 3) * 32 + part * 16; i < rows; ++i) {
      bf16* dst = p.out + (static_cast<int64_t>(row0 + (i >> shift)) * p.H + g * Hg + (i & (Hg - 1))) * kDim + half * kHalfDim;
      reinterpret_cast<uint4*>(dst)[lane] = reinterpret_cast<const uint4*>(smem + i * kOutBytes)[lane];
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 8) {
    fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace latent5
}  // namespace sb
