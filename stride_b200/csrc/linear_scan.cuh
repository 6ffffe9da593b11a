// The recurrence of linear attention over a state kept per request, with one decay a head (lightning attention, retention) or a gate per
// key channel and token (HGRN2):
//
//   S_t = a_t S_(t-1) + k_t v_t^T        S: [D, V] float32 per head; a_t: a constant of the head, or diag(g_t)
//   o_t = S_t^T q_t
//
// Everything is 32-bit. A column of the state depends on no other column, so the value columns may be spread over CTAs and threads in any
// way. The D sums of an output are cut into 32 parts of DL consecutive elements (DL = 2, 4 or 8 by the key size alone; elements beyond D
// are zero, and a part that lies wholly beyond D adds zeros whatever the values, which may be infinite), each two chains of fused multiply-adds
// (even and odd elements, ascending, then added), and the parts are added as a binary tree of neighbours (part 2i + part 2i + 1, and so on).
// None of it depends on the step, so a token's output has the same bits however the sequence was cut into steps, whichever of the two kernels
// below ran, and whatever else the batch holds.
//
// `scan_kernel` is for steps in which an entry brings several tokens; `step_core` is the work of a token for steps of single tokens.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "step_ops.h"

namespace sbscan {

constexpr int kLanes = 32;       // parts of the D sums
constexpr int kWarps = 4;        // computing warps of scan_kernel
constexpr int kChunk = 16;       // tokens staged in shared memory at a time
constexpr int kMaxStages = 3;    // staging buffers of scan_kernel, at most

inline int lane_elements(int D) { return D <= 64 ? 2 : D <= 128 ? 4 : 8; }

struct Params {
  const float* rows;        // [n][width], float32: the tokens' q, k, v (and gates)
  int width;                // elements of a token's row
  int q_off, k_off, v_off, g_off;
  const int32_t* meta;      // [4][meta_stride]: slot, first row, length, first position of every entry
  int meta_stride;
  const float* decay;       // [H]; unused with gates
  float* state;             // [slots][H][D][V]
  float* out;               // [n][H V]
  int H, D, V;
};

// Asynchronous copies from global to shared memory and the wait for all but the newest N groups of a thread's own.
template <int FLOATS>
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if constexpr (FLOATS == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two float32 operations in one instruction (sm_100): each half rounds as the scalar one does.
__device__ __forceinline__ uint64_t bits2(float2 a) { return *reinterpret_cast<const uint64_t*>(&a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
  return *reinterpret_cast<float2*>(&d);
}

// A token's keys, queries and gates of DL elements, as pairs.
template <int DL, bool GATED>
struct Part {
  float2 k[DL / 2], q[DL / 2], g[GATED ? DL / 2 : 1];
  // GAP: floats from one of the part's pieces of four elements to the next
  template <int GAP>
  static __device__ __forceinline__ void fetch(float2 (&to)[DL / 2], const float* from) {
    if constexpr (DL == 2) {
      to[0] = *reinterpret_cast<const float2*>(from);
    } else {
#pragma unroll
      for (int i = 0; i < DL / 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(from + i * GAP);
        to[2 * i] = make_float2(v.x, v.y);
        to[2 * i + 1] = make_float2(v.z, v.w);
      }
    }
  }
  template <int GAP>
  __device__ __forceinline__ void load(const float* sq, const float* sk, const float* sg) {
    fetch<GAP>(k, sk);
    fetch<GAP>(q, sq);
    if constexpr (GATED) fetch<GAP>(g, sg);
  }
};

// One token for one part of one column: S <- a S + k v; the part's share of the output.
template <int DL, bool GATED>
__device__ __forceinline__ float token(float2 (&S)[DL / 2], const Part<DL, GATED>& x, float v, float decay) {
  const float2 v2 = make_float2(v, v), d2 = make_float2(decay, decay);
  float2 acc;
#pragma unroll
  for (int i = 0; i < DL / 2; ++i) {
    S[i] = fma2(GATED ? x.g[GATED ? i : 0] : d2, S[i], mul2(x.k[i], v2));
    acc = i == 0 ? mul2(S[0], x.q[0]) : fma2(S[i], x.q[i], acc);
  }
  return acc.x + acc.y;
}

template <int N>
__device__ __forceinline__ void put(float2 (&S)[N], int i, float v) {
  if (i & 1) S[i / 2].y = v;
  else S[i / 2].x = v;
}
template <int N>
__device__ __forceinline__ float get(const float2 (&S)[N], int i) { return i & 1 ? S[i / 2].y : S[i / 2].x; }

// Every lane holds its part of 32 sums; lane i returns the whole of sum i: 31 exchanges instead of 32 times 5.
__device__ __forceinline__ float transpose_add(float (&a)[32], int lane) {
#pragma unroll
  for (int m = 1; m < 32; m <<= 1) {
    const bool up = lane & m;
#pragma unroll
    for (int i = 0; i < 32; i += 2 * m) {
      const float give = up ? a[i] : a[i + m], keep = up ? a[i + m] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
    }
  }
  return a[0];
}

// Named barriers of scan_kernel (id 0 is __syncthreads): one per buffer and direction.
enum { kBarFull = 1, kBarEmpty = 1 + kMaxStages };
__device__ __forceinline__ void bar_sync(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int count) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }

// A CTA owns (entry, head, 4 PER value columns) and walks the entry's tokens of this step in order. A computing warp owns PER columns, a
// lane one part of each: a token's keys and queries are read from shared memory once a warp, every lane its own, and serve PER columns. The
// parts of 32 / PER tokens' outputs are added up together by exchanges between lanes, so that no part goes through shared memory. One more
// warp keeps the rows of the next two chunks of tokens on their way into the staging buffers; it announces a chunk before it requests
// another, since a request waits until its buffer is free. What bounds the kernel is each warp's wait for its own reads and exchanges, with one
// or two computing warps a scheduler (PER = 2: issue slots 47% busy; PER = 4: without the loads and the exchanges 155 of 220 us are left).
// Measured (16 heads of 128 x 128 without gates, one entry of 2,048 tokens / eight, launches one behind another): eight warps of one column a
// thread, the outputs' parts through shared memory, 611 / 1,600 us; PER = 4 220 / 710 us, PER = 2 187 / 828 us, and 143 us on its own, which it
// takes in a row too (151) now that it starts behind the kernel in front (launch_scan_of): let in early, its CTAs took their places while that
// one still ran, wherever an SM had room, and some SMs got more of them.
// With eight elements a lane: the row's pieces of four lie the even ones first, then the odd ones, so that the lanes' 16-byte reads take
// neighbouring places (side by side they would meet in half the banks), and with gates two staging buffers, which leaves two CTAs an SM.
template <int DL, bool GATED>
__host__ __device__ constexpr int stages_of() { return DL == 8 && GATED ? 2 : kMaxStages; }
template <int DL>
__device__ __forceinline__ int staged_at(int d) { return DL == 8 ? (d >> 2 & 1) * (kLanes * 4) + (d >> 3) * 4 + (d & 3) : d; }

template <int DL, int PER, bool GATED, int VEC, bool PAD>      // PAD: the key size is less than the lanes' elements
__global__ void __launch_bounds__(kWarps * 32 + 32, DL == 8 ? 2 : DL == 4 && PER == 4 ? 3 : 0) scan_kernel(const Params p) {
  extern __shared__ __align__(16) float smem[];
  sb::grid_launch_dependents();
  constexpr int kStages = stages_of<DL, GATED>(), kGap = DL == 8 ? kLanes * 4 : 4;
  constexpr int kCols = kWarps * PER, kGroup = 32 / PER;       // a group: the tokens whose outputs a warp adds up together
  constexpr int Dp = kLanes * DL, NC = kWarps * 32, NQ = GATED ? 3 : 2, stage = kChunk * (NQ * Dp + kCols);
  const int e = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * kCols, vn = min(kCols, p.V - c0);
  const int slot = p.meta[e], row0 = p.meta[p.meta_stride + e], len = p.meta[2 * p.meta_stride + e], pos0 = p.meta[3 * p.meta_stride + e];
  const int chunks = (len + kChunk - 1) / kChunk;
  // nothing copies into the cells beyond D and beyond the CTA's existing columns: they are zero for good
  if (PAD || vn != kCols) {
    auto clear = [](float* at, int floats) {
      for (int i = threadIdx.x * 4; i < floats; i += (kWarps + 1) * 128) *reinterpret_cast<float4*>(at + i) = make_float4(0, 0, 0, 0);
    };
    for (int b = 0; b < kStages; ++b) {
      const int rows = min(kChunk, len - b * kChunk);            // that tokens will use
      if (rows <= 0) break;
      for (int k = 0; k < NQ; ++k) clear(smem + b * stage + k * kChunk * Dp, rows * Dp);
      clear(smem + b * stage + NQ * kChunk * Dp, rows * kCols);
    }
  }
  sb::grid_dependency_wait();
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < kWarps) {
    // ---------------------------------------------------------------- the recurrence
    const float decay = GATED ? 0.0f : p.decay[h];
    const int cl = warp * PER, dn = PAD ? min(DL, p.D - lane * DL) : DL;
    float* st = p.state + ((static_cast<int64_t>(slot) * p.H + h) * p.D + lane * DL) * p.V + c0 + cl;
    float2 S[PER][DL / 2];
    using Columns = typename std::conditional<PER == 4, float4, float2>::type;      // (VEC == 4: a warp's columns all exist, or none)
#pragma unroll
    for (int i = 0; i < DL; ++i) {
      alignas(16) float row[PER];
#pragma unroll
      for (int c = 0; c < PER; ++c) row[c] = 0.0f;
      if constexpr (VEC == 4) {
        if (pos0 > 0 && cl < vn && i < dn) *reinterpret_cast<Columns*>(row) = *reinterpret_cast<const Columns*>(st + static_cast<int64_t>(i) * p.V);
      } else {
#pragma unroll
        for (int c = 0; c < PER; ++c)
          if (pos0 > 0 && cl + c < vn && i < dn) row[c] = st[static_cast<int64_t>(i) * p.V + c];
      }
#pragma unroll
      for (int c = 0; c < PER; ++c) put(S[c], i, row[c]);
    }
    float* out = p.out + static_cast<int64_t>(row0) * p.H * p.V + h * p.V + c0 + cl + (lane & (PER - 1));
    const bool live = cl + (lane & (PER - 1)) < vn;
    for (int c = 0, b = 0; c < chunks; ++c, b = b + 1 == kStages ? 0 : b + 1) {
      const float* sq = smem + b * stage + lane * min(DL, 4);
      const float* sv = smem + b * stage + NQ * kChunk * Dp + cl;
      bar_sync(kBarFull + b, NC + 32);
#pragma unroll 1
      for (int t0 = 0; t0 < kChunk; t0 += kGroup) {
        const int nt = min(kGroup, len - c * kChunk - t0);
        if (nt <= 0) break;
        float sums[32];
        // the next token's operands are on their way while a token is computed; a whole group runs without a test between its tokens, which
        // would keep one token's operations from filling another's waits (320 us in place of 220)
        auto walk = [&](auto whole) {
          Part<DL, GATED> x[2];
          float v[2][PER];
          auto load = [&](int t, int at) {
            const float* row = sq + (t0 + t) * Dp;
            x[at].template load<kGap>(row, row + kChunk * Dp, row + (GATED ? 2 : 0) * kChunk * Dp);
            const float* from = sv + (t0 + t) * kCols;
            if constexpr (PER == 4) {
              const float4 w = *reinterpret_cast<const float4*>(from);
              v[at][0] = w.x, v[at][1] = w.y, v[at][2] = w.z, v[at][3] = w.w;
            } else {
              const float2 w = *reinterpret_cast<const float2*>(from);
              v[at][0] = w.x, v[at][1] = w.y;
            }
          };
          load(0, 0);
#pragma unroll
          for (int t = 0; t < kGroup; ++t) {
            if (t + 1 < kGroup) load(t + 1, (t + 1) & 1);        // (a row beyond the chunk's tokens holds old values, which nothing uses)
            if (decltype(whole)::value || t < nt) {
#pragma unroll
              for (int j = 0; j < PER; ++j) sums[t * PER + j] = token<DL, GATED>(S[j], x[t & 1], v[t & 1][j], decay);
            } else {
#pragma unroll
              for (int j = 0; j < PER; ++j) sums[t * PER + j] = 0.0f;
            }
          }
        };
        if (nt == kGroup) walk(std::true_type{});
        else walk(std::false_type{});
        if (t0 + kGroup >= min(kChunk, len - c * kChunk) && c + kStages < chunks) bar_arrive(kBarEmpty + b, NC + 32);
        if (PAD && dn <= 0) {      // a part beyond D: zeros, whatever 0 times an infinite value is
#pragma unroll
          for (int i = 0; i < 32; ++i) sums[i] = 0.0f;
        }
        const float sum = transpose_add(sums, lane);
        const int t = lane / PER;
        if (live && t < nt) out[static_cast<int64_t>(c * kChunk + t0 + t) * p.H * p.V] = sum;
      }
    }
#pragma unroll
    for (int i = 0; i < DL; ++i) {
      alignas(16) float row[PER];
#pragma unroll
      for (int c = 0; c < PER; ++c) row[c] = get(S[c], i);
      if constexpr (VEC == 4) {
        if (cl < vn && i < dn) *reinterpret_cast<Columns*>(st + static_cast<int64_t>(i) * p.V) = *reinterpret_cast<const Columns*>(row);
      } else {
#pragma unroll
        for (int c = 0; c < PER; ++c)
          if (cl + c < vn && i < dn) st[static_cast<int64_t>(i) * p.V + c] = row[c];
      }
    }
  } else {
    // ---------------------------------------------------------------- the loads
    const int du = p.D / VEC, vu = vn / VEC;      // (VEC == 4 only when every size and offset is a multiple of four)
    const float* src0 = p.rows + static_cast<int64_t>(row0) * p.width;
    auto request = [&](int c, int b) {
      const int nt = min(kChunk, len - c * kChunk);
      float* to = smem + b * stage;
      const float* from = src0 + static_cast<int64_t>(c) * kChunk * p.width;
      for (int u = lane; u < du; u += 32) {
        const float* src = from + h * p.D + u * VEC;
        float* dst = to + staged_at<DL>(u * VEC);
#pragma unroll 4
        for (int t = 0; t < nt; ++t, src += p.width, dst += Dp) {
          copy_async<VEC>(dst, src + p.q_off);
          copy_async<VEC>(dst + kChunk * Dp, src + p.k_off);
          if constexpr (GATED) copy_async<VEC>(dst + 2 * kChunk * Dp, src + p.g_off);
        }
      }
      constexpr int kPieces = kCols / VEC;
      for (int i = lane; i < nt * kPieces; i += 32) {
        const int t = i / kPieces, u = i % kPieces;
        if (u < vu)
          copy_async<VEC>(to + NQ * kChunk * Dp + t * kCols + u * VEC, from + static_cast<int64_t>(t) * p.width + p.v_off + h * p.V + c0 + u * VEC);
      }
      copy_async_commit();
    };
    constexpr int ahead = kStages - 1;
    for (int c = 0; c < ahead && c < chunks; ++c) request(c, c);
    for (int c = 0, b = 0; c < chunks; ++c, b = b + 1 == kStages ? 0 : b + 1) {
      if (c + 1 < chunks) copy_async_wait<ahead - 1>();
      else copy_async_wait<0>();
      bar_arrive(kBarFull + b, NC + 32);
      if (c + ahead < chunks) {
        const int rb = b == 0 ? kStages - 1 : b - 1;
        if (c + ahead >= kStages) bar_sync(kBarEmpty + rb, NC + 32);
        request(c + ahead, rb);
      }
    }
  }
}

// Whether a launch with two columns a warp begins behind the kernel in front instead of early: one or two long CTAs an SM have to be dealt out
// evenly, which CTAs that are let in beside a running kernel are not, and a CTA that begins late lacks 0.4 to 0.9 us. `tokens`: an entry's, on
// average. In a row with the kernels in front and behind, us, early / behind (906 points of 26 shapes of heads). More CTAs than half the SMs, keys
// of 65 to 128: 16 heads of 128 x 128 (256 CTAs) 2 tokens 8.5 / 8.2, 64 tokens 14.3 / 12.6, 2,048 tokens 204 / 153, with gates 8.7 / 7.7, 14.8 /
// 12.6, 236 / 164; 80 CTAs 4 tokens 6.3 / 6.7, 16 tokens 6.6 / 6.6, 256 tokens 28 / 19, with gates 6.4 / 6.1, 6.9 / 6.1, 33 / 19. Keys up to 64: 32
// heads of 64 x 64 4 tokens 6.7 / 7.0, 16 tokens 7.0 / 7.0, 64 tokens 12.2 / 9.9; 256 CTAs of 32 x 32 32 tokens 8.1 / 8.5, 64 tokens 11.8 / 10.7. Keys beyond
// 128, which leave an SM one CTA: 128 CTAs 2 tokens 9.4 / 7.9, 128 tokens 28.6 / 19.5 (with gates 8 tokens 8.6 / 8.9), more CTAs than SMs 2 tokens
// 8.8 / 9.6, 128 tokens 29.0 / 30.5. Up to half the SMs: 64 CTAs of 128 x 128 64 tokens 8.8 / 9.2, 128 tokens 13.9 / 12.2, with gates 16 tokens 6.3 / 6.2, 64
// tokens 9.4 / 8.8; 32 CTAs 128 tokens 10.6 / 12.0, 256 tokens 22 / 18; 16 CTAs 256 tokens 16.5 / 17.3, 512 tokens 34 / 28.
template <int DL, bool GATED>
bool starts_behind(int64_t ctas, int D, int64_t tokens) {
  const int64_t sms = sb::sm_count();
  if (DL == 8) return ctas <= sms;
  if (2 * ctas <= sms) return tokens >= (8 * ctas <= sms ? 512 : 4 * ctas <= sms ? 256 : DL == 4 && GATED ? 32 : 128);
  if (DL == 4) return GATED || 4 * ctas > 3 * sms || tokens >= 16;
  return tokens >= (D > 32 ? 16 : 64);
}

template <int DL, int PER, bool GATED>
int launch_scan_of(const Params& p, int entries, int n, const char* who, cudaStream_t stream) {
  constexpr int kCols = kWarps * PER;
  constexpr size_t smem = sizeof(float) * stages_of<DL, GATED>() * kChunk * ((GATED ? 3 : 2) * kLanes * DL + kCols);
  static_assert(smem <= 200 * 1024, "staging buffers");
  const bool vec = p.D % 4 == 0 && p.V % 4 == 0 && p.width % 4 == 0 && p.q_off % 4 == 0 && p.k_off % 4 == 0 && p.v_off % 4 == 0 &&
                   (!GATED || p.g_off % 4 == 0) &&
                   ((reinterpret_cast<uintptr_t>(p.rows) | reinterpret_cast<uintptr_t>(p.state)) & 15) == 0;
  // (without gates and with two columns a warp the form that looks at the lanes' sizes is the faster one also where they are full: one entry of
  // 2,048 tokens, 16 heads of 128 x 128, 154 us and 178)
  const bool pad = p.D != kLanes * DL || (!GATED && DL == 4 && PER == 2);
  const auto kernel = !vec ? scan_kernel<DL, PER, GATED, 1, true> : pad ? scan_kernel<DL, PER, GATED, 4, true> : scan_kernel<DL, PER, GATED, 4, false>;
  static sb::DeviceOnce once;
  if (once.needed()) {
    for (const auto k : {scan_kernel<DL, PER, GATED, 1, true>, scan_kernel<DL, PER, GATED, 4, true>, scan_kernel<DL, PER, GATED, 4, false>})
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    once.done();
  }
  const dim3 grid(entries, p.H, (p.V + kCols - 1) / kCols), block(kWarps * 32 + 32);
  // (four columns a warp: entries enough to fill the SMs either way; 16 entries of 64 tokens 59 us early, 61 behind)
  if (PER == 2 && starts_behind<DL, GATED>(static_cast<int64_t>(grid.x) * grid.y * grid.z, p.D, n / entries)) sb::launch_behind(kernel, grid, block, smem, stream, p);
  else sb::launch_pdl(kernel, grid, block, smem, stream, p);
  return sb::check_launch(who);
}

// Launches scan_kernel for the key size (at most 256). Four columns a warp make fewer reads a column; two make twice the CTAs, which is the
// faster way for long entries while they all run at once (16 heads of 128 x 128 in a row with the kernels around them, 1,024 tokens: 85 against
// 131 us for 128 CTAs of four, 16 tokens 8.8 against 8.5; alone, eight entries of 2,048 tokens, 828 against 710 us for 1,024).
template <bool GATED>
int launch_scan(const Params& p, int entries, int n, const char* who, cudaStream_t stream) {
  const bool few = static_cast<int64_t>(entries) * p.H * ((p.V + 15) / 16) <= sb::sm_count();
#define SB_SCAN_OF(DL) (few ? launch_scan_of<DL, 2, GATED>(p, entries, n, who, stream) : launch_scan_of<DL, 4, GATED>(p, entries, n, who, stream))
  switch (lane_elements(p.D)) {
    case 2: return SB_SCAN_OF(2);
    case 4: return SB_SCAN_OF(4);
    default: return SB_SCAN_OF(8);
  }
#undef SB_SCAN_OF
}

// Steps with as many tokens as entries: a CTA is (entry, head, 32 value columns), a thread kRows elements of one column (what a warp reads of
// the state is whole 128-byte rows). The state's loads are requested first; `fill(smem, Ds, row)` writes the token's q, k, (g,) v into shared
// memory meanwhile: q, k, g [Ds] each (D in whole warps), zero beyond D, v [32]. The same operations in the same order as scan_kernel: a
// thread adds its own neighbouring parts, the warps' sums are the upper levels of the tree, in which the parts beyond the last warp's are zeros.
constexpr int kRows = 16;
template <int DL, bool GATED, class Fill>
__device__ __forceinline__ void step_token(const Params& p, float* smem, int slot, int row, int pos, int V, Fill fill) {
  constexpr int kParts = kRows / DL, warps = kLanes * DL / kRows;
  const int h = blockIdx.y, c0 = blockIdx.z * 32, warp = threadIdx.x >> 5, cl = threadIdx.x & 31, Ds = blockDim.x / 32 * kRows;
  float* sv = smem + (GATED ? 3 : 2) * Ds;
  float* so = sv + 32;         // [warps][32]
  const bool live = c0 + cl < V;
  const int d0 = warp * kRows, dn = min(kRows, p.D - d0);
  const float decay = GATED ? 0.0f : p.decay[h];
  float* st = p.state + ((static_cast<int64_t>(slot) * p.H + h) * p.D + d0) * V + c0 + cl;
  float2 S[kParts][DL / 2];
#pragma unroll
  for (int i = 0; i < kRows; ++i) put(S[i / DL], i % DL, pos > 0 && live && i < dn ? st[static_cast<int64_t>(i) * V] : 0.0f);
  fill(smem, Ds, row);
  __syncthreads();
  float a[kParts];
#pragma unroll
  for (int j = 0; j < kParts; ++j) {
    const float* sq = smem + d0 + j * DL;
    Part<DL, GATED> x;
    x.template load<4>(sq, sq + Ds, sq + (GATED ? 2 : 0) * Ds);
    a[j] = token<DL, GATED>(S[j], x, j * DL < dn ? sv[cl] : 0.0f, decay);
  }
#pragma unroll
  for (int m = 1; m < kParts; m <<= 1)
#pragma unroll
    for (int j = 0; j < kParts; j += 2 * m) a[j] = a[j] + a[j + m];
  so[warp * 32 + cl] = a[0];
  if (live) {
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      if (i < dn) st[static_cast<int64_t>(i) * V] = get(S[i / DL], i % DL);
  }
  __syncthreads();
  if (warp == 0 && live) {
    float w[warps];
#pragma unroll
    for (int q = 0; q < warps; ++q) w[q] = q * 32 < blockDim.x ? so[q * 32 + cl] : 0.0f;
#pragma unroll
    for (int m = 1; m < warps; m <<= 1)
#pragma unroll
      for (int q = 0; q < warps; q += 2 * m) w[q] = w[q] + w[q + m];
    p.out[static_cast<int64_t>(row) * p.H * V + h * V + c0 + cl] = w[0];
  }
}
template <int DL, bool GATED, class Fill>
__device__ __forceinline__ void step_core(const Params& p, float* smem, int slot, int row0, int len, int pos0, Fill fill) {
  if (len == 1) {
    step_token<DL, GATED>(p, smem, slot, row0, pos0, p.V, fill);
    return;
  }
  // no token, or several: one after the other, the state through memory (a thread reads what it wrote; the token in front has been read when
  // every warp has passed the second barrier)
#pragma unroll 1
  for (int t = 0; t < len; ++t) {
    int V = p.V;
    asm volatile("" : "+r"(V));      // (sixteen addresses kept from one token to the next would cost the usual case its registers)
    step_token<DL, GATED>(p, smem, slot, row0 + t, pos0 + t, V, fill);
  }
}

inline int step_threads(int D) { return (D + kRows - 1) / kRows * 32; }
inline size_t step_smem(int D, bool gated) { return sizeof(float) * ((gated ? 3 : 2) * (step_threads(D) / 32 * kRows) + 32 + step_threads(D)); }

}  // namespace sbscan
