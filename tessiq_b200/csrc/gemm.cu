// GEMM + bias + activation on the 5th-generation tensor cores (tcgen05), for sm_100a.
//
//   C[b] = act(op(A[b]) @ op(B[b]) + bias)      bf16 or f16 operands, f32 accumulation, one rounding
//
// Two kernels share the work by shape (choose_tiling): CTA pairs over 256 x 256, 256 x 192 or 256 x 128 tiles
// (below), and single CTAs over 128 x 128 tiles, several of which may share a tile's K range, or 128 x 256 ones. In both,
// persistent CTAs walk the tiles and ten warps of a CTA have three jobs:
//
//   warp 0, one lane   producer: TMA loads (cp.async.bulk.tensor, 128-byte swizzle) of a 64-wide slice
//                      of A and of B into a ring of stages in shared memory, each stage announced on an
//                      mbarrier by its byte count;
//   warp 1, one lane   issuer: for every stage four tcgen05.mma (16 elements of K each) accumulating in
//                      tensor memory; tcgen05.commit hands the stage back to the producer and, after
//                      the last slice of a tile, hands the accumulator to the epilogue;
//   warps 2..9         epilogue: tcgen05.ld of the f32 accumulator (each warp 32 lanes of tensor
//                      memory by every other 64 columns), + bias, activation in f32, one rounding, a
//                      regrouping through shared memory, whole-line 128-bit stores.
//
// The lanes that issue are chosen by elect.sync: with `lane == 0` in its place a k-block cost at least 560
// cycles whatever the tile's width (8192 x 4096 x 4096, 128 columns a pair: 269 us against 182; 192: 209 / 174),
// which a 256-wide tile hides and a narrow one does not.
//
// A product with few rows is a stream of B. 64 x 4096 x 4096 took 35.2 us as 16 tiles of 256 columns on 16 SMs
// and takes 14.2 as 32 tiles of 128 columns with four CTAs of a cluster on each, which add their partial
// sums through distributed shared memory (kernel times after an L2 flush; in a graph of such launches 12.5. Its bytes: 5.4; the
// launch, the first loads and the two cluster barriers are the rest: 768 x 768 with one row takes 6.3).
//
// Tensor memory holds two f32 accumulators, so the epilogue of tile i
// runs under the MMAs of tile i+1. Either operand may be K-major (row-major A, nn.Linear weight
// [n,k]) or MN-major (A stored [k,m]; B stored [k,n], the `A @ B` form): transposed operands are
// consumed in place through the shared-memory descriptor's major bit, never copied
// (csrc/tessiq/codegen/gemm.cpp:28-53 in the reference does the same through cuBLAS flags).
// No load uses cluster multicast. Every wait is bounded: a wait that gives up sets the device
// status word (see tq_status_poll) and the CTA leaves through the normal teardown, freeing its
// tensor memory.
//
// Replaces launch_gemm + the bias pre-fill (csrc/tessiq/codegen/blas.cpp:92-193,
// csrc/tessiq/codegen/gemm.cpp:186-199) and the custom ops gemm_bias_gelu_tanh
// (csrc/custom_ops/gemm_bias_gelu_tanh/gemm_bias_gelu_tanh.nvcc.cu:219-288) and gemm_bias_gelu
// (csrc/custom_ops/gemm_bias_gelu/gemm_bias_gelu.nvcc.cu:90-158).
#include <cuda.h>

#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.h"
#include "tcgen05.h"

namespace tq {
namespace {

constexpr int kTileM = 128;
constexpr int kSplitTileN = 128;   // of tiles whose K range a cluster shares; otherwise widths are template parameters
constexpr int kTileK = 64;    // 64 two-byte elements = one 128-byte swizzle row
constexpr int kMmaK = 16;
constexpr int kThreads = 320;           // producer warp, issuer warp, eight epilogue warps
constexpr int kEpilogueThreads = 256;
constexpr int kEpilogueWarps = kEpilogueThreads / 32;
constexpr int kStoreColumns = 64;       // columns an epilogue warp regroups at a time
constexpr uint32_t kStoreBytes = 32 * kStoreColumns * 2;   // 4 KiB of staging per epilogue warp
constexpr uint32_t kBytesA = kTileM * kTileK * 2;   // 16 KiB
constexpr uint32_t kChunkBytes = 64 * kTileK * 2;   // one 64-wide MN chunk of an MN-major operand: 8 KiB
constexpr int kMaxSplit = 8;                        // CTAs of a cluster that share one tile's K range

enum WaitCode { kWaitEmpty = 101, kWaitFull = 102, kWaitTmemEmpty = 103, kWaitTmemFull = 104 };

struct GemmParams {
  int m, n, k, batch;
  int tiles_m, tiles_n;
  int split;                       // CTAs of a cluster that share a tile's K range (single-CTA kernel)
  int a_rows;                      // rows of A a stage loads (single-CTA kernel): fewer than a tile has where m is smaller
  long long num_tiles;
  const void* bias;
  const void* residual;            // added after the activation, or null
  long long ldr, stride_r;
  void* c;
  long long ldc, stride_c;
  int activation;
  WaitStatus status;
};

// Instruction descriptor of tcgen05.mma kind::f16: f32 accumulator, A/B format (0 f16, 1 bf16),
// major bits (0 K-major, 1 MN-major), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t instruction_descriptor(bool bf16, bool a_mn_major, bool b_mn_major, int m, int n) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// A barrier of the eight epilogue warps (named barrier 1) that also returns whether `ok` held on every
// one of its threads, so that a bounded wait that gave up on one warp takes all of them out at once.
__device__ __forceinline__ bool epilogue_all(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred mine, every;\n\t"
      "setp.ne.b32 mine, %1, 0;\n\t"
      "bar.red.and.pred every, 1, %2, mine;\n\t"
      "selp.u32 %0, 1, 0, every;\n\t}"
      : "=r"(all)
      : "r"(static_cast<uint32_t>(ok)), "n"(kEpilogueThreads)
      : "memory");
  return all != 0;
}

// The activation of two elements at once with the .f32x2 forms of add, mul and fma, and with the
// activation a compile-time constant: the epilogue of a short-K product (12 k-blocks at K = 768) is
// what the CTA waits for, and it is bound by the instructions its eight warps issue.
template <int ACTIVATION>
__device__ __forceinline__ float2 activate_pair(float2 v) {
  if constexpr (ACTIVATION == TQ_ACT_GELU_TANH) {
    // v / (1 + exp2(v (c0 + c1 v^2))), c0 = -2 k log2(e) = -2.3022082, c1 = 0.044715 c0
    const float2 square = __fmul2_rn(v, v);
    const float2 inner = __ffma2_rn(square, make_float2(-0.10294324f, -0.10294324f), make_float2(-2.302208198144325f, -2.302208198144325f));
    const float2 t = __fmul2_rn(v, inner);
    const float2 denominator = __fadd2_rn(make_float2(exp2_ftz(t.x), exp2_ftz(t.y)), make_float2(1.0f, 1.0f));
    return __fmul2_rn(v, make_float2(rcp_ftz(denominator.x), rcp_ftz(denominator.y)));
  } else if constexpr (ACTIVATION == TQ_ACT_GELU_ERF) {
    // 0.5 v (1 + erf(v / sqrt 2)) = v Phi(v), Phi(v) = 1 - h for v >= 0 and h for v < 0, where
    // h = 0.5 erfc(|v| / sqrt 2) and erfc(z) = exp(-z^2) P(t), t = 1 / (1 + 0.3275911 z), P a polynomial
    // of degree 8 without a constant term fitted to erfc(z) exp(z^2) over 0 <= z <= 10 with a RELATIVE
    // error of 4e-7, so the negative tail keeps its digits (erff's branches cost 25 instructions per
    // element, this is 12). |v| is clamped at 14.2, where erfc has left the f32 range. As with the
    // erff form: +inf gives +inf, -inf gives NaN (inf * 0), NaN stays NaN, -0 stays -0.
    float2 a;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(a.x) : "f"(fabsf(v.x)), "f"(14.2f));
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(a.y) : "f"(fabsf(v.y)), "f"(14.2f));
    auto both = [](float c) { return make_float2(c, c); };
    const float2 denominator = __ffma2_rn(a, both(0.3275911f * 0.70710678118654752440f), both(1.0f));
    const float2 t = make_float2(rcp_ftz(denominator.x), rcp_ftz(denominator.y));
    const float2 exponent = __ffma2_rn(__fmul2_rn(a, a), both(-0.72134752044448170368f), both(-1.0f));   // log2(0.5 exp(-z^2)), z^2 = a^2 / 2
    const float2 decay = make_float2(exp2_ftz(exponent.x), exp2_ftz(exponent.y));
    float2 poly = __ffma2_rn(both(-0.140646293759346f), t, both(0.49450618028640747f));
    poly = __ffma2_rn(poly, t, both(-0.4017721116542816f));
    poly = __ffma2_rn(poly, t, both(0.4490189850330353f));
    poly = __ffma2_rn(poly, t, both(0.02793201059103012f));
    poly = __ffma2_rn(poly, t, both(0.2050340622663498f));
    poly = __ffma2_rn(poly, t, both(0.18088608980178833f));
    poly = __ffma2_rn(poly, t, both(0.18504123389720917f));
    const float2 h = __fmul2_rn(__fmul2_rn(poly, t), decay);
    const float2 upper = __ffma2_rn(h, both(-1.0f), both(1.0f));
    return __fmul2_rn(v, make_float2(v.x >= 0.0f ? upper.x : h.x, v.y >= 0.0f ? upper.y : h.y));
  } else {
    return v;
  }
}

// Eight consecutive columns of one row: accumulators + bias, activation, residual, one rounding.
template <typename T, int ACTIVATION, bool RESIDUAL>
__device__ __forceinline__ uint4 finish_unit(const uint32_t (&r0)[32], const uint32_t (&r1)[32], const float* bias, int unit, const uint4& residual) {
  Vec<T, 8> out;
  const Vec<T, 8> add = *reinterpret_cast<const Vec<T, 8>*>(&residual);
  const float4 bias_low = *reinterpret_cast<const float4*>(bias + unit * 8), bias_high = *reinterpret_cast<const float4*>(bias + unit * 8 + 4);
  const float bias_of[8] = {bias_low.x, bias_low.y, bias_low.z, bias_low.w, bias_high.x, bias_high.y, bias_high.z, bias_high.w};
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const int j = unit * 8 + e;
    const float2 accumulator = make_float2(__uint_as_float(j < 32 ? r0[j] : r1[j - 32]), __uint_as_float(j < 32 ? r0[j + 1] : r1[j - 31]));
    float2 value = activate_pair<ACTIVATION>(__fadd2_rn(accumulator, make_float2(bias_of[e], bias_of[e + 1])));
    if constexpr (RESIDUAL) value = __fadd2_rn(value, make_float2(to_compute(add.v[e]), to_compute(add.v[e + 1])));
    out.v[e] = from_compute<T, float>(value.x);
    out.v[e + 1] = from_compute<T, float>(value.y);
  }
  return *reinterpret_cast<const uint4*>(&out);
}

// Calls `finish` with the activation and the presence of a residual as compile-time constants.
template <typename F>
__device__ __forceinline__ void with_activation(int activation, bool residual, F finish) {
  auto go = [&](auto activation_tag) {
    if (residual) {
      finish(activation_tag, std::true_type{});
    } else {
      finish(activation_tag, std::false_type{});
    }
  };
  if (activation == TQ_ACT_GELU_TANH) {
    go(std::integral_constant<int, TQ_ACT_GELU_TANH>{});
  } else if (activation == TQ_ACT_GELU_ERF) {
    go(std::integral_constant<int, TQ_ACT_GELU_ERF>{});
  } else {
    go(std::integral_constant<int, TQ_ACT_NONE>{});
  }
}

// Tiles in groups of 16 rows of tiles, so that the CTAs running at one time share A and B slices
// in L2.
__device__ __forceinline__ void tile_coordinates(long long tile, const GemmParams& p, int& batch, int& tile_m, int& tile_n) {
  const long long per_batch = static_cast<long long>(p.tiles_m) * p.tiles_n;
  batch = static_cast<int>(tile / per_batch);
  const int t = static_cast<int>(tile % per_batch);
  constexpr int kGroup = 16;
  const int group_span = kGroup * p.tiles_n;
  const int group = t / group_span;
  const int first_m = group * kGroup;
  const int rows = min(kGroup, p.tiles_m - first_m);
  tile_m = first_m + (t % group_span) % rows;
  tile_n = (t % group_span) / rows;
}

// An element of an epilogue warp's staging block (rows of 64 elements, 16-byte units XOR-swizzled by row).
__device__ __forceinline__ uint16_t staged_element(uint32_t staging, int row, int column) {
  uint16_t value;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(value) : "r"(staging + row * 128 + (((column >> 3) ^ (row & 7)) << 4) + (column & 7) * 2) : "memory");
  return value;
}

// One epilogue warp's share of a 128 x TILE_N accumulator: the 32 rows of its tensor-memory lanes by
// every other block of 64 columns, beginning with block `half` (of 192 columns one half gets two blocks
// and the other one; the caller swaps the halves from tile to tile). Per block: tcgen05.ld (lane i holds
// row i), + bias, activation, one rounding, then the 32 x 64 block goes through 4 KiB of this warp's
// shared memory (16-byte units XOR-swizzled by row, conflict-free both ways) so that each store
// instruction writes four whole 128-byte lines of C instead of 32 scattered 16-byte pieces. A residual
// tile (added after the activation, before the one rounding) takes the same road the other way: whole
// lines from global memory into the staging block, then each thread picks up its own row. Where C's rows
// are not made of aligned 16-byte pieces (an odd n) the staged block is written an element a lane, half a row
// per instruction, in place of one element of each of 32 rows. (Four-byte pieces from each row's first
// aligned address were slower: 8192 x 9973 x 768 276 us against 231.)
template <typename T, int TILE_N>
__device__ __forceinline__ void epilogue_rows(uint32_t tmem_accumulator, int quarter, int half, int lane, const float* bias_tile,
                                              T* c_tile, long long ldc, const T* residual_tile, long long ldr, int rows_left,
                                              int columns_left, int activation, unsigned char* staging, bool vector_ok) {
  const uint32_t staging_address = smem_address(staging);
  if (quarter * 32 >= rows_left) return;       // C has none of this warp's rows
#pragma unroll 1
  for (int block = half; block < TILE_N / kStoreColumns; block += 2) {
    const int column0 = block * kStoreColumns;
    uint4 residual_words[8];
    if (residual_tile != nullptr && vector_ok) {      // issued before the tensor-memory load so the two latencies overlap
      const int unit = lane & 7;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = quarter * 32 + i * 4 + (lane >> 3);
        residual_words[i] = make_uint4(0, 0, 0, 0);
        if (r < rows_left && column0 + unit * 8 < columns_left) {
          residual_words[i] = __ldg(reinterpret_cast<const uint4*>(residual_tile + static_cast<long long>(r) * ldr + column0 + unit * 8));
        }
      }
    }
    uint32_t r0[32], r1[32];
    tmem_load_32(tmem_accumulator + column0 + (static_cast<uint32_t>(quarter * 32) << 16), r0);
    tmem_load_32(tmem_accumulator + column0 + 32 + (static_cast<uint32_t>(quarter * 32) << 16), r1);
    tmem_load_wait();
    if (residual_tile != nullptr) {
      if (vector_ok) {
        const int unit = lane & 7;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(staging_address + r * 128 + ((unit ^ (r & 7)) << 4)),
                       "r"(residual_words[i].x), "r"(residual_words[i].y), "r"(residual_words[i].z), "r"(residual_words[i].w)
                       : "memory");
        }
      } else {
        const int rows = min(32, rows_left - quarter * 32);
#pragma unroll 4
        for (int r = 0; r < rows; ++r) {
          const T* residual_row = residual_tile + static_cast<long long>(quarter * 32 + r) * ldr + column0;
          for (int j = lane; j < kStoreColumns && column0 + j < columns_left; j += 32) {
            *reinterpret_cast<T*>(staging + r * 128 + (((j >> 3) ^ (r & 7)) << 4) + (j & 7) * 2) = residual_row[j];
          }
        }
      }
      __syncwarp();
    }
    // (the eight units are worked out side by side and stored afterwards: a store between them would order
    // each unit's bias reads behind the one before, and the chain of a unit is what a warp waits for)
    auto finish = [&](auto activation_tag, auto residual_tag) {
      constexpr int kActivation = decltype(activation_tag)::value;
      constexpr bool kResidual = decltype(residual_tag)::value;
      uint4 words[8];
#pragma unroll
      for (int unit = 0; unit < 8; ++unit) {
        words[unit] = make_uint4(0, 0, 0, 0);
        if constexpr (kResidual) {
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(words[unit].x), "=r"(words[unit].y), "=r"(words[unit].z), "=r"(words[unit].w)
                       : "r"(staging_address + lane * 128 + ((unit ^ (lane & 7)) << 4))
                       : "memory");
        }
      }
#pragma unroll
      for (int unit = 0; unit < 8; ++unit) words[unit] = finish_unit<T, kActivation, kResidual>(r0, r1, bias_tile + column0, unit, words[unit]);
#pragma unroll
      for (int unit = 0; unit < 8; ++unit) {
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(staging_address + lane * 128 + ((unit ^ (lane & 7)) << 4)),
                     "r"(words[unit].x), "r"(words[unit].y), "r"(words[unit].z), "r"(words[unit].w)
                     : "memory");
      }
    };
    with_activation(activation, residual_tile != nullptr, finish);
    __syncwarp();
    if (vector_ok) {
      const int unit = lane & 7;
      if (column0 + unit * 8 < columns_left) {
        uint4 words[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(words[i].x), "=r"(words[i].y), "=r"(words[i].z), "=r"(words[i].w)
                       : "r"(staging_address + r * 128 + ((unit ^ (r & 7)) << 4))
                       : "memory");
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          if (quarter * 32 + r < rows_left) {
            *reinterpret_cast<uint4*>(c_tile + static_cast<long long>(quarter * 32 + r) * ldc + column0 + unit * 8) = words[i];
          }
        }
      }
    } else {
      const int rows = min(32, rows_left - quarter * 32), columns = columns_left - column0;
#pragma unroll 1
      for (int r0 = 0; r0 < rows; r0 += 8) {
        uint16_t low[8], high[8];      // all eight rows are read before the first is written: the compiler must not order one by one
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          low[i] = staged_element(staging_address, r0 + i, lane);
          high[i] = staged_element(staging_address, r0 + i, lane + 32);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint16_t* c_row = reinterpret_cast<uint16_t*>(c_tile + static_cast<long long>(quarter * 32 + r0 + i) * ldc + column0);
          if (r0 + i < rows && lane < columns) c_row[lane] = low[i];
          if (r0 + i < rows && lane + 32 < columns) c_row[lane + 32] = high[i];
        }
      }
    }
    __syncwarp();
  }
}

// The end of a tile whose K range was shared by the CTAs of a cluster: every CTA sends each other one its
// share of the columns as f32 partial sums, through distributed shared memory into the (now idle) stage
// ring, 16-byte units in the order [sender][column / 4][row] so that a warp's store is one 512-byte run.
__device__ __forceinline__ void push_partials(uint32_t tmem_accumulator, int quarter, int half, int lane, uint32_t ring, uint32_t rank, int split,
                                              int rows_left) {
  const int row = quarter * 32 + lane;
  const int owned_units = kSplitTileN / 4 / split;             // a power of two: kSplitTileN, split are
#pragma unroll
  for (int step = 0; step < 2; ++step) {
    const int column0 = half * 64 + step * 32;
    uint32_t r[32];
    tmem_load_32(tmem_accumulator + column0 + (static_cast<uint32_t>(quarter * 32) << 16), r);
    tmem_load_wait();
    if (row < rows_left) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int unit = column0 / 4 + u;
        const uint32_t owner = unit / owned_units;
        const uint32_t local = ring + ((rank * owned_units + unit % owned_units) * kTileM + row) * 16;
        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(peer_address(local, owner)), "r"(r[4 * u]), "r"(r[4 * u + 1]),
                     "r"(r[4 * u + 2]), "r"(r[4 * u + 3])
                     : "memory");
      }
    }
    __syncwarp();
  }
}

// Then each CTA adds the partial sums of its own columns in the order of the senders, sixteen columns of
// a row per thread, and finishes them.
template <typename T>
__device__ __forceinline__ void finish_split(uint32_t ring, uint32_t rank, int split, int epilogue_thread, const float* bias_tile, T* c_tile, long long ldc,
                                             const T* residual_tile, long long ldr, int rows_left, int columns_left, int activation, bool vector_ok) {
  const int owned = kSplitTileN / split;                       // 16, 32 or 64 columns
  for (int item = epilogue_thread; item < kTileM * (owned / 16); item += kEpilogueThreads) {
    const int row = item % kTileM, local0 = (item / kTileM) * 16;
    const int column0 = static_cast<int>(rank) * owned + local0;
    if (row >= rows_left || column0 >= columns_left) continue;
    float2 sum[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] = make_float2(0.f, 0.f);
    for (int sender = 0; sender < split; ++sender) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 part;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(part.x), "=f"(part.y), "=f"(part.z), "=f"(part.w)
                     : "r"(ring + ((sender * (owned / 4) + local0 / 4 + u) * kTileM + row) * 16)
                     : "memory");
        sum[2 * u] = __fadd2_rn(sum[2 * u], make_float2(part.x, part.y));
        sum[2 * u + 1] = __fadd2_rn(sum[2 * u + 1], make_float2(part.z, part.w));
      }
    }
    uint32_t r[32];
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(j % 2 ? sum[j / 2].y : sum[j / 2].x);
    T* c = c_tile + static_cast<long long>(row) * ldc + column0;
    const T* residual = residual_tile == nullptr ? nullptr : residual_tile + static_cast<long long>(row) * ldr + column0;
    auto finish = [&](auto activation_tag, auto residual_tag) {
      constexpr int kActivation = decltype(activation_tag)::value;
      constexpr bool kResidual = decltype(residual_tag)::value;
#pragma unroll
      for (int unit = 0; unit < 2; ++unit) {
        if (column0 + unit * 8 >= columns_left) break;
        uint4 word = make_uint4(0, 0, 0, 0);
        Vec<T, 8>& elements = reinterpret_cast<Vec<T, 8>&>(word);
        if (vector_ok) {
          if constexpr (kResidual) word = __ldg(reinterpret_cast<const uint4*>(residual + unit * 8));
          *reinterpret_cast<uint4*>(c + unit * 8) = finish_unit<T, kActivation, kResidual>(r, r, bias_tile + column0, unit, word);
        } else {
          const int count = min(8, columns_left - column0 - unit * 8);
          if constexpr (kResidual) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (j < count) elements.v[j] = residual[unit * 8 + j];
            }
          }
          word = finish_unit<T, kActivation, kResidual>(r, r, bias_tile + column0, unit, word);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j < count) c[unit * 8 + j] = elements.v[j];
          }
        }
      }
    };
    with_activation(activation, residual != nullptr, finish);
  }
}

// Whether C (and the residual) can be written (read) in aligned units of eight columns.
__device__ __forceinline__ bool whole_units(const GemmParams& p) {
  return (p.ldc % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.c) & 15) == 0) && (p.stride_c % 8 == 0) && (p.n % 8 == 0) &&
         (p.residual == nullptr || ((p.ldr % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.residual) & 15) == 0) && (p.stride_r % 8 == 0)));
}

template <int TILE_N>
struct SingleShape {
  static constexpr uint32_t kBytesB = TILE_N * kTileK * 2;            // 16 or 32 KiB
  static constexpr uint32_t kStageBytes = kBytesA + kBytesB;
  static constexpr int kStages = TILE_N == 128 ? 6 : 3;
  static constexpr uint32_t kTmemColumns = 2 * TILE_N;                // two accumulators
  static constexpr size_t kSmemBytes = 1024 /*alignment slack*/ + static_cast<size_t>(kStages) * kStageBytes + 2 * TILE_N * sizeof(float) /*bias*/ +
                                       256 /*barriers, tmem slot*/ + kEpilogueWarps * kStoreBytes;
};

template <typename T, int TILE_N, bool A_MN, bool B_MN, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bias_act_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
  using Shape = SingleShape<TILE_N>;
  constexpr int kStages = Shape::kStages;
  constexpr uint32_t kBytesB = Shape::kBytesB, kStageBytes = Shape::kStageBytes;
  static_assert(!SPLIT || TILE_N == kSplitTileN, "the partial sums' way through the ring is laid out for one width");
  extern __shared__ unsigned char raw_smem[];
  const uint32_t base = (smem_address(raw_smem) + 1023u) & ~1023u;   // swizzled tiles need 1024-byte alignment
  unsigned char* aligned = raw_smem + (base - smem_address(raw_smem));
  float* bias_smem = reinterpret_cast<float*>(aligned + kStages * kStageBytes);        // [2][TILE_N]
  const uint32_t barriers = base + kStages * kStageBytes + 2 * TILE_N * sizeof(float);
  // barrier slots, 8 bytes each: full[kStages], empty[kStages], tmem_full[2], tmem_empty[2]
  auto full_bar = [&](int s) { return barriers + 8u * s; };
  auto empty_bar = [&](int s) { return barriers + 8u * (kStages + s); };
  auto tmem_full_bar = [&](int a) { return barriers + 8u * (2 * kStages + a); };
  auto tmem_empty_bar = [&](int a) { return barriers + 8u * (2 * kStages + 2 + a); };
  const uint32_t tmem_slot = barriers + 8u * (2 * kStages + 4);
  volatile uint32_t* tmem_slot_pointer =
      reinterpret_cast<volatile uint32_t*>(aligned + kStages * kStageBytes + 2 * TILE_N * sizeof(float) + 8 * (2 * kStages + 4));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // With SPLIT a cluster of p.split CTAs has one tile, each CTA an even share of its k-blocks; otherwise the
  // CTAs walk the tiles and take them whole.
  const uint32_t rank = SPLIT ? cluster_rank() : 0;
  const long long first_tile = SPLIT ? blockIdx.x / p.split : blockIdx.x;
  const long long tile_step = SPLIT ? p.num_tiles : gridDim.x;
  const int all_blocks = (p.k + kTileK - 1) / kTileK;
  const int first_block = SPLIT ? static_cast<int>(static_cast<long long>(all_blocks) * rank / p.split) : 0;
  const int k_blocks = (SPLIT ? static_cast<int>(static_cast<long long>(all_blocks) * (rank + 1) / p.split) : all_blocks) - first_block;

  // One stage of the ring: the k-block's slices of A and B.
  auto load_stage = [&](int s, int kb, int batch, int tile_m, int tile_n) {
    barrier_expect_tx(full_bar(s), kBytesB + p.a_rows * (kTileK * 2));
    const uint32_t smem_a = base + s * kStageBytes;
    const uint32_t smem_b = smem_a + kBytesA;
    const int k0 = (first_block + kb) * kTileK;
    if constexpr (A_MN) {
#pragma unroll
      for (int i = 0; i < kTileM / 64; ++i) tma_load_3d(smem_a + i * kChunkBytes, &map_a, full_bar(s), tile_m * kTileM + i * 64, k0, batch);
    } else {
      tma_load_3d(smem_a, &map_a, full_bar(s), k0, tile_m * kTileM, batch);
    }
    if constexpr (B_MN) {
#pragma unroll
      for (int i = 0; i < TILE_N / 64; ++i) tma_load_3d(smem_b + i * kChunkBytes, &map_b, full_bar(s), tile_n * TILE_N + i * 64, k0, batch);
    } else {
      tma_load_3d(smem_b, &map_b, full_bar(s), k0, tile_n * TILE_N, batch);
    }
  };

  // The producer lane sets the barriers up and fills the ring for the first time before the CTA meets, so
  // that the loads' latency runs under the tensor-memory allocation and the barrier.
  const int early = min(k_blocks, kStages);
  if (warp == 0 && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    if (blockIdx.x == 0) p.status.begin();   // this launch's abort word starts clear
    for (int s = 0; s < kStages; ++s) {
      barrier_init(full_bar(s), 1);
      barrier_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      barrier_init(tmem_full_bar(a), 1);
      barrier_init(tmem_empty_bar(a), kEpilogueThreads / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    int batch, tile_m, tile_n;
    tile_coordinates(first_tile, p, batch, tile_m, tile_n);
    for (int kb = 0; kb < early; ++kb) load_stage(kb, kb, batch, tile_m, tile_n);
  }
  if (warp == 1) tmem_alloc(tmem_slot, Shape::kTmemColumns);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_pointer;

  if (warp == 0) {
    // ---- producer: what did not fit the first filling ------------------------------------------
    if (elect_one()) {
      uint32_t iteration = early;
      bool alive = true;
      for (long long tile = first_tile; alive && tile < p.num_tiles; tile += tile_step) {
        int batch, tile_m, tile_n;
        tile_coordinates(tile, p, batch, tile_m, tile_n);
        for (int kb = tile == first_tile ? early : 0; kb < k_blocks; ++kb, ++iteration) {
          const int s = iteration % kStages;
          const uint32_t phase = (iteration / kStages) & 1;
          if (!barrier_wait(empty_bar(s), phase ^ 1, p.status, kWaitEmpty)) { alive = false; break; }
          load_stage(s, kb, batch, tile_m, tile_n);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ------------------------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc = instruction_descriptor(std::is_same_v<T, __nv_bfloat16>, A_MN, B_MN, kTileM, TILE_N);
      // K-major: 8-row groups are 1024 B apart; a step of 16 along K is 32 B inside the swizzle row.
      // MN-major: 64-wide chunks are kChunkBytes apart, groups of 8 K-rows 1024 B; 16 K-rows = 2048 B.
      constexpr uint32_t lead_a = A_MN ? kChunkBytes : 0, lead_b = B_MN ? kChunkBytes : 0;
      constexpr uint32_t step_a16 = (A_MN ? 2048 : 32) >> 4, step_b16 = (B_MN ? 2048 : 32) >> 4;
      // Descriptors as (low, high) words stepped by one add, stage and phase as counters, no
      // tcgen05 fence per k-block: what this lane does between two k-blocks is time the pipe can run dry.
      constexpr uint32_t kHigh = kDescriptorHigh;
      const uint32_t low_a0 = descriptor_low(base, lead_a), low_b0 = descriptor_low(base + kBytesA, lead_b);
      uint32_t s = 0, phase = 0;
      uint32_t local_tile = 0;
      bool alive = true;
      for (long long tile = first_tile; alive && tile < p.num_tiles; tile += tile_step, ++local_tile) {
        const uint32_t acc = local_tile & 1;
        const uint32_t acc_phase = (local_tile >> 1) & 1;
        if (!barrier_wait(tmem_empty_bar(acc), acc_phase ^ 1, p.status, kWaitTmemEmpty)) break;
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + acc * TILE_N;
        uint32_t accumulate = 0;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!barrier_wait(full_bar(s), phase, p.status, kWaitFull)) { alive = false; break; }
          const uint32_t low_a = low_a0 + s * (kStageBytes >> 4), low_b = low_b0 + s * (kStageBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kTileK / kMmaK; ++kk) {
            mma_f16_split(tmem_d, low_a + kk * step_a16, kHigh, low_b + kk * step_b16, kHigh, idesc, accumulate);
            accumulate = 1;
          }
          mma_commit(empty_bar(s));                        // the stage is free once these MMAs have read it
          if (++s == kStages) { s = 0; phase ^= 1; }
        }
        if (alive) mma_commit(tmem_full_bar(acc));         // the tile is complete
      }
    }
  } else {
    // ---- epilogue: warps 2..9; warp w owns tensor-memory lanes 32 (w % 4) .. +31 and every other
    // block of 64 columns from block (w - 2) / 4 on ----------------------------------------------
    const int epilogue_thread = threadIdx.x - 64;
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    unsigned char* staging = aligned + kStages * kStageBytes + 2 * TILE_N * sizeof(float) + 256 + (warp - 2) * kStoreBytes;
    const bool vector_ok = whole_units(p);
    uint32_t local_tile = 0;
    for (long long tile = first_tile; tile < p.num_tiles; tile += tile_step, ++local_tile) {
      int batch, tile_m, tile_n;
      tile_coordinates(tile, p, batch, tile_m, tile_n);
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_phase = (local_tile >> 1) & 1;
      const int n0 = tile_n * TILE_N;
      float* bias_tile = bias_smem + acc * TILE_N;
      for (int j = epilogue_thread; j < TILE_N; j += kEpilogueThreads) {
        float value = 0.f;
        if (p.bias != nullptr && n0 + j < p.n) value = to_compute(static_cast<const T*>(p.bias)[n0 + j]);
        bias_tile[j] = value;
      }
      // The give-up is decided for the epilogue as a whole: every epilogue thread reaches the named
      // barrier, which also carries the AND of their waits, and all leave together or none does.
      const bool arrived = barrier_wait(tmem_full_bar(acc), acc_phase, p.status, kWaitTmemFull);
      tcgen05_fence_after();
      const bool complete = epilogue_all(arrived);     // also: bias_tile is complete
      if constexpr (!SPLIT) {
        if (!complete) break;
      }
      T* c_tile = static_cast<T*>(p.c) + static_cast<long long>(batch) * p.stride_c + static_cast<long long>(tile_m) * kTileM * p.ldc + n0;
      const T* residual_tile = p.residual == nullptr ? nullptr : static_cast<const T*>(p.residual) + static_cast<long long>(batch) * p.stride_r +
                                                                  static_cast<long long>(tile_m) * kTileM * p.ldr + n0;
      const int rows_left = p.m - tile_m * kTileM, columns_left = p.n - n0;
      if constexpr (SPLIT) {
        // Every thread of the cluster passes both barriers (the other two warps below), also after a wait
        // that gave up. After the first all rings are idle: each CTA's MMAs have completed, so they have
        // read what its loads brought. After the second the partial sums are where they belong.
        __syncwarp();
        cluster_sync_all();
        if (complete) push_partials(tmem_base, quarter, half, lane, base, rank, p.split, rows_left);
        cluster_sync_all();
        if (complete) {
          finish_split<T>(base, rank, p.split, epilogue_thread, bias_tile, c_tile, p.ldc, residual_tile, p.ldr, rows_left, columns_left, p.activation,
                          vector_ok);
        }
      } else {
        epilogue_rows<T, TILE_N>(tmem_base + acc * TILE_N, quarter, half, lane, bias_tile, c_tile, p.ldc, residual_tile, p.ldr, rows_left, columns_left,
                                 p.activation, staging, vector_ok);
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) barrier_arrive(tmem_empty_bar(acc));   // this warp has read its part of the accumulator
      }
    }
  }
  if constexpr (SPLIT) {
    if (warp < 2) {
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  }

  // ---- teardown: every thread arrives here, also after a wait that gave up -----------------
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, Shape::kTmemColumns);
  }
}


// ---------------------------------------------------------------------------------------------
// The CTA-pair variant: two CTAs on neighbouring SMs (a cluster of 2) compute one 256 x 256 tile
// with tcgen05.mma.cta_group::2. Each CTA loads its own 128 rows of A and its own 128 columns of B
// (half the bytes per SM of the single-CTA tile), each CTA's tensor memory holds its 128 rows of the
// accumulator, and each CTA's epilogue warps write those rows. One lane of the even CTA (the
// leader) issues the MMAs for both; the stages' "full" barriers live in the leader and count the
// bytes of both CTAs' TMA loads (the loads name the leader's barrier; they are plain loads, no
// multicast); tcgen05.commit reports to the barriers of both CTAs.

//
// The tile's width is 256 columns, or 192 or 128 where that leaves fewer SMs idle in the last wave (see
// choose_tiling): a narrower tile reads A again for every tile of its row and brings fewer products per byte.

constexpr int kPairTileM = 256;

template <int TILE_N>
struct PairShape {
  static constexpr uint32_t kBytesB = (TILE_N / 2) * kTileK * 2;     // this CTA's half of B: 16, 12 or 8 KiB
  static constexpr uint32_t kStageBytes = kBytesA + kBytesB;          // per CTA
  static constexpr int kStages = TILE_N == 256 ? 5 : TILE_N == 192 ? 6 : 7;
  static constexpr uint32_t kTmemColumns = TILE_N == 128 ? 256 : 512; // an allocation is a power of two
  static constexpr size_t kSmemBytes = 1024 + static_cast<size_t>(kStages) * kStageBytes + 2 * TILE_N * sizeof(float) + 256 + kEpilogueWarps * kStoreBytes;
};

template <typename T, int TILE_N, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bias_act_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
  using Shape = PairShape<TILE_N>;
  constexpr int kPairStages = Shape::kStages;
  constexpr uint32_t kPairStageBytes = Shape::kStageBytes;
  static_assert(!B_MN || (TILE_N / 2) % 64 == 0, "an MN-major B comes in chunks of 64 columns per CTA");
  extern __shared__ unsigned char raw_smem[];
  const uint32_t base = (smem_address(raw_smem) + 1023u) & ~1023u;
  unsigned char* aligned = raw_smem + (base - smem_address(raw_smem));
  float* bias_smem = reinterpret_cast<float*>(aligned + kPairStages * kPairStageBytes);
  const uint32_t barriers = base + kPairStages * kPairStageBytes + 2 * TILE_N * sizeof(float);
  auto full_bar = [&](int s) { return barriers + 8u * s; };                       // used in the leader only
  auto empty_bar = [&](int s) { return barriers + 8u * (kPairStages + s); };       // one per CTA
  auto tmem_full_bar = [&](int a) { return barriers + 8u * (2 * kPairStages + a); };      // one per CTA
  auto tmem_empty_bar = [&](int a) { return barriers + 8u * (2 * kPairStages + 2 + a); }; // used in the leader only
  const uint32_t tmem_slot = barriers + 8u * (2 * kPairStages + 4);
  volatile uint32_t* tmem_slot_pointer =
      reinterpret_cast<volatile uint32_t*>(aligned + kPairStages * kPairStageBytes + 2 * TILE_N * sizeof(float) + 8 * (2 * kPairStages + 4));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();           // 0: leader, 1: peer
  const long long pair = blockIdx.x >> 1;
  const long long pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    if (blockIdx.x == 0) p.status.begin();   // this launch's abort word starts clear
    for (int s = 0; s < kPairStages; ++s) {
      barrier_init(full_bar(s), 2);                // one arrive.expect_tx from each CTA's producer
      barrier_init(empty_bar(s), 1);               // one commit
    }
    for (int a = 0; a < 2; ++a) {
      barrier_init(tmem_full_bar(a), 1);           // one commit
      barrier_init(tmem_empty_bar(a), 2 * (kEpilogueThreads / 32));   // the epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, Shape::kTmemColumns);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();                              // the peer's barriers exist before anything signals them
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_pointer;

  const int k_blocks = (p.k + kTileK - 1) / kTileK;

  if (warp == 0) {
    // ---- producer (one lane in each CTA) -----------------------------------------------------
    if (elect_one()) {
      uint32_t iteration = 0;
      bool alive = true;
      for (long long tile = pair; alive && tile < p.num_tiles; tile += pairs) {
        int batch, tile_m, tile_n;
        tile_coordinates(tile, p, batch, tile_m, tile_n);
        const int m0 = tile_m * kPairTileM + static_cast<int>(rank) * kTileM;
        const int n0 = tile_n * TILE_N + static_cast<int>(rank) * (TILE_N / 2);
        for (int kb = 0; kb < k_blocks; ++kb, ++iteration) {
          const int s = iteration % kPairStages;
          const uint32_t phase = (iteration / kPairStages) & 1;
          if (!barrier_wait(empty_bar(s), phase ^ 1, p.status, kWaitEmpty)) { alive = false; break; }
          const uint32_t leader_full = peer_address(full_bar(s), 0);
          remote_expect_tx(leader_full, kPairStageBytes);
          const uint32_t smem_a = base + s * kPairStageBytes;
          const uint32_t smem_b = smem_a + kBytesA;
          const int k0 = kb * kTileK;
          if constexpr (A_MN) {
#pragma unroll
            for (int i = 0; i < kTileM / 64; ++i) tma_load_3d_pair(smem_a + i * kChunkBytes, &map_a, leader_full, m0 + i * 64, k0, batch);
          } else {
            tma_load_3d_pair(smem_a, &map_a, leader_full, k0, m0, batch);
          }
          if constexpr (B_MN) {
#pragma unroll
            for (int i = 0; i < TILE_N / 2 / 64; ++i) tma_load_3d_pair(smem_b + i * kChunkBytes, &map_b, leader_full, n0 + i * 64, k0, batch);
          } else {
            tma_load_3d_pair(smem_b, &map_b, leader_full, k0, n0, batch);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one lane of the leader CTA, for both ------------------------------------
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = instruction_descriptor(std::is_same_v<T, __nv_bfloat16>, A_MN, B_MN, kPairTileM, TILE_N);
      constexpr uint32_t lead_a = A_MN ? kChunkBytes : 0, lead_b = B_MN ? kChunkBytes : 0;
      constexpr uint32_t step_a = A_MN ? 2048 : 32, step_b = B_MN ? 2048 : 32;
      uint32_t local_tile = 0;
      bool alive = true;
      // The tensor pipe holds only a couple of MMAs ahead of the one it executes, so whatever this
      // lane does between the last MMA of one k-block and the first of the next is time the pipe
      // can run dry: descriptors are (low, high) words stepped by one add, the stage and its
      // phase are counters (no division), and there is no tcgen05 fence per k-block — the
      // operands come from TMA through the full barrier, not from another thread's tcgen05 work.
      constexpr uint32_t kHigh = kDescriptorHigh;
      constexpr uint32_t step_a16 = step_a >> 4, step_b16 = step_b >> 4;
      const uint32_t low_a0 = descriptor_low(base, lead_a), low_b0 = descriptor_low(base + kBytesA, lead_b);
      uint32_t s = 0, phase = 0;
      for (long long tile = pair; alive && tile < p.num_tiles; tile += pairs, ++local_tile) {
        const uint32_t acc = local_tile & 1;
        const uint32_t acc_phase = (local_tile >> 1) & 1;
        if (!barrier_wait(tmem_empty_bar(acc), acc_phase ^ 1, p.status, kWaitTmemEmpty)) break;
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + acc * TILE_N;
        uint32_t accumulate = 0;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!barrier_wait(full_bar(s), phase, p.status, kWaitFull)) { alive = false; break; }
          const uint32_t low_a = low_a0 + s * (kPairStageBytes >> 4), low_b = low_b0 + s * (kPairStageBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kTileK / kMmaK; ++kk) {
            mma_f16_pair_split(tmem_d, low_a + kk * step_a16, kHigh, low_b + kk * step_b16, kHigh, idesc, accumulate);
            accumulate = 1;
          }
          mma_commit_pair(empty_bar(s));
          if (++s == kPairStages) { s = 0; phase ^= 1; }
        }
        if (alive) mma_commit_pair(tmem_full_bar(acc));
      }
    }
  } else {
    // ---- epilogue: this CTA's 128 rows of the pair's tile, eight warps -------------------------
    const int epilogue_thread = threadIdx.x - 64;
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    unsigned char* staging = aligned + kPairStages * kPairStageBytes + 2 * TILE_N * sizeof(float) + 256 + (warp - 2) * kStoreBytes;
    const bool vector_ok = whole_units(p);
    uint32_t local_tile = 0;
    for (long long tile = pair; tile < p.num_tiles; tile += pairs, ++local_tile) {
      int batch, tile_m, tile_n;
      tile_coordinates(tile, p, batch, tile_m, tile_n);
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_phase = (local_tile >> 1) & 1;
      const int n0 = tile_n * TILE_N;
      float* bias_tile = bias_smem + acc * TILE_N;
      for (int j = epilogue_thread; j < TILE_N; j += kEpilogueThreads) {
        float value = 0.f;
        if (p.bias != nullptr && n0 + j < p.n) value = to_compute(static_cast<const T*>(p.bias)[n0 + j]);
        bias_tile[j] = value;
      }
      // The give-up is decided for the epilogue as a whole: every epilogue thread reaches the named
      // barrier, which also carries the AND of their waits, and all leave together or none does.
      const bool arrived = barrier_wait(tmem_full_bar(acc), acc_phase, p.status, kWaitTmemFull);
      tcgen05_fence_after();
      if (!epilogue_all(arrived)) break;   // also: bias_tile is complete

      const int row0 = tile_m * kPairTileM + static_cast<int>(rank) * kTileM;
      T* c_tile = static_cast<T*>(p.c) + static_cast<long long>(batch) * p.stride_c + static_cast<long long>(row0) * p.ldc + n0;
      const T* residual_tile = p.residual == nullptr ? nullptr : static_cast<const T*>(p.residual) + static_cast<long long>(batch) * p.stride_r +
                                                                  static_cast<long long>(row0) * p.ldr + n0;
      epilogue_rows<T, TILE_N>(tmem_base + acc * TILE_N, quarter, half ^ static_cast<int>(acc), lane, bias_tile, c_tile, p.ldc, residual_tile, p.ldr, p.m - row0, p.n - n0,
                       p.activation, staging, vector_ok);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) remote_arrive(peer_address(tmem_empty_bar(acc), 0));   // tell the leader: this part is drained
    }
  }

  // ---- teardown: both CTAs stay until the pair is done (the leader's MMAs read the peer's
  // shared memory and signal its barriers) -----------------------------------------------------
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, Shape::kTmemColumns);
  }
}

// ---------------------------------------------------------------------------------------------
// Host

// A three-axis map over one operand: `inner` contiguous elements, `outer` rows `ld` elements apart,
// `batch` matrices `stride` elements apart; box = box_inner x box_outer x 1, 128-byte swizzle.
tq_status make_map(CUtensorMap* map, tq_dtype dtype, const void* pointer, long long inner, long long outer, long long ld,
                   long long batch, long long stride, int box_inner, int box_outer) {
  EncodeTiled encode = encode_tiled();
  TQ_REQUIRE(encode != nullptr, TQ_EXTERNAL, "the CUDA driver does not provide cuTensorMapEncodeTiled");
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer), static_cast<cuuint64_t>(batch)};
  // A stride of 0 (one operand shared by the whole batch) is not a legal map stride; such a map
  // gets one matrix and the kernel is launched with batch coordinate 0 for it (see below).
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2, static_cast<cuuint64_t>(stride > 0 ? stride : ld * outer) * 2};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_inner), static_cast<cuuint32_t>(box_outer), 1};
  const cuuint32_t element_strides[3] = {1, 1, 1};
  const CUresult result = encode(map, dtype == TQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                                 const_cast<void*>(pointer), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TQ_REQUIRE(result == CUDA_SUCCESS, TQ_UNSUPPORTED, "this operand layout cannot be described to TMA (driver code %d)", static_cast<int>(result));
  return TQ_OK;
}

// How a product is cut up: CTA pairs over 256 x tile_n tiles, or single CTAs over 128 x 128 tiles with
// `split` CTAs of a cluster sharing a tile's K range.
struct Tiling {
  bool pair;
  int tile_n;
  int split;
};

// How many clusters of 1, 2, 4 and 8 single CTAs run at once. Clusters of four and eight do not fill the GPU, since
// one lies within a graphics processing cluster, whose number of SMs differs from unit to unit and from GPU to GPU
// (33 and 15 on the B200 that the choice below was fitted on, which is what is assumed where there is none to ask).
struct ClusterRoom {
  long long of[4];
};

ClusterRoom assumed_room(long long sms) { return {{sms, sms / 2, sms * 33 / 148, sms * 15 / 148}}; }

// The device that is current, asked once.
ClusterRoom cluster_room(int32_t device) {
  static std::mutex mutex;
  static ClusterRoom known[64] = {};
  const ClusterRoom assumed = assumed_room(sm_count(device));
  if (device < 0 || device >= 64) return assumed;
  std::lock_guard<std::mutex> lock(mutex);
  ClusterRoom& room = known[device];
  if (room.of[0] == 0) {
    room = assumed;
    auto kernel = gemm_bias_act_kernel<__nv_bfloat16, kSplitTileN, false, false, true>;
    constexpr size_t kSmem = SingleShape<kSplitTileN>::kSmemBytes;
    bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)) == cudaSuccess;
    for (int i = 1; ok && i < 4; ++i) {
      cudaLaunchConfig_t config = {};
      config.gridDim = dim3(1u << i);
      config.blockDim = dim3(kThreads);
      config.dynamicSmemBytes = kSmem;
      cudaLaunchAttribute attribute[1];
      attribute[0].id = cudaLaunchAttributeClusterDimension;
      attribute[0].val.clusterDim.x = 1u << i;
      attribute[0].val.clusterDim.y = 1;
      attribute[0].val.clusterDim.z = 1;
      config.attrs = attribute;
      config.numAttrs = 1;
      int clusters = 0;
      ok = cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) == cudaSuccess && clusters > 0;
      if (ok) room.of[i] = clusters;
    }
    if (!ok) cudaGetLastError();
  }
  return room;
}

// The tiling with the least expected time, in microseconds. The constants are fitted to kernel times (graphs of launches over
// rotating operands, B200, bf16) of every tiling at 346 shapes: m = 1 ... 8192 for sixteen (k, n) from 64 x 512 to 4096 x
// 16384, and batches of 1 ... 2048 small products. A launch costs `launch`, each wave a k-block of 64 `block` per k-block, and
// each wave but the last at least `tile` (its epilogue, where K is too short to cover it). Over those shapes the choice
// takes 0.6 % longer than the best tiling on average; above 5 % only where a few rows could share K among more or fewer CTAs
// (512 x 1024 x 1024: 9.0 by four against 8.2 by two).
// A narrow tile does fewer products per byte it brings from L2 (a 128 x 128 k-block costs 0.22 where half of a
// 256 x 256 one costs 0.16 per CTA), so it pays only where it saves a wave: 8192 x 3072 x 768 (m, n, k) takes 31 as 256 x 256, 37 as
// 256 x 128; 4096 x 768 x 3072 takes 23.4 as 256 x 256, 21.1 as 256 x 192; 8192 x 768 x 768 14.4 and, as 256 x 128, 13.8.
// A single CTA's 256-wide tile halves the epilogues of products with few rows and a short K: 768 products of 1 x 1000 x 64
// take 54.5 where 128-wide tiles take 67.
// Sharing a tile's K range pays until the GPU is full: 64 x 4096 x 4096 19.3 by one CTA, 14.4 by two, 12.2 by four; but more
// clusters than there is room for take a second wave: 512 x 512 x 2048 is 16 clusters of eight, of which 15 run at once: 15.8
// against 8.8 by four.
Tiling choose_tiling(long long m, long long n, long long k, long long batch, bool b_mn, long long sms, const ClusterRoom& room) {
  const long long blocks = (k + kTileK - 1) / kTileK;
  Tiling best = {};
  double least = 0;
  auto consider = [&](Tiling t, long long tile_m, long long workers, double launch, double block, double tile) {
    const long long tiles = ((m + tile_m - 1) / tile_m) * ((n + t.tile_n - 1) / t.tile_n) * batch;
    const double waves = static_cast<double>((tiles + workers - 1) / workers), share = static_cast<double>((blocks + t.split - 1) / t.split);
    const double cost = launch + share * block + (waves - 1) * (share * block > tile ? share * block : tile);
    if (best.split == 0 || cost < least) {
      best = t;
      least = cost;
    }
  };
  consider({false, 128, 1}, kTileM, sms, 7.51, 0.223, 2.87);
  consider({false, 256, 1}, kTileM, sms, 7.77, 0.501, 5.50);
  double hops = 0;
  for (int i = 1; (1 << i) <= kMaxSplit; ++i) {
    hops += 0.567;
    if (blocks >= (2 << i)) consider({false, kSplitTileN, 1 << i}, kTileM, room.of[i], 8.15 + hops, 0.268, 14.6);
  }
  if (m > kTileM) {
    consider({true, 256, 1}, kPairTileM, sms / 2, 8.48, 0.323, 4.80);
    if (!b_mn) consider({true, 192, 1}, kPairTileM, sms / 2, 9.32, 0.270, 8.14);
    consider({true, 128, 1}, kPairTileM, sms / 2, 7.75, 0.217, 2.77);
  }
  return best;
}

// One launch of `kernel` with clusters of `cluster` CTAs.
template <typename Kernel>
tq_status launch_kernel(Kernel kernel, const char* name, long long ctas, int cluster, size_t smem, const CUtensorMap& map_a, const CUtensorMap& map_b,
                        const GemmParams& p, cudaStream_t stream) {
  TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(ctas));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = cluster;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = cluster > 1 ? 1 : 0;
  TQ_CUDA(cudaLaunchKernelEx(&config, kernel, map_a, map_b, p));
  return check_launch(name);
}

template <typename T, bool A_MN, bool B_MN>
tq_status launch_tiling(const Tiling& tiling, const CUtensorMap& map_a, const CUtensorMap& map_b, const GemmParams& p, int32_t device, cudaStream_t stream) {
  const long long sms = sm_count(device);
  if (!tiling.pair) {
    const long long ctas = tiling.split > 1 ? p.num_tiles * tiling.split : p.num_tiles < sms ? p.num_tiles : sms;
    auto go = [&](auto tile_n, auto split) {
      constexpr int kWidth = decltype(tile_n)::value;
      return launch_kernel(gemm_bias_act_kernel<T, kWidth, A_MN, B_MN, decltype(split)::value>, "gemm_bias_act_kernel", ctas, tiling.split,
                           SingleShape<kWidth>::kSmemBytes, map_a, map_b, p, stream);
    };
    if (tiling.split > 1) return go(std::integral_constant<int, kSplitTileN>{}, std::true_type{});
    if (tiling.tile_n == 256) return go(std::integral_constant<int, 256>{}, std::false_type{});
    return go(std::integral_constant<int, 128>{}, std::false_type{});
  }
  const long long pairs = p.num_tiles < sms / 2 ? p.num_tiles : sms / 2;
  auto go = [&](auto tile_n) {
    constexpr int kWidth = decltype(tile_n)::value;
    return launch_kernel(gemm_bias_act_pair_kernel<T, kWidth, A_MN, B_MN>, "gemm_bias_act_pair_kernel", pairs * 2, 2, PairShape<kWidth>::kSmemBytes, map_a,
                         map_b, p, stream);
  };
  if constexpr (!B_MN) {
    if (tiling.tile_n == 192) return go(std::integral_constant<int, 192>{});
  }
  if (tiling.tile_n == 128) return go(std::integral_constant<int, 128>{});
  return go(std::integral_constant<int, 256>{});
}

template <typename T>
tq_status launch(bool a_mn, bool b_mn, const Tiling& tiling, const CUtensorMap& map_a, const CUtensorMap& map_b, const GemmParams& p, int32_t device,
                 cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_tiling<T, false, false>(tiling, map_a, map_b, p, device, stream);
  if (!a_mn && b_mn) return launch_tiling<T, false, true>(tiling, map_a, map_b, p, device, stream);
  if (a_mn && !b_mn) return launch_tiling<T, true, false>(tiling, map_a, map_b, p, device, stream);
  return launch_tiling<T, true, true>(tiling, map_a, map_b, p, device, stream);
}

}  // namespace
}  // namespace tq

extern "C" tq_status tq_gemm_tiling(int64_t m, int64_t n, int64_t k, int64_t batch, int32_t trans_b, int32_t device, int32_t* ctas, int32_t* tile_n,
                                    int32_t* split) {
  TQ_REQUIRE(ctas != nullptr && tile_n != nullptr && split != nullptr, TQ_INVALID_ARGUMENT, "null out-pointer");
  TQ_REQUIRE(m > 0 && n > 0 && k > 0 && batch > 0, TQ_INVALID_ARGUMENT, "extents must be positive, not m=%lld n=%lld k=%lld batch=%lld", (long long)m,
             (long long)n, (long long)k, (long long)batch);
  tq::ClusterRoom room = tq::assumed_room(148);
  if (device >= 0) {
    tq::DeviceScope device_scope(device);
    if (tq_status s = device_scope.status()) return s;
    room = tq::cluster_room(device);
  }
  const tq::Tiling tiling = tq::choose_tiling(m, n, k, batch, trans_b == 0, room.of[0], room);
  *ctas = tiling.pair ? 2 : 1;
  *tile_n = tiling.tile_n;
  *split = tiling.split;
  return TQ_OK;
}

extern "C" tq_status tq_gemm_bias_act_launch(tq_dtype dtype, tq_activation activation, const void* a, int64_t lda,
                                             int32_t trans_a, const void* b, int64_t ldb, int32_t trans_b,
                                             const void* bias, void* c, int64_t ldc, int64_t m, int64_t n, int64_t k,
                                             int64_t batch, int64_t stride_a, int64_t stride_b, int64_t stride_c,
                                             int32_t device, void* stream) {
  return tq_gemm_bias_act_residual_launch(dtype, activation, a, lda, trans_a, b, ldb, trans_b, bias, nullptr, 0, 0, c, ldc, m, n, k,
                                          batch, stride_a, stride_b, stride_c, device, stream);
}

extern "C" tq_status tq_gemm_bias_act_residual_launch(tq_dtype dtype, tq_activation activation, const void* a, int64_t lda,
                                                      int32_t trans_a, const void* b, int64_t ldb, int32_t trans_b,
                                                      const void* bias, const void* residual, int64_t ldr, int64_t stride_r,
                                                      void* c, int64_t ldc, int64_t m, int64_t n, int64_t k, int64_t batch,
                                                      int64_t stride_a, int64_t stride_b, int64_t stride_c, int32_t device,
                                                      void* stream) {
  TQ_RECORD_OR_RUN([=](int32_t d, void* s) {
    return tq_gemm_bias_act_residual_launch(dtype, activation, a, lda, trans_a, b, ldb, trans_b, bias, residual, ldr, stride_r, c, ldc,
                                            m, n, k, batch, stride_a, stride_b, stride_c, d, s);
  });
  TQ_REQUIRE(dtype == TQ_BF16 || dtype == TQ_F16, TQ_UNSUPPORTED,
             "the tensor-core GEMM takes bf16 or f16 operands, not %s", tq::dtype_name(dtype));
  TQ_REQUIRE(activation >= TQ_ACT_NONE && activation <= TQ_ACT_GELU_TANH, TQ_INVALID_ARGUMENT, "unknown activation %d", activation);
  TQ_REQUIRE(m >= 0 && n >= 0 && k >= 0 && batch >= 0, TQ_INVALID_ARGUMENT, "negative extent in m=%lld n=%lld k=%lld batch=%lld",
             (long long)m, (long long)n, (long long)k, (long long)batch);
  if (m == 0 || n == 0 || batch == 0) return TQ_OK;
  TQ_REQUIRE(k > 0, TQ_UNSUPPORTED, "a product over no elements has no kernel");
  TQ_REQUIRE(a != nullptr && b != nullptr && c != nullptr, TQ_INVALID_ARGUMENT, "null operand or result");
  TQ_REQUIRE(m < (1LL << 31) && n < (1LL << 31) && k < (1LL << 31), TQ_UNSUPPORTED, "extents beyond 2^31 have no kernel");
  // TMA's rules: 16-byte-aligned bases, strides that are multiples of 16 bytes.
  const long long a_inner = trans_a ? m : k, a_outer = trans_a ? k : m;
  const long long b_inner = trans_b ? k : n, b_outer = trans_b ? n : k;
  TQ_REQUIRE(lda >= a_inner && ldb >= b_inner && ldc >= n, TQ_INVALID_ARGUMENT, "a leading dimension is smaller than its row");
  TQ_REQUIRE(tq::aligned_to(a, 16) && tq::aligned_to(b, 16) && lda % 8 == 0 && ldb % 8 == 0 &&
                 (batch == 1 || (stride_a % 8 == 0 && stride_b % 8 == 0)),
             TQ_UNSUPPORTED, "operands must be 16-byte aligned with leading dimensions and batch strides that are multiples of 8 elements");
  TQ_REQUIRE(tq::aligned_to(c, 2) && (bias == nullptr || tq::aligned_to(bias, 2)), TQ_INVALID_ARGUMENT, "misaligned result or bias");
  TQ_REQUIRE(residual == nullptr || (tq::aligned_to(residual, 2) && ldr >= n), TQ_INVALID_ARGUMENT,
             "misaligned residual, or its leading dimension is smaller than a row");
  tq::DeviceScope device_scope(device);
  if (tq_status s = device_scope.status()) return s;
  const tq::WaitStatus status = tq::wait_status_for(device);
  TQ_REQUIRE(status.abort != nullptr, TQ_RESOURCE_EXHAUSTED, "no device memory for the status word");

  const tq::Tiling tiling = tq::choose_tiling(m, n, k, batch, trans_b == 0, tq::sm_count(device), tq::cluster_room(device));
  CUtensorMap map_a, map_b;
  const long long batch_a = stride_a > 0 ? batch : 1, batch_b = stride_b > 0 ? batch : 1;
  // (rows of the tile that A does not have are not brought; what lies there gives rows of C nobody stores)
  const int a_rows = tiling.pair || trans_a || m > tq::kTileM ? tq::kTileM : static_cast<int>((m + 7) / 8 * 8);
  const int b_rows = tiling.pair ? tiling.tile_n / 2 : tiling.tile_n;
  if (tq_status s = tq::make_map(&map_a, dtype, a, a_inner, a_outer, lda, batch_a, stride_a, 64, trans_a ? 64 : a_rows)) return s;
  if (tq_status s = tq::make_map(&map_b, dtype, b, b_inner, b_outer, ldb, batch_b, stride_b, 64, trans_b ? b_rows : 64)) return s;
  TQ_REQUIRE(batch == 1 || (stride_a > 0 && stride_b > 0), TQ_UNSUPPORTED,
             "a batch that shares one operand (stride 0) has no kernel; fold the batch into m instead");

  tq::GemmParams p = {};
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.k = static_cast<int>(k);
  p.batch = static_cast<int>(batch);
  const int tile_m = tiling.pair ? tq::kPairTileM : tq::kTileM;
  p.tiles_m = static_cast<int>((m + tile_m - 1) / tile_m);
  p.tiles_n = static_cast<int>((n + tiling.tile_n - 1) / tiling.tile_n);
  p.split = tiling.split;
  p.a_rows = a_rows;
  p.num_tiles = static_cast<long long>(p.tiles_m) * p.tiles_n * batch;
  p.bias = bias;
  p.residual = residual;
  p.ldr = ldr;
  p.stride_r = stride_r;
  p.c = c;
  p.ldc = ldc;
  p.stride_c = stride_c;
  p.activation = activation;
  p.status = status;
  cudaStream_t cuda_stream = static_cast<cudaStream_t>(stream);
  if (dtype == TQ_BF16) return tq::launch<__nv_bfloat16>(trans_a != 0, trans_b == 0, tiling, map_a, map_b, p, device, cuda_stream);
  return tq::launch<__half>(trans_a != 0, trans_b == 0, tiling, map_a, map_b, p, device, cuda_stream);
}
