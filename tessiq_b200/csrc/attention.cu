// Fused attention on the 5th-generation tensor cores (tcgen05), for sm_100a.
//
//   out[b,h,i,:] = sum_j softmax_j(scale * q[b,h,i,:] . k[b,h,j,:]) v[b,h,j,:]     (j <= i when causal)
//
// bf16 or f16 operands, heads of up to 128 elements, f32 scores and sums, one rounding of the result. The
// score matrix never leaves the SM: one CTA owns 128 query rows of one head and walks the keys 64 or 128 at a
// time (choose_attention_form) with a row reference point and row sum (the online form of softmax).
//
//   warps 0..3          softmax, one thread per query row: tcgen05.ld of the row's f32 scores of a step (held in
//                       registers for both the maximum and the exponentials), ex2, row sum; the
//                       probabilities go back into tensor memory with tcgen05.st as packed bf16/f16 pairs —
//                       the A operand of the second product. The result accumulates in tensor memory
//                       across the steps and is read once, at the end.
//   warp 4, one lane    producer: TMA loads (128-byte swizzle) of the query tile once, then one key tile and
//                       one value tile per step into two rings; the first filling leaves before the CTA's
//                       set-up barrier.
//   warp 5, one lane    issuer: S = Q K^T (128 x keys x head, both operands K-major in shared memory) and
//                       O = P V (128 x head x keys, P from tensor memory, V consumed MN-major exactly as it
//                       lies in memory). The scores of step j + 1 are computed while the softmax warps work
//                       on step j, which hand the columns back as soon as they have them in registers.
//
// softmax is exp(s - m) / sum exp(s - m) for ANY m, so a row keeps the maximum of its first 128 keys
// as its reference point and moves it only when a later tile rises more than 2^8 above it — then,
// and only then, the row's sum and its accumulators in tensor memory are rescaled (a warp-wide
// slow path, rare on real data). Without that, nothing is read back per step: the second product
// accumulates O += P V in place. Probabilities are at most 2^8, well inside bf16 and f16. (With 64 keys a step the second
// tile's scores are computed ahead for it, into the result's columns: from the first 64 keys alone a row's largest
// probability was exactly 1 less often, and the error against 64 bits 1 to 3 % larger.)
//
// A few queries (FEW) leave three of the four softmax warps without a row and the tensor cores idle, so their probabilities
// are taken as two 16-bit operands, the rounded value and what rounding took off: the result is as exact as the
// streaming kernel's, whose probabilities are never rounded (error against 64 bits 1.65e-3 in bf16, all of it the result's
// rounding; 2.3e-3 with one operand).
//
// What bounds it: a step of 64 keys of one CTA is a chain (scores seen, tcgen05.ld, maximum, ex2, tcgen05.st, signal) of about
// 1 500 cycles of which the special-function unit works 512, so an SM needs several chains. Three CTAs of one
// softmax warp per scheduler each (two for heads above 64) keep the unit busy 65 % of the time, and one CTA's
// start and end run under the others' steps; two CTAs with 128 keys a step pay a step's hand-overs half as often and reach
// as much. One CTA an SM with two groups of 128 rows and 128-key steps, as it
// was once, spent 5 000 cycles on every start: 64 x 12 heads, 1024 tokens of 64 causal 256 us, now 229, no mask 377, now 323,
// 4 x 12 x 4096 no mask 332, now 296; 64 x 6 heads of 128, whose second group had idled, 235, now 175.
// Measured beside it (before the reference point took 128 keys, when the first two of those were 225 and 320): two CTAs with two groups each and the probabilities over the scores (four chains, each
// with both products inside it) 216 / 307 / 312 / 205; one exponential in four, or in sixteen, as a polynomial of
// degree 5 on the FMA pipes 328 and 322 instead of 312; scalar instead of two-element FMA and add 311 - 318; the
// row sum after the signal 333; skipping the rows past the diagonal of a whole warp: no change.
//
// The softmax warps run with 120 registers per thread where three CTAs share an SM, 200 where two do, the other four with 40 and 56
// (setmaxnreg). Q, K, V and the result are addressed through (batch, head, token) strides, so the three slices
// of a fused QKV projection are read in place and the result is written directly in [batch, token, head, head_dim]
// order: none of the four packing copies around `bmm -> where -> softmax -> bmm` remains.
//
// Every wait is bounded; a wait that gives up sets the device status word (tq_status_poll) and the
// CTA leaves through the normal teardown, freeing its tensor memory. No load uses multicast.
//
// The reference has no attention kernel: its compiler emits bmm (csrc/tessiq/codegen/gemm.cpp:100-175),
// a host-side mask, the softmax custom op (csrc/custom_ops/softmax/softmax.cu:19-61) and a second bmm
// for the pattern in tests/python/test_models.py:64-67, with the [batch, heads, T, T] scores in memory.
#include <cuda.h>

#include <cmath>
#include <mutex>
#include <type_traits>

#include "common.h"
#include "tcgen05.h"

namespace tq {
namespace {

constexpr int kHeadDim = 64;
constexpr int kRows = 128;            // query rows per CTA
constexpr int kAttnThreads = 256;     // four softmax warps; producer and issuer in a second group of four
constexpr uint32_t kQueryBytes = kRows * kHeadDim * 2;       // 16 KiB: 128 rows of 64 elements, one TMA box, one swizzled operand tile
// D: heads of up to 64 elements, or of up to 128 (two 64-wide sub-tiles side by side in every tile). KEYS: keys per step. FEW:
// the form for a few queries, whose probabilities take two operands (below). Shared memory: the query tile, the key
// ring, the value ring, the barriers. Tensor memory, f32 columns: scores (KEYS), packed probabilities (KEYS / 2, twice with FEW),
// result (D). An allocation is a power of two, so heads of 64 with 64 keys a step take two (scores and result,
// probabilities: 160 columns, and three CTAs have 480 of the 512) and the other forms a single one.
template <int D, int KEYS, bool FEW>
struct AttnLayout {
  static constexpr int kSubTiles = D / kHeadDim;
  static constexpr bool kTwoAllocations = D == kHeadDim && KEYS == 64 && !FEW;
  static constexpr int kCtasPerSm = kTwoAllocations ? 3 : KEYS == 64 || (D == kHeadDim && !FEW) ? 2 : 1;
  static constexpr int kRing = D == kHeadDim && KEYS == 64 ? 3 : 2;          // stages of the key ring and of the value ring
  static constexpr uint32_t kSubTileBytes = KEYS * kHeadDim * 2;            // 8 or 16 KiB: 64 elements of a tile's keys or values
  static constexpr uint32_t kTileBytes = kSubTiles * kSubTileBytes;
  static constexpr uint32_t kOffsetK = kSubTiles * kQueryBytes;
  static constexpr uint32_t kOffsetV = kOffsetK + kRing * kTileBytes;
  static constexpr uint32_t kOffsetBarriers = kOffsetV + kRing * kTileBytes;
  static constexpr size_t kSmemBytes = 1024 + kOffsetBarriers + 256;
  static constexpr uint32_t kColumnP = KEYS, kColumnO = kTwoAllocations ? 64 : D == kHeadDim && !FEW ? KEYS + KEYS / 2 : 2 * KEYS;
  static constexpr uint32_t kTmemColumns = kTwoAllocations ? 128 : kColumnO + D <= 256 ? 256 : 512;      // scores from column 0 on
  static_assert(kTwoAllocations || (kColumnP + (FEW ? KEYS : KEYS / 2) <= kColumnO && kColumnO + D <= kTmemColumns), "the columns overlap");
  static_assert(kTwoAllocations ? kCtasPerSm * 160 <= 512 : kCtasPerSm * kTmemColumns <= 512, "more CTAs an SM than it has tensor memory for");
  static_assert(kCtasPerSm * (kSmemBytes + 1024) <= 228 * 1024, "the staging has to fit as often as there are CTAs an SM");
  // setmaxnreg moves registers inside the CTA's own allocation: what the second group of four warps gives up is
  // at least what the softmax warps take. An increase beyond what was released would wait for ever. (A CTA that has
  // its SM to itself has registers enough from the start.)
  static constexpr int kLaunchRegisters = (65536 / kCtasPerSm / kAttnThreads) / 8 * 8;
  static constexpr int kSoftmaxRegisters = kCtasPerSm == 3 ? 120 : 200, kOtherRegisters = kCtasPerSm == 3 ? 40 : 56;
  static constexpr bool kMovesRegisters = kCtasPerSm > 1;
  static_assert(!kMovesRegisters || 128 * (kSoftmaxRegisters - kLaunchRegisters) <= 128 * (kLaunchRegisters - kOtherRegisters),
                "the softmax warps would wait for registers nobody releases");
};
constexpr uint32_t kTmemColumnsP = 32;       // of the second allocation
constexpr float kSlack = 8.f;                // a row's reference point moves when a tile's maximum is more than 2^kSlack above it

enum AttnWait { kWaitQ = 201, kWaitKeyEmpty = 202, kWaitValueEmpty = 203, kWaitKeyFull = 204, kWaitValueFull = 205,
                kWaitScores = 206, kWaitProbabilities = 207, kWaitPartial = 208, kWaitBufferFree = 209 };

struct AttnParams {
  int batch, heads, q_tokens, k_tokens;
  int head_dim;                    // 8, 16, ... 128: narrower heads ride in tiles of 64 or 128 whose other columns TMA fills with zeros
  int q_blocks;                    // CTAs per head
  int causal;
  float scale_log2;                // scale * log2(e)
  void* out;
  long long out_batch, out_head, out_token;   // element strides
  WaitStatus status;
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// f32 accumulator, A and B of type T, M = 128, N = `n`; B MN-major when `b_mn`.
template <typename T>
__host__ __device__ constexpr uint32_t attn_instruction_descriptor(int n, bool b_mn) {
  constexpr uint32_t format = std::is_same_v<T, __nv_bfloat16> ? 1u : 0u;
  return (1u << 4) | (format << 7) | (format << 10) | ((b_mn ? 1u : 0u) << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(kRows >> 4) << 24);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float low, float high) {
  if constexpr (std::is_same_v<T, __nv_bfloat16>) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
    return *reinterpret_cast<const uint32_t*>(&pair);
  } else {
    const __half2 pair = __floats2half2_rn(low, high);
    return *reinterpret_cast<const uint32_t*>(&pair);
  }
}

// What rounding took off a pair of probabilities, rounded itself.
template <typename T>
__device__ __forceinline__ uint32_t pack_rest(uint32_t rounded, float2 exact) {
  if constexpr (std::is_same_v<T, __nv_bfloat16>) {
    return pack_pair<T>(exact.x - __uint_as_float(rounded << 16), exact.y - __uint_as_float(rounded & 0xffff0000u));
  } else {
    const float2 wide = __half22float2(*reinterpret_cast<const __half2*>(&rounded));
    return pack_pair<T>(exact.x - wide.x, exact.y - wide.y);
  }
}

template <typename T, int D, int KEYS, bool FEW>
__global__ void __launch_bounds__(kAttnThreads, AttnLayout<D, KEYS, FEW>::kCtasPerSm)
attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  using L = AttnLayout<D, KEYS, FEW>;
  constexpr int kKeys = KEYS;
  constexpr bool kAhead = KEYS < 128;      // the reference point takes the second tile's scores too
  constexpr uint32_t kSubTileBytes = L::kSubTileBytes;
  constexpr int kRing = L::kRing;
  constexpr uint32_t kTileBytes = L::kTileBytes, kOffsetK = L::kOffsetK, kOffsetV = L::kOffsetV;
  constexpr uint32_t kOffsetBarriers = L::kOffsetBarriers, kColumnO = L::kColumnO;
  constexpr int kSubTiles = L::kSubTiles;
  extern __shared__ unsigned char raw_smem[];
  const uint32_t base = (smem_address(raw_smem) + 1023u) & ~1023u;
  unsigned char* aligned = raw_smem + (base - smem_address(raw_smem));
  const uint32_t barriers = base + kOffsetBarriers;
  // barrier slots, 8 bytes each
  const uint32_t q_full = barriers;
  auto k_full = [&](int s) { return barriers + 8u * (1 + s); };
  auto k_empty = [&](int s) { return barriers + 8u * (1 + kRing + s); };
  auto v_full = [&](int s) { return barriers + 8u * (1 + 2 * kRing + s); };
  auto v_empty = [&](int s) { return barriers + 8u * (1 + 3 * kRing + s); };
  const uint32_t s_full = barriers + 8u * (1 + 4 * kRing);      // the scores of a step are in tensor memory
  const uint32_t s_free = s_full + 8;                           // ... and in the softmax warps' registers
  const uint32_t p_full = s_full + 16;                          // the probabilities of a step are in tensor memory
  const uint32_t pv_done = s_full + 24;                         // ... and the second product has consumed them
  constexpr int kBarrierCount = 1 + 4 * kRing + 4;
  const uint32_t tmem_slot = barriers + 8u * kBarrierCount;
  volatile uint32_t* tmem_slot_pointer = reinterpret_cast<volatile uint32_t*>(aligned + kOffsetBarriers + 8 * kBarrierCount);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // Which rows of which head: heads in launch order, the long (late) query blocks of a head first.
  const int q_block = p.q_blocks - 1 - static_cast<int>(blockIdx.x % p.q_blocks);
  const int head_index = static_cast<int>(blockIdx.x / p.q_blocks);
  const int head = head_index % p.heads, batch = head_index / p.heads;
  const int q0 = q_block * kRows;
  const int key_tiles = (p.k_tokens + kKeys - 1) / kKeys;
  // under a causal mask only the key tiles that hold a key <= the CTA's last row; at least one step
  const int steps = p.causal ? min(key_tiles, (min(q0 + kRows, p.q_tokens) - 1) / kKeys + 1) : key_tiles;

  auto load_tile = [&](const CUtensorMap* map, uint32_t ring, uint32_t full, int j) {
    barrier_expect_tx(full, kTileBytes);
    for (int h = 0; h < kSubTiles; ++h)
      tma_load_4d(base + ring + (j % kRing) * kTileBytes + h * kSubTileBytes, map, full, h * kHeadDim, j * kKeys, head, batch);
  };

  // The producer lane sets the barriers up and fills the rings for the first time before the CTA meets: the
  // loads' latency runs under the tensor-memory allocation and the barrier.
  const int early = min(steps, kRing);
  if (warp == 4 && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    if (blockIdx.x == 0) p.status.begin();   // this launch's abort word starts clear
    barrier_init(q_full, 1);
    for (int s = 0; s < kRing; ++s) {
      barrier_init(k_full(s), 1);
      barrier_init(k_empty(s), 1);
      barrier_init(v_full(s), 1);
      barrier_init(v_empty(s), 1);
    }
    barrier_init(s_full, 1);
    barrier_init(pv_done, 1);
    barrier_init(p_full, kRows / 32);          // one arrival per softmax warp
    barrier_init(s_free, kRows / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    barrier_expect_tx(q_full, kSubTiles * kQueryBytes);
    for (int h = 0; h < kSubTiles; ++h) tma_load_4d(base + h * kQueryBytes, &map_q, q_full, h * kHeadDim, q0, head, batch);
    for (int j = 0; j < early; ++j) load_tile(&map_k, kOffsetK, k_full(j), j);
    for (int j = 0; j < early; ++j) load_tile(&map_v, kOffsetV, v_full(j), j);
  }
  if (warp == 5) {
    if constexpr (L::kTwoAllocations) {
      tmem_alloc_more(tmem_slot, L::kTmemColumns);
      tmem_alloc(tmem_slot + 4, kTmemColumnsP);
    } else {
      tmem_alloc(tmem_slot, L::kTmemColumns);
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_slot_pointer[0];
  const uint32_t tmem_p = L::kTwoAllocations ? tmem_slot_pointer[1] : tmem_base + L::kColumnP;

  if (L::kMovesRegisters && warp >= 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(L::kOtherRegisters));
  if (warp == 4) {
    // ---- producer: what did not fit the first filling --------------------------------------------
    if (elect_one()) {
      for (int j = early; j < steps; ++j) {
        const int s = j % kRing;
        const uint32_t phase = (j / kRing) & 1;
        if (!barrier_wait(k_empty(s), phase ^ 1, p.status, kWaitKeyEmpty)) break;
        load_tile(&map_k, kOffsetK, k_full(s), j);
        if (!barrier_wait(v_empty(s), phase ^ 1, p.status, kWaitValueEmpty)) break;
        load_tile(&map_v, kOffsetV, v_full(s), j);
      }
    }
  } else if (warp == 5) {
    // ---- issuer ----------------------------------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = attn_instruction_descriptor<T>(kKeys, false);
      constexpr uint32_t idesc_o = attn_instruction_descriptor<T>(kHeadDim, true);
      // Descriptors as (low, high) words: one constant high word, low words stepped by adds.
      constexpr uint32_t kHighWord = kDescriptorHigh;
      const uint32_t low_q = descriptor_low(base, 0), low_k = descriptor_low(base + kOffsetK, 0);
      const uint32_t low_v = descriptor_low(base + kOffsetV, kSubTileBytes);
      // S(i) = Q K_i^T: both operands K-major, 16 elements of K = 32 B in the swizzle row
      auto scores = [&](int i, uint32_t into) {
        const uint32_t k = low_k + (i % kRing) * (kTileBytes >> 4);
        // (a 128-wide head is two 64-wide sub-tiles side by side: the same steps in the second one)
#pragma unroll
        for (int h = 0; h < kSubTiles; ++h) {
#pragma unroll
          for (int kk = 0; kk < kHeadDim / 16; ++kk)
            mma_f16_split(into, low_q + h * (kQueryBytes >> 4) + kk * 2, kHighWord, k + h * (kSubTileBytes >> 4) + kk * 2, kHighWord, idesc_s,
                          (h != 0 || kk != 0) ? 1u : 0u);
        }
      };
      // O += P_i V_i (O = for the first step): P from tensor memory (16 keys = 8 columns), V MN-major
      // from shared memory (16 keys = 2048 B)
      auto partial = [&](int i) {
        const uint32_t v = low_v + (i % kRing) * (kTileBytes >> 4);
        // (a 128-wide head: the second sub-tile of V gives result columns 64..127)
#pragma unroll
        for (int h = 0; h < kSubTiles; ++h) {
#pragma unroll
          for (int kk = 0; kk < kKeys / 16; ++kk)
            mma_f16_tmem_a(tmem_base + kColumnO + h * kHeadDim, tmem_p + kk * 8, v + h * (kSubTileBytes >> 4) + kk * (2048 >> 4), kHighWord, idesc_o,
                           (i != 0 || kk != 0) ? 1u : 0u);
          if constexpr (FEW) {      // ... and what rounding took off the probabilities
#pragma unroll
            for (int kk = 0; kk < kKeys / 16; ++kk)
              mma_f16_tmem_a(tmem_base + kColumnO + h * kHeadDim, tmem_p + kKeys / 2 + kk * 8, v + h * (kSubTileBytes >> 4) + kk * (2048 >> 4), kHighWord,
                             idesc_o, 1u);
          }
        }
        mma_commit(pv_done);
      };
      if (barrier_wait(q_full, 0, p.status, kWaitQ) && barrier_wait(k_full(0), 0, p.status, kWaitKeyFull) &&
          (!kAhead || steps == 1 || barrier_wait(k_full(1), 0, p.status, kWaitKeyFull))) {
        tcgen05_fence_after();
        // (the second tile's scores too, for the reference point: into result columns, which nothing uses before the first
        // product of probabilities and values)
        scores(0, tmem_base);
        if (kAhead && steps > 1) scores(1, tmem_base + kColumnO);
        mma_commit(s_full);
        for (int i = 0; i < steps; ++i) {
          // the scores of step i + 1, once the softmax warps hold those of step i in registers
          if (i + 1 < steps) {
            if (!barrier_wait(k_full((i + 1) % kRing), ((i + 1) / kRing) & 1, p.status, kWaitKeyFull)) break;
            if (!barrier_wait(s_free, i & 1, p.status, kWaitBufferFree)) break;
            tcgen05_fence_after();
            scores(i + 1, tmem_base);
            mma_commit(s_full);
          }
          // the second product of step i, once its probabilities are in tensor memory
          if (!barrier_wait(v_full(i % kRing), (i / kRing) & 1, p.status, kWaitValueFull)) break;
          if (!barrier_wait(p_full, i & 1, p.status, kWaitProbabilities)) break;
          tcgen05_fence_after();
          partial(i);
        }
      }
    }
  } else if (warp < 4) {
    // ---- softmax: warp w owns tensor-memory lanes 32 w .. +31, one thread per query row ------------
    if constexpr (L::kMovesRegisters) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(L::kSoftmaxRegisters));
    const int query = q0 + static_cast<int>(threadIdx.x);
    const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
    const uint32_t tmem_s = tmem_base + lanes, tmem_o = tmem_base + kColumnO + lanes, tmem_mine = tmem_p + lanes;
    float reference = -INFINITY, row_sum = 0.f;     // -inf: the row has seen no finite score yet
    bool alive = true;
    const int last_allowed = p.causal ? min(query, p.k_tokens - 1) : p.k_tokens - 1;   // the last key this row may see
    const int open_until = p.causal ? min(q0, p.k_tokens - 1) : p.k_tokens - 1;         // ... and the last that every row of the CTA may

    if (FEW && q0 + warp * 32 >= p.q_tokens) {
      // A warp without a query takes part in the hand-overs only: its rows of scores and of the result mean nothing.
      for (int j = 0; alive && j < steps; ++j) {
        alive = barrier_wait(s_full, j & 1, p.status, kWaitScores);
        if (alive && lane == 0) barrier_arrive(s_free);
        if (alive && j > 0) alive = barrier_wait(pv_done, (j - 1) & 1, p.status, kWaitPartial);
        if (alive && lane == 0) barrier_arrive(p_full);
        __syncwarp();
      }
      alive = false;
    }

    // the second product of step j has finished: its probabilities and its value tile are spent
    auto wait_product = [&](int j) {
      if (!barrier_wait(pv_done, j & 1, p.status, kWaitPartial)) return false;
      tcgen05_fence_after();
      if (threadIdx.x == 0) barrier_arrive(v_empty(j % kRing));
      return true;
    };

    // One tile's scores: a row per thread, held in registers for both the maximum and the exponentials.
    using Scores = uint32_t[kKeys];
    auto load_scores = [&](Scores& r, uint32_t from) {
#pragma unroll
      for (int i = 0; i < kKeys; i += 32) tmem_load_32(from + i, *reinterpret_cast<uint32_t(*)[32]>(&r[i]));
      tmem_load_wait();
    };
    auto mask = [&](Scores& r, int key0) {
      if (key0 + kKeys - 1 > open_until) {            // uniform in the CTA
        const int limit = last_allowed - key0;        // columns > limit are masked for this row
#pragma unroll
        for (int i = 0; i < kKeys; ++i) {
          if (i > limit) r[i] = 0xff800000u;   // -inf
        }
      }
    };
    // (three-input maximum, and below two-element FMA and add: every element costs half an instruction for
    // the maximum, half for the scaling, one ex2, half for the sum and half for the rounding)
    auto maximum = [&](const Scores& r) {
      float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
      for (int i = 0; i < kKeys; i += 8) {
        m0 = max3(m0, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
        m1 = max3(m1, __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
        m2 = max3(m2, __uint_as_float(r[i + 4]), __uint_as_float(r[i + 5]));
        m3 = max3(m3, __uint_as_float(r[i + 6]), __uint_as_float(r[i + 7]));
      }
      return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
    };

    // The second tile's maximum, for the row's reference point.
    float second_max = -INFINITY;
    if (kAhead && alive && steps > 1) {
      alive = barrier_wait(s_full, 0, p.status, kWaitScores);
      if (alive) {
        Scores r;
        tcgen05_fence_after();
        load_scores(r, tmem_o);
        mask(r, kKeys);
        second_max = maximum(r);
      }
    }
    for (int j = 0; alive && j < steps; ++j) {
      if (!barrier_wait(s_full, j & 1, p.status, kWaitScores)) { alive = false; break; }
      tcgen05_fence_after();
      if (threadIdx.x == 0) barrier_arrive(k_empty(j % kRing));      // the first product has read key tile j
      Scores r;
      load_scores(r, tmem_s);         // the columns go back to the issuer at once
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) barrier_arrive(s_free);
      mask(r, j * kKeys);
      const float tile_max = maximum(r);
      // The reference point: the first two tiles' maximum, moved only when a tile rises more than
      // 2^kSlack above it (from -inf, any finite maximum does). `factor` rescales what the row has
      // gathered so far; it is 1 for a row that stays.
      float factor = 1.f;
      const bool moves = j == 0 || (tile_max - reference) * p.scale_log2 > kSlack;       // false for NaN
      if (moves) {
        if (j != 0) factor = exp2_ftz((reference - tile_max) * p.scale_log2);             // from -inf: 0, and nothing was gathered
        reference = j == 0 ? fmaxf(tile_max, second_max) : tile_max;
      }
      const bool rescale = j != 0 && __any_sync(0xffffffffu, moves);
      const float shift = reference == -INFINITY ? 0.f : -reference * p.scale_log2;       // all scores -inf so far: every probability is 0

      // probabilities and their sum; the probabilities go into tensor memory as the A operand of the second
      // product (16-bit pairs)
      float2 sum0 = make_float2(0.f, 0.f), sum1 = sum0;
      uint32_t packed[kKeys / 2], rest[FEW ? kKeys / 2 : 1];
      const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), shift2 = make_float2(shift, shift);
#pragma unroll
      for (int chunk = 0; chunk < kKeys / 4; ++chunk) {
        const float2 t0 = __ffma2_rn(make_float2(__uint_as_float(r[chunk * 4 + 0]), __uint_as_float(r[chunk * 4 + 1])), scale2, shift2);
        const float2 t1 = __ffma2_rn(make_float2(__uint_as_float(r[chunk * 4 + 2]), __uint_as_float(r[chunk * 4 + 3])), scale2, shift2);
        const float2 e0 = make_float2(exp2_ftz(t0.x), exp2_ftz(t0.y));
        const float2 e1 = make_float2(exp2_ftz(t1.x), exp2_ftz(t1.y));
        sum0 = __fadd2_rn(sum0, e0);
        sum1 = __fadd2_rn(sum1, e1);
        packed[chunk * 2 + 0] = pack_pair<T>(e0.x, e0.y);
        packed[chunk * 2 + 1] = pack_pair<T>(e1.x, e1.y);
        if constexpr (FEW) {
          rest[chunk * 2 + 0] = pack_rest<T>(packed[chunk * 2 + 0], e0);
          rest[chunk * 2 + 1] = pack_rest<T>(packed[chunk * 2 + 1], e1);
        }
      }
      const float2 sum01 = __fadd2_rn(sum0, sum1);
      row_sum = row_sum * factor + (sum01.x + sum01.y);

      // The previous step's product still reads the probability columns and adds into the result: wait for it
      // (it had this step's loads and exponentials to finish), then write.
      if (j > 0) {
        if (!wait_product(j - 1)) { alive = false; break; }
        if (rescale) {       // rare: some row of this warp moved its reference point
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {      // sixteen result columns at a time: the probabilities are still in registers
            uint32_t o[16];
            tmem_load_16(tmem_o + c * 16, o);
            tmem_load_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
            tmem_store_16(tmem_o + c * 16, o);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kKeys / 2; i += 32) {
        tmem_store_32(tmem_mine + i, *reinterpret_cast<uint32_t(*)[32]>(&packed[i]));
        if constexpr (FEW) tmem_store_32(tmem_mine + kKeys / 2 + i, *reinterpret_cast<uint32_t(*)[32]>(&rest[i]));
      }
      tmem_store_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) barrier_arrive(p_full);
    }

    if (alive && wait_product(steps - 1)) {
      // the result row leaves tensor memory 32 columns at a time (the loads are warp-wide: every lane takes
      // part, rows beyond the queries only skip the stores)
      const bool stores = query < p.q_tokens;
      const float inverse = 1.0f / row_sum;
      T* out_row = static_cast<T*>(p.out) + batch * p.out_batch + head * p.out_head + static_cast<long long>(query) * p.out_token;
      const bool vector_ok = (reinterpret_cast<uintptr_t>(out_row) & 15) == 0;
      const int width = p.head_dim;       // a multiple of 8: whole 16-byte vectors
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        if (c * 32 >= width) break;
        uint32_t o[32];
        tmem_load_32(tmem_o + c * 32, o);
        tmem_load_wait();
        if (stores && vector_ok) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (c * 32 + v * 8 < width) {
              uint4 word;
              word.x = pack_pair<T>(__uint_as_float(o[v * 8 + 0]) * inverse, __uint_as_float(o[v * 8 + 1]) * inverse);
              word.y = pack_pair<T>(__uint_as_float(o[v * 8 + 2]) * inverse, __uint_as_float(o[v * 8 + 3]) * inverse);
              word.z = pack_pair<T>(__uint_as_float(o[v * 8 + 4]) * inverse, __uint_as_float(o[v * 8 + 5]) * inverse);
              word.w = pack_pair<T>(__uint_as_float(o[v * 8 + 6]) * inverse, __uint_as_float(o[v * 8 + 7]) * inverse);
              *reinterpret_cast<uint4*>(out_row + c * 32 + v * 8) = word;
            }
          }
        } else if (stores) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (c * 32 + i < width) out_row[c * 32 + i] = from_compute<T, float>(__uint_as_float(o[i]) * inverse);
          }
        }
        __syncwarp();
      }
    }
  }

  // ---- teardown: every thread arrives here, also after a wait that gave up -------------------
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 5) {
    tcgen05_fence_after();
    if constexpr (L::kTwoAllocations) tmem_dealloc(tmem_p, kTmemColumnsP);
    tmem_dealloc(tmem_base, L::kTmemColumns);
  }
}

// A four-axis map over one of Q, K, V: `head_dim` contiguous elements, then tokens, heads, batch with
// the caller's element strides; box = 64 x `rows` x 1 x 1 (128 queries, or a step's keys), 128-byte swizzle. Rows beyond the tokens read
// 0, and so do the columns beyond a head narrower than its tiles: zeros add nothing to q . k and give
// result columns nobody stores, so a narrow head runs through the same 64-wide tiles.
tq_status attention_map(CUtensorMap* map, tq_dtype dtype, const void* pointer, long long head_dim, long long tokens, long long heads,
                        long long batch, const int64_t* strides, int rows) {
  EncodeTiled encode = encode_tiled();
  TQ_REQUIRE(encode != nullptr, TQ_EXTERNAL, "the CUDA driver does not provide cuTensorMapEncodeTiled");
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(head_dim), static_cast<cuuint64_t>(tokens), static_cast<cuuint64_t>(heads),
                              static_cast<cuuint64_t>(batch)};
  // an axis of extent 1 never moves, so its stride only has to be legal
  const long long token_stride = tokens > 1 ? strides[2] : head_dim;
  const long long head_stride = heads > 1 ? strides[1] : head_dim;
  const long long batch_stride = batch > 1 ? strides[0] : head_dim;
  const cuuint64_t byte_strides[3] = {static_cast<cuuint64_t>(token_stride) * 2, static_cast<cuuint64_t>(head_stride) * 2,
                                      static_cast<cuuint64_t>(batch_stride) * 2};
  const cuuint32_t box[4] = {static_cast<cuuint32_t>(kHeadDim), static_cast<cuuint32_t>(rows), 1, 1};
  const cuuint32_t element_strides[4] = {1, 1, 1, 1};
  const CUresult result = encode(map, dtype == TQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                                 const_cast<void*>(pointer), dims, byte_strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TQ_REQUIRE(result == CUDA_SUCCESS, TQ_UNSUPPORTED, "this operand layout cannot be described to TMA (driver code %d)", static_cast<int>(result));
  return TQ_OK;
}

bool legal_strides(const void* pointer, const int64_t* strides, long long head_dim, long long tokens, long long heads, long long batch) {
  if (!aligned_to(pointer, 16)) return false;
  if (tokens > 1 && (strides[2] < head_dim || strides[2] % 8 != 0)) return false;
  if (heads > 1 && (strides[1] <= 0 || strides[1] % 8 != 0)) return false;
  if (batch > 1 && (strides[0] <= 0 || strides[0] % 8 != 0)) return false;
  return true;
}

}  // namespace

// decode.cu
tq_status attention_decode(tq_dtype dtype, const void* q, const void* k, const void* v, void* out, long long batch, long long heads,
                           long long q_tokens, long long k_tokens, long long head_dim, const int64_t* q_strides, const int64_t* k_strides,
                           const int64_t* v_strides, const int64_t* out_strides, float scale_log2, bool causal, int32_t device, cudaStream_t stream);
constexpr int kDecodeQueries = 4;

struct AttentionForm {
  bool decode;      // decode.cu
  int keys;         // keys a step of the tensor-core kernel
  bool few;         // its form for a few queries
};

// Kernel times (graphs of launches over rotating operands, B200, bf16, us) behind the rules. `heads` is batch times heads.
//
// One to four queries: streaming the keys (decode.cu) costs multiply-adds per query, the tensor cores' few-query form does not, but
// it walks a head's keys in one CTA. Four queries of 64 x 12 heads over 1000 keys: heads of 64 streamed 73, few 53; heads of 128
// 143 and 74; two queries of heads of 128 85 and 74, one 75 and 74; but over 100 keys, heads of 64, 14.0 and 17. Where heads do
// not fill the SMs a head's keys are shared when streamed: four queries of 8 heads of 128 over 4000 keys 36 and 47, of 96 heads
// 80 and 50. From there to one head an SM clusters of four no longer fit: one query, 144 heads of 96, 4000 keys 57 and 53.
//
// More queries: 128 keys a step halve the hand-overs of a chain, but only two CTAs share an SM (one for heads above 64)
// where 64 keys let three (two). 1 x 8 x 4096 causal 68.9 with 64, 54.4 with 128; 64 x 12 x 1024 causal 228.7 and 228.7; 5 ... 9 waves
// of 200 to 256 tokens 0 - 4 % better with 64; 64 x 6 x 1024 of 128 174.7 and 225. Without a mask, CTAs that fit
// three an SM but not two are one wave with 64 (384 CTAs over 4096 keys 90.6 and 92.9). Half of a 128-key step may be empty: of the only
// one (64 x 12 x 64 11.4 and 15.5) or of the last (without a mask 64 x 12 x 700 185.4 and 204).
AttentionForm choose_attention_form(long long heads, long long q_tokens, long long k_tokens, long long head_dim, bool causal, long long sms) {
  const bool wide = head_dim > kHeadDim;
  if (q_tokens <= kDecodeQueries) {
    const long long keys = causal && q_tokens < k_tokens ? q_tokens : k_tokens;       // that any query sees
    const bool no_fours = heads * 25 > sms * 24;                                    // clusters of four: 142 of them on 148 SMs
    if (heads > sms) {
      const long long enough = q_tokens >= 3 ? (wide ? heads / 4 : heads / 2) : heads;
      if ((wide ? q_tokens >= 2 : q_tokens >= 3) && keys >= enough && keys >= 64) return {false, 64, true};
    } else if (keys > kHeadDim) {
      const bool half = heads * 2 > sms;
      const bool many = q_tokens >= 3 && (wide ? half || keys <= 512 : keys <= 128 || (half && keys <= 300) || no_fours);
      if (many || (wide && no_fours && keys >= 256)) return {false, 128, true};
    }
    return {true, 0, false};
  }
  const long long ctas = heads * ((q_tokens + kRows - 1) / kRows);
  if (k_tokens <= 64) return {false, 64, false};
  if (wide) return {false, ctas <= sms ? 128 : 64, false};
  const bool thirds = !causal && ctas > 2 * sms && ctas <= 3 * sms;
  const bool half_step = !causal && k_tokens < 1280 && (k_tokens + 63) / 64 % 2 == 1;
  return {false, ctas <= 2 * sms || (k_tokens >= 512 && !thirds && !half_step) ? 128 : 64, false};
}

}  // namespace tq

extern "C" tq_status tq_attention_form(int64_t heads, int64_t q_tokens, int64_t k_tokens, int64_t head_dim, int32_t causal, int32_t device, int32_t* form,
                                       int32_t* keys) {
  TQ_REQUIRE(form != nullptr && keys != nullptr, TQ_INVALID_ARGUMENT, "null out-pointer");
  TQ_REQUIRE(heads > 0 && q_tokens > 0 && k_tokens > 0, TQ_INVALID_ARGUMENT, "extents must be positive, not heads=%lld q_tokens=%lld k_tokens=%lld",
             (long long)heads, (long long)q_tokens, (long long)k_tokens);
  TQ_REQUIRE(head_dim >= 8 && head_dim <= 2 * tq::kHeadDim && head_dim % 8 == 0, TQ_UNSUPPORTED,
             "fused attention has a kernel for heads of 8, 16, ... %d elements, not %lld", 2 * tq::kHeadDim, (long long)head_dim);
  const tq::AttentionForm chosen = tq::choose_attention_form(heads, q_tokens, k_tokens, head_dim, causal != 0, device < 0 ? 148 : tq::sm_count(device));
  *form = chosen.decode ? TQ_ATTENTION_STREAMED : chosen.few ? TQ_ATTENTION_TILES_FEW : TQ_ATTENTION_TILES;
  *keys = chosen.keys;
  return TQ_OK;
}

extern "C" tq_status tq_attention_launch(tq_dtype dtype, const void* q, const void* k, const void* v, void* out, int64_t batch,
                                         int64_t heads, int64_t q_tokens, int64_t k_tokens, int64_t head_dim,
                                         const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides,
                                         const int64_t* out_strides, double scale, int32_t causal, int32_t device, void* stream) {
  TQ_REQUIRE(q_strides != nullptr && k_strides != nullptr && v_strides != nullptr && out_strides != nullptr, TQ_INVALID_ARGUMENT,
             "null strides");
  if (tq::recording()) {
    struct Kept { int64_t q[3], k[3], v[3], out[3]; } kept;
    for (int i = 0; i < 3; ++i) {
      kept.q[i] = q_strides[i];
      kept.k[i] = k_strides[i];
      kept.v[i] = v_strides[i];
      kept.out[i] = out_strides[i];
    }
    return tq::record([=](int32_t d, void* s) {
      return tq_attention_launch(dtype, q, k, v, out, batch, heads, q_tokens, k_tokens, head_dim, kept.q, kept.k, kept.v, kept.out,
                                 scale, causal, d, s);
    });
  }
  TQ_REQUIRE(dtype == TQ_BF16 || dtype == TQ_F16, TQ_UNSUPPORTED, "fused attention takes bf16 or f16 operands, not %s",
             tq::dtype_name(dtype));
  TQ_REQUIRE(batch >= 0 && heads >= 0 && q_tokens >= 0 && k_tokens >= 0, TQ_INVALID_ARGUMENT,
             "negative extent in batch=%lld heads=%lld q_tokens=%lld k_tokens=%lld", (long long)batch, (long long)heads,
             (long long)q_tokens, (long long)k_tokens);
  TQ_REQUIRE(head_dim >= 8 && head_dim <= 2 * tq::kHeadDim && head_dim % 8 == 0, TQ_UNSUPPORTED,
             "fused attention has a kernel for heads of 8, 16, ... %d elements, not %lld", 2 * tq::kHeadDim, (long long)head_dim);
  if (batch == 0 || heads == 0 || q_tokens == 0) return TQ_OK;
  TQ_REQUIRE(k_tokens > 0, TQ_UNSUPPORTED, "a softmax over no keys has no kernel");
  TQ_REQUIRE(std::isfinite(scale) && scale > 0.0, TQ_UNSUPPORTED, "the score scale must be positive and finite, not %g", scale);
  TQ_REQUIRE(q != nullptr && k != nullptr && v != nullptr && out != nullptr, TQ_INVALID_ARGUMENT, "null operand or result");
  TQ_REQUIRE(q_tokens < (1LL << 30) && k_tokens < (1LL << 30) && heads < 65536 && batch * heads < (1LL << 24), TQ_UNSUPPORTED,
             "extents beyond the kernel's index range");
  TQ_REQUIRE(tq::legal_strides(q, q_strides, head_dim, q_tokens, heads, batch) && tq::legal_strides(k, k_strides, head_dim, k_tokens, heads, batch) &&
                 tq::legal_strides(v, v_strides, head_dim, k_tokens, heads, batch),
             TQ_UNSUPPORTED, "Q, K and V must be 16-byte aligned with positive strides that are multiples of 8 elements (TMA's rules)");
  TQ_REQUIRE(tq::aligned_to(out, 2) && out_strides[0] >= 0 && out_strides[1] >= 0 && out_strides[2] >= 0, TQ_INVALID_ARGUMENT,
             "misaligned result or negative result stride");
  tq::DeviceScope device_scope(device);
  if (tq_status s = device_scope.status()) return s;
  const bool wide = head_dim > tq::kHeadDim;             // two sub-tiles side by side
  const tq::AttentionForm form = tq::choose_attention_form(batch * heads, q_tokens, k_tokens, head_dim, causal != 0, tq::sm_count(device));
  // (The decoding form's batch * heads * split CTAs stay below 2^28.)
  if (form.decode) {
    return tq::attention_decode(dtype, q, k, v, out, batch, heads, q_tokens, k_tokens, head_dim, q_strides, k_strides, v_strides, out_strides,
                                static_cast<float>(scale * 1.4426950408889634), causal != 0, device, static_cast<cudaStream_t>(stream));
  }
  const tq::WaitStatus status = tq::wait_status_for(device);
  TQ_REQUIRE(status.abort != nullptr, TQ_RESOURCE_EXHAUSTED, "no device memory for the status word");

  CUtensorMap map_q, map_k, map_v;
  if (tq_status s = tq::attention_map(&map_q, dtype, q, head_dim, q_tokens, heads, batch, q_strides, tq::kRows)) return s;
  if (tq_status s = tq::attention_map(&map_k, dtype, k, head_dim, k_tokens, heads, batch, k_strides, form.keys)) return s;
  if (tq_status s = tq::attention_map(&map_v, dtype, v, head_dim, k_tokens, heads, batch, v_strides, form.keys)) return s;

  tq::AttnParams p = {};
  p.batch = static_cast<int>(batch);
  p.heads = static_cast<int>(heads);
  p.q_tokens = static_cast<int>(q_tokens);
  p.k_tokens = static_cast<int>(k_tokens);
  p.head_dim = static_cast<int>(head_dim);
  p.q_blocks = static_cast<int>((q_tokens + tq::kRows - 1) / tq::kRows);
  p.causal = causal != 0;
  p.scale_log2 = static_cast<float>(scale * 1.4426950408889634);
  p.out = out;
  p.out_batch = out_strides[0];
  p.out_head = out_strides[1];
  p.out_token = out_strides[2];
  p.status = status;
  const long long ctas = static_cast<long long>(p.q_blocks) * heads * batch;
  TQ_REQUIRE(ctas < (1LL << 31), TQ_UNSUPPORTED, "too many query blocks for one launch");
  cudaStream_t cuda_stream = static_cast<cudaStream_t>(stream);
  auto go = [&](auto width, auto keys, auto few) -> tq_status {
    constexpr int kWidth = decltype(width)::value, kKeys = decltype(keys)::value;
    constexpr bool kFew = decltype(few)::value;
    constexpr size_t smem = tq::AttnLayout<kWidth, kKeys, kFew>::kSmemBytes;
    auto start = [&](auto kernel) -> tq_status {
      TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
      kernel<<<static_cast<unsigned>(ctas), tq::kAttnThreads, smem, cuda_stream>>>(map_q, map_k, map_v, p);
      return tq::check_launch("attention_kernel");
    };
    if (dtype == TQ_BF16) return start(tq::attention_kernel<__nv_bfloat16, kWidth, kKeys, kFew>);
    return start(tq::attention_kernel<__half, kWidth, kKeys, kFew>);
  };
  auto with_width = [&](auto keys, auto few) {
    return wide ? go(std::integral_constant<int, 2 * tq::kHeadDim>{}, keys, few) : go(std::integral_constant<int, tq::kHeadDim>{}, keys, few);
  };
  auto with_keys = [&](auto few) {
    return form.keys == 128 ? with_width(std::integral_constant<int, 128>{}, few) : with_width(std::integral_constant<int, 64>{}, few);
  };
  return form.few ? with_keys(std::true_type{}) : with_keys(std::false_type{});
}
