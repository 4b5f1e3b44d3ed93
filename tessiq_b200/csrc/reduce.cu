// Reductions over a packed [outer, reduce, inner] view: sum, mean, amax, amin, argmax.
//
// Three kernel shapes, chosen on the host by plan():
//   warp-per-slice   inner == 1, many slices of moderate length: each warp streams one slice with
//                    128-bit loads and finishes with shuffles; no shared memory, no barrier.
//   cta-per-slice    inner == 1, long or few slices: `split` CTAs stream one slice; warp shuffle,
//                    then shared memory, then distributed shared memory across the thread-block
//                    cluster, then (only when a slice spans more than one cluster) per-cluster
//                    partials in scratch memory that the last cluster to arrive combines.
//   columns          inner > 1: threads run along `inner` (coalesced), warps along `reduce`;
//                    the same cluster / scratch steps when `reduce` is split.
// No wait anywhere: the "last to arrive" step uses a ticket, not a spin.
//
// Semantics follow the reference's reduction kernels (csrc/tessiq/codegen/cuda_emitter.cpp:159-210):
// mean divides once after the sum, amax/amin propagate NaN. argmax returns the first index of the
// maximum with NaN counted as the maximum, which is what aten.argmax computes on the reference's
// host device.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <limits>
#include <mutex>
#include <type_traits>

#include "common.h"
#include "reducers.h"
#include "tcgen05.h"

namespace cg = cooperative_groups;

namespace tq {
namespace {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
constexpr int kUnroll = 4;
constexpr int kMaxCluster = 8;
constexpr int kRingDepth = 8;   // columns kernel: rows in flight per thread (cp.async ring)

// ---------------------------------------------------------------------------------------------
// Reducers

template <typename T>
struct SumReducer {
  static constexpr bool kSeeded = false;   // no seed / step_seeded / set_count protocol (see MomentsReducer)
  using C = typename Compute<T>::type;
  using Acc = std::conditional_t<std::is_integral_v<C>, long long, C>;
  using Out = std::conditional_t<std::is_same_v<T, int>, long long, T>;
  __device__ static Acc identity() { return Acc(0); }
  __device__ static Acc lift(T v, long long) { return static_cast<Acc>(to_compute(v)); }
  __device__ static Acc combine(Acc a, Acc b) { return a + b; }
  __device__ static Acc shuffle(Acc a, int offset) { return shfl_xor(a, offset); }
  template <int VEC> using Local = Acc;
  template <int VEC> __device__ static Acc local_identity() { return identity(); }
  template <int VEC> __device__ static void step(Acc& local, T v, long long) { local += static_cast<Acc>(to_compute(v)); }
  // (a vector is summed in a tree of its own first: few lanes a slice make a lane's chain of additions long, which sums of
  // 32 bits show; 16-bit results are rounded far above it)
  template <int VEC> __device__ static void step_vector(Acc& local, const Vec<T, VEC>& x, long long) {
    if constexpr (sizeof(T) == 2) {
#pragma unroll
      for (int e = 0; e < VEC; ++e) local += static_cast<Acc>(to_compute(x.v[e]));
    } else {
      Acc part[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) part[e] = static_cast<Acc>(to_compute(x.v[e]));
#pragma unroll
      for (int width = VEC / 2; width > 0; width /= 2) {
#pragma unroll
        for (int e = 0; e < width; ++e) part[e] += part[e + width];
      }
      local += part[0];
    }
  }
  // Two rows, or four, of neighbouring columns: added to one another first (floating types of 32 and 64 bits).
  static constexpr bool kPairs = std::is_floating_point_v<T>;
  template <int V> __device__ static void step_pair(Acc* local, const Vec<T, V>& a, const Vec<T, V>& b) {
#pragma unroll
    for (int e = 0; e < V; ++e) local[e] += static_cast<Acc>(to_compute(a.v[e])) + static_cast<Acc>(to_compute(b.v[e]));
  }
  template <int V> __device__ static void step_four(Acc* local, const Vec<T, V> (&x)[4]) {
#pragma unroll
    for (int e = 0; e < V; ++e)
      local[e] += (static_cast<Acc>(to_compute(x[0].v[e])) + static_cast<Acc>(to_compute(x[1].v[e]))) +
                  (static_cast<Acc>(to_compute(x[2].v[e])) + static_cast<Acc>(to_compute(x[3].v[e])));
  }
  template <int V> __device__ static void step_single(Acc* local, const Vec<T, V>& a) {
#pragma unroll
    for (int e = 0; e < V; ++e) local[e] += static_cast<Acc>(to_compute(a.v[e]));
  }
  template <int VEC> __device__ static Acc to_acc(Acc local) { return local; }
  __device__ static Out finish(Acc a, long long count, bool mean) {
    if constexpr (!std::is_integral_v<C>) {
      if (mean) a = a / static_cast<Acc>(count);
      return from_compute<Out, Acc>(a);
    } else {
      return static_cast<Out>(a);
    }
  }
};


template <typename C>
struct alignas(16) Indexed {
  C value;
  long long index;
};

template <typename T>
struct ArgmaxReducer {
  static constexpr bool kSeeded = false;   // no seed / step_seeded / set_count protocol (see MomentsReducer)
  using C = typename Compute<T>::type;
  using Acc = Indexed<C>;
  using Out = long long;
  __device__ static Acc identity() {
    Acc a;
    if constexpr (std::is_integral_v<C>) {
      a.value = std::numeric_limits<C>::lowest();
    } else {
      a.value = -std::numeric_limits<C>::infinity();
    }
    a.index = std::numeric_limits<long long>::max();
    return a;
  }
  __device__ static Acc lift(T v, long long index) {
    Acc a;
    a.value = to_compute(v);
    a.index = index;
    return a;
  }
  // A total order: NaN above everything, then the value, then the lower index.
  __device__ static Acc combine(Acc a, Acc b) {
    bool a_nan = false, b_nan = false;
    if constexpr (!std::is_integral_v<C>) {
      a_nan = a.value != a.value;
      b_nan = b.value != b.value;
    }
    bool take_b;
    if (a_nan || b_nan) {
      take_b = (a_nan && b_nan) ? (b.index < a.index) : b_nan;
    } else if (a.value == b.value) {
      take_b = b.index < a.index;
    } else {
      take_b = b.value > a.value;
    }
    return take_b ? b : a;
  }
  __device__ static Acc shuffle(Acc a, int offset) {
    Acc b;
    b.value = shfl_xor(a.value, offset);
    b.index = shfl_xor(a.index, offset);
    return b;
  }
  // Within one thread the positions only grow, so a strict comparison keeps the first of equal
  // values and the thread needs no index comparison. A thread looks at one vector at a time: the
  // vector's NaN-propagating maximum (packed two-at-a-time for the half types) is compared with
  // the best so far, and a vector that beats it is kept whole together with its position; which
  // element of the kept vector won is resolved once, at the end. Positions are kept in 32 bits
  // (the host declines longer slices). `!(m <= best)` is true for a larger value and for a NaN;
  // the second test freezes the state once `best` itself is a NaN.
  template <int VEC>
  struct Local {
    C best;
    unsigned base;
    Vec<T, VEC> winner;
  };
  static constexpr unsigned kNone = 0xffffffffu;
  template <int VEC> __device__ static Local<VEC> local_identity() {
    Local<VEC> l;
    l.best = identity().value;
    l.base = kNone;
#pragma unroll
    for (int e = 0; e < VEC; ++e) l.winner.v[e] = T();
    return l;
  }
  __device__ static bool beats(C value, C best) {
    if constexpr (std::is_integral_v<C>) {
      return value > best;
    } else {
      return !(value <= best) && (best == best);
    }
  }
  template <int VEC> __device__ static void step(Local<VEC>& local, T v, long long index) {
    const C value = to_compute(v);
    if (beats(value, local.best)) {
      local.best = value;
      local.base = static_cast<unsigned>(index);
#pragma unroll
      for (int e = 0; e < VEC; ++e) local.winner.v[e] = v;
    }
  }
  // (Testing once per row of V neighbouring columns whether any of them beats its best, as the softmax
  // statistics do, measured 123 us against 86 at [32768, 4096]: a column of random values has a new
  // maximum in about ln(n) of its n rows, and with 32 lanes x V columns per warp nearly every row has one
  // somewhere in the warp, so the rare path ran for every row.)
  template <int VEC> __device__ static C vector_max(const Vec<T, VEC>& x) {
    if constexpr (std::is_same_v<T, __nv_bfloat16> && VEC % 2 == 0) {
      const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&x);
      __nv_bfloat162 m = pairs[0];
#pragma unroll
      for (int i = 1; i < VEC / 2; ++i) m = __hmax2_nan(m, pairs[i]);
      return ExtremeReducer<float, true>::combine(__low2float(m), __high2float(m));
    } else if constexpr (std::is_same_v<T, __half> && VEC % 2 == 0) {
      const __half2* pairs = reinterpret_cast<const __half2*>(&x);
      __half2 m = pairs[0];
#pragma unroll
      for (int i = 1; i < VEC / 2; ++i) m = __hmax2_nan(m, pairs[i]);
      return ExtremeReducer<float, true>::combine(__low2float(m), __high2float(m));
    } else {
      C m = to_compute(x.v[0]);
#pragma unroll
      for (int e = 1; e < VEC; ++e) m = ExtremeReducer<C, true>::combine(m, to_compute(x.v[e]));
      return m;
    }
  }
  template <int VEC> __device__ static void step_vector(Local<VEC>& local, const Vec<T, VEC>& x, long long index) {
    const C m = vector_max<VEC>(x);
    if (beats(m, local.best)) {
      local.best = m;
      local.base = static_cast<unsigned>(index);
      local.winner = x;
    }
  }
  template <int VEC> __device__ static Acc to_acc(const Local<VEC>& local) {
    Acc a;
    a.value = local.best;
    a.index = std::numeric_limits<long long>::max();
    if (local.base != kNone) {
      int offset = 0;
#pragma unroll
      for (int e = VEC - 1; e >= 0; --e) {
        const C w = to_compute(local.winner.v[e]);
        const bool same = (w == local.best) || (w != w && local.best != local.best);
        if (same) offset = e;
      }
      a.index = static_cast<long long>(local.base) + offset;
    }
    return a;
  }
  // No position was ever taken only if every element equals the identity (-inf, or the lowest
  // integer): the first of equal values is position 0.
  __device__ static Out finish(Acc a, long long, bool) {
    return a.index == std::numeric_limits<long long>::max() ? 0 : a.index;
  }
};



// The local part of a reduction over a tensor that is split over several GPUs (collective.cu): the
// result is a two-float partial that an all-reduce can combine. A sum's partial is {sum in f32, 0}
// (the f32 accumulator itself: a bf16 tensor's partial is not rounded to bf16 first).
template <typename T>
struct SumPartialReducer : SumReducer<T> {
  using Out = float2;
  using Acc = typename SumReducer<T>::Acc;
  __device__ static Out finish(Acc a, long long, bool) { return make_float2(static_cast<float>(a), 0.f); }
};

// A maximum's partial is {maximum with a NaN replaced by -inf, 1 if a NaN was seen}, to be combined
// with MAX on both words; a minimum's {minimum with a NaN replaced by +inf, -1 if a NaN was seen},
// combined with MIN: a collective's maximum does not promise to propagate NaN, the flag does.
template <typename T, bool kMax>
struct ExtremePartialReducer : ExtremeReducer<T, kMax> {
  using Out = float2;
  using Acc = typename ExtremeReducer<T, kMax>::Acc;
  __device__ static Out finish(Acc a, long long, bool) {
    const float value = static_cast<float>(a);
    if (value != value) return make_float2(kMax ? -std::numeric_limits<float>::infinity() : std::numeric_limits<float>::infinity(), kMax ? 1.f : -1.f);
    return make_float2(value, 0.f);
  }
};

// Reads a partial another CTA wrote, from L2 (never a stale L1 line).
template <typename A>
__device__ __forceinline__ A load_partial(const A* pointer) {
  if constexpr (sizeof(A) == 16) {
    uint4 raw = __ldcg(reinterpret_cast<const uint4*>(pointer));
    return *reinterpret_cast<A*>(&raw);
  } else if constexpr (sizeof(A) == 8) {
    unsigned long long raw = __ldcg(reinterpret_cast<const unsigned long long*>(pointer));
    return *reinterpret_cast<A*>(&raw);
  } else {
    static_assert(sizeof(A) == 4, "accumulators are 4, 8 or 16 bytes");
    unsigned raw = __ldcg(reinterpret_cast<const unsigned*>(pointer));
    return *reinterpret_cast<A*>(&raw);
  }
}

// Over each aligned set of LANES lanes of the warp.
template <typename R, int LANES = 32>
__device__ __forceinline__ typename R::Acc warp_reduce(typename R::Acc a) {
#pragma unroll
  for (int offset = LANES / 2; offset > 0; offset >>= 1) a = R::combine(a, R::shuffle(a, offset));
  return a;
}

// All threads call; the result is valid on thread 0.
template <typename R>
__device__ __forceinline__ typename R::Acc block_reduce(typename R::Acc a, typename R::Acc* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  a = warp_reduce<R>(a);
  __syncthreads();  // scratch may still be read from an earlier use
  if (lane == 0) scratch[warp] = a;
  __syncthreads();
  if (warp == 0) {
    a = lane < kWarps ? scratch[lane] : R::identity();
    a = warp_reduce<R>(a);
  }
  return a;
}

// Folds elements [begin, end) of `row` into `acc`, `threads` threads cooperating, this one being
// `tid`. The span is cut into a scalar head up to the first 16-byte boundary, a body of VEC-wide
// streaming loads, and a scalar tail, so that any element-aligned pointer works.
template <typename T, typename R, int VEC>
__device__ __forceinline__ void fold_span(const T* __restrict__ row, long long begin, long long end,
                                          int tid, int threads, typename R::template Local<VEC>& acc) {
  if (begin >= end) return;
  const T* start = row + begin;
  long long head = 0;
  if constexpr (VEC > 1) {
    const unsigned misaligned =
        static_cast<unsigned>(reinterpret_cast<uintptr_t>(start) % (sizeof(T) * VEC)) / sizeof(T);
    head = misaligned ? (VEC - misaligned) : 0;
    if (head > end - begin) head = end - begin;
    if (tid < head) R::template step<VEC>(acc, start[tid], begin + tid);
  }
  const long long body = begin + head;
  const long long vectors = (end - body) / VEC;
  const T* vector_base = row + body;
  for (long long v = tid; v < vectors; v += static_cast<long long>(threads) * kUnroll) {
    Vec<T, VEC> x[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long vi = v + static_cast<long long>(u) * threads;
      if (vi < vectors) x[u] = load_stream<T, VEC>(vector_base + vi * VEC);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long vi = v + static_cast<long long>(u) * threads;
      if (vi < vectors) R::template step_vector<VEC>(acc, x[u], body + vi * VEC);
    }
  }
  const long long tail = body + vectors * VEC + tid;
  if (tail < end) R::template step<VEC>(acc, row[tail], tail);
}

// ---------------------------------------------------------------------------------------------
// Kernels

// LANES lanes per slice: a warp, or eight or sixteen lanes for short slices, of which a warp then has four or two
// under way where one of 256 bytes left it with half its lanes idle: 10^6 x 64 f32 sum 187 us with 32 lanes, 53 with
// eight (bytes: 40). (Eight is also as many lanes as a slice can have elements before its first vector.)
// grid.x * kBlock / LANES >= outer.
template <typename T, typename R, int VEC, int LANES>
__global__ void __launch_bounds__(kBlock)
reduce_warp_per_slice(const T* __restrict__ in, typename R::Out* __restrict__ out, long long outer,
                      long long reduce, int mean) {
  static_assert(LANES >= VEC, "a slice's head and tail are one element per lane");
  const int lane = threadIdx.x % LANES;
  const long long slice = static_cast<long long>(blockIdx.x) * (kBlock / LANES) + threadIdx.x / LANES;
  if (LANES == 32 && slice >= outer) return;
  typename R::template Local<VEC> local = R::template local_identity<VEC>();
  // (lanes without a slice stay for the shuffles)
  if (LANES == 32 || slice < outer) fold_span<T, R, VEC>(in + slice * reduce, 0, reduce, lane, LANES, local);
  __syncwarp();
  typename R::Acc acc = warp_reduce<R, LANES>(R::template to_acc<VEC>(local));
  if (lane == 0 && (LANES == 32 || slice < outer)) out[slice] = R::finish(acc, reduce, mean != 0);
}

// `split` CTAs per slice, `cluster` of them in one thread-block cluster (cluster divides split).
// blockIdx.x = slice * split + part.
template <typename T, typename R, int VEC>
__global__ void __launch_bounds__(kBlock)
reduce_cta_per_slice(const T* __restrict__ in, typename R::Out* __restrict__ out, long long reduce,
                     int split, int cluster, int mean, typename R::Acc* __restrict__ partials,
                     unsigned* __restrict__ tickets) {
  using Acc = typename R::Acc;
  __shared__ Acc warp_scratch[kWarps];
  __shared__ Acc cluster_scratch[kMaxCluster];
  __shared__ bool is_last;

  const long long slice = blockIdx.x / split;
  const int part = static_cast<int>(blockIdx.x % split);
  // Parts are cut on multiples of the vector width so that only the first can be misaligned.
  long long chunk = (reduce + split - 1) / split;
  chunk = (chunk + VEC - 1) / VEC * VEC;
  const long long begin = static_cast<long long>(part) * chunk;
  long long end = begin + chunk;
  if (end > reduce) end = reduce;

  if (cluster > 1) cluster_start();
  typename R::template Local<VEC> local = R::template local_identity<VEC>();
  fold_span<T, R, VEC>(in + slice * reduce, begin, end, threadIdx.x, kBlock, local);
  Acc acc = block_reduce<R>(R::template to_acc<VEC>(local), warp_scratch);

  if (cluster > 1) {
    cg::cluster_group group = cg::this_cluster();
    const unsigned rank = group.block_rank();
    cluster_started();
    if (threadIdx.x == 0) {
      Acc* leader = group.map_shared_rank(cluster_scratch, 0);
      leader[rank] = acc;
    }
    group.sync();
    if (rank != 0) return;
    if (threadIdx.x == 0) {
      acc = cluster_scratch[0];
      for (int j = 1; j < cluster; ++j) acc = R::combine(acc, cluster_scratch[j]);
    }
  }

  const int clusters = split / cluster;
  if (clusters == 1) {
    if (threadIdx.x == 0) out[slice] = R::finish(acc, reduce, mean != 0);
    return;
  }

  if (threadIdx.x == 0) {
    partials[slice * clusters + part / cluster] = acc;
    __threadfence();
    const unsigned ticket = atomicAdd(&tickets[slice], 1u);
    is_last = ticket == static_cast<unsigned>(clusters - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  Acc total = R::identity();
  for (int j = threadIdx.x; j < clusters; j += kBlock) {
    total = R::combine(total, load_partial(partials + slice * clusters + j));
  }
  total = block_reduce<R>(total, warp_scratch);
  if (threadIdx.x == 0) out[slice] = R::finish(total, reduce, mean != 0);
}

// inner > 1. Thread layout: tx = threadIdx.x % lanes_x runs along inner (VEC columns each),
// ty = threadIdx.x / lanes_x along reduce. grid = (column tiles, split, outer); the cluster, when
// there is one, runs along grid.y.
//
// RAGGED (with the ring and 32 lanes): rows that do not start on a vector's boundary, because inner is odd or
// the tensor starts in between. A warp takes every eighth row, and eight rows of any width are a whole number
// of 16-byte units, so all rows of a warp have their vectors at the same place: `before` columns to the
// left of the tile's first. A tile is 31 vectors wide and the 32 lanes cover it wherever that is; what they
// read beside it are elements of its neighbours, gathered and never used. Only a vector that would begin before
// the tensor (its first row) or end behind it (its last) is read column by column. Rows of odd length used
// to be read an element, or four bytes, a lane: 40256 x 709 bf16 44.6 us a reduction where the bytes take 8.8.
//
// Sums are brought together in trees and pairs throughout: with a chain of additions in its place the error against 64 bits of an f32 sum or
// LayerNorm grew by up to a seventh when clusters took over from tickets and a thread's rows became more.
//
// What the kernel would divide by comes as shifts and quotients from the host: a small reduction is as long as its chain
// of instructions, and a dozen divisions were a tenth of it.
struct ColumnArgs {
  long long reduce, inner;
  long long chunk;          // rows of a CTA: reduce / split, rounded up
  int lanes_shift;          // log2 of the threads along inner
  int shares_shift;         // log2 of the threads that fold an item of the CTA's tile
  int split, cluster_shift, clusters;      // CTAs of a column tile, of a cluster (log2), clusters of a tile
  int mean;
};

// `count` accumulators (a power of two), `stride` apart, as a tree.
template <typename R>
__device__ __forceinline__ typename R::Acc fold_tree(const typename R::Acc* from, int count, int stride) {
  using Acc = typename R::Acc;
  if constexpr (rescales<R>::value) {
    float m = from[0].m;
    for (int i = 1; i < count; ++i) m = R::larger(m, from[i * stride].m);
    float s = R::scaled(from[0], m);
    for (int i = 1; i < count; i += 2) s += i + 1 < count ? R::scaled(from[i * stride], m) + R::scaled(from[(i + 1) * stride], m) : R::scaled(from[i * stride], m);
    return Acc{m, s};
  } else {
    Acc total = from[0];
    if (count >= 2) total = R::combine(total, from[stride]);
    if (count >= 4) total = R::combine(total, R::combine(from[2 * stride], from[3 * stride]));
    for (int i = 4; i < count; i += 4)
      total = R::combine(total, R::combine(R::combine(from[i * stride], from[(i + 1) * stride]), R::combine(from[(i + 2) * stride], from[(i + 3) * stride])));
    return total;
  }
}

// Five CTAs an SM, four where the state needs the registers: accumulators of 16 bytes, and f64 sums by plain loads, whose four rows in flight
// and their sum did not fit 48 registers any more (us with five and four: 3158 x 464 of 32 slices 108 and 57.5, 62403 x 1415 293 and
// 196, 50 x 16168 of 32 49.5 and 37.4; f64 extremes over 32768 x 2048, in more CTAs than run at once by fours, 115 and 129).
template <typename T, typename R, int VEC, bool RING, bool RAGGED = false>
__global__ void __launch_bounds__(kBlock, sizeof(typename R::Acc) > 8 || (std::is_same_v<R, SumReducer<double>> && !RING) ? 4 : 5)
reduce_columns(const T* __restrict__ in, typename R::Out* __restrict__ out, const ColumnArgs args,
               typename R::Acc* __restrict__ partials, unsigned* __restrict__ tickets) {
  using Acc = typename R::Acc;
  constexpr int kVecShift = VEC == 8 ? 3 : VEC == 4 ? 2 : VEC == 2 ? 1 : 0;
  static_assert(VEC == 1 << kVecShift);
  const long long reduce = args.reduce, inner = args.inner;
  const int lanes_x = 1 << args.lanes_shift, cluster = 1 << args.cluster_shift;
  extern __shared__ __align__(16) unsigned char dynamic_smem[];
  Acc* rows_scratch = reinterpret_cast<Acc*>(dynamic_smem);              // [kBlock * VEC]
  Acc* cluster_scratch = rows_scratch + kBlock * VEC;                    // [lanes_x * VEC]
  __shared__ bool is_last;

  if (cluster > 1) cluster_start();
  const int tx = threadIdx.x & (lanes_x - 1);
  const int ty = threadIdx.x >> args.lanes_shift;
  const int lanes_y = kBlock >> args.lanes_shift;
  const long long slice = blockIdx.z;
  const int part = blockIdx.y;
  const int tile_columns = RAGGED ? (lanes_x - 1) * VEC : lanes_x * VEC;
  const long long first_column = static_cast<long long>(blockIdx.x) * tile_columns;

  const long long begin = static_cast<long long>(part) * args.chunk;
  long long end = begin + args.chunk;
  if (end > reduce) end = reduce;

  int before = 0;
  if constexpr (RAGGED) {
    const T* row_start = in + (slice * reduce + begin + ty) * inner + first_column;
    before = static_cast<int>(reinterpret_cast<uintptr_t>(row_start) / sizeof(T) % VEC);
  }
  const long long column = first_column + tx * VEC - before;       // of this thread's vectors
  const bool in_range = column < inner;

  // A thread of the ring takes many rows. Sums of 32 and 64 bits take them two at a time into four chains, so that they
  // lose no digits by it (moments of 32-bit elements into two: their state is larger).
  constexpr int kMoreChains = !RING ? 0 : std::is_same_v<R, SumReducer<float>> || std::is_same_v<R, SumReducer<double>> ? 3 : std::is_same_v<R, MomentsReducer<float>> ? 1 : 0;
  typename R::template Local<1> local[VEC], more[kMoreChains ? kMoreChains * VEC : 1];
#pragma unroll
  for (int e = 0; e < VEC; ++e) local[e] = R::template local_identity<1>();
#pragma unroll
  for (int i = 0; i < kMoreChains * VEC; ++i) more[i] = local[0];

  if (in_range) {
    const T* base = in + slice * reduce * inner + column;
    constexpr int kBytes = static_cast<int>(sizeof(T)) * VEC;
    constexpr int UNROLL = kUnroll;
    if constexpr (RING && (kBytes == 4 || kBytes == 8 || kBytes == 16)) {
      // Each thread streams its own column vector through a private ring of kRingDepth slots in
      // shared memory with cp.async: the copies in flight cost no registers, so a thread keeps
      // kRingDepth - 1 rows (up to 112 bytes) on their way from HBM while it folds the oldest.
      // A slot is written and read by the same thread only, so no barrier is involved.
      // The loop is unrolled by the ring's depth, so slot addresses are constants, the source is a
      // pointer that advances by one stride, and the count is 32 bits: per row a wait, a shared
      // load, a copy, a commit and a pointer add besides the reducer's own work (the rolled form
      // with 64-bit index arithmetic spent 18 instructions per element on 4-byte moments and made
      // every 2-byte column reduction issue-bound).
      Vec<T, VEC>* ring = reinterpret_cast<Vec<T, VEC>*>(cluster_scratch + lanes_x * VEC) + threadIdx.x;     // slot d at + d * kBlock
      const uint32_t ring_address = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
      constexpr uint32_t kSlotBytes = static_cast<uint32_t>(kBlock) * kBytes;
      long long first = begin + ty;
      int count = first < end ? static_cast<int>((end - first + lanes_y - 1) / lanes_y) : 0;   // the host keeps this below 2^31
      // (RAGGED) the row whose vector would leave the tensor: column by column
      auto by_columns = [&](long long row) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          if (column + e >= 0 && column + e < inner) R::template step<1>(local[e], base[row * inner + e], row);
        }
      };
      bool leaves = false;
      if constexpr (RAGGED) {
        const long long at = slice * reduce * inner + column;      // element of the tensor, of the vector in row 0
        if (count > 0 && at + first * inner < 0) {
          by_columns(first);
          first += lanes_y;
          --count;
        }
        if (count > 0 && at + (first + static_cast<long long>(count - 1) * lanes_y) * inner + VEC > static_cast<long long>(gridDim.z) * reduce * inner) {
          leaves = true;
          --count;
        }
      }
      const T* source = base + first * inner;
      const long long stride = static_cast<long long>(lanes_y) * inner;
      long long ri = first;
      auto copy = [&](int slot) {
        if constexpr (kBytes == 16) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring_address + slot * kSlotBytes), "l"(source) : "memory");
        } else {
          asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(ring_address + slot * kSlotBytes), "l"(source), "n"(kBytes) : "memory");
        }
        source += stride;
      };
      if constexpr (R::kSeeded) {
        if (count > 0) {
          const Vec<T, VEC> x = load_stream<T, VEC>(source);
#pragma unroll
          for (int e = 0; e < VEC; ++e) {
            R::template seed<1>(local[e], x.v[e]);
            if constexpr (kMoreChains > 0) more[e] = local[e];
          }
        }
      }
#pragma unroll
      for (int d = 0; d < kRingDepth - 1; ++d) {
        if (d < count) copy(d);
        asm volatile("cp.async.commit_group;" ::: "memory");   // one group per row, empty past the end
      }
      Vec<T, VEC> held;      // the first row of a pair
      for (int i = 0; i < count; i += kRingDepth) {
#pragma unroll
        for (int d = 0; d < kRingDepth; ++d) {
          if (i + d < count) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kRingDepth - 2) : "memory");   // row i + d has landed
            const Vec<T, VEC> x = ring[d * kBlock];
            if constexpr (has_pairs<R>::value) {
              if (d % 2 == 0) {
                held = x;
              } else {
                constexpr int kChains = kMoreChains + 1;
                R::template step_pair<VEC>(d / 2 % kChains ? more + (d / 2 % kChains - 1) * VEC : local, held, x);
              }
            } else if constexpr (R::kSeeded) {
#pragma unroll
              for (int e = 0; e < VEC; ++e) R::template step_seeded<1>(local[e], x.v[e]);
            } else if constexpr (has_column_step<R>::value) {
              R::template step_columns<VEC>(local, x, ri);
              ri += lanes_y;
            } else {
#pragma unroll
              for (int e = 0; e < VEC; ++e) R::template step<1>(local[e], x.v[e], ri);
              ri += lanes_y;
            }
            if (i + d + kRingDepth - 1 < count) copy((d + kRingDepth - 1) % kRingDepth);   // into the slot read one row ago
            asm volatile("cp.async.commit_group;" ::: "memory");
          }
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if constexpr (has_pairs<R>::value) {
        if (count % 2 != 0) R::template step_single<VEC>(local, held);
      }
      if constexpr (R::kSeeded) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) R::template set_count<1>(local[e], count);
      }
      if constexpr (RAGGED) {
        if (leaves) by_columns(first + static_cast<long long>(count) * lanes_y);
      }
    } else {
      for (long long r = begin + ty; r < end; r += static_cast<long long>(lanes_y) * UNROLL) {
        Vec<T, VEC> x[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const long long ri = r + static_cast<long long>(u) * lanes_y;
          if (ri < end) x[u] = load_stream<T, VEC>(base + ri * inner);
        }
        if constexpr (has_pairs<R>::value && !R::kSeeded) {
          static_assert(UNROLL == 4);
          if (r + 3ll * lanes_y < end) {
            if constexpr (std::is_same_v<R, SumReducer<T>>) {
              R::template step_four<VEC>(local, x);
            } else {
              R::template step_pair<VEC>(local, x[0], x[1]);
              R::template step_pair<VEC>(local, x[2], x[3]);
            }
            continue;
          }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const long long ri = r + static_cast<long long>(u) * lanes_y;
          if (ri < end) {
            if constexpr (has_column_step<R>::value) {
              R::template step_columns<VEC>(local, x[u], ri);
            } else {
#pragma unroll
              for (int e = 0; e < VEC; ++e) R::template step<1>(local[e], x[u].v[e], ri);
            }
          }
        }
      }
    }
  }

  // Across the rows of the CTA, in a fixed order and by every thread: shuffles bring a warp's rows together (where whole
  // vectors line up), then a thread folds its share of an item's rows in shared memory.
  Acc acc[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    if constexpr (kMoreChains == 1) R::template add_chain<1>(local[e], more[e]);
    acc[e] = R::template to_acc<1>(local[e]);
    if constexpr (kMoreChains == 3) acc[e] = (acc[e] + more[e]) + (more[VEC + e] + more[2 * VEC + e]);
  }
  const int items = lanes_x * VEC;                // at most kBlock
  int rows = lanes_y, row = ty;
  bool writes = true;
  if constexpr (!RAGGED) {
    if (lanes_x < 32) {
      if constexpr (rescales<R>::value) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          float m = acc[e].m;
          for (int offset = lanes_x; offset < 32; offset *= 2) m = R::larger(m, shfl_xor(m, offset));
          float s = R::scaled(acc[e], m);
          for (int offset = lanes_x; offset < 32; offset *= 2) s += shfl_xor(s, offset);
          acc[e] = Acc{m, s};
        }
      } else {
        for (int offset = lanes_x; offset < 32; offset *= 2) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[e] = R::combine(acc[e], R::shuffle(acc[e], offset));
        }
      }
      rows = kWarps;
      row = threadIdx.x / 32;
      writes = (threadIdx.x & 31) < lanes_x;
    }
  }
  if (writes) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const int item = tx * VEC + e - before;
      if (!RAGGED || (item >= 0 && item < tile_columns)) rows_scratch[row * items + item] = acc[e];
    }
  }
  __syncthreads();
  const int shares = 1 << args.shares_shift;      // threads an item
  const int my_item = threadIdx.x & (items - 1), share = threadIdx.x >> (args.lanes_shift + kVecShift);
  Acc total = R::identity();
  if (share < shares && (!RAGGED || my_item < tile_columns))
    total = fold_tree<R>(rows_scratch + share * items + my_item, rows >> args.shares_shift, items << args.shares_shift);
  if (shares > 1) {
    __syncthreads();
    if (share > 0 && share < shares) rows_scratch[share * items + my_item] = total;
    __syncthreads();
    if (share == 0 && (!RAGGED || my_item < tile_columns)) {
      rows_scratch[my_item] = total;
      total = fold_tree<R>(rows_scratch + my_item, shares, items);
    }
  }
  const bool holder = share == 0 && (!RAGGED || my_item < tile_columns);

  // Across the CTAs of the cluster: a reduce-scatter through distributed shared memory. The
  // tile's `items` accumulators are cut into `cluster` equal slices; every CTA sends slice q of
  // its accumulators to CTA q, one cluster barrier, and CTA q folds what it received in rank
  // order. Each CTA then owns items [rank * slice_items, (rank + 1) * slice_items) of the tile.
  const int slice_shift = args.lanes_shift + kVecShift - args.cluster_shift, slice_items = 1 << slice_shift;      // cluster <= items
  unsigned rank = 0;
  typename R::Out* out_row = out + slice * inner;
  const long long tile_column = first_column;
  // what of the tile's items is a column of this tile
  const long long live = inner - tile_column < tile_columns ? inner - tile_column : tile_columns;
  const int clusters = args.clusters;
  const long long tile = slice * gridDim.x + blockIdx.x;
  Acc* tile_partials = partials + tile * clusters * items;

  if (cluster > 1) {
    cg::cluster_group group = cg::this_cluster();
    rank = group.block_rank();
    cluster_started();
    if (holder) group.map_shared_rank(cluster_scratch, my_item >> slice_shift)[rank * slice_items + (my_item & (slice_items - 1))] = total;
    group.sync();
    // Thread t < slice_items now finishes item rank * slice_items + t.
    if (threadIdx.x < slice_items) {
      const Acc total = fold_tree<R>(cluster_scratch + threadIdx.x, cluster, slice_items);
      const int item = rank * slice_items + threadIdx.x;
      if (clusters == 1) {
        if (item < live) out_row[tile_column + item] = R::finish(total, reduce, args.mean != 0);
      } else {
        tile_partials[(part >> args.cluster_shift) * items + item] = total;
      }
    }
    if (clusters == 1) return;
  } else {
    if (clusters == 1) {
      if (holder && my_item < live) out_row[tile_column + my_item] = R::finish(total, reduce, args.mean != 0);
      return;
    }
    if (holder) tile_partials[part * items + my_item] = total;
  }

  // Across clusters: every CTA has written its share of its cluster's partial; the last CTA of
  // the tile to take a ticket folds the `clusters` partials of every item, all threads at work,
  // eight loads in flight each, in a fixed order.
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned ticket = atomicAdd(&tickets[tile], 1u);
    is_last = ticket == static_cast<unsigned>(args.split - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  for (int item = threadIdx.x; item < items; item += kBlock) {
    if (item >= live) continue;
    Acc total = R::identity();
    for (int j = 0; j < clusters; j += 4) {
      Acc batch[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (j + u < clusters) batch[u] = load_partial(tile_partials + static_cast<long long>(j + u) * items + item);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (j + u < clusters) total = R::combine(total, batch[u]);
      }
    }
    out_row[tile_column + item] = R::finish(total, reduce, args.mean != 0);
  }
}

// ---------------------------------------------------------------------------------------------
// inner > 1, large tensors: the persistent streaming form. The tensor is cut into panels of columns
// (512 bytes of every row) and a panel into units of 64 rows; a unit is one TMA tile (32 KiB). The
// units, panel after panel, are dealt out as one contiguous range per CTA (one CTA per SM), so every
// SM streams the same number of bytes (to within one unit) and a panel is shared by the few CTAs
// whose ranges meet it. One lane issues the tile loads into a ring of shared-memory stages; eight
// consumer warps fold the rows (warp w rows w, w + 8, ... of a unit, a lane 16 bytes of a row). Where
// a CTA's range leaves a panel it folds its eight warps' accumulators through shared memory and, if
// it is not the panel's only CTA, leaves one partial per column in scratch; the last CTA of the panel
// to take a ticket folds the partials in row order and writes the results. Replaces the thread-level
// loads of reduce_columns for the shapes where those leave the memory system short of requests:
// per 16 bytes a consumer spends a shared-memory load and the reducer's own work, nothing else.
// Consumer warps: eight, or sixteen for the softmax statistics of 2-byte elements, whose per-element work
// (a scaling, a test, an exponential, an add; 8 elements per 16 bytes) binds before HBM does with eight.
// Measured on B200 at [32768, 4096] bf16: softmax over the view's statistics + normalise 190 us with
// sixteen against 228 with eight (177 against 190 once the reducer stepped eight columns behind one
// test); argmax 63.5 us with sixteen against 58.6 with eight, the moments equal.
template <typename T, typename R>
constexpr int stream_consumers() { return (sizeof(T) == 2 && std::is_same_v<R, SoftmaxStatReducer<T>>) ? 16 : 8; }
constexpr int kStreamPieceBytes = 512;
constexpr int kStreamUnitRows = 64;
constexpr int kStreamStageBytes = kStreamUnitRows * kStreamPieceBytes;
constexpr int kStreamStages = 5;                 // with eight consumer warps; four with sixteen (their accumulators take the room)
constexpr int kStatusStreamData = 0x53544d31;    // "STM1": a unit's data never arrived
constexpr int kStatusStreamRing = 0x53544d32;    // "STM2": a stage was never handed back

struct StreamArgs {
  long long reduce, inner;
  long long units;            // outer * panels per slice * units per panel
  int units_per_panel;        // reduce / 64
  int panels_per_slice;       // inner / columns per panel
  int slots;                  // partial rows reserved per panel
  int mean;
  WaitStatus status;
};

// units * grid stays below 2^32 (the plan declines otherwise), so the kernel's divisions are 32-bit ones:
// a 64-bit division is about a hundred dependent instructions, and a segment's end runs six of them.
__device__ __forceinline__ long long stream_first_unit(long long cta, long long units, long long grid) {
  return static_cast<unsigned>(cta * units) / static_cast<unsigned>(grid);
}

// The CTA whose range holds `unit`.
__device__ __forceinline__ int stream_owner(long long unit, long long units, int grid) {
  long long c = static_cast<unsigned>(unit * grid) / static_cast<unsigned>(units);
  while (c + 1 < grid && stream_first_unit(c + 1, units, grid) <= unit) ++c;
  while (c > 0 && stream_first_unit(c, units, grid) > unit) --c;
  return static_cast<int>(c);
}

template <typename T, typename R>
__global__ void __launch_bounds__((stream_consumers<T, R>() + 1) * 32, 1)
reduce_columns_stream(const __grid_constant__ CUtensorMap map, const StreamArgs args, typename R::Out* __restrict__ out,
                      typename R::Acc* __restrict__ partials, unsigned* __restrict__ tickets) {
  using Acc = typename R::Acc;
  constexpr int V = 16 / static_cast<int>(sizeof(T));
  constexpr int kColumns = 32 * V;
  constexpr int kStreamConsumers = stream_consumers<T, R>();
  constexpr int kStreamStages = kStreamConsumers == 8 ? 5 : 4;      // (hides the namespace's value)
  constexpr int kConsumerThreads = kStreamConsumers * 32;
  constexpr int kRowsPerWarp = kStreamUnitRows / kStreamConsumers;
  extern __shared__ __align__(128) unsigned char stream_smem[];
  __shared__ int is_last;
  unsigned char* ring = stream_smem;
  Acc* scratch = reinterpret_cast<Acc*>(ring + kStreamStages * kStreamStageBytes);   // [8 warps][columns]
  uint64_t* barriers = reinterpret_cast<uint64_t*>(scratch + kStreamConsumers * kColumns);
  const uint32_t full0 = smem_address(barriers), empty0 = full0 + 8 * kStreamStages;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStreamStages; ++s) {
      barrier_init(full0 + 8 * s, 1);
      barrier_init(empty0 + 8 * s, kStreamConsumers);
    }
    if (blockIdx.x == 0) args.status.begin();
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  const long long first = stream_first_unit(cta, args.units, grid), last = stream_first_unit(cta + 1, args.units, grid);
  const int upp = args.units_per_panel;
  int stage = 0;
  uint32_t phase = 0;

  if (warp == kStreamConsumers) {
    // ---- producer ---------------------------------------------------------------------------------
    if (lane == 0) {
      for (long long u = first; u < last; ++u) {
        const long long panel = static_cast<unsigned>(u) / static_cast<unsigned>(upp);
        const int unit = static_cast<int>(u - panel * upp);
        const long long slice = static_cast<unsigned>(panel) / static_cast<unsigned>(args.panels_per_slice);
        const int column = static_cast<int>(panel - slice * args.panels_per_slice) * kColumns;
        if (!barrier_wait(empty0 + 8 * stage, phase ^ 1, args.status, kStatusStreamRing)) break;
        barrier_expect_tx(full0 + 8 * stage, kStreamStageBytes);
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                         smem_address(ring) + stage * kStreamStageBytes),
                     "l"(&map), "r"(full0 + 8 * stage), "r"(column), "r"(static_cast<int>(slice * args.reduce + static_cast<long long>(unit) * kStreamUnitRows))
                     : "memory");
        if (++stage == kStreamStages) {
          stage = 0;
          phase ^= 1;
        }
      }
      // nothing may still be on its way into this CTA's shared memory when it leaves: the consumers
      // wait for every tile they were promised, and after a give-up the loads already issued are
      // waited for here (a stage that was never armed answers at once)
      if (args.status.aborted()) {
        for (int s = 0; s < kStreamStages; ++s) {
          const uint32_t parity = s < stage ? phase : phase ^ 1;
          for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
            if (barrier_try_wait(full0 + 8 * s, parity)) break;
          }
        }
      }
    }
    return;
  }

  // ---- consumers: a segment is the part of the CTA's range that lies in one panel --------------------
  bool alive = true;
  for (long long u = first; u < last && alive;) {
    const long long panel = static_cast<unsigned>(u) / static_cast<unsigned>(upp);
    const long long panel_first = panel * upp;
    long long segment_end = panel_first + upp;
    if (segment_end > last) segment_end = last;
    typename R::template Local<1> local[V];
#pragma unroll
    for (int e = 0; e < V; ++e) local[e] = R::template local_identity<1>();
    const long long segment_first = u;
    for (; u < segment_end; ++u) {
      if (!barrier_wait(full0 + 8 * stage, phase, args.status, kStatusStreamData)) {
        alive = false;
        break;
      }
      const Vec<T, V>* mine = reinterpret_cast<const Vec<T, V>*>(ring + static_cast<size_t>(stage) * kStreamStageBytes +
                                                                 static_cast<size_t>(warp) * kStreamPieceBytes) + lane;
      long long row = (u - panel_first) * kStreamUnitRows + warp;   // within the slice
      if constexpr (R::kSeeded) {
        if (u == segment_first) {
          const Vec<T, V> x = mine[0];
#pragma unroll
          for (int e = 0; e < V; ++e) R::template seed<1>(local[e], x.v[e]);
        }
      }
#pragma unroll
      for (int i = 0; i < kRowsPerWarp; ++i) {
        const Vec<T, V> x = mine[i * kStreamConsumers * (kStreamPieceBytes / 16)];
        if constexpr (has_column_step<R>::value) {
          R::template step_columns<V>(local, x, row);
        } else {
#pragma unroll
          for (int e = 0; e < V; ++e) {
            if constexpr (R::kSeeded) {
              R::template step_seeded<1>(local[e], x.v[e]);
            } else {
              R::template step<1>(local[e], x.v[e], row);
            }
          }
        }
        row += kStreamConsumers;
      }
      __syncwarp();
      if (lane == 0) barrier_arrive(empty0 + 8 * stage);
      if (++stage == kStreamStages) {
        stage = 0;
        phase ^= 1;
      }
    }
    if (!alive) break;
    if constexpr (R::kSeeded) {
#pragma unroll
      for (int e = 0; e < V; ++e) R::template set_count<1>(local[e], static_cast<int>(segment_end - segment_first) * kRowsPerWarp);
    }
    // the eight warps' accumulators meet in shared memory (the first barrier: everyone is done reading
    // what the previous segment left there), one thread per column folds them in warp order
    asm volatile("bar.sync 1, %0;" ::"n"(kConsumerThreads) : "memory");
#pragma unroll
    for (int e = 0; e < V; ++e) scratch[warp * kColumns + lane * V + e] = R::template to_acc<1>(local[e]);
    asm volatile("bar.sync 1, %0;" ::"n"(kConsumerThreads) : "memory");
    const int owner_first = stream_owner(panel_first, args.units, grid);
    const int owner_last = stream_owner(panel_first + upp - 1, args.units, grid);
    const int sharers = owner_last - owner_first + 1;
    const long long slice = static_cast<unsigned>(panel) / static_cast<unsigned>(args.panels_per_slice);
    typename R::Out* out_row = out + slice * args.inner + (panel - slice * args.panels_per_slice) * kColumns;
    Acc* panel_partials = partials + panel * args.slots * kColumns;
    for (int column = threadIdx.x; column < kColumns; column += kConsumerThreads) {
      Acc total = scratch[column];
#pragma unroll
      for (int w = 1; w < kStreamConsumers; ++w) total = R::combine(total, scratch[w * kColumns + column]);
      if (sharers == 1) {
        out_row[column] = R::finish(total, args.reduce, args.mean != 0);
      } else {
        panel_partials[(cta - owner_first) * kColumns + column] = total;
      }
    }
    if (sharers > 1) {
      // the last CTA of the panel to take a ticket folds the partials in CTA order, which is row order
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(kConsumerThreads) : "memory");
      if (threadIdx.x == 0) is_last = atomicAdd(&tickets[panel], 1u) == static_cast<unsigned>(sharers - 1) ? 1 : 0;
      asm volatile("bar.sync 1, %0;" ::"n"(kConsumerThreads) : "memory");
      if (is_last) {
        __threadfence();
        for (int column = threadIdx.x; column < kColumns; column += kConsumerThreads) {
          Acc total = R::identity();
          for (int j = 0; j < sharers; j += 12) {
            Acc batch[12];
#pragma unroll
            for (int k = 0; k < 12; ++k) {
              if (j + k < sharers) batch[k] = load_partial(panel_partials + (j + k) * kColumns + column);
            }
#pragma unroll
            for (int k = 0; k < 12; ++k) {
              if (j + k < sharers) total = R::combine(total, batch[k]);
            }
          }
          out_row[column] = R::finish(total, args.reduce, args.mean != 0);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Host: the plan and the launch

enum class Shape { kWarpPerSlice, kCtaPerSlice, kColumns, kColumnStream };

struct Plan {
  Shape shape = Shape::kWarpPerSlice;
  int split = 1;      // CTAs per slice (or per column tile)
  int cluster = 1;    // CTAs per thread-block cluster; divides split
  int lanes_x = 32;   // columns kernel: threads along inner
  int vec = 1;        // columns kernel: elements per thread along inner
  bool ring = false;  // columns kernel: stream through the per-thread cp.async ring
  bool ragged = false;   // columns kernel: rows that do not start on a vector's boundary
  long long tiles = 0;        // ticketed outputs: slices, or outer * column tiles
  long long column_tiles = 0;
  size_t acc_bytes = 0;
  size_t partial_bytes = 0;   // scratch for partials (0 when one cluster covers a slice)
  size_t ticket_bytes = 0;
  size_t reported = 0;        // what the workspace query answers: the need of the form with partials, also where another one runs
  size_t need() const { return partial_bytes + ticket_bytes; }      // what a launch of this plan uses, and asks for
  // the streaming columns kernel
  int device = 0;
  int grid = 0;               // CTAs: one per SM
  long long units = 0;        // outer * panels per slice * units per panel
  int units_per_panel = 0;
  int panels_per_slice = 0;
  int slots = 0;              // partial rows per panel
};

// Whether the persistent streaming kernel takes a column reduction, and its tiling. Measured on B200
// at [32768, 4096] against reduce_columns: bf16 sum / mean / amax 51-52 us against 54-55, bf16 argmax
// 60 against 72, f32 argmax 93 against 103, bf16 moments (inside LayerNorm over a transposed view) 18 us
// less; f32 sum / mean / amax 89-91 us against 82-85, so those stay with reduce_columns. The streaming
// kernel moves 5.9-6.0 TB/s whatever the reducer until the reducer's instructions bind (bf16 argmax);
// what it loses is fixed: about 2 us until the first tile lands and 3 us for the last panel's fold.
bool plan_stream(Plan& p, tq_reduce_op op, tq_dtype dtype, long long outer, long long reduce, long long inner, int32_t device,
                 int vec_bytes_limit) {
  const int size = dtype_size(dtype);
  if (dtype != TQ_F32 && dtype != TQ_F16 && dtype != TQ_BF16) return false;
  if (!(size == 2 || op == TQ_ARGMAX || static_cast<int>(op) >= kOpSoftmaxStat)) return false;
  if (vec_bytes_limit != 16 || (inner * size) % kStreamPieceBytes != 0 || reduce % kStreamUnitRows != 0) return false;
  if (outer * reduce >= (1ll << 31) || inner >= (1ll << 31)) return false;   // TMA coordinates are 32 bits
  if (outer * reduce * inner * size < (64ll << 20)) return false;
  const int sms = sm_count(device);
  const long long panels = outer * (inner * size / kStreamPieceBytes);
  const long long units = panels * (reduce / kStreamUnitRows);
  if (units < 4ll * sms || panels > (1ll << 24)) return false;
  if (units * (sms + 1) >= (1ll << 32)) return false;   // the kernel divides unit x CTA products as 32-bit numbers
  p.shape = Shape::kColumnStream;
  p.device = device;
  p.grid = sms;
  p.units = units;
  p.units_per_panel = static_cast<int>(reduce / kStreamUnitRows);
  p.panels_per_slice = static_cast<int>(inner * size / kStreamPieceBytes);
  p.slots = static_cast<int>((p.units_per_panel + units / sms - 1) / (units / sms)) + 1;
  p.tiles = panels;
  const long long columns = kStreamPieceBytes / size;
  p.partial_bytes = (static_cast<size_t>(panels) * p.slots * columns * p.acc_bytes + 255) / 256 * 256;
  p.ticket_bytes = (static_cast<size_t>(panels) * sizeof(unsigned) + 255) / 256 * 256;
  return true;
}

int log2_of(int power) {
  int shift = 0;
  while ((1 << (shift + 1)) <= power) ++shift;
  return shift;
}

// Expected times, us, of a column reduction over `bytes` by the streaming kernel, and in the shape that the reduction's split gives it: fits to
// measured times, no bounds (part of a tensor is in L2 when a program calls, so that their rates may pass that of HBM).
//
// By clusters that meet over tickets the clearing of the tickets, partials in memory and the last CTA's fold are the fixed part; more for
// accumulators of 16 bytes and where rows start between vectors. Kernel times of [5184 x 1000] f16, [3072 x 4096], [16384 x 1024],
// [131072 x 128] f32, [40000 x 300], [262144 x 128] bf16 sums by tickets: 12.4, 16.3, 19.9, 23.1, 18.6, 30.9. (With plain loads and all CTAs
// in one wave of five an SM HBM is reached in the end: 32768 x 4096 f32 86; 16384 x 8192, whose 768 CTAs are more, 108.) f64 takes longer
// (us, so and by one-cluster tiles: 32768 x 2048 sum 113 and 86, extreme 115 and 86; sum 7977 x 424 of 32 slices 190 and 148, 62403 x 1415 196 and
// 123, 6749 x 5879 95 and 62); only of a few rows plain loads are as quick (35 x 69685 of two slices 13.4 and 18.8).
//
// Where one cluster covers a tile by itself there are no tickets to pay for, and from some size on that tells: plain loads of 16 bytes run near
// HBM's rate, less a third of what a last wave leaves idle (us of the split and of one-cluster tiles: 1060 x 44716 f32 30 and 36, 3897 x 29600
// 70 and 77, 2 x 6431 x 11176 90 and 103, 237 x 30096 of two slices 12.2 and 14; i32 sums, added up in 64 bits, 1494 x 17040 of two 40 and 39).
double stream_time(tq_reduce_op op, int size, long long bytes) { return 8.0 + bytes / 6.0e6 + (op == TQ_ARGMAX && size == 2 ? 6.0 : 0.0); }
double split_time(const Plan& p, tq_reduce_op op, tq_dtype dtype, long long reduce, long long bytes, int sms) {
  const bool light = op != TQ_ARGMAX && op < kOpSoftmaxStat, tickets = p.split > p.cluster;
  const bool whole_loads = p.vec * dtype_size(dtype) == 16;
  if (light && dtype == TQ_F64 && (tickets || (bytes >= 30000000 && reduce >= 80))) return 9.0 + bytes / (whole_loads ? 3.5e6 : 2.5e6);
  const double ticketed = !p.ring && p.tiles * p.split <= 5ll * sms
                              ? std::min(9.0 + bytes / 5.2e6, 14.0 + bytes / 7.4e6)
                              : 9.0 + bytes / 5.2e6 + (light || op == kOpSoftmaxStat ? 0.0 : 8.0) + (p.ragged ? 4.0 : 0.0);
  if (!light || tickets || p.ring || !whole_loads || dtype_size(dtype) != 4 || (op == TQ_SUM && dtype == TQ_I32) || bytes < 120000000) return ticketed;
  const double waves = static_cast<double>(p.tiles) * p.split / (5.0 * sms);
  return std::min(ticketed, 3.0 + bytes / 7.0e6 * (waves > 1.0 ? 1.0 + 0.35 * (std::ceil(waves) - waves) / waves : 1.0));
}

// Whether one cluster (or one CTA) takes a tile of columns whole: no partials, no tickets, nothing to clear. The tile's width (lanes) and
// the cluster are chosen by expected time: the launch and the folds; every CTA's bytes at the 38 KB a us that the
// cp.async ring gets through one CTA of an SM, 48 for two and more together (30 and 32 where a row's piece is 64 bytes, 16 and 20
// where it is 32); the reducer's work per row of a thread (argmax, the statistics); HBM, of which pieces of 256 bytes get most
// (32768 x 4096 f32 sum 85.5 us in 256 bytes by clusters of four, 90 in 512 by eight, 110 in 128 by two); and what CTAs beyond two
// an SM cost (1 us per further wave of 296: 256 CTAs measured best at every size). us, before and now: 5003 x 1250 bf16 sum 12.4 and
// 6.0, argmax 16.6 and 9.2; 1000 x 1000 f32 sum 10.3 and 3.8; 5184 x 1000 f16 LayerNorm over the view 40.7 and 13.9; 3072 x 4096
// f32 sum 17.2 and 11.6, argmax 39 and 12.3; 16384 x 8192 f32 sum 108 and 85; 20000 x 64 bf16 sum 10.3 and 6.1. Tall and narrow
// tensors of some size have too few tiles for it (131072 x 128 f32 sum 23 by tickets, 28 so), and argmax and statistics over
// 200 MB and more stay with the streaming kernel (32768 x 4096 argmax from a cold L2 bf16 56.5 and 66, f32 91.9 and 98).
bool plan_one_cluster(Plan& p, tq_reduce_op op, int size, long long outer, long long reduce, long long inner, int sms, double others) {
  const long long groups = (inner + p.vec - 1) / p.vec;
  const long long bytes = outer * reduce * inner * size;
  const bool statistic = op >= kOpSoftmaxStat, heavy = op == TQ_ARGMAX || op == kOpMoments;       // accumulators of 16 bytes
  if ((op == TQ_ARGMAX || statistic) && bytes >= (200ll << 20)) return false;
  if (reduce >= (1ll << 31)) return false;              // the ring counts a thread's rows in 32 bits
  if (outer > 65535) return false;                      // planes of a grid; the streaming kernel has no such limit
  double best = 0.95 * others;
  bool found = false;
  for (int lanes = p.ragged || p.vec > kBlock / 64 ? 32 : 64; lanes >= 2; lanes /= 2) {
    const int piece = lanes * p.vec * size;
    if (piece < 32 || (p.ragged && lanes < 4)) break;
    const long long tiles = p.ragged ? (inner + (lanes - 1) * p.vec - 1) / ((lanes - 1) * p.vec) : (groups + lanes - 1) / lanes;
    const int rows_at_once = kBlock / lanes;
    const double one = piece >= 128 ? 38e3 : piece >= 64 ? 30e3 : 16e3;        // bytes a us
    const double together = piece >= 128 ? 48e3 : piece >= 64 ? 32e3 : 20e3;
    for (int cluster = 1; cluster <= kMaxCluster; cluster *= 2) {
      if (cluster > lanes * p.vec || (cluster > 1 && reduce < 2ll * cluster * rows_at_once)) break;
      const long long ctas = tiles * outer * cluster;
      const long long rows = (reduce + cluster - 1) / cluster;
      const double an_sm = static_cast<double>((ctas + sms - 1) / sms);
      const double cta_bytes = static_cast<double>(rows) * piece;
      // (up to six rows a thread are two trips of plain loads, which start sooner: 512 x 768 f32 sum 2.8 and 3.1, 1000 x 1000 3.7 and 4.0)
      const bool few = rows <= 6ll * rows_at_once && size >= 4 && op != TQ_ARGMAX && !statistic && !p.ragged;
      if (lanes > 32 && !few) break;      // (larger clusters of 64 lanes could be few again, and were the expected best of none of 700 shapes of 20 to 200 rows)
      const double rate = an_sm > 1 ? std::min(together, an_sm * one) : one;
      const double work = static_cast<double>(rows) / rows_at_once *
                          (op == TQ_ARGMAX ? 0.1 : op == kOpMoments ? 0.03 * an_sm : op == kOpSoftmaxStat ? (size == 2 ? 0.11 : 0.05) * std::max(an_sm, 1.7) : 0.03);
      const double moving = std::max({bytes / (piece >= 256 ? 6.2e6 : 5.8e6), an_sm * cta_bytes / rate, work}) * (piece == 256 ? 0.96 : 1.0);
      const double time = 2.3 + (cluster > 1 ? (heavy ? 1.6 : 0.8) : 0.0) + (heavy ? 0.15 : 0.05) * log2_of(std::max(32 / lanes, 1)) + (few ? 0.0 : 0.4) +
                          moving + std::max(0.0, static_cast<double>(ctas) / (2.0 * sms) - 1.0);
      if (time >= best) continue;
      best = time;
      found = true;
      p.lanes_x = lanes;
      p.split = p.cluster = cluster;
      p.column_tiles = tiles;
      p.tiles = tiles * outer;
      p.ring = !few;
    }
  }
  return found;
}

int floor_pow2(long long v) {
  int p = 1;
  while (static_cast<long long>(p) * 2 <= v) p *= 2;
  return p;
}

// Partials and tickets, where a slice or a tile of columns is shared by more than one cluster.
void add_scratch(Plan& p) {
  const int clusters = p.split / p.cluster;
  if (clusters > 1) {
    const long long items = p.shape == Shape::kColumns ? p.lanes_x * p.vec : 1;
    p.partial_bytes = static_cast<size_t>(p.tiles) * clusters * items * p.acc_bytes;
    p.partial_bytes = (p.partial_bytes + 255) / 256 * 256;
    p.ticket_bytes = (static_cast<size_t>(p.tiles) * sizeof(unsigned) + 255) / 256 * 256;
  }
  p.reported = p.need();
}

Plan plan(tq_reduce_op op, tq_dtype dtype, long long outer, long long reduce, long long inner,
          int32_t device, int vec_bytes_limit, bool may_be_ragged = true) {
  Plan p;
  p.device = device;
  const int size = dtype_size(dtype);
  const int sms = sm_count(device);
  const long long target_ctas = static_cast<long long>(sms) * 4;
  p.acc_bytes = (op == TQ_ARGMAX || op == kOpMoments) ? 16 : 8;  // upper bound; every other Acc fits 8 bytes
  if (inner == 1) {
    const int vec = 16 / size;
    const long long slice_bytes = reduce * size;
    if (slice_bytes <= 4096 || (outer >= static_cast<long long>(sms) * 16 && slice_bytes <= 65536)) {
      p.shape = Shape::kWarpPerSlice;
      return p;
    }
    p.shape = Shape::kCtaPerSlice;
    long long want = (target_ctas + outer - 1) / outer;
    const long long per_pass = static_cast<long long>(kBlock) * vec * kUnroll;
    long long most = reduce / per_pass;
    if (most < 1) most = 1;
    if (want > most) want = most;
    if (want < 1) want = 1;
    if (want <= kMaxCluster) {
      p.split = floor_pow2(want);
      p.cluster = p.split;
    } else {
      if (want > 1024) want = 1024;
      p.split = static_cast<int>((want + kMaxCluster - 1) / kMaxCluster * kMaxCluster);
      p.cluster = kMaxCluster;
    }
    p.tiles = outer;
  } else {
    Plan stream = p;
    const bool may_stream = plan_stream(stream, op, dtype, outer, reduce, inner, device, vec_bytes_limit);
    p.shape = Shape::kColumns;
    int vec = vec_bytes_limit / size;
    if (vec > 8) vec = 8;
    if (vec < 1) vec = 1;
    while (vec > 1 && inner % vec != 0) vec /= 2;
    if ((op == TQ_ARGMAX || op == kOpMoments) && vec > 4) vec = 4;  // their per-column state is large; 16-byte loads measured no better (argmax) or worse (moments)
    // Rows no whole vector fits go to the ragged form, unless they are so short that most of its lanes would
    // have no column, or the pass is one of statistics (their callers ask for whole vectors).
    const int whole = (op == TQ_ARGMAX ? 4 : 8) < 16 / size ? (op == TQ_ARGMAX ? 4 : 8) : 16 / size;
    // ... or they are few and their bytes too: up to so many rows the plain form needs no tickets, and is done while the
    // ragged one folds (us, plain and ragged: 200 x 709 bf16 sum 3.2 and 4.4, argmax 3.5 and 6.8; 17 x 3001 f32 sum 2.4 and 2.8, argmax
    // 2.7 and 5.2, 128 x 3001 argmax 4.4 and 6.2; but 300 x 9999 bf16 sum 10.8 and 5.7, 1000 x 50 f32 sum 8.2 and 4.1, argmax 9.3 and
    // 7.5, 64 x 1000001 f32 sum 100 and 49).
    const long long rows_without_tickets = size == 2 || op == TQ_ARGMAX ? 288 : 144;
    const long long elements = outer * reduce * inner;
    const bool small = reduce < rows_without_tickets && elements * size < (op == TQ_ARGMAX ? 4ll << 20 : 1ll << 20);
    // ... or argmax of four-byte elements two columns a load (or a row within one tile) over 60 to 300 MB, where the plain
    // form's waves fill (us, plain and ragged: 40000 x 502 f32 36.6 and 40.5, 160000 x 98 41.8 and 51.8; but 40000 x 370 .8, 10000 x 1002
    // .78, 2000 x 1250 .39 of the plain form's time, 40000 x 2002 .99, 32768 x 4098 .93).
    // (Both measured where the split had tickets; few rows need none by either kind of load now. The one-cluster form below takes the kind
    // that is chosen here and has not been measured with the other: 200 x 709 bf16 sum 3.2, argmax 3.4, 40000 x 502 f32 argmax 20.1,
    // 160000 x 98 35.8. Plain loads of one two-byte column, which no ring carries, are slower there than its estimate says: 20000 x 65
    // bf16 sum 15.0 for 8.6, with tickets 18.7.)
    const bool plain_fills = op == TQ_ARGMAX && size == 4 && elements >= 15500000 && elements < 75000000 && (vec >= 2 || inner <= 31 * whole);
    p.ragged = may_be_ragged && vec < whole && (size == 2 || size == 4) && op < kOpSoftmaxStat && inner >= 12 * whole && reduce < (1ll << 31) && !small &&
               !plain_fills;
    if (p.ragged) vec = whole;
    p.vec = vec;
    const long long groups = (inner + vec - 1) / vec;
    Plan whole_tiles = p;
    // A warp reads 32 vectors (512 bytes) of one row; the CTA's 8 warps read 8 consecutive rows.
    // Measured on B200 at [32768, 4096]: 4-byte sums and extremes are fastest with plain unrolled
    // loads, 64 lanes along `inner` and one wave of CTAs; 2-byte types and argmax (whose state
    // costs registers) with the cp.async ring and 32 lanes.
    p.ring = (size <= 2 || op == TQ_ARGMAX || op >= kOpSoftmaxStat) && reduce < (1ll << 31);   // the ring counts a thread's rows in 32 bits
    if (p.ragged) p.ring = true;
    int lanes = p.ring || vec > kBlock / 64 ? 32 : 64;      // an item of the tile a thread, at most
    while (lanes > 1 && lanes / 2 >= groups && !p.ragged) lanes /= 2;
    p.lanes_x = lanes;
    p.column_tiles = p.ragged ? (inner + (lanes - 1) * vec - 1) / ((lanes - 1) * vec) : (groups + lanes - 1) / lanes;
    const long long base_ctas = p.column_tiles * outer;
    // One or two waves of CTAs (all of a wave resident at once, equal work each).
    const int waves = (p.ring && !(op == TQ_ARGMAX && size <= 2)) ? 2 : 1;
    long long want = (target_ctas * waves + base_ctas - 1) / base_ctas;
    // (the ragged form: at least twice the ring's depth of rows a thread; 5003 x 1250 split finer is all folding, f32 sum 18.2 us against 14.5)
    const long long per_pass = static_cast<long long>(kBlock / lanes) * (p.ragged ? 2 * kRingDepth : kUnroll);
    long long most = reduce / per_pass;
    if (most < 1) most = 1;
    if (want > most) want = most;
    // Argmax's accumulators leave room for four CTAs an SM, of which clusters of eight fill 24 of 25: whole waves of those. 6 tiles
    // shared by 200 CTAs each were 150 clusters where 142 run at once: 40256 x 709 f32 49.4 us, now 46.
    const long long wave = target_ctas * 24 / 25;
    if (p.ragged && op == TQ_ARGMAX && want * base_ctas > wave) want = want * base_ctas / wave * wave / base_ctas;
    if (want < 1) want = 1;
    // The cluster's reduce-scatter gives every CTA a whole number of threads' accumulators.
    int max_cluster = kMaxCluster;
    while (max_cluster > lanes) max_cluster /= 2;
    if (want <= max_cluster) {
      p.split = floor_pow2(want);
      p.cluster = p.split;
    } else {
      if (want > 1024) want = 1024;
      // (rounded down in the ragged form, whose waves are counted out)
      p.split = static_cast<int>((p.ragged ? want : want + max_cluster - 1) / max_cluster * max_cluster);
      p.cluster = max_cluster;
    }
    p.tiles = base_ctas;
    add_scratch(p);
    if (may_stream) stream.reported = stream.need();
    const Plan& other = may_stream ? stream : p;
    const double others = may_stream ? stream_time(op, size, elements * size) : split_time(p, op, dtype, reduce, elements * size, sms);
    if (!plan_one_cluster(whole_tiles, op, size, outer, reduce, inner, sms, others)) return other;
    whole_tiles.reported = other.reported;
    return whole_tiles;
  }
  add_scratch(p);
  return p;
}

template <typename Kernel, typename... Args>
tq_status launch_clustered(Kernel kernel, dim3 grid, dim3 cluster, size_t smem, cudaStream_t stream,
                           Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(kBlock);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = cluster.x;
  attribute[0].val.clusterDim.y = cluster.y;
  attribute[0].val.clusterDim.z = cluster.z;
  config.attrs = attribute;
  config.numAttrs = (cluster.x * cluster.y * cluster.z > 1) ? 1 : 0;
  TQ_CUDA(cudaLaunchKernelEx(&config, kernel, args...));
  return TQ_OK;
}

template <typename T, typename R>
tq_status run(const Plan& p, const void* in, void* out, long long outer, long long reduce,
              long long inner, bool mean, void* workspace, cudaStream_t stream) {
  using Acc = typename R::Acc;
  using Out = typename R::Out;
  static_assert(sizeof(Acc) <= 16, "accumulators are sized as at most 16 bytes in plan()");
  const T* input = static_cast<const T*>(in);
  Out* output = static_cast<Out*>(out);
  Acc* partials = static_cast<Acc*>(workspace);
  unsigned* tickets =
      reinterpret_cast<unsigned*>(static_cast<unsigned char*>(workspace) + p.partial_bytes);
  if (p.ticket_bytes) TQ_CUDA(cudaMemsetAsync(tickets, 0, p.ticket_bytes, stream));
  constexpr int kVec = 16 / sizeof(T);
  switch (p.shape) {
    case Shape::kWarpPerSlice: {
      // Short slices share a warp, of many slices also longer ones; of few, eight or sixteen lanes only make each slice's chain
      // longer. Measured (us with 32 / 16 / 8 lanes): 300000 slices of 500 bf16 sum 98.7 / 61.3 / 53.6, argmax 154.8 / 90.4 / 66.9; of 250 f32
      // sum 78.0 / 51.9 / 50.2; of 500 f32 sum 89.6 / 94.3 / 101, argmax 116 / 95 / 102; 40000 of 96 f64 sum 12.3 / 8.0 / 9.4; 1000
      // slices of 1000 bf16 sum 2.1 / 2.5 / 3.3, argmax 2.7 / 3.2 / 4.4, 12000 6.5 / 6.9 / 6.9 and 8.8 / 8.5 / 7.9; 1000 of
      // 250 f32 3.1 / 3.2 / 4.0.
      const long long slice_bytes = reduce * static_cast<long long>(sizeof(T));
      constexpr bool kArgmax = std::is_same_v<R, ArgmaxReducer<T>>, kBusy = sizeof(T) == 2 || kArgmax;
      const long long per_sm = outer / sm_count(p.device);
      const int lanes = slice_bytes <= 512                            ? 8
                        : slice_bytes <= 1024 && per_sm >= 16        ? (sizeof(T) == 2 && per_sm >= 64 ? 8 : 16)
                        : slice_bytes <= (sizeof(T) == 2 && !kArgmax ? 1536 : 2048) && kBusy && per_sm >= 96 ? 16
                                                                     : 32;
      const int slices = kBlock / lanes;
      const long long blocks = (outer + slices - 1) / slices;
      TQ_REQUIRE(blocks <= 0x7fffffffLL, TQ_UNSUPPORTED, "%lld slices are more than a grid holds", outer);
      if (lanes == 16) {
        reduce_warp_per_slice<T, R, kVec, 16><<<static_cast<unsigned>(blocks), kBlock, 0, stream>>>(input, output, outer, reduce, mean ? 1 : 0);
      } else if (lanes == 8) {
        reduce_warp_per_slice<T, R, kVec, 8><<<static_cast<unsigned>(blocks), kBlock, 0, stream>>>(input, output, outer, reduce, mean ? 1 : 0);
      } else {
        reduce_warp_per_slice<T, R, kVec, 32><<<static_cast<unsigned>(blocks), kBlock, 0, stream>>>(input, output, outer, reduce, mean ? 1 : 0);
      }
      return check_launch("reduce_warp_per_slice");
    }
    case Shape::kCtaPerSlice: {
      const long long blocks = outer * p.split;
      TQ_REQUIRE(blocks <= 0x7fffffffLL, TQ_UNSUPPORTED, "%lld slices are more than a grid holds", outer);
      if (tq_status s = launch_clustered(reduce_cta_per_slice<T, R, kVec>,
                                         dim3(static_cast<unsigned>(blocks)), dim3(p.cluster), 0,
                                         stream, input, output, reduce, p.split, p.cluster,
                                         mean ? 1 : 0, partials, tickets)) {
        return s;
      }
      return check_launch("reduce_cta_per_slice");
    }
    case Shape::kColumns: {
      TQ_REQUIRE(outer <= 65535, TQ_UNSUPPORTED,
                 "a reduction with kept axes on both sides and %lld leading slices has no kernel", outer);
      dim3 grid(static_cast<unsigned>(p.column_tiles), p.split, static_cast<unsigned>(outer));
      auto go = [&](auto kernel, int vec) -> tq_status {
        const size_t fixed = static_cast<size_t>(kBlock) * vec * sizeof(Acc) + static_cast<size_t>(kRingDepth) * kBlock * vec * sizeof(T);
        const size_t smem = fixed + static_cast<size_t>(p.lanes_x) * vec * sizeof(Acc);
        // The kernel's limit is always that of its widest tile, an item a thread: another thread's launch of a narrower one does not lower it
        // between this setting and this launch.
        const size_t most = fixed + kBlock * sizeof(Acc);
        if (most > 40 * 1024) {
          TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most)));
        }
        ColumnArgs args = {};
        args.reduce = reduce;
        args.inner = inner;
        args.chunk = (reduce + p.split - 1) / p.split;
        args.lanes_shift = log2_of(p.lanes_x);
        const int items = p.lanes_x * vec, rows = p.ragged || p.lanes_x > 32 ? kBlock / p.lanes_x : kWarps;
        while ((items << (args.shares_shift + 1)) <= kBlock && (2 << args.shares_shift) <= rows) ++args.shares_shift;
        args.split = p.split;
        args.cluster_shift = log2_of(p.cluster);
        args.clusters = p.split / p.cluster;
        args.mean = mean ? 1 : 0;
        if (tq_status s = launch_clustered(kernel, grid, dim3(1, p.cluster, 1), smem, stream, input, output, args, partials, tickets)) {
          return s;
        }
        return check_launch("reduce_columns");
      };
      constexpr int kColumnVec = kVec > 8 ? 8 : kVec;
      if (p.ragged) {
        if constexpr (sizeof(T) == 2 || sizeof(T) == 4) {
          constexpr int kWhole = std::is_same_v<Acc, Indexed<typename Compute<T>::type>> ? 4 : kColumnVec;
          return p.vec == kWhole ? go(reduce_columns<T, R, kWhole, true, true>, kWhole)
                                 : fail(TQ_INTERNAL, "no ragged column kernel for %d elements per thread", p.vec);
        }
      }
      if (p.vec == 1) return p.ring ? go(reduce_columns<T, R, 1, true>, 1) : go(reduce_columns<T, R, 1, false>, 1);
      if constexpr (kColumnVec >= 2) {
        if (p.vec == 2) return p.ring ? go(reduce_columns<T, R, 2, true>, 2) : go(reduce_columns<T, R, 2, false>, 2);
      }
      if constexpr (kColumnVec >= 4) {
        if (p.vec == 4) return p.ring ? go(reduce_columns<T, R, 4, true>, 4) : go(reduce_columns<T, R, 4, false>, 4);
      }
      if constexpr (kColumnVec >= 8) {
        if (p.vec == 8) return p.ring ? go(reduce_columns<T, R, 8, true>, 8) : go(reduce_columns<T, R, 8, false>, 8);
      }
      return fail(TQ_INTERNAL, "no column kernel for %d elements per thread", p.vec);
    }
    case Shape::kColumnStream: {
      if constexpr (std::is_same_v<T, float> || std::is_same_v<T, __half> || std::is_same_v<T, __nv_bfloat16>) {
        constexpr int kColumns = kStreamPieceBytes / static_cast<int>(sizeof(T));
        EncodeTiled encode = encode_tiled();
        TQ_REQUIRE(encode != nullptr, TQ_EXTERNAL, "the CUDA driver does not provide cuTensorMapEncodeTiled");
        // in[outer * reduce, inner] as a two-axis map; a tile is one unit: 512 bytes of 64 consecutive rows
        CUtensorMap map;
        const cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer * reduce)};
        const cuuint64_t strides[1] = {static_cast<cuuint64_t>(inner) * sizeof(T)};
        const cuuint32_t box[2] = {static_cast<cuuint32_t>(kColumns), static_cast<cuuint32_t>(kStreamUnitRows)};
        const cuuint32_t element_strides[2] = {1, 1};
        const CUtensorMapDataType type = std::is_same_v<T, float>    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                         : std::is_same_v<T, __half> ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                     : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        const CUresult encoded = encode(&map, type, 2, const_cast<T*>(input), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        TQ_REQUIRE(encoded == CUDA_SUCCESS, TQ_EXTERNAL, "cuTensorMapEncodeTiled refused the reduction's input (%d)", static_cast<int>(encoded));
        StreamArgs args = {};
        args.reduce = reduce;
        args.inner = inner;
        args.units = p.units;
        args.units_per_panel = p.units_per_panel;
        args.panels_per_slice = p.panels_per_slice;
        args.slots = p.slots;
        args.mean = mean ? 1 : 0;
        args.status = wait_status_for(p.device);
        TQ_REQUIRE(args.status.abort != nullptr, TQ_RESOURCE_EXHAUSTED, "no device memory for the status word");
        auto kernel = reduce_columns_stream<T, R>;
        constexpr int kConsumers = stream_consumers<T, R>();
        constexpr int kStages = kConsumers == 8 ? kStreamStages : 4;
        const size_t smem = static_cast<size_t>(kStages) * kStreamStageBytes + static_cast<size_t>(kConsumers) * kColumns * sizeof(Acc) + 2 * kStages * 8;
        TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        kernel<<<static_cast<unsigned>(p.grid), (kConsumers + 1) * 32, smem, stream>>>(map, args, output, partials, tickets);
        return check_launch("reduce_columns_stream");
      } else {
        return fail(TQ_INTERNAL, "the streaming columns kernel was planned for an element type it does not serve");
      }
    }
  }
  return fail(TQ_INTERNAL, "unreachable reduction shape");
}

template <typename T>
tq_status run_op(tq_reduce_op op, const Plan& p, const void* in, void* out, long long outer,
                 long long reduce, long long inner, void* workspace, cudaStream_t stream) {
  switch (op) {
    case TQ_SUM: return run<T, SumReducer<T>>(p, in, out, outer, reduce, inner, false, workspace, stream);
    case TQ_MEAN: return run<T, SumReducer<T>>(p, in, out, outer, reduce, inner, true, workspace, stream);
    case TQ_AMAX: return run<T, ExtremeReducer<T, true>>(p, in, out, outer, reduce, inner, false, workspace, stream);
    case TQ_AMIN: return run<T, ExtremeReducer<T, false>>(p, in, out, outer, reduce, inner, false, workspace, stream);
    case TQ_ARGMAX: return run<T, ArgmaxReducer<T>>(p, in, out, outer, reduce, inner, false, workspace, stream);
    default: return fail(TQ_INVALID_ARGUMENT, "unknown reduction %d", op);
  }
}

tq_status validate(tq_reduce_op op, tq_dtype dtype, long long outer, long long reduce, long long inner) {
  TQ_REQUIRE(op >= TQ_SUM && op <= TQ_ARGMAX, TQ_INVALID_ARGUMENT, "unknown reduction %d", op);
  TQ_REQUIRE(dtype_size(dtype) != 0 && dtype != TQ_BOOL, TQ_UNSUPPORTED,
             "reductions have no kernel for element type %s", dtype_name(dtype));
  TQ_REQUIRE(outer >= 0 && reduce >= 0 && inner >= 0, TQ_INVALID_ARGUMENT,
             "negative extent in [%lld, %lld, %lld]", outer, reduce, inner);
  TQ_REQUIRE(reduce > 0, TQ_UNSUPPORTED, "a reduction over no elements has no kernel");
  TQ_REQUIRE(!(op == TQ_ARGMAX && reduce >= 0xffffffffLL), TQ_UNSUPPORTED,
             "argmax over %lld elements has no kernel (positions are kept in 32 bits)", reduce);
  TQ_REQUIRE(!(op == TQ_MEAN && (dtype == TQ_I32 || dtype == TQ_I64)), TQ_UNSUPPORTED,
             "mean of an integer tensor has no kernel");
  return TQ_OK;
}

// The columns kernel needs vector loads aligned in every row: inner * size and the base pointer
// must both be multiples of the vector's bytes.
int column_vec_bytes(const void* in, long long inner, int size) {
  int bytes = 16;
  while (bytes > size && (!aligned_to(in, bytes) || (inner * size) % bytes != 0)) bytes /= 2;
  return bytes;
}

template <typename T>
tq_status run_stats(int kind, const Plan& p, const void* in, void* out, long long outer, long long reduce,
                    long long inner, void* workspace, cudaStream_t stream) {
  if (kind == kOpSoftmaxStat) return run<T, SoftmaxStatReducer<T>>(p, in, out, outer, reduce, inner, false, workspace, stream);
  return run<T, MomentsReducer<T>>(p, in, out, outer, reduce, inner, false, workspace, stream);
}

// ---------------------------------------------------------------------------------------------
// Scratch that exists without anyone allocating it, for tq_reduce_launch_static.
//
// The array lives in the library's device image: every GPU that loads the library carries these
// bytes from load until the process exits. In host code the array's name is only a stand-in for
// the symbol, not a device address, so the host asks the runtime for the real address once per
// device (with that device current) and hands that pointer to the kernels.
constexpr size_t kStaticScratchBytes = TQ_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

std::mutex g_static_mutex;
void* g_static_address[64] = {nullptr};

// Looks the address up on first use for `device`, which must be current.
tq_status static_scratch_for(int32_t device, void** address) {
  TQ_REQUIRE(device >= 0 && device < 64, TQ_INVALID_ARGUMENT, "device ordinal %d is out of range", device);
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (g_static_address[device] == nullptr) {
    void* found = nullptr;
    const cudaError_t status = cudaGetSymbolAddress(&found, g_static_scratch);
    if (status != cudaSuccess || found == nullptr) {
      return fail(TQ_EXTERNAL, "cannot find the built-in scratch on device %d: %s", device,
                  cudaGetErrorString(status));
    }
    g_static_address[device] = found;
  }
  *address = g_static_address[device];
  return TQ_OK;
}

}  // namespace

// Per-slice statistics for the transposed softmax / LayerNorm (rownorm.cu): `kind` 0 writes
// (max, 1 / sum exp(x - max)), `kind` 1 writes (mean, biased variance), as two floats per slice,
// for a packed [outer, reduce, inner] input of a floating type (f32, f16, bf16).
size_t slice_stats_workspace_bytes(int kind, tq_dtype dtype, long long outer, long long reduce, long long inner, int32_t device) {
  size_t bytes = 0;
  const int op = kind == 0 ? kOpSoftmaxStat : kOpMoments;
  for (int limit = 16; limit >= dtype_size(dtype); limit /= 2) {
    const Plan p = plan(op, dtype, outer, reduce, inner, device, limit);
    bytes = std::max(bytes, p.reported);
  }
  return bytes;
}

tq_status slice_stats_launch(int kind, tq_dtype dtype, const void* in, void* stats, long long outer, long long reduce,
                             long long inner, void* workspace, size_t workspace_bytes, int32_t device, cudaStream_t stream) {
  const int op = kind == 0 ? kOpSoftmaxStat : kOpMoments;
  const int size = dtype_size(dtype);
  const Plan p = plan(op, dtype, outer, reduce, inner, device, inner == 1 ? 16 : column_vec_bytes(in, inner, size));
  const size_t need = p.need();
  TQ_REQUIRE(need == 0 || (workspace != nullptr && workspace_bytes >= need && aligned_to(workspace, 16)), TQ_INVALID_ARGUMENT,
             "the statistics pass needs %zu bytes of 16-byte-aligned scratch and was given %zu", need, workspace_bytes);
  switch (dtype) {
    case TQ_F32: return run_stats<float>(op, p, in, stats, outer, reduce, inner, workspace, stream);
    case TQ_F16: return run_stats<__half>(op, p, in, stats, outer, reduce, inner, workspace, stream);
    case TQ_BF16: return run_stats<__nv_bfloat16>(op, p, in, stats, outer, reduce, inner, workspace, stream);
    default: return fail(TQ_UNSUPPORTED, "slice statistics have no kernel for element type %s", dtype_name(dtype));
  }
}

}  // namespace tq

extern "C" {

tq_status tq_reduce_workspace_bytes(tq_reduce_op op, tq_dtype dtype, int64_t outer, int64_t reduce,
                                    int64_t inner, int32_t device, size_t* bytes) {
  TQ_REQUIRE(bytes != nullptr, TQ_INVALID_ARGUMENT, "bytes out-pointer is null");
  if (tq_status s = tq::validate(op, dtype, outer, reduce, inner)) return s;
  *bytes = 0;
  if (outer == 0 || inner == 0) return TQ_OK;
  // The input's alignment is unknown here and decides the vector width of the columns kernel,
  // which changes its tiling: answer with the largest need over the widths it may pick. (An answer that does not change
  // with the rule that picks between the forms: where one cluster takes a tile of columns whole, a launch needs none of it.)
  for (int limit = 16; limit >= tq::dtype_size(dtype); limit /= 2) {
    tq::Plan p = tq::plan(op, dtype, outer, reduce, inner, device, limit);
    *bytes = std::max(*bytes, p.reported);
  }
  return TQ_OK;
}

tq_status tq_reduce_launch(tq_reduce_op op, tq_dtype dtype, const void* in, void* out, int64_t outer,
                           int64_t reduce, int64_t inner, void* workspace, size_t workspace_bytes,
                           int32_t device, void* stream) {
  TQ_RECORD_OR_RUN([=](int32_t d, void* s) {
    return tq_reduce_launch(op, dtype, in, out, outer, reduce, inner, workspace, workspace_bytes, d, s);
  });
  if (tq_status s = tq::validate(op, dtype, outer, reduce, inner)) return s;
  if (outer == 0 || inner == 0) return TQ_OK;
  TQ_REQUIRE(in != nullptr && out != nullptr, TQ_INVALID_ARGUMENT, "null input or output");
  const int size = tq::dtype_size(dtype);
  TQ_REQUIRE(tq::aligned_to(in, size), TQ_INVALID_ARGUMENT, "input pointer is not aligned to its element type");
  tq::DeviceScope device_scope(device);
  if (tq_status s = device_scope.status()) return s;
  tq::Plan p = tq::plan(op, dtype, outer, reduce, inner, device,
                        inner == 1 ? 16 : tq::column_vec_bytes(in, inner, size));
  const size_t need = p.need();
  TQ_REQUIRE(need == 0 || (workspace != nullptr && workspace_bytes >= need), TQ_INVALID_ARGUMENT,
             "this reduction needs %zu bytes of scratch and was given %zu", need, workspace_bytes);
  TQ_REQUIRE(need == 0 || tq::aligned_to(workspace, 16), TQ_INVALID_ARGUMENT,
             "scratch memory must be 16-byte aligned");
  const auto held = tq::hold_scratch(p.ticket_bytes != 0 ? workspace : nullptr);
  cudaStream_t cuda_stream = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case TQ_F32: return tq::run_op<float>(op, p, in, out, outer, reduce, inner, workspace, cuda_stream);
    case TQ_F64: return tq::run_op<double>(op, p, in, out, outer, reduce, inner, workspace, cuda_stream);
    case TQ_F16: return tq::run_op<__half>(op, p, in, out, outer, reduce, inner, workspace, cuda_stream);
    case TQ_BF16: return tq::run_op<__nv_bfloat16>(op, p, in, out, outer, reduce, inner, workspace, cuda_stream);
    case TQ_I32: return tq::run_op<int>(op, p, in, out, outer, reduce, inner, workspace, cuda_stream);
    case TQ_I64: return tq::run_op<long long>(op, p, in, out, outer, reduce, inner, workspace, cuda_stream);
    default: return tq::fail(TQ_UNSUPPORTED, "reductions have no kernel for element type %s", tq::dtype_name(dtype));
  }
}

tq_status tq_reduce_partial_launch(tq_reduce_op op, tq_dtype dtype, const void* in, void* partial, int64_t count, void* workspace,
                                   size_t workspace_bytes, int32_t device, void* stream) {
  TQ_RECORD_OR_RUN([=](int32_t d, void* s) { return tq_reduce_partial_launch(op, dtype, in, partial, count, workspace, workspace_bytes, d, s); });
  TQ_REQUIRE(op == TQ_SUM || op == TQ_MEAN || op == TQ_AMAX || op == TQ_AMIN, TQ_UNSUPPORTED, "no global partial for operation %d", op);
  TQ_REQUIRE(dtype == TQ_F32 || dtype == TQ_F16 || dtype == TQ_BF16, TQ_UNSUPPORTED,
             "the two-float partial serves f32, f16 and bf16 tensors, not %s", tq::dtype_name(dtype));
  TQ_REQUIRE(count > 0, TQ_UNSUPPORTED, "a reduction over no elements has no kernel");
  TQ_REQUIRE(in != nullptr && partial != nullptr && tq::aligned_to(partial, 8), TQ_INVALID_ARGUMENT, "null input, or a partial that is not 8-byte aligned");
  const int size = tq::dtype_size(dtype);
  TQ_REQUIRE(tq::aligned_to(in, size), TQ_INVALID_ARGUMENT, "input pointer is not aligned to its element type");
  tq::DeviceScope device_scope(device);
  if (tq_status s = device_scope.status()) return s;
  // the plan of the plain reduction over [1, count, 1]: same kernels, same scratch, another finish
  const tq::Plan p = tq::plan(op == TQ_MEAN ? TQ_SUM : op, dtype, 1, count, 1, device, 16);
  const size_t need = p.need();
  TQ_REQUIRE(need == 0 || (workspace != nullptr && workspace_bytes >= need && tq::aligned_to(workspace, 16)), TQ_INVALID_ARGUMENT,
             "this reduction needs %zu bytes of 16-byte-aligned scratch (tq_reduce_workspace_bytes) and was given %zu", need, workspace_bytes);
  const auto held = tq::hold_scratch(p.ticket_bytes != 0 ? workspace : nullptr);
  cudaStream_t cuda_stream = static_cast<cudaStream_t>(stream);
#define TQ_PARTIAL(T)                                                                                                                      \
  switch (op) {                                                                                                                            \
    case TQ_AMAX: return tq::run<T, tq::ExtremePartialReducer<T, true>>(p, in, partial, 1, count, 1, false, workspace, cuda_stream);        \
    case TQ_AMIN: return tq::run<T, tq::ExtremePartialReducer<T, false>>(p, in, partial, 1, count, 1, false, workspace, cuda_stream);       \
    default: return tq::run<T, tq::SumPartialReducer<T>>(p, in, partial, 1, count, 1, false, workspace, cuda_stream);                        \
  }
  switch (dtype) {
    case TQ_F32: TQ_PARTIAL(float)
    case TQ_F16: TQ_PARTIAL(__half)
    default: TQ_PARTIAL(__nv_bfloat16)
  }
#undef TQ_PARTIAL
}

tq_status tq_reduce_launch_static(tq_reduce_op op, tq_dtype dtype, const void* in, void* out,
                                  int64_t outer, int64_t reduce, int64_t inner, int32_t device,
                                  void* stream) {
  // recorded like every other launch: the replay looks the built-in array up for the device it runs on
  TQ_RECORD_OR_RUN([=](int32_t d, void* s) { return tq_reduce_launch_static(op, dtype, in, out, outer, reduce, inner, d, s); });
  if (tq_status s = tq::validate(op, dtype, outer, reduce, inner)) return s;
  if (outer == 0 || inner == 0) return TQ_OK;
  TQ_REQUIRE(in != nullptr && out != nullptr, TQ_INVALID_ARGUMENT, "null input or output");
  const int size = tq::dtype_size(dtype);
  TQ_REQUIRE(tq::aligned_to(in, size), TQ_INVALID_ARGUMENT, "input pointer is not aligned to its element type");
  tq::DeviceScope device_scope(device);
  if (tq_status s = device_scope.status()) return s;
  const int limit = inner == 1 ? 16 : tq::column_vec_bytes(in, inner, size);
  tq::Plan p = tq::plan(op, dtype, outer, reduce, inner, device, limit);
  if (p.need() > tq::kStaticScratchBytes) p = tq::plan(op, dtype, outer, reduce, inner, device, limit, false);
  const size_t need = p.need();
  TQ_REQUIRE(need <= tq::kStaticScratchBytes, TQ_RESOURCE_EXHAUSTED,
             "this reduction needs %zu bytes of scratch; the built-in scratch of tq_reduce_launch_static holds %zu. "
             "Use tq_reduce_launch with caller-provided scratch for extents this large",
             need, tq::kStaticScratchBytes);
  void* scratch = nullptr;
  if (need != 0) {
    if (tq_status s = tq::static_scratch_for(device, &scratch)) return s;
  }
  const auto held = tq::hold_scratch(scratch);
  // Partials are overwritten before they are read and the ticket words are cleared by the launch
  // itself (a memset node on `stream`), so whatever the previous call left behind does not matter.
  cudaStream_t cuda_stream = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case TQ_F32: return tq::run_op<float>(op, p, in, out, outer, reduce, inner, scratch, cuda_stream);
    case TQ_F64: return tq::run_op<double>(op, p, in, out, outer, reduce, inner, scratch, cuda_stream);
    case TQ_F16: return tq::run_op<__half>(op, p, in, out, outer, reduce, inner, scratch, cuda_stream);
    case TQ_BF16: return tq::run_op<__nv_bfloat16>(op, p, in, out, outer, reduce, inner, scratch, cuda_stream);
    case TQ_I32: return tq::run_op<int>(op, p, in, out, outer, reduce, inner, scratch, cuda_stream);
    case TQ_I64: return tq::run_op<long long>(op, p, in, out, outer, reduce, inner, scratch, cuda_stream);
    default: return tq::fail(TQ_UNSUPPORTED, "reductions have no kernel for element type %s", tq::dtype_name(dtype));
  }
}

}  // extern "C"
