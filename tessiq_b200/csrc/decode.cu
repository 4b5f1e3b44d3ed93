// Attention of a few new tokens against many keys (decoding), for sm_100a.
//
//   out[b,h,i,:] = sum_j softmax_j(scale * q[b,h,i,:] . k[b,h,j,:]) v[b,h,j,:]     (j <= i when causal), i < 4
//
// With one or two query rows there is nothing for the tensor cores to reuse: each key and value is read
// once and takes part in a handful of multiply-adds, so the kernel is a stream of K and V (bound: HBM). Three or
// four come here only where sharing a head's keys among CTAs is worth more (choose_attention_form).
// The tensor-core kernel, which pads the queries to a tile and walks a head's keys in one CTA, took 77.9 us for 64 x 12
// heads of 64 over 1000 keys when its tile was 256 rows, where the bytes take 30.5; this one takes 41.1 (4.8 TB/s; 64 x 16
// heads over 3000 keys 129 = 6.1 TB/s).
//
// A key's row is spread over LANES neighbouring lanes, 16 bytes each, so that a load instruction of a warp
// covers 32 / LANES whole rows; a lane keeps kUnroll keys and as many values in flight (8 KiB a warp for one
// query). The lanes of a row agree on its score by shuffles and then hold the matching 16 bytes of the
// value, so a probability never moves: each set of LANES lanes runs an online softmax of its own over its
// keys (maximum, sum and result in f32, probabilities never rounded), and the sets meet once, at the end:
// by shuffles in the warp, through shared memory in the CTA, and through distributed shared memory in the
// cluster of up to eight CTAs that share one head's keys when there are too few heads to fill the GPU.
#include <mutex>

#include "common.h"
#include "tcgen05.h"

namespace tq {
namespace {

constexpr int kDecodeThreads = 128;
constexpr int kDecodeWarps = kDecodeThreads / 32;
constexpr int kDecodeMaxSplit = 8;

struct DecodeParams {
  const void *q, *k, *v;
  void* out;
  long long q_strides[3], k_strides[3], v_strides[3], out_strides[3];   // batch, head, token, in elements
  int heads, q_tokens, k_tokens, head_dim;
  int split;                       // CTAs of a cluster that share a head's keys
  int causal;
  float scale_log2;                // scale * log2(e)
};

// Two neighbouring 16-bit elements as f32.
template <typename T>
__device__ __forceinline__ float2 widen(uint32_t pair) {
  if constexpr (std::is_same_v<T, __nv_bfloat16>) {
    return make_float2(__uint_as_float(pair << 16), __uint_as_float(pair & 0xffff0000u));
  } else {
    return __half22float2(*reinterpret_cast<const __half2*>(&pair));
  }
}

// The factor that brings what was gathered against the reference point `from` to the reference point `to`.
// Where nothing finite has been seen on either side it is 1: there is nothing, or a NaN, to bring along.
__device__ __forceinline__ float rescaling(float from, float to) { return from == to ? 1.f : exp2_ftz(from - to); }

__device__ __forceinline__ uint4 load_streaming(const void* pointer) {
  uint4 word;
  asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(word.x), "=r"(word.y), "=r"(word.z), "=r"(word.w) : "l"(pointer));
  return word;
}

__device__ __forceinline__ float remote_float(uint32_t cluster_address) {
  float value;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(value) : "r"(cluster_address) : "memory");
  return value;
}

template <typename T, int LANES, int QUERIES>
__global__ void __launch_bounds__(kDecodeThreads, 4) attention_decode_kernel(const DecodeParams p) {
  constexpr int kSets = 32 / LANES;                    // rows a load instruction covers
  constexpr int kUnroll = QUERIES == 1 ? 8 : 4;        // keys in flight per lane
  constexpr int kWidth = LANES * 8;                    // head elements, rounded up to a power of two
  constexpr int kChunk = kSets * kUnroll;              // keys a warp takes at a time
  struct Part {
    float maximum, sum;
    float result[kWidth];
  };
  __shared__ Part parts[kDecodeWarps][QUERIES];
  __shared__ Part merged[QUERIES];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int set = lane / LANES, column = (lane % LANES) * 8;
  const bool live = column < p.head_dim;               // heads of 24 or 40 elements leave lanes without columns
  const int rank = static_cast<int>(blockIdx.x) % p.split;
  const int head_index = static_cast<int>(blockIdx.x) / p.split;
  const int head = head_index % p.heads, batch = head_index / p.heads;

  float2 query[QUERIES][4];
#pragma unroll
  for (int n = 0; n < QUERIES; ++n) {
    uint4 word = make_uint4(0, 0, 0, 0);
    if (live && n < p.q_tokens) {
      word = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.q) + batch * p.q_strides[0] + head * p.q_strides[1] + n * p.q_strides[2] + column);
    }
    query[n][0] = widen<T>(word.x);
    query[n][1] = widen<T>(word.y);
    query[n][2] = widen<T>(word.z);
    query[n][3] = widen<T>(word.w);
  }

  // This CTA's keys: an even share. Under a causal mask no query sees a key beyond its own index.
  const int keys = p.causal ? min(p.k_tokens, p.q_tokens) : p.k_tokens;
  const int first = static_cast<int>(static_cast<long long>(keys) * rank / p.split);
  const int last = static_cast<int>(static_cast<long long>(keys) * (rank + 1) / p.split);
  const T* k_base = static_cast<const T*>(p.k) + batch * p.k_strides[0] + head * p.k_strides[1] + column;
  const T* v_base = static_cast<const T*>(p.v) + batch * p.v_strides[0] + head * p.v_strides[1] + column;

  float maximum[QUERIES], sum[QUERIES];
  float2 result[QUERIES][4];
#pragma unroll
  for (int n = 0; n < QUERIES; ++n) {
    maximum[n] = -INFINITY;
    sum[n] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) result[n][j] = make_float2(0.f, 0.f);
  }

  for (int base = first + warp * kChunk; base < last; base += kDecodeWarps * kChunk) {
    uint4 k[kUnroll], v[kUnroll];
    auto load = [&](uint4 (&into)[kUnroll], const T* from, long long stride) {
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int key = base + u * kSets + set;
        into[u] = make_uint4(0, 0, 0, 0);
        if (live && key < last) into[u] = load_streaming(from + key * stride);
      }
    };
    load(k, k_base, p.k_strides[2]);
    load(v, v_base, p.v_strides[2]);
    float score[QUERIES][kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const float2 k0 = widen<T>(k[u].x), k1 = widen<T>(k[u].y), k2 = widen<T>(k[u].z), k3 = widen<T>(k[u].w);
      const int key = base + u * kSets + set;
#pragma unroll
      for (int n = 0; n < QUERIES; ++n) {
        float2 dot = __fmul2_rn(query[n][0], k0);
        dot = __ffma2_rn(query[n][1], k1, dot);
        dot = __ffma2_rn(query[n][2], k2, dot);
        dot = __ffma2_rn(query[n][3], k3, dot);
        float s = dot.x + dot.y;
#pragma unroll
        for (int offset = LANES / 2; offset > 0; offset /= 2) s += __shfl_xor_sync(0xffffffffu, s, offset);
        const bool seen = key < last && (!p.causal || key <= n);
        score[n][u] = seen ? s * p.scale_log2 : -INFINITY;
      }
    }
#pragma unroll
    for (int n = 0; n < QUERIES; ++n) {
      float top = maximum[n];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) top = fmaxf(top, score[n][u]);
      const float factor = rescaling(maximum[n], top);
      const float reference = top == -INFINITY ? 0.f : top;
      maximum[n] = top;
      sum[n] *= factor;
#pragma unroll
      for (int j = 0; j < 4; ++j) result[n][j] = __fmul2_rn(result[n][j], make_float2(factor, factor));
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        score[n][u] = exp2_ftz(score[n][u] - reference);
        sum[n] += score[n][u];
      }
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const float2 v0 = widen<T>(v[u].x), v1 = widen<T>(v[u].y), v2 = widen<T>(v[u].z), v3 = widen<T>(v[u].w);
#pragma unroll
      for (int n = 0; n < QUERIES; ++n) {
        const float2 weight = make_float2(score[n][u], score[n][u]);
        result[n][0] = __ffma2_rn(weight, v0, result[n][0]);
        result[n][1] = __ffma2_rn(weight, v1, result[n][1]);
        result[n][2] = __ffma2_rn(weight, v2, result[n][2]);
        result[n][3] = __ffma2_rn(weight, v3, result[n][3]);
      }
    }
  }

  // The sets of a warp meet by shuffles.
#pragma unroll
  for (int n = 0; n < QUERIES; ++n) {
#pragma unroll
    for (int offset = LANES; offset < 32; offset *= 2) {
      const float other = __shfl_xor_sync(0xffffffffu, maximum[n], offset);
      const float top = fmaxf(maximum[n], other);
      const float factor = rescaling(maximum[n], top);
      maximum[n] = top;
      sum[n] *= factor;
      sum[n] += __shfl_xor_sync(0xffffffffu, sum[n], offset);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        result[n][j] = __fmul2_rn(result[n][j], make_float2(factor, factor));
        result[n][j].x += __shfl_xor_sync(0xffffffffu, result[n][j].x, offset);
        result[n][j].y += __shfl_xor_sync(0xffffffffu, result[n][j].y, offset);
      }
    }
    if (set == 0) {
      Part& part = parts[warp][n];
      if (lane == 0) {
        part.maximum = maximum[n];
        part.sum = sum[n];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        part.result[column + 2 * j] = result[n][j].x;
        part.result[column + 2 * j + 1] = result[n][j].y;
      }
    }
  }
  __syncthreads();

  // The warps meet in shared memory; a CTA that has its head's keys to itself is done then.
  for (int item = threadIdx.x; item < QUERIES * kWidth; item += kDecodeThreads) {
    const int n = item / kWidth, c = item % kWidth;
    float top = parts[0][n].maximum;
#pragma unroll
    for (int w = 1; w < kDecodeWarps; ++w) top = fmaxf(top, parts[w][n].maximum);
    float total = 0.f, value = 0.f;
#pragma unroll
    for (int w = 0; w < kDecodeWarps; ++w) {
      const float factor = rescaling(parts[w][n].maximum, top);
      total += parts[w][n].sum * factor;
      value += parts[w][n].result[c] * factor;
    }
    if (p.split == 1) {
      if (n < p.q_tokens && c < p.head_dim) {
        static_cast<T*>(p.out)[batch * p.out_strides[0] + head * p.out_strides[1] + n * p.out_strides[2] + c] = from_compute<T, float>(value / total);
      }
    } else {
      merged[n].result[c] = value;
      if (c == 0) {
        merged[n].maximum = top;
        merged[n].sum = total;
      }
    }
  }
  if (p.split == 1) return;

  // The CTAs of the cluster meet in the first one's registers, in the order of their ranks.
  __syncwarp();
  cluster_sync_all();
  if (rank == 0) {
    for (int item = threadIdx.x; item < QUERIES * kWidth; item += kDecodeThreads) {
      const int n = item / kWidth, c = item % kWidth;
      if (n >= p.q_tokens || c >= p.head_dim) continue;
      const uint32_t maximum_at = smem_address(&merged[n].maximum), sum_at = smem_address(&merged[n].sum), value_at = smem_address(&merged[n].result[c]);
      float top = -INFINITY, total = 0.f, value = 0.f;
      float tops[kDecodeMaxSplit], sums[kDecodeMaxSplit], values[kDecodeMaxSplit];
#pragma unroll
      for (int r = 0; r < kDecodeMaxSplit; ++r) {
        if (r < p.split) {
          tops[r] = remote_float(peer_address(maximum_at, r));
          sums[r] = remote_float(peer_address(sum_at, r));
          values[r] = remote_float(peer_address(value_at, r));
        }
      }
#pragma unroll
      for (int r = 0; r < kDecodeMaxSplit; ++r) {
        if (r < p.split) top = fmaxf(top, tops[r]);
      }
#pragma unroll
      for (int r = 0; r < kDecodeMaxSplit; ++r) {
        if (r < p.split) {
          const float factor = rescaling(tops[r], top);
          total += sums[r] * factor;
          value += values[r] * factor;
        }
      }
      static_cast<T*>(p.out)[batch * p.out_strides[0] + head * p.out_strides[1] + n * p.out_strides[2] + c] = from_compute<T, float>(value / total);
    }
  }
  __syncwarp();
  cluster_sync_all();       // the others' shared memory stays until the first has read it
}

template <typename T, int LANES, int QUERIES>
tq_status launch_decode(const DecodeParams& p, long long heads_in_all, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(heads_in_all * p.split));
  config.blockDim = dim3(kDecodeThreads);
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = p.split;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = p.split > 1 ? 1 : 0;
  TQ_CUDA(cudaLaunchKernelEx(&config, attention_decode_kernel<T, LANES, QUERIES>, p));
  return check_launch("attention_decode_kernel");
}

template <typename T, int LANES>
tq_status launch_queries(const DecodeParams& p, long long heads_in_all, cudaStream_t stream) {
  if (p.q_tokens == 1) return launch_decode<T, LANES, 1>(p, heads_in_all, stream);
  if (p.q_tokens == 2) return launch_decode<T, LANES, 2>(p, heads_in_all, stream);
  return launch_decode<T, LANES, 4>(p, heads_in_all, stream);
}

template <typename T>
tq_status launch_width(const DecodeParams& p, long long heads_in_all, cudaStream_t stream) {
  if (p.head_dim <= 8) return launch_queries<T, 1>(p, heads_in_all, stream);
  if (p.head_dim <= 16) return launch_queries<T, 2>(p, heads_in_all, stream);
  if (p.head_dim <= 32) return launch_queries<T, 4>(p, heads_in_all, stream);
  if (p.head_dim <= 64) return launch_queries<T, 8>(p, heads_in_all, stream);
  return launch_queries<T, 16>(p, heads_in_all, stream);
}

// How many clusters of 1, 2, 4 and 8 CTAs run at once (148 SMs: 592, 296, 142 and 71), asked once per device; every form of the
// kernel is built for four CTAs an SM.
struct DecodeRoom {
  long long of[4];
};

DecodeRoom decode_room(int32_t device) {
  static std::mutex mutex;
  static DecodeRoom known[64] = {};
  const long long sms = sm_count(device);
  const DecodeRoom assumed = {{4 * sms, 2 * sms, sms * 24 / 25, sms * 12 / 25}};
  if (device < 0 || device >= 64) return assumed;
  std::lock_guard<std::mutex> lock(mutex);
  DecodeRoom& room = known[device];
  if (room.of[0] == 0) {
    room = assumed;
    for (int i = 1; i < 4; ++i) {
      cudaLaunchConfig_t config = {};
      config.gridDim = dim3(1u << i);
      config.blockDim = dim3(kDecodeThreads);
      cudaLaunchAttribute attribute[1];
      attribute[0].id = cudaLaunchAttributeClusterDimension;
      attribute[0].val.clusterDim.x = 1u << i;
      attribute[0].val.clusterDim.y = 1;
      attribute[0].val.clusterDim.z = 1;
      config.attrs = attribute;
      config.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, attention_decode_kernel<__nv_bfloat16, 8, 1>, &config) != cudaSuccess || clusters <= 0) {
        cudaGetLastError();
        break;
      }
      room.of[i] = clusters;
    }
  }
  return room;
}

}  // namespace

// Called by tq_attention_launch, which has checked the arguments: 1 to kDecodeQueries query rows.
tq_status attention_decode(tq_dtype dtype, const void* q, const void* k, const void* v, void* out, long long batch, long long heads,
                           long long q_tokens, long long k_tokens, long long head_dim, const int64_t* q_strides, const int64_t* k_strides,
                           const int64_t* v_strides, const int64_t* out_strides, float scale_log2, bool causal, int32_t device, cudaStream_t stream) {
  DecodeParams p = {};
  p.q = q;
  p.k = k;
  p.v = v;
  p.out = out;
  for (int i = 0; i < 3; ++i) {
    p.q_strides[i] = q_strides[i];
    p.k_strides[i] = k_strides[i];
    p.v_strides[i] = v_strides[i];
    p.out_strides[i] = out_strides[i];
  }
  p.heads = static_cast<int>(heads);
  p.q_tokens = static_cast<int>(q_tokens);
  p.k_tokens = static_cast<int>(k_tokens);
  p.head_dim = static_cast<int>(head_dim);
  p.causal = causal;
  p.scale_log2 = scale_log2;
  // Share a head's keys as long as all clusters run at once (four CTAs an SM, less what graphics processing clusters leave over) and have some
  // keys each: 96 heads of 4000 keys take 46.8, 30.6, 22.3, 26.1 us shared by 1, 2, 4, 8 CTAs, 144 heads, for which
  // clusters of four are two more than run at once, 48.4, 33.3, 38.7, 37.7, 768 of 1000 keys 44.4, 43.9, 49.9, 64.8, and 1024 of 3000
  // keys 129.6, 138.9, 145.1, 161.8.
  const long long keys = causal && q_tokens < k_tokens ? q_tokens : k_tokens;
  const DecodeRoom room = decode_room(device);
  p.split = 1;
  for (int i = 1; i < 4 && batch * heads <= room.of[i] && keys >= (96LL << (i - 1)); ++i) p.split = 1 << i;
  if (dtype == TQ_BF16) return launch_width<__nv_bfloat16>(p, batch * heads, stream);
  return launch_width<__half>(p, batch * heads, stream);
}

}  // namespace tq
