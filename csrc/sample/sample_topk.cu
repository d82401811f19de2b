// Next-token sampling in one kernel per batch: temperature, top-k filter, softmax, multinomial.
//
// One CTA per row of fp32 logits [B, V]:
//   1. (top-k) the k-th largest logit is found exactly by a 4-pass, 8-bit radix select over
//      order-preserving integer keys; every logit >= that value is kept, ties included, which is
//      what masking with `logits < topk(logits, k).values[-1]` keeps
//      (nn/gpt2/modules.py:131-133 of the reference);
//   2. a uniform number from a counter-based generator (Philox 4x32-10 keyed by seed, counter
//      = offset + row) picks the token by inverse CDF over exp((x - max) / T) of the kept logits:
//      per-thread segment sums, a block scan of those, and a serial walk inside the one segment that
//      contains the target.
// The result depends only on (logits, temperature, k, seed, offset): integer counts aside no atomics, no
// scheduling-dependent order. Replaces softmax + torch.multinomial (modules.py:134-135).
//
// One CTA works on a row, so what bounds it is latency: up to six passes over V logits. Rows of up to
// kCachedColumns are read once into shared memory and passed over there (CACHED). k = 1 needs no select.
// Otherwise logits crowd into few values of the first digit, so lanes with equal digits count together
// before they touch the histogram; the digit scan is a warp's, and the select ends as soon as the
// threshold's bin is kept whole.
#include "../common/launch.cuh"
#include <cstdint>

namespace z2h {
namespace {

constexpr int kThreads = 1024;
constexpr int kCachedColumns = 55 * 1024;  // 220 KiB

__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // larger float <-> larger key
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

__device__ __forceinline__ uint32_t mulhilo(uint32_t a, uint32_t b, uint32_t* hi) {
  const uint64_t p = (uint64_t)a * b;
  *hi = (uint32_t)(p >> 32);
  return (uint32_t)p;
}
// Philox 4x32 with 10 rounds; returns the first output word as a float in [0, 1).
__device__ float philox_uniform(uint64_t seed, uint64_t counter) {
  uint32_t c0 = (uint32_t)counter, c1 = (uint32_t)(counter >> 32), c2 = 0, c3 = 0;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0, hi1;
    const uint32_t lo0 = mulhilo(0xD2511F53u, c0, &hi0);
    const uint32_t lo1 = mulhilo(0xCD9E8D57u, c2, &hi1);
    const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return (c0 >> 8) * (1.0f / 16777216.0f);
}

__device__ __forceinline__ float block_reduce(float v, float* sh, bool is_max) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float t = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmaxf(v, t) : v + t;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = is_max ? -INFINITY : 0.f;
  for (int w = 0; w < kThreads / 32; ++w) r = is_max ? fmaxf(r, sh[w]) : r + sh[w];
  return r;
}

template <bool CACHED>
__global__ void __launch_bounds__(kThreads)
sample_topk_kernel(const float* __restrict__ logits, long long* __restrict__ out, long long out_stride, int V,
                   long long ld, float inv_temperature, int top_k, uint64_t seed, uint64_t offset) {
  extern __shared__ float cache[];
  __shared__ unsigned int hist[256];
  __shared__ float sh[kThreads / 32];
  __shared__ float seg_prefix[kThreads];
  __shared__ uint32_t s_prefix_key;
  __shared__ int s_remaining, s_whole;
  const int row = blockIdx.x, lane = threadIdx.x & 31;
  const float* x = logits + (long long)row * ld;
  float m = -INFINITY;  // of the whole row: its largest logit is kept whatever k is
  bool odd = false;     // a NaN somewhere
#pragma unroll 16
  for (int i = threadIdx.x; i < V; i += kThreads) {
    const float v = x[i];
    if (CACHED) cache[i] = v;
    m = fmaxf(m, v);
    odd |= v != v;
  }
  if (CACHED) x = cache;
  m = block_reduce(m, sh, true);
  odd = __syncthreads_or(odd);

  // ---- 1. threshold = k-th largest logit (or -inf when no top-k filter applies)
  float threshold = -INFINITY;
  if (top_k == 1 && V > 1 && !odd) {
    threshold = m;
  } else if (top_k > 0 && top_k < V) {
    uint32_t prefix = 0, mask = 0;
    int remaining = top_k;
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      for (int i = threadIdx.x; i < 256; i += kThreads) hist[i] = 0;
      __syncthreads();
      for (int i0 = 0; i0 < V; i0 += kThreads) {  // whole warps stay for the match
        const int i = i0 + threadIdx.x;
        const uint32_t k = i < V ? order_key(x[i]) : 0u;
        const bool in = i < V && (k & mask) == prefix;
        if (!__any_sync(0xffffffffu, in)) continue;
        const uint32_t digit = in ? (k >> shift) & 255u : 256u;
        const uint32_t same = __match_any_sync(0xffffffffu, digit);
        if (in && lane == __ffs(same) - 1) atomicAdd(&hist[digit], (unsigned)__popc(same));
      }
      __syncthreads();
      if (threadIdx.x < 32) {  // lane 0 holds the eight largest digits, lane 31 the smallest
        int mine = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) mine += (int)hist[255 - 8 * lane - j];
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += t;
        }
        const uint32_t reach = __ballot_sync(0xffffffffu, upto >= remaining);
        const int who = reach != 0u ? __ffs(reach) - 1 : 31;
        if (lane == who) {
          int rem = remaining - (upto - mine), b = 255 - 8 * lane;
          for (const int last = b - 7; b > last; --b) {  // walk from the largest digit down
            if ((int)hist[b] >= rem) break;
            rem -= (int)hist[b];
          }
          s_prefix_key = prefix | ((uint32_t)b << shift);
          s_remaining = rem;
          s_whole = (int)hist[b] == rem;
        }
      }
      __syncthreads();
      prefix = s_prefix_key;
      remaining = s_remaining;
      mask |= 255u << shift;
      // everything with this prefix is kept: its smallest key is threshold enough (0.0 is not: it would let
      // -0.0 in as well)
      if (s_whole && prefix != 0x80000000u) break;
      __syncthreads();
    }
    threshold = key_to_float(prefix);
    if (prefix < 0x007fffffu) threshold = -INFINITY;  // the lowest bin's smallest key is a NaN's
  }

  // ---- 2. inverse-CDF draw over contiguous per-thread segments
  const int seg = (V + kThreads - 1) / kThreads;
  const int i0 = threadIdx.x * seg, i1 = min(V, i0 + seg);
  float local = 0.f;
  for (int i = i0; i < i1; ++i) {
    const float v = x[i];
    if (v >= threshold) local += __expf((v - m) * inv_temperature);
  }
  seg_prefix[threadIdx.x] = local;
  __syncthreads();
  // inclusive Hillis-Steele scan over the 1024 segment sums
  for (int off = 1; off < kThreads; off <<= 1) {
    float t = 0.f;
    if (threadIdx.x >= off) t = seg_prefix[threadIdx.x - off];
    __syncthreads();
    seg_prefix[threadIdx.x] += t;
    __syncthreads();
  }
  const float total = seg_prefix[kThreads - 1];
  const float target = philox_uniform(seed, offset + row) * total;
  const float before = threadIdx.x == 0 ? 0.f : seg_prefix[threadIdx.x - 1];
  const float upto = seg_prefix[threadIdx.x];
  // exactly one non-empty segment satisfies before <= target < upto (the last one also takes
  // target == total, which rounding can produce)
  const bool last_nonempty = (upto == total) && (before < total);
  if (local > 0.f && target >= before && (target < upto || last_nonempty)) {
    float acc = before;
    int pick = -1;
    for (int i = i0; i < i1; ++i) {
      const float v = x[i];
      if (v >= threshold) {
        acc += __expf((v - m) * inv_temperature);
        pick = i;  // the last kept index so far: the fallback when rounding leaves acc < target
        if (acc > target) break;
      }
    }
    if (pick >= 0) out[row * out_stride] = pick;
  }
}

}  // namespace

int sample_topk(const float* logits, long long* out, long long out_stride, int B, int V, long long ld,
                float temperature, int top_k, unsigned long long seed, unsigned long long offset,
                cudaStream_t stream) {
  if (B <= 0) return 0;
  if (V <= 0 || !(temperature > 0.f)) return 1;
  if (V > kCachedColumns) {
    sample_topk_kernel<false><<<B, kThreads, 0, stream>>>(logits, out, out_stride, V, ld, 1.0f / temperature, top_k,
                                                          seed, offset);
  } else {
    static std::atomic<unsigned long long> seen{0};
    if (first_use_on_current_device(seen) &&
        cudaFuncSetAttribute(sample_topk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kCachedColumns * 4) != cudaSuccess)
      return 3;
    sample_topk_kernel<true><<<B, kThreads, (size_t)V * 4, stream>>>(logits, out, out_stride, V, ld, 1.0f / temperature,
                                                                     top_k, seed, offset);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace z2h

// The id of row b is written to out[b * out_stride].
extern "C" int z2h_sample_topk_strided(const float* logits, long long* out, long long out_stride, int B, int V,
                                       long long ld, float temperature, int top_k, unsigned long long seed,
                                       unsigned long long offset, void* stream) {
  return z2h::sample_topk(logits, out, out_stride, B, V, ld, temperature, top_k, seed, offset, (cudaStream_t)stream);
}
