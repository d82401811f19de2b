// Activations of the MLP outside the GEMMs: ReLU, and the backward of GELU (dx = dy * gelu'(x) for a saved
// bf16 x) and ReLU (dx = 0 where the output is zero or less, dy elsewhere, at a NaN too), with the column
// sums of dx (the bias gradient of the layer that produced x) added up on the way.
//
// Bound by memory: 6 bytes an element. A CTA takes 256 columns (32 lanes x 8) of a slab of rows, one row
// per warp; a thread keeps its 8 column sums in registers over the slab, the 8 warps fold theirs in
// shared memory and one atomic per column joins the slabs. tanh comes from the hardware exponential
// (error around 1e-6, as exact as the bf16 output can show).
#include "../common/launch.cuh"
#include "../common/ptx.cuh"

namespace z2h {
namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ float gelu_tanh_grad_exact(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float u = fminf(fmaxf(k0 * (x + k1 * x * x * x), -15.f), 15.f);
  const float t = 1.f - __fdividef(2.f, __expf(2.f * u) + 1.f);
  const float d = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
  return fabsf(x) >= 12.f ? (x > 0.f ? 1.f : 0.f) : d;  // 0 * inf beyond fp32's range of x^3
}

template <bool RELU>
__global__ void __launch_bounds__(kWarps * 32)
act_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ pre,
                __nv_bfloat16* __restrict__ dx, float* __restrict__ db, int M, int N, int rows_per_slab) {
  __shared__ float sums[kWarps][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  const int r1 = min(M, (int)(blockIdx.y + 1) * rows_per_slab);
  float s[8] = {};
  if (col < N) {
#pragma unroll 4
    for (int r = blockIdx.y * rows_per_slab + warp; r < r1; r += kWarps) {
      const long long at = (long long)r * N + col;
      const uint4 g = *reinterpret_cast<const uint4*>(dy + at), x = *reinterpret_cast<const uint4*>(pre + at);
      const uint32_t *gw = &g.x, *xw = &x.x;
      uint4 o;
      uint32_t* ow = &o.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = unpack_bf16x2(gw[j]), b = unpack_bf16x2(xw[j]);
        ow[j] = RELU ? pack_bf16x2(b.x <= 0.f ? 0.f : a.x, b.y <= 0.f ? 0.f : a.y)
                     : pack_bf16x2(a.x * gelu_tanh_grad_exact(b.x), a.y * gelu_tanh_grad_exact(b.y));
        const float2 q = unpack_bf16x2(ow[j]);  // the sums are those of the stored values
        s[2 * j] += q.x;
        s[2 * j + 1] += q.y;
      }
      *reinterpret_cast<uint4*>(dx + at) = o;
    }
  }
  if (db == nullptr) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) sums[warp][lane * 8 + j] = s[j];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < N) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += sums[w][threadIdx.x];
    atomicAdd(db + c, t);
  }
}

// max(x, 0), NaN kept
__global__ void __launch_bounds__(256) relu_kernel(uint4* x, long long vecs) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < vecs; i += gridDim.x * 256ll) {
    uint4 u = x[i];
    uint32_t* w = &u.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(w[j]);
      w[j] = pack_bf16x2(f.x < 0.f ? 0.f : f.x, f.y < 0.f ? 0.f : f.y);
    }
    x[i] = u;
  }
}

}  // namespace

template <bool RELU>
static int act_bwd(const void* dy, const void* pre, void* dx, float* db, int M, int N, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (N % 8 || ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(dx)) & 15))
    return 1;
  const int cols = (N + 255) / 256;
  // about eight CTAs per SM, at least four rows per warp
  int slabs = (8 * sm_count_current_device() + cols - 1) / cols;
  int rows = (M + slabs - 1) / slabs;
  if (rows < 4 * kWarps) rows = 4 * kWarps;
  slabs = (M + rows - 1) / rows;
  act_bwd_kernel<RELU><<<dim3(cols, slabs), kWarps * 32, 0, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)pre,
                                                                     (__nv_bfloat16*)dx, db, M, N, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int gelu_bwd(const void* dy, const void* pre, void* dx, float* db, int M, int N, cudaStream_t stream) {
  return act_bwd<false>(dy, pre, dx, db, M, N, stream);
}
int relu_bwd(const void* dy, const void* out, void* dx, float* db, int M, int N, cudaStream_t stream) {
  return act_bwd<true>(dy, out, dx, db, M, N, stream);
}
int relu(void* x, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) return 1;
  const long long ctas = (n / 8 + 255) / 256, most = 8 * sm_count_current_device();
  relu_kernel<<<(int)(ctas < most ? ctas : most), 256, 0, stream>>>((uint4*)x, n / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace z2h

// dy, pre, dx: bf16 [M, N], tight; db: fp32 [N], added to, or null
extern "C" int z2h_gelu_bwd(const void* dy, const void* pre, void* dx, float* db, int M, int N, void* stream) {
  return z2h::gelu_bwd(dy, pre, dx, db, M, N, (cudaStream_t)stream);
}
// the same for y = max(x, 0), from y
extern "C" int z2h_relu_bwd(const void* dy, const void* out, void* dx, float* db, int M, int N, void* stream) {
  return z2h::relu_bwd(dy, out, dx, db, M, N, (cudaStream_t)stream);
}
// in place over n bf16
extern "C" int z2h_relu(void* x, long long n, void* stream) { return z2h::relu(x, n, (cudaStream_t)stream); }
