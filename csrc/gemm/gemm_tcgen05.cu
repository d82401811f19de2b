// The one-CTA GEMM (gemm_onecta.cuh) with 128x256 tiles, and the choice between the GEMM kernels.
#include "gemm_onecta.cuh"

namespace z2h {

static int g_algo = 2;
void gemm_set_algo(int algo) { g_algo = algo; }
int gemm_get_algo() { return g_algo; }

// Tile width of the one-CTA kernel. A wave of 128 x BN tiles costs 4 * (44 + BN / 2) tensor-pipe cycles a
// k-block (64 deep; no less than about 400, what issuing and waiting take) and some 1,500 + 4 BN to fill and
// drain. Narrow tiles are less efficient each, but where 256 columns leave SMs without a tile they finish
// first. Measured at 256 / 128 / 64 columns, us: M1024 N768 K768 9.4 / 8.4 / 7.8, M1024 N2304 K768
// 9.8 / 9.2 / 12.7, M2545 N1152 K384 8.0 / 9.2 / 10.9, M512 N384 K128 6.2 / 5.3 / 4.4.
static int pick_bn(long long M, long long N, long long K, long long sms) {
  const long long kb = (K + 63) / 64, tm = (M + 127) / 128;
  int best = 256;
  long long best_cost = 0;
  for (int bn = 256; bn >= 64; bn /= 2) {
    const long long waves = (tm * ((N + bn - 1) / bn) + sms - 1) / sms, mma = 4 * (44 + bn / 2);
    const long long cost = waves * (kb * (mma < 400 ? 400 : mma) + 1500 + 4 * bn);
    if (bn == 256 || cost < best_cost) { best = bn; best_cost = cost; }
  }
  return best;
}

// Whether pairs of SMs would need another wave for a few 256 x 256 tiles where single SMs do not. A wave of
// pairs is the shorter one (0.8 of a wave of single SMs at K 768), so one wave less pays while there are few:
// single / pairs, us, at 2 waves of pairs (M808 N4800 K1600) 14.3 / 22.2, 3 (M1920 N4800 K768) 16.5 / 19.9, 6
// (M2331 N9600 K768) 32.4 / 33.1; but at 8 (M640 N50264 K768) 66.7 / 58.8, at 27 (M2331 N50264 K768) 211 / 176.
// A short contraction is bound by its stores, alike in both: K 192 at 27 waves 150 to 161 / 160.
static bool pairs_spill_over(long long M, long long N, long long K, long long sms) {
  const long long tn = (N + 255) / 256;
  const long long pairs = ((M + 255) / 256 * tn + sms / 2 - 1) / (sms / 2);
  return ((M + 127) / 128 * tn + sms - 1) / sms < pairs && (pairs <= 6 || K <= 192);
}

// The kernel for a product without split K on `sms` SMs: 2 = CTA pairs, else the tile width of the one-CTA
// kernel.
static int pick_kernel(long long M, long long N, long long K, long long sms) {
  const long long tiles = (M + 255) / 256 * ((N + 255) / 256);
  if (M >= 256 && tiles >= sms / 2 && !pairs_spill_over(M, N, K, sms)) return 2;
  return pick_bn(M, N, K, sms);
}

int gemm_bf16(const GemmArgs& g, cudaStream_t stream) {
  // argument checks: everything the TMA descriptors and the vector epilogue rely on
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(g.A) & 15) || (reinterpret_cast<uintptr_t>(g.B) & 15) ||
      (reinterpret_cast<uintptr_t>(g.C) & 15))
    return 1;
  if ((g.lda % 8) || (g.ldb % 8) || (g.ldc % 8)) return 1;
  if ((g.epi == kEpiAtomicAdd || g.epi == kEpiAccumulate) && !g.out_fp32) return 1;
  if (g.split_k > 1 && g.epi != kEpiAtomicAdd && g.epi != kEpiSliceStore) return 1;
  if (g.epi == kEpiSliceStore && (!g.out_fp32 || g.split_k < 1 || g.bias != nullptr ||
                                  g.slice_stride < (long long)(g.M - 1) * g.ldc + g.N || (g.slice_stride % 4)))
    return 1;
  if (g.epi == kEpiResidual && (g.residual == nullptr || (g.ldr % 8))) return 1;
  if (g.epi == kEpiGelu && (g.aux_out == nullptr || (g.ldaux % 8))) return 1;
  if (g.epi == kEpiGeluGrad && (g.aux_in == nullptr || (g.ldaux % 8))) return 1;
  if (g.epi == kEpiGeluSaveGrad && (g.aux_out == nullptr || (g.ldaux % 8) || g.out_fp32)) return 1;
  if (g.epi == kEpiMulAux && (g.aux_in == nullptr || (g.ldaux % 8) || g.out_fp32)) return 1;
  if (g.epi < kEpiNone || g.epi > kEpiSliceStore) return 1;
  if (reinterpret_cast<uintptr_t>(g.bias) & 7) return 1;
  if (g.colsum != nullptr && (g.out_fp32 || g.split_k != 1 || (g.M % 32) || (g.N % 32) ||
                              (reinterpret_cast<uintptr_t>(g.colsum) & 3)))
    return 1;
  if ((reinterpret_cast<uintptr_t>(g.residual) & 15) || (reinterpret_cast<uintptr_t>(g.aux_out) & 15) ||
      (reinterpret_cast<uintptr_t>(g.aux_in) & 15))
    return 1;
  int kernel = g_algo == 0 ? 256 : g_algo == 1 ? (g.M >= 256 ? 2 : 256) : g_algo;
  if (g_algo == 2) {
    const bool stream_k = g.split_k <= 0 && g.epi == kEpiAtomicAdd;  // fills every SM whatever the tile count
    // split-K and stream-K launches always take the pair kernel: it measured faster at every factor
    if (stream_k || g.split_k > 1) kernel = g.M >= 256 ? 2 : 256;
    else kernel = pick_kernel(g.M, g.N, g.K, sm_count_current_device());
    if (kernel != 2 && g.max_ctas > 0) kernel = 256;
  }
  switch (kernel) {
    case 2: return gemm_bf16_pair(g, stream);
    case 64: return gemm_bf16_narrow64(g, stream);
    case 128: return gemm_bf16_narrow128(g, stream);
    default: return launch_onecta<256>(g, stream);
  }
}

}  // namespace z2h

#ifdef Z2H_KERNEL_TRACE
extern "C" int z2h_gemm_trace_read(long long* host_out) {
  return (int)cudaMemcpyFromSymbol(host_out, g_kernel_trace, sizeof(g_kernel_trace));
}
#endif
extern "C" void z2h_gemm_set_algo(int algo) { z2h::gemm_set_algo(algo); }
extern "C" void z2h_gemm_set_fixup(int on) { z2h::gemm_set_fixup(on); }
// Which kernel the automatic choice takes for a product without split K (see pick_kernel).
extern "C" int z2h_gemm_pick_kernel(int M, int N, int K, int sms) { return z2h::pick_kernel(M, N, K, sms); }
extern "C" int z2h_gemm_get_algo() { return z2h::gemm_get_algo(); }
namespace z2h {
namespace {
__global__ void fold_slices_kernel(const float* __restrict__ slices, int num_slices, long long n4,
                                   float* __restrict__ dst) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4;
       i += (long long)gridDim.x * blockDim.x) {
    float4 acc = reinterpret_cast<const float4*>(dst)[i];
    for (int s = 0; s < num_slices; ++s) {  // slice order: the sum is the same bits every time
      const float4 v = reinterpret_cast<const float4*>(slices)[(long long)s * n4 + i];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    reinterpret_cast<float4*>(dst)[i] = acc;
  }
}
}  // namespace
int gemm_fold_slices(const float* slices, int num_slices, long long n, float* dst, cudaStream_t stream) {
  if (n % 4 != 0 || num_slices < 1 || (reinterpret_cast<uintptr_t>(slices) & 15) ||
      (reinterpret_cast<uintptr_t>(dst) & 15))
    return 1;
  const long long n4 = n / 4;
  const int grid = (int)((n4 + 255) / 256 < 148 * 8 ? (n4 + 255) / 256 : 148 * 8);
  fold_slices_kernel<<<grid < 1 ? 1 : grid, 256, 0, stream>>>(slices, num_slices, n4, dst);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}
}  // namespace z2h

extern "C" int z2h_gemm_fold_slices(const float* slices, int num_slices, long long n, float* dst, void* stream) {
  return z2h::gemm_fold_slices(slices, num_slices, n, dst, reinterpret_cast<cudaStream_t>(stream));
}

// z2h_gemm_bf16 plus the column-sum by-product (GemmArgs::colsum) and the K-slice stride of
// kEpiSliceStore (GemmArgs::slice_stride).
extern "C" int z2h_gemm_bf16_ex(const void* A, int a_mn, long long lda, const void* B, int b_mn,
                                long long ldb, void* C, long long ldc, int out_fp32, int M, int N, int K,
                                int epi, int split_k, const void* bias, const void* residual,
                                long long ldr, void* aux_out, const void* aux_in, long long ldaux,
                                int* status, int max_ctas, void* colsum, long long slice_stride, void* stream) {
  z2h::GemmArgs g;
  g.A = A; g.a_mn = a_mn; g.lda = lda;
  g.B = B; g.b_mn = b_mn; g.ldb = ldb;
  g.C = C; g.ldc = ldc; g.out_fp32 = out_fp32;
  g.M = M; g.N = N; g.K = K;
  g.epi = epi; g.split_k = split_k;
  g.bias = bias; g.residual = residual; g.ldr = ldr;
  g.aux_out = aux_out; g.aux_in = aux_in; g.ldaux = ldaux;
  g.status = status; g.max_ctas = max_ctas;
  g.colsum = colsum;
  g.slice_stride = slice_stride;
  return z2h::gemm_bf16(g, reinterpret_cast<cudaStream_t>(stream));
}
extern "C" int z2h_gemm_bf16_colsum(const void* A, int a_mn, long long lda, const void* B, int b_mn,
                                    long long ldb, void* C, long long ldc, int out_fp32, int M, int N, int K,
                                    int epi, int split_k, const void* bias, const void* residual,
                                    long long ldr, void* aux_out, const void* aux_in, long long ldaux,
                                    int* status, int max_ctas, void* colsum, void* stream) {
  return z2h_gemm_bf16_ex(A, a_mn, lda, B, b_mn, ldb, C, ldc, out_fp32, M, N, K, epi, split_k, bias, residual,
                          ldr, aux_out, aux_in, ldaux, status, max_ctas, colsum, 0, stream);
}
extern "C" int z2h_gemm_bf16(const void* A, int a_mn, long long lda, const void* B, int b_mn,
                             long long ldb, void* C, long long ldc, int out_fp32, int M, int N, int K,
                             int epi, int split_k, const void* bias, const void* residual,
                             long long ldr, void* aux_out, const void* aux_in, long long ldaux,
                             int* status, int max_ctas, void* stream) {
  return z2h_gemm_bf16_colsum(A, a_mn, lda, B, b_mn, ldb, C, ldc, out_fp32, M, N, K, epi, split_k, bias,
                              residual, ldr, aux_out, aux_in, ldaux, status, max_ctas, nullptr, stream);
}
