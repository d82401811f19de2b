// The one-CTA GEMM with 128x128 tiles (see pick_bn in gemm_tcgen05.cu).
#include "gemm_onecta.cuh"

namespace z2h {
int gemm_bf16_narrow128(const GemmArgs& args, cudaStream_t stream) { return launch_onecta<128>(args, stream); }
}  // namespace z2h
