// The one-CTA GEMM with 128x64 tiles (see pick_bn in gemm_tcgen05.cu).
#include "gemm_onecta.cuh"

namespace z2h {
int gemm_bf16_narrow64(const GemmArgs& args, cudaStream_t stream) { return launch_onecta<64>(args, stream); }
}  // namespace z2h
