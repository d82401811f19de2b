// Cross-entropy host API.
#pragma once
#include <cuda_runtime.h>
namespace z2h {
// logits: bf16 [M, ld] (ld >= V_pad, multiple of 8); overwritten with dlogits when write_grad.
// losses: fp32 [M] per-row loss (may be null). Rows whose target equals ignore_index (or is out
// of range) contribute zero loss and zero gradient.
int ce_fwd_bwd(void* logits, const void* targets, int idx_is_64, float* losses, int M, int V_real,
               int V_pad, long long ld, float grad_scale, int write_grad, int ignore_index,
               cudaStream_t stream);
// The pair behind autograd: the forward leaves the logits alone (any pitch and 2-byte alignment; rows of
// up to 57,300 columns) and writes losses, every row's maximum and logarithm of the sum of exp(x - maximum)
// (`stats`, two floats a row) and, unless null, a copy of the logits with zeros up to the next multiple of 8
// columns; the backward turns that copy (same pitch) into (softmax - onehot) * scale * *upstream.
// `strict`: a label that is neither a class nor ignore_index gives a NaN (loss and gradient row) and
// kBadArgument in *status instead of counting as ignored. *status also reports a wait that ran out.
int ce_fwd_save(const void* logits, long long ld, const void* targets, int idx_is_64, float* losses, float* stats,
                void* copy, long long ld_copy, int M, int V, int V_real, int ignore_index, int strict, int* status,
                cudaStream_t stream);
int ce_bwd(const void* x, const void* targets, int idx_is_64, const float* stats, const float* upstream, float scale,
           void* grad, long long ld, int M, int V, int V_real, int ignore_index, int strict, cudaStream_t stream);
// dst (tight bf16 rows of N) = src (rows of pitch ld)
int compact_rows(const void* src, long long ld, void* dst, int M, int N, cudaStream_t stream);
int reduce_sum(const float* x, int n, float scale, float* out, int accumulate, cudaStream_t stream);
}  // namespace z2h
