// Products with at most 96 rows (gemm_rows.cu); rb_gemm_bf16 sends calls here.
#pragma once
#include <cuda_runtime.h>

#include "gemm_tcgen05.h"

namespace rbhost {
// Whether `gemm_rows` computes this call (arguments already checked by rb_gemm_bf16).
bool gemm_rows_takes(const RbGemmArgs& g);
// Whether it can take the rows through the norm that the call names.
bool gemm_rows_norm_takes(const RbGemmArgs& g);
int gemm_rows(const RbGemmArgs& g, cudaStream_t stream);
}  // namespace rbhost
