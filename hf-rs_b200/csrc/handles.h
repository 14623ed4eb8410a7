// The cuBLAS and cuSOLVER handles of a context.
#pragma once
#include <cublas_v2.h>
#include <cusolverDn.h>

#include "hfg_ctx.h"

namespace hfg {

// The context's handles on its stream, created on first use and released
// with the context: creating the two costs milliseconds, as much as a small
// factor's whole build, and one stream's work never shares a workspace with
// another's.  The context's lock is held.
int ctx_handles(hfg_ctx* ctx, cublasHandle_t* blas, cusolverDnHandle_t* solver);

}  // namespace hfg
