// What the library's own parts need of a context beyond the C interface.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

#include "../../include/dagc.h"

namespace dagc {

// A device allocation on a context's account: failed ones are counted, and
// retried once the context's cache and the process's idle brick tables are
// given back. Freed with cudaFree.
cudaError_t context_malloc(dagc_context ctx, void** p, size_t bytes);

}  // namespace dagc
