// What the library's own parts need of a context beyond the C interface.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/dagc.h"

namespace dagc {

// A device allocation on a context's account: failed ones are counted, and
// retried once the context's cache and the process's idle brick tables are
// given back. Freed with cudaFree.
cudaError_t context_malloc(dagc_context ctx, void** p, size_t bytes);

// Bytes of the brick table (DAGC_OPT_BRICK_TABLE) that a call may take, beyond
// dagc_create_footprint, and that a context holds now.
uint64_t brick_table_bytes(uint64_t n, int depth);
uint64_t brick_table_held(dagc_context ctx);

}  // namespace dagc
