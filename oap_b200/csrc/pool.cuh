// The library's stream-ordered workspace pools (gram.cu): memory freed to them
// is kept for the next call instead of being unmapped at the next
// synchronisation; oapb_gram_trim gives it back.
#pragma once

#include <cuda_runtime.h>

namespace oapb {

// the current device's pool, null when it cannot be created; a bounded one
// keeps 1 GiB at most
cudaMemPool_t workspace_pool(bool bounded);

}  // namespace oapb
