// Range-walk SpMM instantiations for c64_t values (see fsb_spmm_walk.cuh).
#include "fsb_spmm_walk.cuh"

namespace fsb {
FSB_SEQ_DECL(walk_dispatch_c64) {
    return walk_dispatch_for<c64_t>(A, B, ldb, n_dense, C, ldc, out_dtype, acc_mode, plan, workspace, workspace_bytes, st);
}
}  // namespace fsb
