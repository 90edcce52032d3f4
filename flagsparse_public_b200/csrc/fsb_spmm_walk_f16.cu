// Range-walk SpMM instantiations for __half values (see fsb_spmm_walk.cuh).
#include "fsb_spmm_walk.cuh"

namespace fsb {
FSB_SEQ_DECL(walk_dispatch_f16) {
    return walk_dispatch_for<__half>(A, B, ldb, n_dense, C, ldc, out_dtype, acc_mode, plan, workspace, workspace_bytes, st);
}
}  // namespace fsb
