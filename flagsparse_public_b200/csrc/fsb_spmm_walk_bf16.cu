// Range-walk SpMM instantiations for __nv_bfloat16 values (see fsb_spmm_walk.cuh).
#include "fsb_spmm_walk.cuh"

namespace fsb {
FSB_SEQ_DECL(walk_dispatch_bf16) {
    return walk_dispatch_for<__nv_bfloat16>(A, B, ldb, n_dense, C, ldc, out_dtype, acc_mode, plan, workspace, workspace_bytes, st);
}
}  // namespace fsb
