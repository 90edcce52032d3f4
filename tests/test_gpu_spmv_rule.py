"""The SpMV plan rules: the native copy (one-shot calls) and the Python copy
(prepared calls) agree over the ranges where a limit lies, and the rule's row
groups are not far from the best of all group widths on long rows."""

import ctypes

import pytest
import torch

from flagsparse_public_b200 import _native as nat
from flagsparse_public_b200 import _plan
from tests.test_gpu_split_rows import _graph_us

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _even(rows, mean, extra=0, cols=4096):
    """``rows`` rows of ``mean`` nonzeros (the middle one ``extra`` more)."""
    lens = torch.full((rows,), mean, dtype=torch.int64, device=DEV)
    lens[rows // 2] += extra
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = lens.cumsum(0)
    return ptr, torch.randint(0, cols, (int(ptr[-1]),), device=DEV), cols


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32, torch.float64, torch.complex64, torch.complex128])
@pytest.mark.parametrize("index_dtype", [torch.int32, torch.int64])
def test_native_and_python_rules_agree(dtype, index_dtype):
    lib = nat.library()
    cases = [(r, m, 0) for r in (37, 5000, 151552) for m in (1, 11, 12, 23, 24)]
    cases += [(r, m, 0) for r in (37, 5000) for m in (63, 64, 79, 80, 127, 128, 199, 200, 511, 512)]
    cases += [(2000, m, e) for m in (8, 31, 32, 33, 127, 128) for e in (900, 1100, 2100, 4200, 9000)]
    cases += [(60000, 34, 600), (61700, 34, 600)]  # either side of 2^21 nonzeros
    for rows, mean, extra in cases:
        ptr, col, cols = _even(rows, mean, extra)
        col = col.to(index_dtype)
        data = torch.ones(col.numel(), dtype=dtype, device=DEV)
        x, y = torch.ones(cols, dtype=dtype, device=DEV), torch.empty(rows, dtype=dtype, device=DEV)
        cm = nat.make_csr(data, col, ptr, rows, cols)
        nbytes = int(lib.fsb_spmv_csr_checked_workspace_bytes(cm, nat.ACC_NATIVE, nat.dtype_code(dtype)))
        ws = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
        fig, plan = (ctypes.c_int64 * 8)(), nat.FsbPlan()
        rc = lib.fsb_spmv_csr_checked(cm, nat.ptr(x), nat.ptr(y), nat.dtype_code(dtype), nat.ACC_NATIVE, nat.ptr(ws),
                                      nbytes, fig, plan, nat.stream_handle(y.device))
        nat.check(rc, "fsb_spmv_csr_checked")
        ref = _plan.default_spmv_plan(_plan.matrix_stats(ptr, rows, cols), dtype, index_bytes=col.element_size())
        assert plan.algo == ref.algo, (rows, mean, extra)
        if ref.algo == nat.ALGO_ROWS:
            assert plan.lanes == ref.lanes, (rows, mean, extra)
        else:
            assert plan.items_per_unit == ref.items_per_unit, (rows, mean, extra)


@pytest.mark.parametrize("dtype,index_dtype,rows,mean", [
    (torch.bfloat16, torch.int64, 10000, 1000), (torch.float64, torch.int32, 10000, 1000),
    (torch.complex128, torch.int32, 30000, 300), (torch.float32, torch.int32, 5000, 3000)])
def test_rows_of_hundreds_take_many_lanes(dtype, index_dtype, rows, mean):
    """The rule's lanes take at most 1.3 times the best of 2 to 32."""
    ptr, col, cols = _even(rows, mean, cols=rows)
    col = col.to(index_dtype)
    data = torch.ones(col.numel(), device=DEV).to(dtype)
    x, y = torch.ones(cols, device=DEV).to(dtype), torch.empty(rows, dtype=dtype, device=DEV)
    plan = _plan.default_spmv_plan(_plan.matrix_stats(ptr, rows, cols), dtype, index_bytes=col.element_size())
    us = {lanes: _graph_us(lambda: _plan.run_spmv(data, col, ptr, rows, cols, x, y, nat.ACC_NATIVE,
                                                  _plan.KernelPlan(nat.ALGO_ROWS, lanes=lanes)))
          for lanes in (2, 4, 8, 16, 32)}
    assert plan.algo == nat.ALGO_ROWS and us[plan.lanes] <= 1.3 * min(us.values()), (plan.lanes, us)
