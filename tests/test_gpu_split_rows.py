"""Rows split over many merge-path units: the sums of their partials
(k_spmv_merge_fixup by lane and by warp, k_spmm_merge_fixup with its loads
ahead) at the run lengths where a form of the loop begins or ends, against the
FP64 oracle; and that a long row costs no more in small units than in large
ones.

Bounds (condition-scaled, tests/numerics.py): those of the other SpMV / SpMM
forms; float32 sums of n products err by about (log2 n + chain) * 2^-24 of
their magnitude with chains of at most 400 additions here, 3e-5."""

import pytest
import torch

from flagsparse_public_b200 import _native as nat
from flagsparse_public_b200 import _plan
from oracle import oracle as orc
from tests.gpu_cases import csr_from_lengths, dense
from tests.numerics import REL_BOUND, scaled_error

pytestmark = pytest.mark.gpu
DEV = "cuda"
ITEMS = 128
MODES = [(torch.float32, nat.ACC_NATIVE, 3e-5), (torch.float32, nat.ACC_WIDE, REL_BOUND[torch.float32]),
         (torch.float64, nat.ACC_NATIVE, REL_BOUND[torch.float64]),
         (torch.complex128, nat.ACC_NATIVE, REL_BOUND[torch.complex128])]


@pytest.mark.parametrize("units", [1, 2, 5, 6, 33, 37, 38, 133, 134, 300])
@pytest.mark.parametrize("mode", MODES, ids=lambda m: f"{str(m[0])[6:]}-{m[1]}")
def test_row_over_units(units, mode):
    """A row over ``units`` units, beside a second one over three, single-unit
    rows and empty ones."""
    dtype, acc, bound = mode
    lengths = [3, 0, units * ITEMS - 40, 1, 0, 0, 3 * ITEMS, 5, ITEMS, 2]
    data, indices, indptr, (n_rows, n_cols) = csr_from_lengths(lengths, 300 * ITEMS, seed=units, dtype=dtype)
    d = (data.to(DEV), indices.to(DEV), indptr.to(DEV))
    x = dense((n_cols,), 71, dtype)
    exact, mag = orc.spmv_csr_exact(data, indices, indptr, x)
    y = torch.full((n_rows,), float("nan"), dtype=dtype, device=DEV)
    _plan.run_spmv(*d, n_rows, n_cols, x.to(DEV), y, acc, _plan.KernelPlan(nat.ALGO_MERGE, items_per_unit=ITEMS))
    assert scaled_error(y, exact, mag) <= bound
    for n_dense in (1, 33, 100):
        B = dense((n_cols, n_dense), 72, dtype)
        exact, mag = orc.spmm_csr_exact(data, indices, indptr, B)
        for flags in (0, nat.PLAN_WALK):
            out = []
            for runs in (None, False):  # finished in the kernel, and by the fix-up kernel
                plan = _plan.KernelPlan(nat.ALGO_SEQ, items_per_unit=ITEMS, flags=flags)
                plan.runs = runs
                C = torch.full((n_rows, n_dense), float("nan"), dtype=dtype, device=DEV)
                _plan.run_spmm(*d, n_rows, n_cols, B.to(DEV), C, acc, plan)
                out.append(C)
            assert torch.equal(out[0], out[1]), (n_dense, flags)
            assert scaled_error(out[0], exact, mag) <= bound, (n_dense, flags)


def _graph_us(fn, launches=10):
    """Best of five replays, us per call of ``fn``."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(launches):
            fn()
    best = float("inf")
    for _ in range(5):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(end) * 1e3 / launches)
    return best


def _arrow(n, dtype):
    """n rows of 2 nonzeros, one of them with n."""
    lens = torch.full((n,), 2, dtype=torch.int64, device=DEV)
    lens[n // 3] = n
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = lens.cumsum(0)
    g = torch.Generator(device=DEV).manual_seed(5)
    nnz = int(ptr[-1])
    col = torch.randint(0, n, (nnz,), generator=g, device=DEV, dtype=torch.int32)
    return torch.rand(nnz, generator=g, device=DEV).to(dtype) - 0.5, col, ptr


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_dense_row_in_default_spmv_units(dtype):
    """The default plan's units (128 items here, 782 of them on the row) take
    no longer than twice the time of the largest ones."""
    n = 100000
    data, col, ptr = _arrow(n, dtype)
    x, y = torch.rand(n, device=DEV).to(dtype), torch.empty(n, dtype=dtype, device=DEV)
    default = _plan.default_spmv_plan(_plan.matrix_stats(ptr, n, n), dtype)
    assert default.algo == nat.ALGO_MERGE and default.items_per_unit < 1024
    us = [_graph_us(lambda: _plan.run_spmv(data, col, ptr, n, n, x, y, nat.ACC_NATIVE, plan))
          for plan in (default, _plan.KernelPlan(nat.ALGO_MERGE, items_per_unit=1024))]
    assert us[0] <= 2.0 * us[1], us


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_dense_row_by_the_spmm_fixup(dtype):
    """128 columns: the separate fix-up (one-shot products) takes no longer
    than twice the time of the finish inside the kernel."""
    n, n_dense = 100000, 128
    data, col, ptr = _arrow(n, dtype)
    B, C = torch.rand(n, n_dense, device=DEV).to(dtype), torch.empty(n, n_dense, dtype=dtype, device=DEV)
    us = []
    for runs in (False, None):
        plan = _plan.default_spmm_plan(_plan.matrix_stats(ptr, n, n), n_dense, dtype)
        plan.runs = runs
        us.append(_graph_us(lambda: _plan.run_spmm(data, col, ptr, n, n, B, C, nat.ACC_NATIVE, plan)))
    assert us[0] <= 2.0 * us[1], us
