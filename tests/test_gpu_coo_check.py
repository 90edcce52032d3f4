"""The COO index check (fsb_coo_check) and the permuted entries
(fsb_take_entries) against torch, at the sizes where a warp, a CTA or the
16-byte loads end; integers and copied bytes compare equal."""

import pytest
import torch

import flagsparse_public_b200 as fs
from flagsparse_public_b200 import _native as nat
from flagsparse_public_b200 import _plan
from flagsparse_public_b200.sparse_operations.spmm_coo import _run_spmm_coo_route
from tests.numerics import REL_BOUND, scaled_error

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 31, 33, 257, 2049, 300001])
@pytest.mark.parametrize("row_dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("col_dtype", [torch.int32, torch.int64])
def test_coo_check_and_take(n, row_dtype, col_dtype):
    g = torch.Generator().manual_seed(n)
    row = torch.randint(-5, 1 << 20, (n,), generator=g).to(row_dtype)
    col = torch.randint(0, 1 << 30, (n,), generator=g).to(col_dtype)
    figs, r32, c32 = nat.coo_check(row.to(DEV), col.to(DEV))
    assert figs == [int(row.min()), int(row.max()), int(col.min()), int(col.max())]
    assert r32.dtype == c32.dtype == torch.int32
    assert torch.equal(r32.cpu(), row.to(torch.int32)) and torch.equal(c32.cpu(), col.to(torch.int32))
    order = torch.randperm(n, generator=g)
    for dtype in (torch.float16, torch.float32, torch.float64, torch.complex128):
        values = torch.randn(n, generator=g, dtype=torch.float64).to(dtype)
        v, c = _plan.take_entries(values.to(DEV), c32, order.to(DEV))
        assert torch.equal(v.cpu(), values[order]) and torch.equal(c.cpu(), col.to(torch.int32)[order])


def test_coo_check_sees_wide_out_of_range_indices():
    """Bounds come from the 64-bit indices, before any narrowing."""
    row = torch.tensor([3, 1 << 40, -(1 << 35)], device=DEV)
    col = torch.tensor([0, 2, 1 << 33], device=DEV)
    assert nat.coo_check(row, col)[0] == [-(1 << 35), 1 << 40, 0, 1 << 33]


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128, torch.float32])
@pytest.mark.parametrize("nnz", [1, 3000])
@pytest.mark.parametrize("route", ["rowrun", "atomic"])
def test_coo_spmm_of_lazy_views(dtype, nnz, route):
    """Values and B given as conjugate (complex) or negative (real) views of
    their memory: the product of what they mean, not of that memory."""
    g = torch.Generator().manual_seed(nnz)
    row, col = torch.randint(0, 70, (nnz,), generator=g), torch.randint(0, 50, (nnz,), generator=g)
    wide = torch.complex128 if dtype.is_complex else torch.float64
    lazy = torch.conj if dtype.is_complex else torch._neg_view
    data, B = torch.randn(nnz, generator=g, dtype=wide).to(dtype), torch.randn(50, 9, generator=g, dtype=wide).to(dtype)
    d, b = lazy(data.to(DEV)), lazy(B.to(DEV))
    assert (d.is_conj() or d.is_neg()) and d.is_contiguous()
    for dv, bv, da, ba in ((d, B.to(DEV), lazy(data), B), (data.to(DEV), b, data, lazy(B)), (d, b, lazy(data), lazy(B))):
        A = torch.zeros(70, 50, dtype=wide).index_put_((row, col), da.to(wide), accumulate=True)
        mag = torch.zeros(70, 50, dtype=torch.float64).index_put_((row, col), da.abs().double(), accumulate=True)
        C = _run_spmm_coo_route(dv, row.to(DEV), col.to(DEV), bv, (70, 50), route=route)
        assert scaled_error(C, A @ ba.to(wide), mag @ ba.abs().double()) <= REL_BOUND[dtype]


def test_coo_spmm_refuses_lazy_complex32_values():
    """A conjugate view of complex32 values cannot be reinterpreted as 32-bit
    patterns: refused, as torch refuses the reinterpretation."""
    z = torch.randn(4, dtype=torch.complex64).to(torch.complex32).to(DEV)
    idx = torch.tensor([3, 0, 2, 1], device=DEV)
    B = torch.zeros(4, 2, dtype=torch.complex64).to(torch.complex32).to(DEV)
    with pytest.raises(RuntimeError):
        fs.flagsparse_spmm_coo(z.conj(), idx, idx, B, (4, 4))
