"""The COO index check (fsb_coo_check) and the permuted entries
(fsb_take_entries) against torch, at the sizes where a warp, a CTA or the
16-byte loads end; integers and copied bytes compare equal."""

import pytest
import torch

from flagsparse_public_b200 import _native as nat
from flagsparse_public_b200 import _plan

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
