"""The range-walk form of the batched merge-path SpMM (FSB_PLAN_WALK) against
the FP64 oracle where it can go wrong: rows at the edges of batches (8), chunks
(256), units and sub-group ranges, ranges without a nonzero, rows that end
where a unit begins, runs of empty rows, and every lane layout (whole 16-byte
lane vectors and strided columns: every compiled columns x lanes pair by a
width that picks it), B and C with rows further apart than their width or off
the 16-byte grid.

Bounds (condition-scaled, tests/numerics.py): those of the other SpMM forms.
A float32 sum's chains are at most 4 products of a batch, 2 sums of pairs, the
range's batches (at most 256 / 8 in a chunk) and the chunks: below 45
additions for the longest row here (511), 45 * 2^-24 = 2.7e-6 of the magnitude
and one rounding of the result, so 1e-5 holds with room; the 3e-5 of the
float32 modes also covers one serial chain of 500."""

import pytest
import torch

from flagsparse_public_b200 import _native as nat
from flagsparse_public_b200 import _plan
from oracle import oracle as orc
from tests.gpu_cases import csr_from_lengths, dense
from tests.numerics import REL_BOUND, scaled_error
from tests.test_gpu_split_rows import _graph_us

pytestmark = pytest.mark.gpu
DEV = "cuda"

PATTERNS = {
    "few": [2, 0, 1],
    "single": [1],
    "batch_edges": [7, 8, 9, 1, 16, 15, 17, 0, 8],
    "chunk_edges": [255, 1, 256, 257, 0, 511, 2, 300],
    "unit_start_end": [100, 100, 64, 36, 0, 0, 0, 200],
    "ones": [1] * 300,
    "empty_runs": [0] * 70 + [5] + [0] * 40 + [3, 0, 290] + [0] * 33,
}
MODES = [(torch.float32, nat.ACC_NATIVE, torch.float32, 3e-5),
         (torch.float32, nat.ACC_WIDE, torch.float32, REL_BOUND[torch.float32]),
         (torch.float64, nat.ACC_NATIVE, torch.float64, REL_BOUND[torch.float64]),
         (torch.bfloat16, nat.ACC_NATIVE, torch.float32, 3e-5),
         (torch.float16, nat.ACC_NATIVE, torch.float32, 3e-5),
         (torch.complex64, nat.ACC_NATIVE, torch.complex64, 3e-5),
         (torch.complex64, nat.ACC_WIDE, torch.complex64, REL_BOUND[torch.complex64]),
         (torch.complex128, nat.ACC_NATIVE, torch.complex128, REL_BOUND[torch.complex128])]


def _id(m):
    return f"{str(m[0])[6:]}-{['native', 'wide'][m[1]]}"


@pytest.mark.parametrize("pattern", sorted(PATTERNS))
@pytest.mark.parametrize("mode", MODES, ids=_id)
def test_walk_matches_oracle(pattern, mode):
    dtype, acc, out_dtype, bound = mode
    wide_idx = pattern in ("ones", "chunk_edges")  # 64-bit columns with 32-bit offsets on two patterns
    data, indices, indptr, (n_rows, n_cols) = csr_from_lengths(
        PATTERNS[pattern], 600, seed=61, dtype=dtype, index_dtype=torch.int64 if wide_idx else torch.int32,
        ptr_dtype=torch.int32 if wide_idx else torch.int64)
    d = (data.to(DEV), indices.to(DEV), indptr.to(DEV))
    for n_dense in (1, 2, 3, 5, 6, 9, 13, 16, 19, 33, 40, 51, 64, 67, 95, 100, 130):
        B = dense((n_cols, n_dense), 62, dtype)
        exact, mag = orc.spmm_csr_exact(data, indices, indptr, B)
        Bd = B.to(DEV)
        for items, snap, n_tile, grid in ((16, 0, 0, 0), (100, 0, 0, 0), (256, 64, 0, 0), (2048, 64, 0, 1), (77, 0, 8, 2)):
            plan = _plan.KernelPlan(nat.ALGO_SEQ, items_per_unit=items, snap=snap, n_tile=n_tile, grid_blocks=grid,
                                    flags=nat.PLAN_WALK)
            out = []
            for finish_in_kernel in (True, False):
                C = torch.full((n_rows, n_dense), float("nan"), dtype=out_dtype, device=DEV)
                if not finish_in_kernel:
                    plan.runs = False  # split rows finished by the fix-up kernel: the same sums
                _plan.run_spmm(*d, n_rows, n_cols, Bd, C, acc, plan)
                out.append(C)
            assert torch.equal(out[0], out[1]), (n_dense, items)
            assert scaled_error(out[0], exact, mag) <= bound, (n_dense, items, n_tile)


def test_walk_leaves_non_finite_b_rows_alone():
    """Lanes without a nonzero in a ragged batch touch no B row: infinities
    and NaN in rows that no nonzero names stay out of the result."""
    data, indices, indptr, (n_rows, n_cols) = csr_from_lengths([3, 0, 5, 1], 64, seed=63)
    B = dense((n_cols, 64), 64, torch.float32)
    used = torch.zeros(n_cols, dtype=torch.bool)
    used[indices.long()] = True
    B[~used] = float("nan")
    B[0 if not used[0] else int((~used).nonzero()[0])] = float("inf")
    exact, mag = orc.spmm_csr_exact(data, indices, indptr, torch.where(used[:, None], B, torch.zeros_like(B)))
    C = torch.empty((n_rows, 64), device=DEV)
    _plan.run_spmm(data.to(DEV), indices.to(DEV), indptr.to(DEV), n_rows, n_cols, B.to(DEV), C, nat.ACC_NATIVE,
                   _plan.KernelPlan(nat.ALGO_SEQ, items_per_unit=128, flags=nat.PLAN_WALK))
    assert scaled_error(C, exact, mag) <= 3e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16, torch.complex64])
@pytest.mark.parametrize("view", ["pitch", "column", "row_pitch_odd"])
def test_walk_on_views_of_b_and_c(dtype, view):
    """B and C as column ranges of wider arrays: rows a multiple of 16 bytes
    apart (lane vectors), the same starting off the 16-byte grid and an odd row
    pitch (strided columns); columns beside C's stay as they were."""
    data, indices, indptr, (n_rows, n_cols) = csr_from_lengths(PATTERNS["chunk_edges"], 600, seed=65, dtype=dtype)
    first, pitch = {"pitch": (0, 80), "column": (1, 80), "row_pitch_odd": (0, 67)}[view]
    out_dtype = torch.float32 if dtype == torch.float16 else dtype
    for n_dense in (8, 64):
        wide = dense((n_cols, pitch), 66, dtype)
        B = wide[:, first:first + n_dense]
        exact, mag = orc.spmm_csr_exact(data, indices, indptr, B.contiguous())
        Cw = torch.full((n_rows, pitch), 7.0, dtype=out_dtype, device=DEV)
        C = Cw[:, first:first + n_dense]
        _plan.run_spmm(data.to(DEV), indices.to(DEV), indptr.to(DEV), n_rows, n_cols,
                       wide.to(DEV)[:, first:first + n_dense], C, nat.ACC_NATIVE,
                       _plan.KernelPlan(nat.ALGO_SEQ, items_per_unit=256, snap=64, flags=nat.PLAN_WALK))
        assert scaled_error(C, exact, mag) <= (REL_BOUND[dtype] if dtype == torch.float64 else 3e-5)
        assert bool((Cw[:, :first] == 7).all()) and bool((Cw[:, first + n_dense:] == 7).all())


@pytest.mark.parametrize("dtype,n_dense,mean", [(torch.complex128, 1, 400), (torch.complex128, 4, 60),
                                                (torch.float64, 3, 400), (torch.float64, 4, 100),
                                                (torch.float32, 32, 60), (torch.float64, 8, 20)])
def test_default_form_is_the_faster_one(dtype, n_dense, mean):
    """The default plan's form takes at most 1.15 times the other one."""
    rows = 20000
    ptr = torch.arange(rows + 1, device=DEV) * mean
    col = torch.randint(0, rows, (rows * mean,), device=DEV, dtype=torch.int32)
    data, B = torch.ones(rows * mean, dtype=dtype, device=DEV), torch.ones(rows, n_dense, dtype=dtype, device=DEV)
    C = torch.empty_like(B)
    st = _plan.matrix_stats(ptr, rows, rows)
    default = _plan.default_spmm_plan(st, n_dense, dtype)
    other = _plan.KernelPlan(nat.ALGO_SEQ, snap=default.snap, flags=default.flags ^ nat.PLAN_WALK,
                             items_per_unit=default.items_per_unit)
    us = [_graph_us(lambda: _plan.run_spmm(data, col, ptr, rows, rows, B, C, nat.ACC_NATIVE, plan))
          for plan in (default, other)]
    assert us[0] <= 1.15 * us[1], us
