"""Performance cases of the sparse products, through the public entry points.

A case is a dict of plain values.  ``prepare`` makes what a caller holds
before a product (the matrix, the dense operand and, where the call takes one,
the prepared handle), ``run`` is one product, ``exact`` the same product in
64-bit torch without this package, ``work`` the bytes and operations that the
product cannot do without.

Matrix patterns: "poisson" (Poisson row lengths, uniform columns), "zipf"
(power-law row lengths, exponent 1.8, capped), "banded" (a 64-wide band, four
scattered nonzeros per row, one row in a hundred with 8192 nonzeros) and
"blocks" (dense 16 x 16 blocks).
"""

import math

import torch

import flagsparse_public_b200 as fs
from flagsparse_public_b200 import batched, bsr, synthetic

DEVICE = "cuda"
BAND, OFF_BAND, LONG_RATE, LONG_LEN = 64, 4, 0.01, 8192
ZIPF_ALPHA, ZIPF_CAP = 1.8, 20000
BATCH_MEAN_LOW, BATCH_MEAN_HIGH = 2.0, 64.0


def listed():
    return [
        # The smallest call: one step of an iterative solver on a small
        # matrix, prepared once; launch latency and the host path count.
        {"name": "spmv_small_prepared", "op": "spmv", "api": "prepared", "pattern": "poisson", "rows": 16384,
         "cols": 16384, "mean": 16.0, "dtype": "float32", "index": "int32", "opt": False, "trans": False},
        # A matrix seen once (assembled, multiplied, dropped), ragged sizes:
        # the structural check and the plan belong to the call.
        {"name": "spmv_oneshot_ragged", "op": "spmv", "api": "oneshot", "pattern": "poisson", "rows": 99991,
         "cols": 77773, "mean": 23.0, "dtype": "float32", "index": "int32", "opt": False, "trans": False},
        # Graph-like matrix in double precision, prepared: a power-iteration
        # step; skewed rows, larger than the L2 cache.
        {"name": "spmv_powerlaw_f64", "op": "spmv", "api": "prepared", "pattern": "zipf", "rows": 1500000,
         "cols": 1500000, "mean": 16.0, "dtype": "float64", "index": "int32", "opt": True, "trans": False},
        # A small one-shot product with an odd width: unaligned rows of B and
        # C, float64 accumulation of float32 data (the plain algorithm).
        {"name": "spmm_oneshot_odd", "op": "spmm", "api": "oneshot", "pattern": "poisson", "rows": 50021,
         "cols": 25013, "mean": 24.0, "n": 33, "dtype": "float32", "index": "int32", "opt": False},
        # The headline product: power-law rows, 64 dense columns, float32
        # accumulation, prepared (graph aggregation with 64 features).
        {"name": "spmm_powerlaw", "op": "spmm", "api": "prepared", "pattern": "zipf", "rows": 262144,
         "cols": 262144, "mean": 12.0, "n": 64, "dtype": "float32", "index": "int32", "opt": True},
        # A block Krylov step in double precision: even rows, wide B, an
        # operand well past the L2 cache.
        {"name": "spmm_wide_f64", "op": "spmm", "api": "prepared", "pattern": "poisson", "rows": 400000,
         "cols": 400000, "mean": 32.0, "n": 128, "dtype": "float64", "index": "int32", "opt": True},
        # 16-bit storage, float32 result: banded matrix with long rows,
        # prepared once and multiplied by 32 columns.
        {"name": "mixed_spmm_banded", "op": "mixed_spmm", "rows": 1048576, "n": 32, "dtype": "bfloat16"},
        # The same form with one vector, in float16.
        {"name": "mixed_spmv_banded", "op": "mixed_spmv", "rows": 1048576, "dtype": "float16"},
        # Many uneven matrices multiplied in one launch (a batch of graphs).
        {"name": "batched_uneven", "op": "batch", "count": 64, "rows_low": 1024, "rows_high": 65536, "n": 32,
         "dtype": "float32"},
        # Unsorted triplets straight from an assembly, multiplied once: the
        # sort belongs to the call.
        {"name": "spmm_coo_unsorted", "op": "coo_spmm", "pattern": "poisson", "rows": 131072, "cols": 131072,
         "mean": 16.0, "n": 32, "dtype": "float32", "index": "int64"},
        # Attention-like scores on a power-law pattern: one dot product of 64
        # per stored position.
        {"name": "sddmm_powerlaw", "op": "sddmm", "pattern": "zipf", "rows": 262144, "cols": 262144, "mean": 12.0,
         "k": 64, "dtype": "float32", "beta": 0.0},
        # Block-sparse weights times 128 columns of activations on the
        # tensor cores, 16-bit storage and float32 result.
        {"name": "bsr_blocks", "op": "bsr", "block_rows": 65536, "blocks_per_row": 4, "n": 128,
         "dtype": "bfloat16"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the listed ranges: sizes over their logarithm (odd
    ones among them), value and index types, patterns and call forms."""
    op = rng.choice(["spmv", "spmv", "spmm", "spmm", "spmm", "mixed_spmm", "mixed_spmv", "batch", "coo_spmm",
                     "coo_spmv", "sddmm", "bsr"])
    if op in ("spmv", "coo_spmv"):
        mean = round(rng.uniform(4.0, 48.0), 1)
        rows = _log_int(rng, 4096, min(1500000, int(24e6 / mean)))
        c = {"op": op, "pattern": rng.choice(["poisson", "zipf"]), "rows": rows,
             "cols": max(4096, int(rows * rng.choice([0.5, 1.0, 1.0, 1.7]))), "mean": mean,
             "dtype": rng.choice(["float32", "float32", "float64", "float16", "bfloat16", "complex64"]),
             "index": rng.choice(["int32", "int32", "int64"])}
        if op == "spmv":
            c["api"] = rng.choice(["prepared", "prepared", "oneshot"])
            c["opt"] = rng.random() < 0.5
            c["trans"] = c["api"] == "prepared" and rng.random() < 0.3
        else:
            if c["dtype"] in ("float16", "bfloat16"):
                c["dtype"] = "float32"
        return c
    if op in ("spmm", "coo_spmm"):
        mean = round(rng.uniform(4.0, 40.0), 1)
        n = rng.choice([1, 8, 16, 32, 32, 64, 64, 128, rng.randint(2, 127)])
        rows = _log_int(rng, 4096, min(400000, int(8e8 / (mean * n))))
        c = {"op": op, "pattern": rng.choice(["poisson", "zipf"]), "rows": rows,
             "cols": max(4096, int(rows * rng.choice([0.5, 1.0, 1.0, 1.7]))), "mean": mean, "n": n,
             "dtype": rng.choice(["float32", "float32", "float32", "float64"]),
             "index": rng.choice(["int32", "int32", "int64"])}
        if op == "spmm":
            c["api"] = rng.choice(["prepared", "prepared", "oneshot"])
            c["opt"] = c["api"] == "prepared" or rng.random() < 0.3
            if not c["opt"]:
                c["dtype"] = rng.choice(["float32", "float32", "float64", "float16", "bfloat16", "complex64"])
        return c
    if op in ("mixed_spmm", "mixed_spmv"):
        c = {"op": op, "rows": _log_int(rng, 65536, 1048576), "dtype": rng.choice(["bfloat16", "float16"])}
        if op == "mixed_spmm":
            c["n"] = rng.choice([16, 32, 32])
        return c
    if op == "batch":
        low = _log_int(rng, 256, 4096)
        return {"op": op, "count": _log_int(rng, 8, 64), "rows_low": low,
                "rows_high": _log_int(rng, 4 * low, 65536), "n": rng.choice([8, 16, 32, 32, 33]), "dtype": "float32"}
    if op == "sddmm":
        mean = round(rng.uniform(4.0, 40.0), 1)
        k = rng.choice([16, 32, 64, 64, 128, rng.randint(3, 200)])
        rows = _log_int(rng, 4096, min(262144, int(4e8 / (mean * k))))
        return {"op": op, "pattern": rng.choice(["poisson", "zipf"]), "rows": rows,
                "cols": max(4096, int(rows * rng.choice([0.5, 1.0, 1.7]))), "mean": mean, "k": k,
                "dtype": rng.choice(["float32", "float32", "float64"]), "beta": rng.choice([0.0, 0.0, 0.5])}
    return {"op": op, "block_rows": _log_int(rng, 1024, 65536), "blocks_per_row": rng.randint(1, 6),
            "n": 8 * rng.randint(1, 16), "dtype": rng.choice(["bfloat16", "float16"])}


def _dtype(case):
    return getattr(torch, case["dtype"])


def _values(n, dtype, seed):
    """U(-1, 1) values (both parts of complex ones)."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    real = torch.float64 if dtype in (torch.float64, torch.complex128) else torch.float32
    if dtype.is_complex:
        return torch.complex(torch.rand(n, generator=g, device=DEVICE, dtype=real) * 2 - 1,
                             torch.rand(n, generator=g, device=DEVICE, dtype=real) * 2 - 1)
    return (torch.rand(n, generator=g, device=DEVICE, dtype=real) * 2 - 1).to(dtype)


def _normal(shape, dtype, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    if dtype.is_complex:
        return torch.randn(shape, generator=g, device=DEVICE, dtype=dtype)
    real = torch.float64 if dtype == torch.float64 else torch.float32
    return torch.randn(shape, generator=g, device=DEVICE, dtype=real).to(dtype)


def _csr(case, seed):
    """(data, indices, indptr, shape) of the case's pattern and types."""
    if case["pattern"] == "zipf":
        _, idx, ptr, shape = synthetic.zipf_powerlaw(case["rows"], case["cols"], alpha=ZIPF_ALPHA, mean=case["mean"],
                                                     cap=min(ZIPF_CAP, case["cols"] // 4), seed=seed,
                                                     device=DEVICE)
    else:
        _, idx, ptr, shape = synthetic.poisson_uniform(case["rows"], case["cols"], mean=case["mean"], seed=seed,
                                                       device=DEVICE)
    idx = idx.to(getattr(torch, case.get("index", "int32")))
    return _values(idx.numel(), _dtype(case), seed + 1), idx, ptr, shape


def _positions(case, seed):
    """The sampled positions of a case: as many for every seed (the result has
    one value per position), in columns relabelled by the seed."""
    data, idx, ptr, shape = _csr(case, 0)
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed + 2)
    relabel = torch.randperm(shape[1], generator=g, device=DEVICE)
    key = _row_ids(ptr, idx.numel()) * shape[1] + relabel[idx.to(torch.int64)]
    idx = (torch.sort(key)[0] % shape[1]).to(idx.dtype)
    return _values(idx.numel(), _dtype(case), seed + 1), idx, ptr, shape


def _banded(case, seed):
    return synthetic.banded_plus_random(case["rows"], band=BAND, off_band=OFF_BAND, long_rate=LONG_RATE,
                                        long_len=LONG_LEN, seed=seed, dtype=_dtype(case), device=DEVICE)


def _blocks(case, seed):
    return synthetic.block_sparse(case["block_rows"], case["blocks_per_row"], seed=seed, dtype=_dtype(case),
                                  device=DEVICE)


def _batch_sizes(case):
    """(rows, mean row length) of every matrix: rows spread evenly over the
    logarithm of their range, means over theirs, in mixed order."""
    out = []
    for i in range(case["count"]):
        t = (i * 0.6180339887498949) % 1.0
        u = (i * 0.7548776662466927) % 1.0
        rows = int(round(case["rows_low"] * (case["rows_high"] / case["rows_low"]) ** t))
        out.append((rows, round(BATCH_MEAN_LOW + (BATCH_MEAN_HIGH - BATCH_MEAN_LOW) * u, 2)))
    return out


def _batch(case, seed):
    return [synthetic.poisson_uniform(rows, rows, mean=mean, seed=seed * 1000 + i, dtype=_dtype(case), device=DEVICE)
            for i, (rows, mean) in enumerate(_batch_sizes(case))]


def _row_ids(ptr, nnz):
    lens = ptr[1:] - ptr[:-1]
    return torch.repeat_interleave(torch.arange(lens.numel(), device=ptr.device), lens, output_size=nnz)


def _triplets(case, seed):
    """The pattern's entries in a random order."""
    data, idx, ptr, shape = _csr(case, seed)
    row = _row_ids(ptr, idx.numel()).to(idx.dtype)
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed + 2)
    order = torch.randperm(idx.numel(), generator=g, device=DEVICE)
    return data[order], row[order], idx[order], shape


def prepare(case, seed):
    op, dt = case["op"], None if "dtype" not in case else _dtype(case)
    if op == "spmv":
        data, idx, ptr, shape = _csr(case, seed)
        x = _normal(shape[0] if case["trans"] else shape[1], dt, seed + 3)
        handle = None
        if case["api"] == "prepared":
            handle = fs.prepare_spmv_csr(data, idx, ptr, shape, op="trans" if case["trans"] else "non")
        return {"case": case, "csr": (data, idx, ptr), "shape": shape, "x": x, "handle": handle}
    if op == "spmm":
        data, idx, ptr, shape = _csr(case, seed)
        handle = fs.prepare_spmm_csr_opt(data, idx, ptr, shape) if case["api"] == "prepared" else None
        return {"case": case, "csr": (data, idx, ptr), "shape": shape, "handle": handle,
                "b": _normal((shape[1], case["n"]), dt, seed + 3)}
    if op in ("mixed_spmm", "mixed_spmv"):
        data, idx, ptr, shape = _banded(case, seed)
        width = (shape[1], case["n"]) if op == "mixed_spmm" else shape[1]
        return {"case": case, "handle": fs.prepare_csr_mixed(data, idx, ptr, shape),
                "b": _normal(width, dt, seed + 3)}
    if op == "batch":
        handle = batched.prepare_spmm_csr_batch(_batch(case, seed), case["n"])
        for i, view in enumerate(handle.b_views):
            view.copy_(_normal(tuple(view.shape), dt, seed * 1000 + 500 + i))
        return {"case": case, "handle": handle}
    if op in ("coo_spmm", "coo_spmv"):
        data, row, col, shape = _triplets(case, seed)
        width = (shape[1], case["n"]) if op == "coo_spmm" else shape[1]
        return {"case": case, "coo": (data, row, col), "shape": shape, "b": _normal(width, dt, seed + 3)}
    if op == "sddmm":
        data, idx, ptr, shape = _positions(case, seed)
        return {"case": case, "handle": fs.prepare_sddmm_csr(idx, ptr, shape, k_hint=case["k"]),
                "data": data if case["beta"] else None, "x": _normal((shape[0], case["k"]), dt, seed + 3),
                "y": _normal((shape[1], case["k"]), dt, seed + 4)}
    if op == "bsr":
        data, idx, ptr, shape = _blocks(case, seed)
        blocks = bsr.csr_to_bsr16(data, idx, ptr, shape)
        return {"case": case, "handle": bsr.prepare_spmm_bsr(*blocks, shape),
                "b": _normal((shape[1], case["n"]), dt, seed + 3)}
    raise ValueError(op)


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "spmv":
        if state["handle"] is not None:
            return fs.flagsparse_spmv_csr(x=state["x"], prepared=state["handle"], use_opt=case["opt"])
        data, idx, ptr = state["csr"]
        return fs.flagsparse_spmv_csr(data, idx, ptr, state["x"], state["shape"], use_opt=case["opt"])
    if op == "spmm":
        if state["handle"] is not None:
            return fs.flagsparse_spmm_csr_opt(B=state["b"], prepared=state["handle"])
        data, idx, ptr = state["csr"]
        if case["opt"]:
            return fs.flagsparse_spmm_csr_opt(data, idx, ptr, state["b"], state["shape"])
        return fs.flagsparse_spmm_csr(data, idx, ptr, state["b"], state["shape"])
    if op == "mixed_spmm":
        return fs.flagsparse_spmm_csr_mixed(B=state["b"], prepared=state["handle"])
    if op == "mixed_spmv":
        return fs.flagsparse_spmv_csr_mixed(x=state["b"], prepared=state["handle"])
    if op == "batch":
        return state["handle"].run()
    if op == "coo_spmm":
        data, row, col = state["coo"]
        return fs.flagsparse_spmm_coo(data, row, col, state["b"], state["shape"])
    if op == "coo_spmv":
        data, row, col = state["coo"]
        return fs.flagsparse_spmv_coo(data, row, col, state["b"], state["shape"])
    if op == "sddmm":
        return fs.flagsparse_sddmm_csr(data=state["data"], x=state["x"], y=state["y"], prepared=state["handle"],
                                       beta=case["beta"])
    return bsr.flagsparse_spmm_bsr(B=state["b"], prepared=state["handle"])


_SIZE = {"float16": 2, "bfloat16": 2, "float32": 4, "float64": 8, "complex64": 8, "int32": 4, "int64": 8}


def work(case):
    op = case["op"]
    if op in ("mixed_spmm", "mixed_spmv"):
        rows, n = case["rows"], case.get("n", 1)
        nnz = rows * ((1 - LONG_RATE) * (BAND + OFF_BAND) + LONG_RATE * LONG_LEN)
        return {"bytes": nnz * 6 + rows * 8 + rows * n * 2 + rows * n * 4, "flops": 2 * nnz * n}
    if op == "batch":
        n, b, f = case["n"], 0, 0
        for rows, mean in _batch_sizes(case):
            b += rows * mean * 8 + rows * 8 + 2 * rows * n * 4
            f += 2 * rows * mean * n
        return {"bytes": b, "flops": f}
    if op == "bsr":
        rows, blocks = case["block_rows"] * 16, case["block_rows"] * case["blocks_per_row"]
        return {"bytes": blocks * (512 + 4) + case["block_rows"] * 8 + rows * case["n"] * 6,
                "flops": 2 * blocks * 256 * case["n"]}
    rows, cols, nnz = case["rows"], case["cols"], case["rows"] * case["mean"]
    sv = _SIZE[case["dtype"]]
    mul = 8 if case["dtype"].startswith("complex") else 2
    if op == "sddmm":
        values = 2 if case["beta"] else 1
        # the row of every position is part of the prepared pattern
        return {"bytes": nnz * (4 + values * sv) + rows * 8 + (rows + cols) * case["k"] * sv,
                "flops": 2 * nnz * case["k"]}
    si, n = _SIZE[case["index"]], case.get("n", 1)
    # triplets carry a row index per entry, compressed rows an offset per row
    structure = nnz * 2 * si if op.startswith("coo") else nnz * si + (rows + 1) * 8
    return {"bytes": nnz * sv + structure + (rows + cols) * n * sv, "flops": mul * nnz * n}


def _wide(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _product(rows, cols, values, dense, n_rows):
    """sum of values * dense[cols] by row in 64 bits, in slices of entries."""
    one = dense.ndim == 1
    d = _wide(dense).reshape(dense.shape[0], -1)
    out = torch.zeros((n_rows, d.shape[1]), dtype=d.dtype, device=d.device)
    step = max(1, (1 << 27) // max(1, d.shape[1]))
    for s in range(0, values.numel(), step):
        part = _wide(values[s:s + step])[:, None] * d[cols[s:s + step].to(torch.int64)]
        r = rows[s:s + step].to(torch.int64)
        if part.is_complex():
            torch.view_as_real(out).index_add_(0, r, torch.view_as_real(part))
        else:
            out.index_add_(0, r, part)
    return out[:, 0] if one else out


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        out = []
        for i, (data, idx, ptr, shape) in enumerate(_batch(case, seed)):
            b = _normal((shape[1], case["n"]), _dtype(case), seed * 1000 + 500 + i)
            out.append(_product(_row_ids(ptr, idx.numel()), idx, data, b, shape[0]))
        return out
    if op in ("coo_spmm", "coo_spmv"):
        data, row, col, shape = _triplets(case, seed)
        width = (shape[1], case["n"]) if op == "coo_spmm" else shape[1]
        return _product(row, col, data, _normal(width, _dtype(case), seed + 3), shape[0])
    if op in ("mixed_spmm", "mixed_spmv"):
        data, idx, ptr, shape = _banded(case, seed)
    elif op == "bsr":
        data, idx, ptr, shape = _blocks(case, seed)
    elif op == "sddmm":
        data, idx, ptr, shape = _positions(case, seed)
    else:
        data, idx, ptr, shape = _csr(case, seed)
    rows = _row_ids(ptr, idx.numel())
    if op == "sddmm":
        x, y = _normal((shape[0], case["k"]), _dtype(case), seed + 3), _normal((shape[1], case["k"]), _dtype(case),
                                                                              seed + 4)
        out = torch.empty(idx.numel(), dtype=torch.float64, device=DEVICE)
        step = max(1, (1 << 27) // case["k"])
        for s in range(0, out.numel(), step):
            out[s:s + step] = (_wide(x)[rows[s:s + step]] * _wide(y)[idx[s:s + step].to(torch.int64)]).sum(1)
        return out + case["beta"] * _wide(data) if case["beta"] else out
    if op == "spmv" and case["trans"]:
        return _product(idx, rows, data, _normal(shape[0], _dtype(case), seed + 3), shape[1])
    width = (shape[1], case["n"]) if "n" in case else shape[1]
    return _product(rows, idx, data, _normal(width, _dtype(case), seed + 3), shape[0])
