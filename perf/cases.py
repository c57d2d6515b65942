"""The calls whose speed this repository stands for, as a user's program makes them.

The library's public boundary is the C ABI of ``include/flag4j_cuda.h`` on
device-resident buffer handles: a Java program reaches it through the Foreign
Function & Memory API, a Python one through ``flag4j_gb300``.  A program keeps
its operands, its results' buffers and its CSR handles on the GPU across calls,
so ``prepare`` makes those and ``run`` is the product call itself.  The one
exception is the host-buffer product, whose operands and result are host arrays
by its nature.

Sizes are those of the library's own workloads (1024, 2048, 4096 and 8192
dense, 2^20 rows of about 16 nonzeros sparse) and ragged ones of the same
range; ``draw`` spreads over the whole of it.
"""
import ctypes

import numpy as np
import torch

from flag4j_gb300 import _lib, default_context, pinned_empty
from flag4j_gb300.device import DeviceBuffer, check

OPS = {"N": _lib.OP_N, "T": _lib.OP_T, "C": _lib.OP_C}


def listed():
    return [
        # Matrix.mult of small matrices: a call is one launch and its latency
        {"name": "mult_small", "op": "mult", "m": 96, "n": 80, "k": 64, "values": "uniform", "opB": "N", "mode": "auto"},
        # Matrix.mult at 1024^3, the library's first dense workload
        {"name": "mult_1024", "op": "mult", "m": 1024, "n": 1024, "k": 1024, "values": "uniform", "opB": "N",
         "mode": "auto"},
        # Matrix.multTranspose on ragged sizes and N(0, 1) entries
        {"name": "mult_transpose_ragged", "op": "mult", "m": 2111, "n": 1777, "k": 1543, "values": "normal", "opB": "T",
         "mode": "auto"},
        # Matrix.mult at 8192^3 on row- and column-scaled entries, the headline workload
        {"name": "mult_8192", "op": "mult", "m": 8192, "n": 8192, "k": 8192, "values": "scaled", "opB": "N",
         "mode": "auto"},
        # the bit-identical mode: the reference's own order and rounding
        {"name": "mult_exact", "op": "mult", "m": 700, "n": 500, "k": 600, "values": "uniform", "opB": "N",
         "mode": "exact"},
        # CMatrix.mult
        {"name": "cmult_2048", "op": "cmult", "m": 2048, "n": 2048, "k": 2048, "values": "uniform", "opB": "N"},
        # training step of a dense product: forward, then both gradients
        {"name": "mult_adjoint", "op": "adjoint", "m": 4096, "n": 4096, "k": 2048, "values": "normal"},
        # Matrix.mult on host arrays (page-locked), as a JVM binding calls it
        {"name": "mult_host_4096", "op": "host", "m": 4096, "n": 4096, "k": 4096, "values": "scaled"},
        # CsrMatrix.mult(Vector)
        {"name": "spmv", "op": "spmv", "rows": 1 << 20, "cols": 1 << 20, "per_row": 16, "mode": "exact"},
        # CsrMatrix.mult(Matrix), 32 columns
        {"name": "spmm_32", "op": "spmm", "rows": 1 << 20, "cols": 1 << 20, "per_row": 16, "ncols": 32, "mode": "exact"},
        # training step of a CSR product: both gradients of C = S X
        {"name": "spmm_adjoint", "op": "spadj", "rows": 1 << 18, "cols": 1 << 18, "per_row": 16, "ncols": 64},
        # CooMatrix.toCsr, then CsrMatrix.T()
        {"name": "coo_to_csr", "op": "coo", "rows": 1 << 20, "cols": 1 << 20, "per_row": 16},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("small", "mult", "mult", "mult", "exact", "cmult", "adjoint", "host", "spmv", "spmm", "spadj",
                       "coo"))
    dims = lambda lo, hi: {d: _log_int(rng, lo, hi) for d in ("m", "n", "k")}
    values = rng.choice(("uniform", "normal", "scaled"))
    if kind == "small":
        return {"op": "mult", **dims(8, 192), "values": values, "opB": rng.choice("NT"), "mode": "auto"}
    if kind == "mult":
        return {"op": "mult", **dims(256, 8192), "values": values, "opB": rng.choice("NT"), "mode": "auto"}
    if kind == "exact":
        return {"op": "mult", **dims(128, 1024), "values": values, "opB": rng.choice("NT"), "mode": "exact"}
    if kind == "cmult":
        return {"op": "cmult", **dims(192, 3000), "values": values, "opB": rng.choice("NC")}
    if kind == "adjoint":
        return {"op": "adjoint", **dims(384, 4096), "values": values}
    if kind == "host":
        return {"op": "host", **dims(512, 5000), "values": values}
    sparse = {"rows": _log_int(rng, 1 << 12, 1 << 20), "cols": _log_int(rng, 1 << 12, 1 << 20),
              "per_row": _log_int(rng, 4, 16)}
    if kind == "spmv":
        return {"op": "spmv", **sparse, "mode": rng.choice(("exact", "fma"))}
    if kind == "spmm":
        return {"op": "spmm", **sparse, "ncols": _log_int(rng, 2, 64), "mode": rng.choice(("exact", "fma"))}
    if kind == "spadj":
        return {"op": "spadj", **sparse, "ncols": rng.choice((16, 32, 64, _log_int(rng, 4, 96)))}
    return {"op": "coo", **sparse}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _dense(rows, cols, values, g, per, cplx=False):
    """Uniform[-1, 1), N(0, 1), or u 2^e with an integer e ~ U[-8, 8] per row (A) or column (B)."""
    shape = (rows, cols, 2) if cplx else (rows, cols)
    if values == "normal":
        x = torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    else:
        x = torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0
    if values == "scaled":
        e = torch.randint(-8, 9, (rows if per == "row" else cols,), device="cuda", generator=g).double()
        s = torch.exp2(e)
        s = s[:, None] if per == "row" else s[None, :]
        x = x * (s[..., None] if cplx else s)
    return x


def _operands(case, seed):
    """A (m x k) and B as stored (k x n, or n x k for a transposed operand)."""
    g = _generator(seed)
    cplx = case["op"] == "cmult"
    A = _dense(case["m"], case["k"], case["values"], g, "row", cplx)
    if case.get("opB", "N") == "N":
        B = _dense(case["k"], case["n"], case["values"], g, "col", cplx)
    else:
        B = _dense(case["n"], case["k"], case["values"], g, "row", cplx)
    W = _dense(case["m"], case["n"], "normal", g, "row") if case["op"] == "adjoint" else None
    return A, B, W


def _csr(case, seed):
    """rows x per_row nonzeros in uniformly drawn rows (lengths near Poisson(per_row), some rows empty
    when per_row is small), distinct sorted columns in each row, N(0, 1) values."""
    g = _generator(seed)
    rows, cols = case["rows"], case["cols"]
    row = torch.randint(0, rows, (rows * case["per_row"],), device="cuda", generator=g).sort().values
    lens = torch.bincount(row, minlength=rows)
    key = row * cols + torch.randint(0, cols, row.shape, device="cuda", generator=g)
    while True:
        key = key.sort().values
        dup = torch.nonzero(key[1:] == key[:-1]).squeeze(1) + 1
        if not dup.numel():
            break
        key[dup] = key[dup] // cols * cols + torch.randint(0, cols, dup.shape, device="cuda", generator=g)
    rowptr = torch.zeros(rows + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = lens.cumsum(0).int()
    vals = torch.randn(row.shape, dtype=torch.float64, device="cuda", generator=g)
    return row.int(), rowptr, (key % cols).int(), vals, g


def _sparse_inputs(case, seed):
    row, rowptr, col, vals, g = _csr(case, seed)
    nc = case.get("ncols", 1)
    X = torch.randn((case["cols"], nc), dtype=torch.float64, device="cuda", generator=g)
    W = torch.randn((case["rows"], nc), dtype=torch.float64, device="cuda", generator=g) if case["op"] == "spadj" else None
    return row, rowptr, col, vals, X, W


# ------------------------------------------------------------------ states
class _Csr:
    """A CSR handle, freed with the object."""

    def __init__(self, ctx, handle):
        self.ctx, self.handle = ctx, handle

    def __del__(self):
        self.ctx.lib.f4j_csr_free(self.ctx.handle, self.handle)


class _Array:
    """A CSR handle's device array, for torch to read in place; keeps the handle alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "strides": None,
                                         "version": 3}


def _buf(ctx, t):
    return DeviceBuffer(ctx, t.numel() * t.element_size(), wrap_ptr=t.data_ptr())


def _out(*shape):
    return torch.empty(shape, dtype=torch.float64, device="cuda")


def _wrap_csr(ctx, case, rowptr, col, vals):
    bufs = (_buf(ctx, rowptr), _buf(ctx, col), _buf(ctx, vals))
    h = ctypes.c_void_p()
    check(ctx.lib.f4j_csr_wrap(ctx.handle, case["rows"], case["cols"], vals.numel(), bufs[0].handle, bufs[1].handle,
                               bufs[2].handle, 0, ctypes.byref(h)))
    return _Csr(ctx, h), bufs


def prepare(case, seed):
    ctx = default_context()
    op = case["op"]
    s = {"case": case, "ctx": ctx}
    if op in ("mult", "cmult", "adjoint"):
        A, B, W = _operands(case, seed)
        m, n, k = case["m"], case["n"], case["k"]
        outs = {"C": _out(m, n, 2) if op == "cmult" else _out(m, n)}
        if op == "adjoint":
            outs.update(dA=_out(m, k), dB=_out(k, n))
        ins = {"A": A, "B": B}
        if W is not None:
            ins["W"] = W
    elif op == "host":
        s["host"] = []
        for t in _operands(case, seed)[:2]:
            a = pinned_empty(tuple(t.shape))
            torch.from_numpy(a).copy_(t)
            s["host"].append(a)
        s["host"].append(pinned_empty((case["m"], case["n"])))
        return s
    else:
        row, rowptr, col, vals, X, W = _sparse_inputs(case, seed)
        if op == "coo":
            ins, outs = {"row": row, "col": col, "vals": vals}, {}
        else:
            s["S"], s["S_bufs"] = _wrap_csr(ctx, case, rowptr, col, vals)
            s["S_arrays"] = (rowptr, col, vals)
            nc = case.get("ncols", 1)
            if op == "spadj":
                ins = {"X": X, "W": W}
                outs = {"dX": _out(case["cols"], nc), "dS": _out(vals.numel())}
            else:
                ins, outs = {"X": X}, {"Y": _out(case["rows"], nc)}
    s["tensors"] = {**ins, **outs}
    s["outs"] = list(outs)
    s["buf"] = {name: _buf(ctx, t) for name, t in s["tensors"].items()}
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    return s


# ------------------------------------------------------------------ one pass
def _structure(s):
    ctx, case = s["ctx"], s["case"]
    rows, cols, nnz = case["rows"], case["cols"], s["tensors"]["vals"].numel()
    h, t = ctypes.c_void_p(), ctypes.c_void_p()
    b = {name: x.handle for name, x in s["buf"].items()}
    check(ctx.lib.f4j_csr_from_coo(ctx.handle, rows, cols, nnz, b["row"], b["col"], b["vals"], ctypes.byref(h)))
    S = _Csr(ctx, h)
    check(ctx.lib.f4j_csr_transpose(ctx.handle, S.handle, ctypes.byref(t)))
    out = []
    for owner, n in ((S, rows), (_Csr(ctx, t), cols)):
        p = [ctypes.c_void_p() for _ in range(3)]
        check(ctx.lib.f4j_csr_buffers(owner.handle, *[ctypes.byref(x) for x in p]))
        for x, count, kind in zip(p, (n + 1, nnz, nnz), ("<i4", "<i4", "<f8")):
            a = _Array(owner, ctx.lib.f4j_buf_device_ptr(x), (count,), kind)
            out.append(torch.as_tensor(a, device="cuda"))
    return out


def run(s):
    ctx, case = s["ctx"], s["case"]
    lib, h, op = ctx.lib, ctx.handle, case["op"]
    if op == "host":
        A, B, C = s["host"]
        check(lib.f4j_dgemm_host(h, case["m"], case["n"], case["k"], A.ctypes.data, _lib.OP_N, B.ctypes.data,
                                 _lib.OP_N, C.ctypes.data, _lib.MODE_AUTO, None))
        return C
    if op == "coo":
        return _structure(s)
    b = s["buf"]
    if op == "mult":
        check(lib.f4j_dgemm(h, case["m"], case["n"], case["k"], b["A"].handle, _lib.OP_N, b["B"].handle,
                            OPS[case["opB"]], b["C"].handle, _lib.MODES[case["mode"]], None))
    elif op == "cmult":
        check(lib.f4j_zgemm(h, case["m"], case["n"], case["k"], b["A"].handle, _lib.OP_N, b["B"].handle,
                            OPS[case["opB"]], b["C"].handle, _lib.MODE_AUTO, None))
    elif op == "adjoint":
        m, n, k = case["m"], case["n"], case["k"]
        check(lib.f4j_dgemm(h, m, n, k, b["A"].handle, _lib.OP_N, b["B"].handle, _lib.OP_N, b["C"].handle,
                            _lib.MODE_AUTO, None))
        check(lib.f4j_dgemm_adjoint(h, m, n, k, b["A"].handle, b["B"].handle, b["W"].handle, b["dA"].handle,
                                    b["dB"].handle, _lib.MODE_AUTO, None))
    elif op == "spmv":
        check(lib.f4j_spmv_ex(h, s["S"].handle, b["X"].handle, b["Y"].handle, _lib.SPARSE_MODES[case["mode"]], None))
    elif op == "spmm":
        check(lib.f4j_spmm_ex(h, s["S"].handle, b["X"].handle, case["ncols"], b["Y"].handle,
                              _lib.SPARSE_MODES[case["mode"]], None))
    elif op == "spadj":
        nc = case["ncols"]
        check(lib.f4j_spmm_t(h, s["S"].handle, b["W"].handle, nc, b["dX"].handle, None))
        check(lib.f4j_sddmm(h, s["S"].handle, b["W"].handle, b["X"].handle, nc, b["dS"].handle, None))
    return [s["tensors"][name] for name in s["outs"]]


# ------------------------------------------------------------------ accounts
def work(case):
    """Bytes: each input read once, each result written once.  Flops: the product's own multiply-adds."""
    op = case["op"]
    if op in ("mult", "host", "cmult", "adjoint"):
        m, n, k = case["m"], case["n"], case["k"]
        elems, flops = m * k + k * n + m * n, 2 * m * n * k
        if op == "cmult":
            return {"bytes": 16 * elems, "flops": 4 * flops}
        if op == "adjoint":  # A, B, W in; C, dA, dB out
            return {"bytes": 8 * 2 * elems, "flops": 3 * flops}
        return {"bytes": 8 * elems, "flops": flops}
    rows, cols, nnz, nc = case["rows"], case["cols"], case["rows"] * case["per_row"], case.get("ncols", 1)
    pattern = 4 * nnz + 4 * (rows + 1)
    if op == "coo":  # row, column, value of each triplet; both CSR results
        return {"bytes": 16 * nnz + 2 * 12 * nnz + 4 * (rows + cols + 2), "flops": 0}
    if op == "spadj":  # pattern, values, W, X in; dX and dS out
        return {"bytes": pattern + 16 * nnz + 8 * nc * (rows + 2 * cols), "flops": 4 * nnz * nc}
    return {"bytes": pattern + 8 * nnz + 8 * nc * (rows + cols), "flops": 2 * nnz * nc}


def exact(case, seed):
    op = case["op"]
    if op in ("mult", "host", "cmult", "adjoint"):
        A, B, W = _operands(case, seed)
        if op == "cmult":
            a, b = torch.view_as_complex(A), torch.view_as_complex(B)
            return [torch.view_as_real(a @ (b if case["opB"] == "N" else b.conj().T))]
        if op == "adjoint":
            return [A @ B, W @ B.T, A.T @ W]
        C = A @ (B if case.get("opB", "N") == "N" else B.T)
        return C.cpu().numpy() if op == "host" else [C]
    row, rowptr, col, vals, X, W = _sparse_inputs(case, seed)
    r, c = row.long(), col.long()
    if op == "coo":
        perm = torch.sort(c, stable=True).indices
        t_rowptr = torch.zeros(case["cols"] + 1, dtype=torch.int32, device="cuda")
        t_rowptr[1:] = torch.bincount(c, minlength=case["cols"]).cumsum(0).int()
        return [rowptr, col, vals, t_rowptr, row[perm], vals[perm]]
    if op == "spadj":
        dX = torch.zeros_like(X)
        dX.index_add_(0, c, vals[:, None] * W[r])
        return [dX, (W[r] * X[c]).sum(1)]
    Y = torch.zeros((case["rows"], X.shape[1]), dtype=torch.float64, device="cuda")
    Y.index_add_(0, r, vals[:, None] * X[c])
    return [Y]
