"""Calls inside a stream capture: what a call captures has to be complete in the graph, and what it keeps
beyond the call must not belong to the graph."""
import contextlib
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def capturing_context(f4j):
    """A context of its own on a stream that torch can capture; yields (ctx, capture(fn) -> graph)."""
    import torch
    from flag4j_gb300.device import check
    ctx = f4j.Context(0)
    stream = torch.cuda.Stream()
    check(ctx.lib.f4j_set_stream(ctx.handle, ctypes.c_void_p(stream.cuda_stream)))

    def capture(fn, mode="global"):
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode=mode):
            fn()
        return g

    try:
        yield ctx, capture
    finally:
        torch.cuda.synchronize()
        check(ctx.lib.f4j_set_stream(ctx.handle, None))


def test_first_residue_product_of_a_context_in_a_capture(f4j):
    """The residue form's constants are part of the library: with workspace enough from a sliced product, a
    context's first residue product allocates and copies nothing, so it can be captured."""
    import torch
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    g = np.random.default_rng(11)
    A, B = g.integers(-(1 << 19), 1 << 19, (300, 300)).astype(float), g.integers(-1000, 1000, (300, 300)).astype(float)
    with capturing_context(f4j) as (ctx, capture):
        big = ctx.from_numpy(g.standard_normal((1024, 1024)))
        out = ctx.alloc(8 << 20)
        check(ctx.lib.f4j_dgemm(ctx.handle, 1024, 1024, 1024, big.handle, 0, big.handle, 0, out.handle, _lib.MODE_SPLIT,
                                None))
        dA, dB, dC = ctx.from_numpy(A), ctx.from_numpy(B), ctx.alloc(8 * 300 * 300)
        dC.zero()
        ctx.sync()
        graph = capture(lambda: check(ctx.lib.f4j_dgemm(ctx.handle, 300, 300, 300, dA.handle, 0, dB.handle, 0, dC.handle,
                                                        _lib.MODE_AUTO, None)))
        assert not dC.to_numpy(np.float64, 300 * 300).any()
        for _ in range(2):
            dC.zero()
            ctx.sync()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(dC.to_numpy(np.float64, 300 * 300).reshape(300, 300), A @ B)  # below 2^53: exact


def _pattern(g, rows, cols, nnz):
    row = np.sort(g.integers(0, rows, nnz))
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum(np.bincount(row, minlength=rows), out=rp[1:])
    return row, rp, g.integers(0, cols, nnz).astype(np.int32)


@pytest.mark.parametrize("first", ["spmm_t", "sddmm", "both"])
@pytest.mark.parametrize("ncols,cols", [(64, 900), (16, 5000), (33, 5000)])
def test_first_sparse_gradient_of_a_handle_in_a_capture(f4j, oracle, first, ncols, cols):
    """S^T W and the SDDMM as a handle's first calls inside a capture: calls on the handle outside of the graph,
    before it ever runs, do not meet arrays that the graph owns, and the graph runs any number of times."""
    import torch
    from flag4j_gb300.device import check
    g = np.random.default_rng(ncols + cols)
    rows, nnz = 700, 9000
    row, rp, ci = _pattern(g, rows, cols, nnz)
    v, W, X = g.standard_normal(nnz), g.standard_normal((rows, ncols)), g.standard_normal((cols, ncols))
    trp, tci, tv, _ = oracle.csr_transpose(rows, cols, rp, ci, v)
    dX_ref = oracle.spmm(trp, tci, tv, W)
    terms = W[row].astype(np.longdouble) * X[ci].astype(np.longdouble)
    bound = 2 * ncols * 2.0 ** -53 * np.abs(terms).sum(1)

    with capturing_context(f4j) as (ctx, capture):
        bufs = [ctx.from_numpy(a) for a in (rp, ci, v)]
        h = ctypes.c_void_p()
        check(ctx.lib.f4j_csr_wrap(ctx.handle, rows, cols, nnz, *[b.handle for b in bufs], 0, ctypes.byref(h)))
        dW, dX, dXin, dS = ctx.from_numpy(W), ctx.alloc(8 * cols * ncols), ctx.from_numpy(X), ctx.alloc(8 * nnz)

        def spmm_t():
            check(ctx.lib.f4j_spmm_t(ctx.handle, h, dW.handle, ncols, dX.handle, None))

        def sddmm():
            check(ctx.lib.f4j_sddmm(ctx.handle, h, dW.handle, dXin.handle, ncols, dS.handle, None))

        def verify(which):
            if which != "sddmm":
                assert np.array_equal(dX.to_numpy(np.float64, cols * ncols).reshape(cols, ncols), dX_ref)
            if which != "spmm_t":
                assert np.all(np.abs(dS.to_numpy(np.float64, nnz) - terms.sum(1)) <= bound)
            dX.zero()
            dS.zero()
            ctx.sync()

        def captured():
            if first != "sddmm":
                spmm_t()
            if first != "spmm_t":
                sddmm()

        graph = capture(captured)
        spmm_t()
        sddmm()
        verify("both")
        for _ in range(3):
            graph.replay()
            torch.cuda.synchronize()
            verify(first)
        spmm_t()
        sddmm()
        verify("both")
        again = capture(captured)  # with the handle's own arrays now
        again.replay()
        torch.cuda.synchronize()
        verify(first)
        check(ctx.lib.f4j_csr_free(ctx.handle, h))
        del graph, again


def test_transpose_permutation_in_a_capture(f4j):
    import torch
    from flag4j_gb300.device import check
    g = np.random.default_rng(3)
    rows, cols, nnz = 500, 3000, 7000
    _, rp, ci = _pattern(g, rows, cols, nnz)
    with capturing_context(f4j) as (ctx, capture):
        bufs = [ctx.from_numpy(a) for a in (rp, ci, g.standard_normal(nnz))]
        h = ctypes.c_void_p()
        check(ctx.lib.f4j_csr_wrap(ctx.handle, rows, cols, nnz, *[b.handle for b in bufs], 0, ctypes.byref(h)))
        perm = ctx.alloc(4 * nnz)
        call = lambda: check(ctx.lib.f4j_csr_transpose_perm(ctx.handle, h, perm.handle))
        graph = capture(call)
        want = np.argsort(ci, kind="stable")
        for run in (graph.replay, call, graph.replay):
            perm.zero()
            ctx.sync()
            run()
            torch.cuda.synchronize()
            assert np.array_equal(perm.to_numpy(np.int32, nnz), want)
        check(ctx.lib.f4j_csr_free(ctx.handle, h))
