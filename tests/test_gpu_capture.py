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
