"""The residue form's workspace: what a product does when it cannot have it, and that the host-buffer products
agree with the device's in AUTO, whichever form that is."""
import ctypes

import numpy as np
import pytest

from test_gpu_capture import capturing_context

pytestmark = pytest.mark.gpu


def product(ctx, A, B, mode, opB=0, host=False):
    from flag4j_gb300.device import check
    m, k = A.shape
    n = B.shape[1 if opB == 0 else 0]
    if host:
        C = np.empty((m, n), A.dtype)
        fn = ctx.lib.f4j_zgemm_host if np.iscomplexobj(A) else ctx.lib.f4j_dgemm_host
        check(fn(ctx.handle, m, n, k, A.ctypes.data, 0, B.ctypes.data, opB, C.ctypes.data, mode, None))
        return C
    dA, dB, dC = ctx.from_numpy(A), ctx.from_numpy(B), ctx.alloc(A.dtype.itemsize * m * n)
    fn = ctx.lib.f4j_zgemm if np.iscomplexobj(A) else ctx.lib.f4j_dgemm
    check(fn(ctx.handle, m, n, k, dA.handle, 0, dB.handle, opB, dC.handle, mode, None))
    return dC.to_numpy(A.dtype, m * n).reshape(m, n)


def operands(m, n, k, seed=1, cplx=False):
    g = np.random.default_rng(seed)
    mk = lambda *s: g.standard_normal(s) + 1j * g.standard_normal(s) if cplx else g.standard_normal(s)
    return mk(m, k), mk(k, n)


@pytest.mark.parametrize("m,n,k", [(2111, 1777, 700), (2000, 2000, 640)])
def test_no_room_for_the_residues_takes_the_slices(f4j, monkeypatch, m, n, k):
    """With its workspace capped an AUTO product is the sliced one, on the device and from host arrays; with the
    cap gone the same context takes the residues."""
    from flag4j_gb300 import _lib
    A, B = operands(m, n, k)
    ctx = f4j.Context(0)
    sliced = product(ctx, A, B, _lib.MODE_SPLIT)  # f4j_dgemm_split_noalloc accepts these shapes
    monkeypatch.setenv("F4J_WORKSPACE_MB", "48")
    other = f4j.Context(0)
    for _ in range(2):
        assert np.array_equal(product(other, A, B, _lib.MODE_AUTO), sliced)
        assert np.array_equal(product(other, A, B, _lib.MODE_AUTO, host=True), sliced)
    monkeypatch.delenv("F4J_WORKSPACE_MB")
    residues = product(other, A, B, _lib.MODE_AUTO)
    assert not np.array_equal(residues, sliced)
    assert np.array_equal(residues, product(ctx, A, B, _lib.MODE_AUTO))
    assert np.array_equal(residues, product(ctx, A, B, _lib.MODE_AUTO, host=True))


def test_a_refused_workspace_costs_nothing_again(f4j, monkeypatch):
    """Once refused, a product neither allocates nor frees nor waits: it can be captured."""
    import torch
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    A, B = operands(2000, 1900, 640)
    monkeypatch.setenv("F4J_WORKSPACE_MB", "48")
    with capturing_context(f4j) as (ctx, capture):
        want = product(ctx, A, B, _lib.MODE_AUTO)
        dA, dB, dC = ctx.from_numpy(A), ctx.from_numpy(B), ctx.alloc(8 * 2000 * 1900)
        dC.zero()
        ctx.sync()
        graph = capture(lambda: check(ctx.lib.f4j_dgemm(ctx.handle, 2000, 1900, 640, dA.handle, 0, dB.handle, 0, dC.handle,
                                                        _lib.MODE_AUTO, None)))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(dC.to_numpy(np.float64, 2000 * 1900).reshape(2000, 1900), want)


@pytest.mark.parametrize("m,n,k,opB,cplx", [
    (300, 300, 300, 0, False), (1024, 1024, 1024, 0, False), (1300, 700, 512, 1, False),    # in turn; SPLIT: slices
    (129, 2048, 300, 0, False), (1300, 1300, 449, 0, False), (600, 500, 400, 2, True),
    (2111, 1777, 700, 0, False), (1777, 2111, 900, 1, False), (513, 400, 8193, 1, False),   # in parts
    (1500, 1300, 900, 0, True), (1300, 1500, 901, 1, True), (1301, 1400, 1000, 2, True),
])
def test_host_product_is_the_device_product_in_auto(f4j, m, n, k, opB, cplx):
    """f4j_dgemm_host and f4j_zgemm_host in AUTO: bit for bit f4j_dgemm's and f4j_zgemm's AUTO."""
    from flag4j_gb300 import _lib
    A, B = operands(m, n, k, m + k, cplx)
    B = B if opB == 0 else np.ascontiguousarray(B.T if opB == 1 else B.conj().T)
    ctx = f4j.default_context()
    dev, host = (product(ctx, A, B, _lib.MODE_AUTO, opB=opB, host=h) for h in (False, True))
    assert np.array_equal(host, dev)
    want = A[:40] @ (B if opB == 0 else B.T if opB == 1 else B.conj().T)
    assert np.abs(dev[:40] - want).max() <= 1e-9


@pytest.mark.parametrize("m,n,k,cplx", [
    (12000, 12100, 330, False),    # C's residues past 4 GiB: row blocks on the device, all at once from the host
    (2200000, 160, 330, False),    # and more than 65535 blocks of rows of A
    (8100, 9000, 170, True),
])
def test_large_results_in_row_blocks(f4j, m, n, k, cplx):
    """Integer operands whose sums stay below 2^53: C is the exact product, and the host-buffer product the same."""
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    g = np.random.default_rng(m)
    mk = lambda *s: g.integers(-30000, 30000, s, dtype=np.int32).astype(np.float64)
    A, B = mk(m, k), mk(k, n)
    if cplx:
        A, B = A + 1j * mk(m, k), B + 1j * mk(k, n)
    ctx = f4j.Context(0)  # its workspace goes with it
    want = A @ B
    assert np.array_equal(product(ctx, A, B, _lib.MODE_AUTO), want)
    assert np.array_equal(product(ctx, A, B, _lib.MODE_AUTO, host=True), want)
    ctx.close()
