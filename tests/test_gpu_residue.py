"""The split GEMM's residue form (f4j_crt.cuh): products the slice form leaves
to it, at the edges of its 256 x 256 tiles, 128-byte K blocks and 8192-term
accumulations.

Integer operands below 2^20 lose nothing in the fixed-point form (F >= 49
bits), and the reconstruction is exact, so C is the exact integer product as
long as that is below 2^53: bit for bit the int64 product.  Elsewhere the bar
is the form's own bound: every element is rounded to half a unit 2^(e - F), so
|C - C_true| <= 2^-(F+1) (2^e_i |b_j|_1 + 2^f_j |a_i|_1) + k 2^-(2F+2) 2^(e_i+f_j)
+ u |C|.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(f4j, A, B, opA=0, opB=0, host=False):
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    ctx = f4j.default_context()
    cplx = np.iscomplexobj(A)
    m, k = A.shape if opA == 0 else A.shape[::-1]
    n = B.shape[1] if opB == 0 else B.shape[0]
    rep, dt = _lib.f4j_report(), np.complex128 if cplx else np.float64
    if host:
        C = np.empty((m, n), dt)
        fn = ctx.lib.f4j_zgemm_host if cplx else ctx.lib.f4j_dgemm_host
        check(fn(ctx.handle, m, n, k, A.ctypes.data, opA, B.ctypes.data, opB, C.ctypes.data, _lib.MODE_SPLIT,
                 ctypes.byref(rep)))
        return C, rep
    dA, dB, dC = ctx.from_numpy(A), ctx.from_numpy(B), ctx.alloc(C_bytes(m, n, cplx))
    fn = ctx.lib.f4j_zgemm if cplx else ctx.lib.f4j_dgemm
    check(fn(ctx.handle, m, n, k, dA.handle, opA, dB.handle, opB, dC.handle, _lib.MODE_SPLIT, ctypes.byref(rep)))
    return dC.to_numpy(dt, m * n).reshape(m, n), rep


def C_bytes(m, n, cplx):
    return m * n * (16 if cplx else 8)


def ints(shape, seed, cplx=False):
    g = np.random.default_rng(seed)
    x = g.integers(-(1 << 19), 1 << 19, shape)
    return x + 1j * g.integers(-(1 << 19), 1 << 19, shape) if cplx else x.astype(np.float64)


def int_product(A, B):
    """Exact product of integer-valued float arrays (|sums| < 2^53)."""
    if np.iscomplexobj(A):
        r = lambda X, Y: int_product(np.ascontiguousarray(X), np.ascontiguousarray(Y))
        return (r(A.real, B.real) - r(A.imag, B.imag)) + 1j * (r(A.real, B.imag) + r(A.imag, B.real))
    # float64 BLAS on 10-bit halves is exact: |sums| < k 2^40 < 2^53 for each of the four
    hi, lo = np.floor(A / 1024.0), A - 1024.0 * np.floor(A / 1024.0)
    bh, bl = np.floor(B / 1024.0), B - 1024.0 * np.floor(B / 1024.0)
    return (hi @ bh) * 1048576.0 + ((hi @ bl) + (lo @ bh)) * 1024.0 + lo @ bl


@pytest.mark.parametrize("m,n,k,opA,opB", [
    (384, 385, 4100, 0, 0),    # two tiles each way, a ragged K block
    (513, 400, 8193, 0, 1),    # one row past two tiles, one term past an accumulation
    (400, 700, 16500, 1, 0),   # three accumulations
    (2049, 385, 1100, 0, 0),   # nine tile rows
    (1029, 1023, 1400, 1, 1),
])
def test_residue_form_is_exact_on_integers(f4j, m, n, k, opA, opB):
    A, B = ints((m, k), m), ints((k, n), n)
    ref = int_product(A, B)
    a = A if opA == 0 else np.ascontiguousarray(A.T)
    b = B if opB == 0 else np.ascontiguousarray(B.T)
    C, rep = run(f4j, a, b, opA, opB)
    assert rep.mode_used == 1 and rep.slices >= 10
    assert np.array_equal(C, ref)
    if opA == 0:
        assert np.array_equal(run(f4j, a, b, 0, opB, host=True)[0], ref)


@pytest.mark.parametrize("m,n,k,opA,opB", [(384, 193, 301, 0, 0), (500, 333, 4099, 0, 2), (391, 250, 700, 2, 1)])
def test_residue_form_complex_is_exact_on_integers(f4j, m, n, k, opA, opB):
    A, B = ints((m, k), m, True), ints((k, n), n, True)
    ref = int_product(A, B)
    tr = {0: lambda X: X, 1: lambda X: np.ascontiguousarray(X.T), 2: lambda X: np.ascontiguousarray(X.conj().T)}
    C, rep = run(f4j, tr[opA](A), tr[opB](B), opA, opB)
    assert rep.mode_used == 1 and np.array_equal(C, ref)
    if opA == 0:
        assert np.array_equal(run(f4j, A, tr[opB](B), 0, opB, host=True)[0], ref)


@pytest.mark.parametrize("v,w", [(17, 17), (-17, 17), (850, 850), (-801, 1584), (24, -25), (524287, -524288)])
def test_residue_form_largest_accumulations(f4j, v, w):
    """Constant operands: every term of a modulus's sum is the same product of digits.  17 and 850
    (= 17 + 17 * 49) take the digit -32 modulo 49, so the sums of 8192 terms reach 2^24, the most the FP32
    accumulator holds exactly."""
    k = 8192
    C, rep = run(f4j, np.full((384, k), float(v)), np.full((k, 400), float(w)))
    assert rep.mode_used == 1
    assert np.all(C == float(k * v * w))


@pytest.mark.parametrize("case", ["uniform", "normal", "scaled", "tiny_row", "zero"])
def test_residue_form_within_its_bound(f4j, oracle, case):
    from flag4j_gb300 import synth
    m, n, k = 400, 500, 3333
    A, B = synth.uniform(m, k, 1), synth.uniform(k, n, 2)
    if case == "normal":
        A, B = synth.normal(m, k, 1), synth.normal(k, n, 2)
    elif case == "scaled":
        A, B = synth.scaled(m, k, 300, 1, "row"), synth.scaled(k, n, 300, 2, "col")
    elif case == "tiny_row":
        A[7] *= 2.0 ** -1060
        A[8] *= 2.0 ** 980
        B[:, 3] = 0.0
    elif case == "zero":
        A[:] = 0.0
    C, rep = run(f4j, A, B)
    assert rep.mode_used == 1
    F = rep.frac_bits
    e = np.frexp(np.abs(A).max(axis=1))[1].astype(int)
    f = np.frexp(np.abs(B).max(axis=0))[1].astype(int)
    An, Bn = np.ldexp(A, -e[:, None]), np.ldexp(B, -f[None, :])  # rows and columns below 1
    truth, absab = oracle.dgemm(An, Bn), np.abs(An) @ np.abs(Bn)
    tol = (np.abs(Bn).sum(axis=0)[None, :] + np.abs(An).sum(axis=1)[:, None]) * 2.0 ** -(F + 1) + k * 2.0 ** -(2 * F + 2)
    # the oracle's own rounding (k u |A||B|), and one rounding of C
    tol = tol + (k + 1) * 2.0 ** -53 * absab
    X = e[:, None] + f[None, :]
    normal = X > -900
    got = np.ldexp(C, -np.where(normal, X, 0))
    assert np.all(np.abs(got - truth)[normal] <= tol[normal])
    assert np.all(np.abs(C - np.ldexp(truth, X))[~normal] <= np.ldexp(tol, X)[~normal] + 2.0 ** -1074)
    if case == "zero":
        assert not C.any()
    if case == "tiny_row":
        assert not C[:, 3].any()


def test_residue_form_launches_in_order(f4j):
    """Products queued back to back without a wait, each from the one before (its kernels start while the
    previous kernel's last blocks run), with a non-finite operand that stands the form down in between: bit
    for bit the products of a queue that waits after each."""
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    ctx = f4j.default_context()
    g = np.random.default_rng(5)
    shapes = [(300, 1100, 900), (300, 1500, 1100), (300, 260, 1500), (300, 2048, 260)]
    X0 = g.standard_normal((300, 900))
    Bs = [g.standard_normal((k, n)) for _, n, k in shapes]
    bad = Bs[1].copy()
    bad[3, 4] = np.nan
    outs = []
    for wait in (True, False):
        dX, dB, dbad = ctx.from_numpy(X0), [ctx.from_numpy(B) for B in Bs], ctx.from_numpy(bad)
        dC = [ctx.alloc(C_bytes(m, n, False)) for m, n, _ in shapes]
        dD = ctx.alloc(C_bytes(300, 1500, False))
        for _ in range(3):
            src = dX
            for (m, n, k), b, c in zip(shapes, dB, dC):
                if n == 1500:  # the same sizes with a NaN: the plain product, from the same workspace
                    check(ctx.lib.f4j_dgemm(ctx.handle, m, n, k, src.handle, 0, dbad.handle, 0, dD.handle,
                                            _lib.MODE_AUTO, None))
                check(ctx.lib.f4j_dgemm(ctx.handle, m, n, k, src.handle, 0, b.handle, 0, c.handle, _lib.MODE_AUTO,
                                        None))
                if wait:
                    ctx.sync()
                src = c
        outs.append([c.to_numpy(np.float64, m * n) for c, (m, n, _) in zip(dC, shapes)] +
                    [dD.to_numpy(np.float64, 300 * 1500)])
    for w, q in zip(*outs):
        assert np.array_equal(w, q, equal_nan=True)
    assert np.isnan(outs[0][-1]).any() and not np.isnan(outs[0][0]).any()


@pytest.mark.parametrize("m,n,k", [
    (129, 700, 256), (700, 129, 300), (129, 2048, 288), (255, 257, 4100),   # one tile wide, just past a slice tile
    (1254, 1254, 512), (1300, 1300, 288), (1300, 1300, 449), (1300, 1300, 513),  # short sums of a large C
    (4100, 4100, 320),
])
def test_narrow_and_short_products_take_the_residue_form(f4j, m, n, k):
    """AUTO at the edges of the shapes that the residue form takes: exact on integers, which the slices are
    not, for every order of the operands."""
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    ctx = f4j.default_context()
    A, B = ints((m, k), m), ints((k, n), n + 1)
    want = int_product(A, B)
    for opA, opB in ((0, 0), (0, 1), (1, 0), (1, 1)):
        dA = ctx.from_numpy(A if opA == 0 else np.ascontiguousarray(A.T))
        dB = ctx.from_numpy(B if opB == 0 else np.ascontiguousarray(B.T))
        dC, rep = ctx.alloc(C_bytes(m, n, False)), _lib.f4j_report()
        check(ctx.lib.f4j_dgemm(ctx.handle, m, n, k, dA.handle, opA, dB.handle, opB, dC.handle, _lib.MODE_AUTO,
                                ctypes.byref(rep)))
        assert rep.mode_used == _lib.MODE_SPLIT
        assert np.array_equal(dC.to_numpy(np.float64, m * n).reshape(m, n), want), (opA, opB)
