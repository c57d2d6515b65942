"""Which form a split product takes, seen in its bits.

45-bit integers fill more of the fixed-point form than the slices multiply out: they drop the products of two
low slices, so some of their entries are not the exact sum rounded once.  The residue form keeps the exact
sum, so every entry is.  An entry's own sum is formed with Python integers."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ints45(shape, seed):
    g = np.random.default_rng(seed)
    return g.integers(-(1 << 45) + 1, 1 << 45, shape)


def rounded_once(A, B, C, samples=1200, seed=9):
    """How many of `samples` entries of C are the exact sum of A B (integers) rounded once."""
    g = np.random.default_rng(seed)
    i, j = g.integers(0, A.shape[0], samples), g.integers(0, B.shape[1], samples)
    exact = 0
    for r, c in zip(i, j):
        s = sum(int(x) * int(y) for x, y in zip(A[r], B[:, c]))
        exact += C[r, c] == float(s)  # int to float rounds to nearest, ties to even
    return exact, samples


def product(f4j, A, B, mode, opA=0, opB=0, host=False):
    from flag4j_gb300 import _lib
    from flag4j_gb300.device import check
    ctx = f4j.default_context()
    (m, k), n = A.shape, B.shape[1]
    a = np.ascontiguousarray((A if opA == 0 else A.T).astype(np.float64))
    b = np.ascontiguousarray((B if opB == 0 else B.T).astype(np.float64))
    rep, C = _lib.f4j_report(), np.empty((m, n))
    if host:
        check(ctx.lib.f4j_dgemm_host(ctx.handle, m, n, k, a.ctypes.data, opA, b.ctypes.data, opB, C.ctypes.data, mode,
                                     ctypes.byref(rep)))
    else:
        dA, dB, dC = ctx.from_numpy(a), ctx.from_numpy(b), ctx.alloc(8 * m * n)
        check(ctx.lib.f4j_dgemm(ctx.handle, m, n, k, dA.handle, opA, dB.handle, opB, dC.handle, mode, ctypes.byref(rep)))
        C = dC.to_numpy(np.float64, m * n).reshape(m, n)
    assert rep.mode_used == _lib.MODE_SPLIT and rep.frac_bits >= 49
    return C


@pytest.mark.parametrize("m,n,k,form", [
    (129, 700, 256, "residues"), (128, 700, 300, "slices"), (700, 129, 300, "residues"),       # one slice tile
    (300, 300, 300, "residues"), (400, 400, 255, "slices"), (400, 400, 256, "residues"),       # the shortest sums
    (1254, 1254, 512, "residues"), (1300, 1300, 512, "slices"), (1300, 1300, 513, "residues"),  # whole slice chunks
    (1300, 1300, 288, "residues"), (1300, 1300, 449, "slices"), (1300, 1300, 448, "residues"),
    (4100, 4100, 319, "slices"), (4100, 4100, 320, "residues"), (255, 257, 4100, "residues"),
])
def test_auto_takes_the_form_its_rule_says(f4j, m, n, k, form):
    from flag4j_gb300 import _lib
    A, B = ints45((m, k), m), ints45((k, n), n + 1)
    for opA, opB in ((0, 0), (1, 1)):
        good, of = rounded_once(A, B, product(f4j, A, B, _lib.MODE_AUTO, opA, opB))
        assert (good == of) == (form == "residues"), (good, of)


@pytest.mark.parametrize("m,n,k,form", [
    (1024, 1024, 1344, "slices"), (1024, 1024, 1408, "residues"),  # what f4j_dgemm_split_noalloc accepts, and not
    (513, 400, 8193, "residues"), (384, 385, 4100, "residues"), (384, 300, 4000, "slices"),
])
def test_split_mode_keeps_the_slices_of_the_no_allocation_shapes(f4j, m, n, k, form):
    from flag4j_gb300 import _lib
    A, B = ints45((m, k), m), ints45((k, n), n + 1)
    for host in (False, True):
        good, of = rounded_once(A, B, product(f4j, A, B, _lib.MODE_SPLIT, host=host))
        assert (good == of) == (form == "residues"), (good, of, host)


def test_auto_with_split_configured_by_name_is_split(f4j, tmp_path):
    """gpuGemmMode = split: AUTO's bits are F4J_MODE_SPLIT's, from the device and from host arrays, where the
    default takes the residues."""
    from flag4j_gb300 import _lib, configs
    A, B = ints45((700, 300), 1), ints45((300, 600), 2)
    sliced = product(f4j, A, B, _lib.MODE_SPLIT)
    try:
        (tmp_path / "GeneralConfigs.properties").write_text("gpuGemmMode = split\n")
        configs.load(tmp_path)
        for host in (False, True):
            assert np.array_equal(product(f4j, A, B, _lib.MODE_AUTO, host=host), sliced)
        (tmp_path / "GeneralConfigs.properties").write_text("gpuGemmMode = auto\n")
        configs.load(tmp_path)
        for host in (False, True):
            C = product(f4j, A, B, _lib.MODE_AUTO, host=host)
            assert not np.array_equal(C, sliced) and len(set(rounded_once(A, B, C))) == 1
    finally:
        configs.reset()
