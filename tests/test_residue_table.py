"""The residue form's constants (CrtTable in f4j_crt.cuh), checked with Python integers (no GPU needed).

tests/native/residue_table_check.cu includes the kernel source and prints the table, which has to be a
compile-time constant."""
import json
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    exe = str(tmp_path_factory.mktemp("residue") / "residue_table_check")
    csrc = os.path.join(ROOT, "flag4j_gb300", "csrc")
    cmd = ["nvcc", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
           "-I", os.path.join(ROOT, "include"), "-o", exe, os.path.join(HERE, "native", "residue_table_check.cu"),
           os.path.join(csrc, "f4j_core.cu"), os.path.join(csrc, "f4j_dense.cu"), os.path.join(csrc, "f4j_config.cu")]
    subprocess.run(cmd, check=True, capture_output=True, timeout=600)
    return json.loads(subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout)


def number(words):
    return sum(w << (32 * i) for i, w in enumerate(words))


def test_every_configuration_reconstructs(table):
    """Per configuration: coprime moduli, weights, group multipliers and word constants, all against M."""
    last = 0
    for c in table["cfgs"]:
        p = [int(m[0]) for m in c["mods"]]
        assert len(p) == c["nmod"] and all(math.gcd(a, b) == 1 for i, a in enumerate(p) for b in p[:i])
        assert all(math.isqrt(q) ** 2 == q for q in p[:c["nsq"]])
        M, top = math.prod(p), 32 * c["words"]
        assert M > last  # rising
        last = M
        assert 2 ** (top - 2) <= M << c["sh"] < 2 ** (top - 1)
        assert number(c["NM"]) == 2 ** top - (M << c["sh"])
        assert abs(c["bits"] - math.log2(M)) < 1e-5
        assert abs(c["qinv"] / float(2 ** (top - 18) / (M << c["sh"])) - 1) < 2 ** -23
        P = [math.prod(int(m[0]) for m in c["mods"] if m[4] == g) for g in range(7)]
        for q, (_, inv, u, cl, g) in zip(p, c["mods"]):
            assert np.float32(inv) == np.float32(1) / np.float32(q)
            assert abs(2 * u) <= q and (M // q * int(u)) % q == 1 % q
            assert cl == P[g] // q
        for g, (z0, *W) in enumerate(c["groups"]):
            if any(m[4] == g for m in c["mods"]):
                assert z0 == 2 * P[g] and number(W) == (M // P[g]) << c["sh"]
            else:
                assert z0 == 0 and not any(W)


def test_picked_configuration_holds_the_sum_and_is_the_cheapest(table):
    """k products of F-bit integers and a sign fit below M; no cheaper entry of the table does."""
    bits = [math.log2(math.prod(int(m[0]) for m in c["mods"])) for c in table["cfgs"]]
    cost = [c["nmod"] + 2 * c["nsq"] for c in table["cfgs"]]
    assert cost == sorted(cost)
    for k, s, i in table["picks"]:
        need = 2 * (4 + 5 * (s - 1)) + math.log2(k) + 1
        assert i >= 0 and bits[i] > need
        assert i == 0 or bits[i - 1] < need + 0.02
