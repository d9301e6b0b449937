"""The Fp product whose reduction is a byte matrix product (tensor_mul.cuh), built
for the host with the matrix product in integers, against Python integers."""
import ctypes
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
R = 1 << 384


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tm") / "libtm.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", out,
                           os.path.join(ROOT, "tests", "tensor_mul_shim.cpp")])
    lib = ctypes.CDLL(out)
    lib.shim_tm_largest.restype = ctypes.c_uint64
    return lib


def words(x):
    return (ctypes.c_uint32 * 12)(*[(x >> (32 * i)) & 0xFFFFFFFF for i in range(12)])


def test_matrix_rows(shim):
    """Row i of part z: 2^(8 i) 2^32 / R times the part's Karatsuba factor."""
    base = pow(2, 32 - 384, P)
    factors = (1 - (1 << 191), (1 << 382) - (1 << 191), 1 << 191)
    row = (ctypes.c_uint8 * 48)()
    for z, f in enumerate(factors):
        for i in range(48):
            shim.shim_tm_row(48 * z + i, row)
            assert int.from_bytes(bytes(row), "little") == base * f * (1 << (8 * i)) % P


@pytest.mark.parametrize("sqr", [0, 1])
def test_products(shim, sqr):
    """Congruent to a b / R, below p + 2^365, for operands up to 2^382 (the split's
    halves and their sum at their largest)."""
    rng = random.Random(11)
    edge = [0, 1, 2, P - 1, P, P + (1 << 365) - 1, 2 * P - 1, (1 << 382) - 1, (1 << 191) - 1, 1 << 191, (1 << 191) + 1,
            ((1 << 191) - 1) << 191, R % P, (1 << 381) - 1, (1 << 382) - (1 << 191)]
    vals = edge + [rng.randrange(P) for _ in range(400)] + [rng.randrange(1 << 382) for _ in range(100)]
    out = (ctypes.c_uint32 * 12)()
    rinv = pow(R, -1, P)
    for k, a in enumerate(vals):
        b = vals[(5 * k + 2) % len(vals)]
        for x, y in ((a, b), (a, edge[k % len(edge)])):
            shim.shim_tm_mul(words(x), words(y), sqr, out)
            got = sum(out[i] << (32 * i) for i in range(12))
            assert got % P == x * (x if sqr else y) * rinv % P
            assert got < P + (1 << 365)
    assert shim.shim_tm_largest() < 1 << 32
