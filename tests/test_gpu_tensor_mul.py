"""The Fp products reduced on the tensor cores (tensor_mul.cuh) on the device against
Python integers, one after another and through the pipeline, and their bounded
wait: one that runs out marks the error words and ends, and the device is as usable
as before."""
import random
import time

import numpy as np
import pytest

import vkzg_b200
from conftest import random_blobs
from test_tensor_mul import P, R

pytestmark = pytest.mark.gpu


def operands():
    """Values below 2^382: the ends of the range, of a product's range and of the
    Karatsuba halves, then random ones below p and up to the end."""
    rng = random.Random(11)
    edge = [0, 1, 2, P - 1, P, P + (1 << 365) - 1, 2 * P - 1, (1 << 382) - 1, (1 << 191) - 1, 1 << 191, (1 << 191) + 1,
            ((1 << 191) - 1) << 191, R % P, (1 << 381) - 1, (1 << 382) - (1 << 191)]
    return edge + [rng.randrange(P) for _ in range(400)] + [rng.randrange(1 << 382) for _ in range(100)]


def _words(vals):
    return np.array([[(x >> (32 * i)) & 0xFFFFFFFF for i in range(12)] for x in vals], np.uint32)


def _ints(words):
    return [int.from_bytes(row.astype("<u4").tobytes(), "little") for row in words]


def _check_products(a, b, out):
    rinv = pow(R, -1, P)
    ab, aa, bb = ([x * y * rinv % P for x, y in zip(u, v)] for u, v in ((a, b), (a, a), (b, b)))
    for got, want in ((out[0], ab), (out[1], aa)):  # not reduced below p
        got = _ints(got)
        assert [x % P for x in got] == want
        assert max(got) < P + (1 << 365)
    for got, want in ((out[2], ab), (out[3], bb), (out[4], aa)):
        assert _ints(got) == want


@pytest.mark.parametrize("n", [1, 255, 256, 515])
def test_products(n):
    vals = operands()
    assert len(vals) == 515
    a = vals[:n]
    b = [vals[(5 * k + 2) % len(vals)] for k in range(n)]
    out, marked = vkzg_b200.tensor_mul_selftest(_words(a), _words(b))
    assert marked == 0
    _check_products(a, b, out)


def test_wait_runs_out(oracle, mainnet_tables, monkeypatch):
    vals = operands()
    b = vals[::-1]
    t0 = time.perf_counter()
    out, marked = vkzg_b200.tensor_mul_selftest(_words(vals), _words(b), give_up=True)
    assert time.perf_counter() - t0 < 30
    assert marked == 8
    _check_products(vals, b, out)  # made before that wait
    out, marked = vkzg_b200.tensor_mul_selftest(_words(vals), _words(b))
    assert marked == 0
    _check_products(vals, b, out)
    monkeypatch.delenv("VKZG_TABLES_PATH", raising=False)
    monkeypatch.setenv("VKZG_PLAN", "4")
    blobs = random_blobs(2, 77)
    with vkzg_b200.Prover(max_batch_size=2) as p:
        got = np.zeros(2 * 6144, np.uint8)
        assert p.compute_proofs_raw(got, blobs, 2) == 0
    rc, want = oracle.compute_proofs(mainnet_tables, blobs)
    assert rc == 0 and np.array_equal(got, np.asarray(want).reshape(-1))
