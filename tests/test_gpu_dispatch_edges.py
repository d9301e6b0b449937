"""Blob counts on both sides of the lines where the launchers choose another
kernel (148 SMs: reduction by warps up to 4 and 9 blobs, tails of phase A's lists
up to 9 and 37, clusters of eight up to 18, ladder lanes up to 37 and 74, Horner
lanes up to 37): every count gives the bytes of the same blobs in a larger call,
and the adversarial ones and a random one are the oracle's."""
import numpy as np
import pytest

import vkzg_b200
from conftest import adversarial_blobs, random_blobs

pytestmark = pytest.mark.gpu

LARGEST = 80
COUNTS = [1, 4, 5, 9, 10, 18, 19, 37, 38, 74, 75]


@pytest.fixture(scope="module")
def blobs():
    return np.concatenate([adversarial_blobs(), random_blobs(LARGEST - 4, 9091)])


def proofs(p, blobs, n):
    out = np.zeros(n * 6144, np.uint8)
    assert p.compute_proofs_raw(out, np.ascontiguousarray(blobs[:n]), n) == 0
    return out


@pytest.mark.parametrize("plan", [0, 3, 4])
def test_proofs_at_the_lines(blobs, oracle, mainnet_tables, monkeypatch, plan):
    monkeypatch.delenv("VKZG_TABLES_PATH", raising=False)
    monkeypatch.setenv("VKZG_PLAN", str(plan))
    monkeypatch.setenv("VKZG_COMB_BITS", "9")
    with vkzg_b200.Prover(max_batch_size=LARGEST) as p:
        whole = proofs(p, blobs, LARGEST)
        for n in COUNTS:
            assert np.array_equal(proofs(p, blobs, n), whole[:n * 6144]), n
    rc, want = oracle.compute_proofs(mainnet_tables, np.ascontiguousarray(blobs[:5]))
    assert rc == 0
    assert np.array_equal(whole[:5 * 6144], np.asarray(want).reshape(-1))


def test_cells_and_recovery_at_the_lines(blobs, oracle):
    rng = np.random.default_rng(5)
    with vkzg_b200.Prover(max_batch_size=LARGEST) as p:
        cells = np.zeros((LARGEST, 262144), np.uint8)
        assert p.compute_cells_raw(cells, blobs, LARGEST) == 0
        present = np.zeros((LARGEST, 128), np.uint8)
        for b in range(LARGEST):
            present[b, rng.choice(128, int(rng.integers(64, 128)), replace=False)] = 1
        present[0], present[1] = np.arange(128) < 64, np.arange(128) % 2
        erased = cells.reshape(LARGEST, 128, 2048) * present[:, :, None]
        for n in (1, 18, 19):
            some = np.zeros((n, 262144), np.uint8)
            assert p.compute_cells_raw(some, np.ascontiguousarray(blobs[:n]), n) == 0
            assert np.array_equal(some, cells[:n]), n
            some[:] = 0
            assert p.recover_cells_raw(some, np.ascontiguousarray(erased[:n]), np.ascontiguousarray(present[:n]), n) == 0
            assert np.array_equal(some, cells[:n]), n
    for b in (0, 3, 4):
        rc, want = oracle.compute_cells(blobs[b])
        assert rc == 0 and np.array_equal(cells[b], np.asarray(want).reshape(-1)), b


def test_device_calls_at_the_lines(blobs, monkeypatch):
    """The device entry points at the same counts: the bytes of the host calls."""
    torch = pytest.importorskip("torch")
    monkeypatch.delenv("VKZG_TABLES_PATH", raising=False)
    monkeypatch.setenv("VKZG_PLAN", "3")
    monkeypatch.setenv("VKZG_COMB_BITS", "9")
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(6)
    present = np.zeros((LARGEST, 128), np.uint8)
    for b in range(LARGEST):
        present[b, rng.choice(128, int(rng.integers(64, 128)), replace=False)] = 1
    with vkzg_b200.Prover(max_batch_size=LARGEST) as p:
        cells, want = np.zeros((LARGEST, 262144), np.uint8), np.zeros(LARGEST * 6144, np.uint8)
        assert p.compute_cells_and_proofs_raw(cells, want, blobs, LARGEST) == 0
        erased = cells.reshape(LARGEST, 128, 2048) * present[:, :, None]
        d_blobs, d_cells, d_present = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (blobs, erased, present))
        stream = torch.cuda.current_stream(dev).cuda_stream
        for n in COUNTS:
            d_out, d_ext = (torch.zeros(n * w, dtype=torch.uint8, device=dev) for w in (6144, 262144))
            d_err, d_miss = (torch.ones(n, dtype=torch.int32, device=dev) for _ in range(2))
            assert p.compute_proofs_device(d_out.data_ptr(), d_blobs.data_ptr(), d_err.data_ptr(), n, stream) == 0
            assert p.recover_cells_device(d_ext.data_ptr(), d_cells.data_ptr(), d_present.data_ptr(),
                                          d_miss.data_ptr(), n, stream) == 0
            assert not d_err.any() and not d_miss.any(), n
            assert np.array_equal(d_out.cpu().numpy(), want[:n * 6144]), n
            assert np.array_equal(d_ext.cpu().numpy(), cells[:n].reshape(-1)), n
