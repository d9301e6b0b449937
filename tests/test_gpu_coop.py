"""Plans 3-4 with each phase's grid-wide rounds in one cooperative launch
(grid barriers between the passes; $VKZG_COOP=1) against the same plans in
three launches per round (the default), and the grid barrier's bounded wait: a barrier that can never complete
gives up after its poll limit, sets the failure flag and marks the error words,
and the launch ends."""
import time

import numpy as np
import pytest

import vkzg_b200
from conftest import random_blobs

pytestmark = pytest.mark.gpu


def test_grid_barrier_completes():
    passed, flag, marked = vkzg_b200.grid_sync_selftest(0, 1 << 20, 5)
    blocks = passed // 5
    assert passed == 5 * blocks and blocks >= 2
    assert flag == 0 and marked == 0


def test_grid_barrier_wait_runs_out():
    t0 = time.perf_counter()
    passed, flag, marked = vkzg_b200.grid_sync_selftest(1, 20000, 3)
    assert time.perf_counter() - t0 < 30
    assert passed == 0  # no barrier can complete: it waits for a block that does not exist
    assert flag == 1 and marked == 8
    # the device is still usable afterwards
    passed, flag, marked = vkzg_b200.grid_sync_selftest(0, 1 << 20, 2)
    assert flag == 0 and passed > 0


@pytest.mark.parametrize("plan", [3, 4])
def test_cooperative_rounds_match_round_launches(monkeypatch, plan):
    monkeypatch.delenv("VKZG_TABLES_PATH", raising=False)
    monkeypatch.setenv("VKZG_PLAN", str(plan))
    monkeypatch.setenv("VKZG_COMB_BITS", "10")
    blobs = random_blobs(40, 808)
    outs, launches = {}, {}
    for coop in ("1", "0"):
        monkeypatch.setenv("VKZG_COOP", coop)
        with vkzg_b200.Prover(max_batch_size=40) as p:
            out = np.zeros(40 * 6144, np.uint8)
            assert p.compute_proofs_raw(out, blobs, 40) == 0  # captures the pipeline's graph
            k0 = vkzg_b200.kernel_launches()
            assert p.compute_proofs_raw(out, blobs, 40) == 0
            launches[coop] = vkzg_b200.kernel_launches() - k0
            outs[coop] = out
    assert np.array_equal(outs["1"], outs["0"])
    assert launches["1"] <= 10 < launches["0"]


def test_failed_chunk_is_reported_by_every_entry_point(monkeypatch):
    """Grid barriers that give up at once ($VKZG_SYNC_POLLS=0): every call that makes
    proofs reports the failure and leaves no proof in the output, recovery alone
    is unaffected, and a prover without the limit works in the same process."""
    torch = pytest.importorskip("torch")
    monkeypatch.delenv("VKZG_TABLES_PATH", raising=False)
    monkeypatch.setenv("VKZG_PLAN", "3")
    monkeypatch.setenv("VKZG_COMB_BITS", "9")
    n = 3
    blobs = random_blobs(n, 809)
    cells, want = np.zeros(n * 262144, np.uint8), np.zeros(n * 6144, np.uint8)
    present = np.ones((n, 128), np.uint8)
    present[:, ::2] = 0
    with vkzg_b200.Prover(max_batch_size=4) as p:
        assert p.compute_cells_and_proofs_raw(cells, want, blobs, n) == 0
    erased = cells.reshape(n, 128, 2048) * present[:, :, None]
    out, got = np.zeros_like(cells), np.zeros_like(want)
    with monkeypatch.context() as m:
        m.setenv("VKZG_COOP", "1")
        m.setenv("VKZG_SYNC_POLLS", "0")
        with vkzg_b200.Prover(max_batch_size=4) as p:
            assert p.compute_proofs_raw(got, blobs, n) == vkzg_b200.ERR_GPU
            assert not got.any()
            assert p.compute_cells_and_proofs_raw(out, got, blobs, n) == vkzg_b200.ERR_GPU
            assert not got.any() and not out.any()
            assert p.recover_cells_and_proofs_raw(out, got, erased, present, n) == vkzg_b200.ERR_GPU
            assert not got.any()
            dev = torch.device("cuda", 0)
            d_in, d_out = torch.from_numpy(blobs.reshape(-1).copy()).to(dev), torch.zeros(n * 6144, dtype=torch.uint8, device=dev)
            d_err = torch.zeros(n, dtype=torch.int32, device=dev)
            assert p.compute_proofs_device(d_out.data_ptr(), d_in.data_ptr(), d_err.data_ptr(), n,
                                           torch.cuda.current_stream(dev).cuda_stream) == 0
            assert (d_err.cpu().numpy() < 0).all()  # bit 31
            out[:] = 0
            assert p.recover_cells_raw(out, erased, present, n) == 0
            assert np.array_equal(out, cells)
    with vkzg_b200.Prover(max_batch_size=4) as p:
        out[:] = 0
        assert p.recover_cells_and_proofs_raw(out, got, erased, present, n) == 0
    assert np.array_equal(out, cells) and np.array_equal(got, want)
