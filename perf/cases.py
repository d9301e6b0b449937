"""The calls a user of this library makes, as measurable cases.

The library turns blobs (4096 field elements, 131072 bytes each) into cell
proofs and cells, and recovers missing cells.  A case is one call, or one burst
of requests to the serving loop, through the public Python interface of
`vkzg_b200` (which is the C ABI with its status codes), on

- "host" buffers: plain numpy arrays, as a client's own allocations are,
- "pinned" buffers: page-locked memory, as a service that cares allocates once,
- "device" buffers: data already in HBM, enqueued on the current stream.

Everything is left at its defaults: the prover of a batch service is sized for
256 blobs and tuned once (digit tables within the default budget), the other
prover is the default one (`max_batch_size` 0).  Provers and the server live as
long as the process, as they do in a program that uses them.

Outputs are whole numbers (bytes and status words), so they compare exactly.
"""
import math

import numpy as np
import torch

import vkzg_b200 as vk

BATCH = 256  # blobs that the batch prover is sized for

# Products per blob that the methods in use cannot do without, and 32-bit
# multiply-adds per product (n^2 for the product, n^2 + n for its reduction).
# Proofs: 64 x 23 table points per output (the default table budget) summed by
# affine additions of 6 products, phase B's 67 k additions, the reduction and
# the ladder.  Recovery: four transforms of 8192 with 13 stages.  Cells: two of 4096.
FP_PER_PROOF_BLOB = 1.85e6
FR_PER_RECOVERY_BLOB = 0.28e6
FR_PER_CELLS_BLOB = 0.057e6
OPS_FP, OPS_FR = 2 * (2 * 144 + 12), 2 * (2 * 64 + 8)

# Requests of a served burst, in the order that they arrive: geometric-looking
# sizes with a mean near 6, three in ten of them recoveries.
BURST_SIZES = (1, 6, 3, 11, 2, 19, 5, 1, 8, 4, 1, 13, 2, 7, 3)
BURST_RECOVERY = (2, 5, 9)  # index mod 10

OPS = ("proofs", "cells", "cells_proofs", "recover", "recover_proofs", "served")


def listed():
    return [
        # one blob on the default prover: a wallet or a test; latency and launches count
        dict(name="proofs_host_1_default", op="proofs", place="host", blobs=1, prover="default"),
        # the blobs of one ordinary block, built by a block producer
        dict(name="proofs_host_6", op="proofs", place="host", blobs=6, prover="batch"),
        # an odd count that is already on the device, from another stage of a pipeline
        dict(name="proofs_device_37", op="proofs", place="device", blobs=37, prover="batch"),
        # the headline: a full batch of a proving service
        dict(name="proofs_device_256", op="proofs", place="device", blobs=256, prover="batch"),
        # the extension alone, of a full block's blobs
        dict(name="cells_host_9", op="cells", place="host", blobs=9, prover="batch"),
        # cells and proofs from one upload (a publisher of sidecars), page-locked buffers
        dict(name="cells_proofs_pinned_96", op="cells_proofs", place="pinned", blobs=96, prover="batch"),
        # recovery of one block's blobs with half of the columns or more
        dict(name="recover_host_6", op="recover", place="host", blobs=6, prover="batch", present="uneven"),
        # the fewest cells that can be recovered from, exactly 64 of 128
        dict(name="recover_device_16_half", op="recover", place="device", blobs=16, prover="batch", present="half"),
        # a full batch with uneven surviving sets
        dict(name="recover_device_256", op="recover", place="device", blobs=256, prover="batch", present="uneven"),
        # more than the prover holds: two chunks, the second one ragged
        dict(name="recover_pinned_300", op="recover", place="pinned", blobs=300, prover="batch", present="uneven"),
        # a node that restores columns and serves them again: cells and their proofs
        dict(name="recover_proofs_pinned_21", op="recover_proofs", place="pinned", blobs=21, prover="batch",
             present="uneven"),
        # requests of several clients at once, in page-locked buffers, through the serving loop
        dict(name="served_burst_100", op="served", place="pinned", blobs=100, present="uneven"),
    ]


def draw(rng):
    op = rng.choice(OPS)
    case = dict(op=op)
    most = {"served": 200, "recover": 300, "cells": 300}.get(op, 256)
    n = min(most, max(1, round(math.exp(rng.uniform(0.0, math.log(most))))))
    case["blobs"] = n
    if op == "served":
        case["place"] = "pinned"
        case["blobs"] = max(n, 2)
    else:
        places = ["host", "pinned"] + (["device"] if op in ("proofs", "recover") else [])
        case["place"] = rng.choice(places)
        case["prover"] = "default" if n <= 4 and rng.random() < 0.5 else "batch"
    if op in ("recover", "recover_proofs", "served"):
        case["present"] = rng.choice(("uneven", "half"))
    return case


# ------------------------------------------------------------- what a program keeps
_kept = {}


def _prover(kind):
    if kind not in _kept:
        if kind == "batch":
            p = vk.Prover(max_batch_size=BATCH)
            p.autotune(BATCH)
        else:
            p = vk.Prover()
            p.autotune()
        _kept[kind] = p
    return _kept[kind]


def _server():
    if "server" not in _kept:
        _kept["server"] = vk.Server()
    return _kept["server"]


# ------------------------------------------------------------------------- inputs
def _blobs(n, seed):
    """n blobs of canonical field elements (big-endian, below the modulus, whose
    leading bytes are 73 ed), on the device.  Every eighth blob's data ends
    partway and zeros follow, as when a rollup posts less than a full blob."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    b = torch.randint(0, 256, (n, 4096, 32), dtype=torch.uint8, device="cuda", generator=g)
    b[:, :, 0] %= 0x74
    top = b[:, :, 0] == 0x73
    b[:, :, 1] = torch.where(top, b[:, :, 1] % 0xED, b[:, :, 1])
    ends = np.random.default_rng(seed).integers(1, 4096, size=n)
    for k in range(7, n, 8):
        b[k, int(ends[k]):] = 0
    return b.reshape(n, vk.BYTES_PER_BLOB)


def _present(n, seed, kind):
    """Which cells survive, per blob: exactly 64, or 64 to 127 of them; among the
    uneven ones a contiguous half and every other cell."""
    rng = np.random.default_rng(seed)
    m = np.zeros((n, vk.CELL_PROOFS_PER_BLOB), np.uint8)
    for k in range(n):
        m[k, rng.permutation(128)[:64 if kind == "half" else int(rng.integers(64, 128))]] = 1
    if kind == "uneven" and n >= 4:
        m[1] = np.arange(128) < 64
        m[2] = np.arange(128) % 2
    return m


def _extension(d_blobs):
    """The cells of the blobs (a valid codeword each), as a host array."""
    n = d_blobs.shape[0]
    host = d_blobs.cpu().numpy()
    out = np.empty((n, vk.BYTES_PER_EXT_BLOB), np.uint8)
    _check(_prover("batch").compute_cells_raw(out, host, n))
    return out


def _erased(cells, present):
    n = cells.shape[0]
    return (cells.reshape(n, 128, vk.BYTES_PER_CELL) * present[:, :, None]).reshape(n, vk.BYTES_PER_EXT_BLOB)


def _put(a, place):
    """The array where the case has its buffers."""
    if place == "device":
        return torch.as_tensor(a).cuda()
    if place == "pinned":
        t = torch.empty(tuple(a.shape), dtype=torch.uint8, pin_memory=True)
        t.copy_(torch.as_tensor(a))
        return t
    return a.cpu().numpy() if isinstance(a, torch.Tensor) else np.ascontiguousarray(a)


def _out(n, width, place):
    if place == "device":
        return torch.zeros((n, width), dtype=torch.uint8, device="cuda")
    if place == "pinned":
        return torch.zeros((n, width), dtype=torch.uint8, pin_memory=True)
    return np.zeros((n, width), np.uint8)


def _ptr(a):
    return a.data_ptr() if isinstance(a, torch.Tensor) else a


def _check(status):
    if status:
        raise RuntimeError("vkzg status %d" % status)


PROOF_BYTES = vk.CELL_PROOFS_PER_BLOB * vk.BYTES_PER_PROOF


def _burst(case, seed):
    """The requests of a served burst: (kind, input, mask, output, blobs) each."""
    sizes, total = [], 0
    while total < case["blobs"]:
        s = min(BURST_SIZES[len(sizes) % len(BURST_SIZES)], case["blobs"] - total)
        sizes.append(s)
        total += s
    d = _blobs(total, seed)
    reqs, at = [], 0
    for i, s in enumerate(sizes):
        part = d[at:at + s]
        at += s
        if i % 10 in BURST_RECOVERY:
            m = _present(s, seed + i, case["present"])
            reqs.append(("recover", _put(_erased(_extension(part), m), "pinned"), _put(m, "pinned"),
                         _out(s, vk.BYTES_PER_EXT_BLOB, "pinned"), s))
        else:
            reqs.append(("proofs", _put(part, "pinned"), None, _out(s, PROOF_BYTES, "pinned"), s))
    return reqs


def prepare(case, seed):
    op, n, place = case["op"], case["blobs"], case["place"]
    if op == "served":
        return dict(op=op, server=_server(), requests=_burst(case, seed))
    s = dict(op=op, place=place, n=n, prover=_prover(case["prover"]))
    d = _blobs(n, seed)
    if op in ("recover", "recover_proofs"):
        m = _present(n, seed, case["present"])
        s["in"], s["mask"] = _put(_erased(_extension(d), m), place), _put(m, place)
    else:
        s["in"] = _put(d, place)
    if op != "proofs":
        s["cells"] = _out(n, vk.BYTES_PER_EXT_BLOB, place)
    if op not in ("cells", "recover"):
        s["proofs"] = _out(n, PROOF_BYTES, place)
    if place == "device":
        s["err"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    return s


def run(s):
    op = s["op"]
    if op == "served":
        server, tickets = s["server"], []
        for kind, src, mask, out, n in s["requests"]:
            if kind == "proofs":
                tickets.append(server.submit_proofs(out.data_ptr(), src.data_ptr(), n))
            else:
                tickets.append(server.submit_recovery(out.data_ptr(), src.data_ptr(), mask.data_ptr(), n))
        for t in tickets:
            _check(server.wait(t))
        return [r[3] for r in s["requests"]]
    p, n = s["prover"], s["n"]
    if s["place"] == "device":
        stream = torch.cuda.current_stream().cuda_stream
        if op == "proofs":
            _check(p.compute_proofs_device(s["proofs"].data_ptr(), s["in"].data_ptr(), s["err"].data_ptr(), n, stream))
            return s["proofs"], s["err"]
        _check(p.recover_cells_device(s["cells"].data_ptr(), s["in"].data_ptr(), s["mask"].data_ptr(),
                                      s["err"].data_ptr(), n, stream))
        return s["cells"], s["err"]
    src = _ptr(s["in"])
    if op == "proofs":
        _check(p.compute_proofs_raw(_ptr(s["proofs"]), src, n))
        return s["proofs"]
    if op == "cells":
        _check(p.compute_cells_raw(_ptr(s["cells"]), src, n))
        return s["cells"]
    if op == "cells_proofs":
        _check(p.compute_cells_and_proofs_raw(_ptr(s["cells"]), _ptr(s["proofs"]), src, n))
        return s["cells"], s["proofs"]
    if op == "recover":
        _check(p.recover_cells_raw(_ptr(s["cells"]), src, _ptr(s["mask"]), n))
        return s["cells"]
    _check(p.recover_cells_and_proofs_raw(_ptr(s["cells"]), _ptr(s["proofs"]), src, _ptr(s["mask"]), n))
    return s["cells"], s["proofs"]


def _unit(op):
    """(bytes, operations) of one blob."""
    blob, ext = vk.BYTES_PER_BLOB, vk.BYTES_PER_EXT_BLOB
    proof = FP_PER_PROOF_BLOB * OPS_FP
    return {
        "proofs": (blob + PROOF_BYTES, proof),
        "cells": (blob + ext, FR_PER_CELLS_BLOB * OPS_FR),
        "cells_proofs": (blob + ext + PROOF_BYTES, proof + FR_PER_CELLS_BLOB * OPS_FR),
        "recover": (2 * ext + 128, FR_PER_RECOVERY_BLOB * OPS_FR),
        "recover_proofs": (2 * ext + 128 + PROOF_BYTES, proof + FR_PER_RECOVERY_BLOB * OPS_FR),
    }[op]


def work(case):
    if case["op"] == "served":
        (pb, pf), (rb, rf) = _unit("proofs"), _unit("recover")
        return {"bytes": case["blobs"] * (0.7 * pb + 0.3 * rb), "flops": case["blobs"] * (0.7 * pf + 0.3 * rf)}
    b, f = _unit(case["op"])
    return {"bytes": case["blobs"] * b, "flops": case["blobs"] * f}


def tolerance(case):
    return "exact"
