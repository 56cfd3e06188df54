"""What a user of this framework has it do: proofs of hash batches, through the public calls.

A case is one call: ``form`` says which one, the rest its sizes.

  prove   Setup.prove_fast_bytes on host records (the ordinary call)
  device  Setup.prove_fast_device_bytes on records that are in device memory already
  union   UnionSetup.prove_bytes: several hash types, any declared counts, one proof
  batch   ProofServer.prove_batch: independent proofs of several shapes at once
  cap     flock_gb300_commit_cap_noalloc: the commitment alone, without device allocations

Every output is a proof bundle (or a Merkle cap) in bytes: they are exact, and the same for
the same records and transcript domain, whoever computes them.
"""
import ctypes

import numpy as np
import torch

import flock_gb300
from flock_gb300 import BLAKE3, KECCAK, SHA256

KINDS = {"blake3": BLAKE3, "sha256": SHA256, "keccak": KECCAK}
# log2 of a block's bits, and its 128-bit columns that carry data
K_LOG = {"blake3": 14, "sha256": 15, "keccak": 16}
USED_COLS = {"blake3": 92, "sha256": 199, "keccak": 333}
# the smallest batch of each hash that the protocol has parameters for (2^22 witness bits),
# the largest of the served range, and the largest that the static working set of `cap` takes
LOG_MIN = {"blake3": 8, "sha256": 7, "keccak": 6}
LOG_MAX = 18
LOG_CAP_MAX = {"blake3": 11, "sha256": 10, "keccak": 9}
UNION_TYPES = ["keccak,sha256,blake3", "sha256,blake3", "keccak,blake3", "keccak,sha256"]


def listed():
    return [
        # one small proof: latency, launches and host round trips
        {"name": "blake3_2p8", "form": "prove", "hash": "blake3", "log_n": 8, "domain": 19},
        # a small batch with the records on the device already
        {"name": "keccak_2p10_device", "form": "device", "hash": "keccak", "log_n": 10, "domain": 8},
        # the benchmark's BLAKE3 batch
        {"name": "blake3_2p12", "form": "prove", "hash": "blake3", "log_n": 12, "domain": 18},
        # a middle of the served sizes
        {"name": "sha256_2p13", "form": "prove", "hash": "sha256", "log_n": 13, "domain": 18},
        # the benchmark's SHA-256 batch
        {"name": "sha256_2p16", "form": "prove", "hash": "sha256", "log_n": 16, "domain": 18},
        # the largest BLAKE3 batch that is served, records on the device
        {"name": "blake3_2p18_device", "form": "device", "hash": "blake3", "log_n": 18, "domain": 18},
        # the benchmark's headline: the largest single proof
        {"name": "keccak_2p18", "form": "prove", "hash": "keccak", "log_n": 18, "domain": 18},
        # two types with few declared rows each (a partly used registry)
        {"name": "union2_partial", "form": "union", "types": "sha256,blake3", "nu": 10, "counts": "50,37", "domain": 19},
        # three types, ragged counts: the general layout at a size where kernels matter
        {"name": "union3_ragged", "form": "union", "types": "keccak,sha256,blake3", "nu": 13,
         "counts": "5003,3001,7777", "domain": 12},
        # independent proofs of mixed sizes and hashes on one server
        {"name": "batch_mixed", "form": "batch", "requests": "blake3:12,keccak:10,sha256:14,blake3:15,keccak:13,sha256:11",
         "domain": 10},
        # a commitment inside a reserved memory budget
        {"name": "cap_blake3_2p11", "form": "cap", "hash": "blake3", "log_n": 11, "domain": 0},
    ]


def draw(rng):
    form = rng.choice(["prove", "prove", "prove", "device", "device", "union", "union", "batch", "cap"])
    domain = rng.randint(0, 200)
    if form == "union":
        types = rng.choice(UNION_TYPES)
        nu = rng.randint(7, 14)
        counts = [0 if rng.random() < 0.1 else max(1, min(1 << nu, int(2 ** rng.uniform(2, nu + 0.3))))
                  for _ in types.split(",")]
        counts[0] = max(1, counts[0])
        return {"form": form, "types": types, "nu": nu, "counts": ",".join(map(str, counts)), "domain": domain}
    if form == "batch":
        reqs = ["%s:%d" % (rng.choice(sorted(KINDS)), rng.randint(10, 15)) for _ in range(rng.randint(2, 8))]
        return {"form": form, "requests": ",".join(reqs), "domain": domain}
    h = rng.choice(sorted(KINDS))
    top = LOG_CAP_MAX[h] if form == "cap" else LOG_MAX
    case = {"form": form, "hash": h, "log_n": rng.randint(LOG_MIN[h], top), "domain": domain}
    if form == "cap":
        case["domain"] = 0
        case["stream"] = rng.randint(0, 1)  # the default stream, or one of the caller's own
    return case


def _records(rng, hash_name, n):
    """n packed records of uniform words (what a hash's state and message words are)."""
    kind = KINDS[hash_name]
    out = np.zeros(n, dtype=flock_gb300.SETUPS[kind].DTYPE)
    if hash_name == "keccak":
        out["lanes"] = rng.integers(0, 1 << 64, size=(n, 25), dtype=np.uint64)
        return out
    words = rng.integers(0, 1 << 32, size=(n, 24), dtype=np.uint32)
    if hash_name == "sha256":
        out["h"], out["w"] = words[:, :8], words[:, 8:]
    else:
        out["cv"], out["m"] = words[:, :8], words[:, 8:]
        out["counter"] = np.arange(n, dtype=np.uint64)
        out["block_len"] = 64
    return out


def _on_device(recs):
    return torch.from_numpy(recs.view(np.uint8).reshape(-1)).to("cuda:0")


def _requests(case):
    return [(h, int(log_n)) for h, log_n in (r.split(":") for r in case["requests"].split(","))]


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    form = case["form"]
    st = {"form": form, "domain": rng.integers(0, 256, size=case["domain"], dtype=np.uint8).tobytes()}
    if form == "union":
        types = case["types"].split(",")
        st["setup"] = flock_gb300.UnionSetup([KINDS[t] for t in types], case["nu"])
        st["counts"] = [int(c) for c in case["counts"].split(",")]  # the types are in slot order
        st["records"] = [_records(rng, t, c) for t, c in zip(types, st["counts"])]
    elif form == "batch":
        st["server"] = flock_gb300.ProofServer()
        st["requests"] = [(KINDS[h], _records(rng, h, 1 << log_n), st["domain"] + b"%d" % i)
                          for i, (h, log_n) in enumerate(_requests(case))]
    else:
        kind, n = KINDS[case["hash"]], 1 << case["log_n"]
        recs = _records(rng, case["hash"], n)
        st.update(kind=kind, n=n)
        if form == "cap":
            st["records"] = _on_device(recs)
            st["lib"] = flock_gb300.load()
            st["out"] = np.zeros(1 << 16, dtype=np.uint8)
            st["stream"] = torch.cuda.Stream() if case.get("stream") else None
        else:
            st["setup"] = flock_gb300.SETUPS[kind](n)
            st["records"] = recs if form == "prove" else _on_device(recs)
        torch.cuda.synchronize()
    return st


def _array(blob):
    return np.frombuffer(blob, dtype=np.uint8)


def run(state):
    form, domain = state["form"], state["domain"]
    if form == "prove":
        return _array(state["setup"].prove_fast_bytes(state["records"], domain))
    if form == "device":
        return _array(state["setup"].prove_fast_device_bytes(state["records"].data_ptr(), state["n"], domain))
    if form == "union":
        return _array(state["setup"].prove_bytes(state["counts"], state["records"], domain))
    if form == "batch":
        return [_array(o.bundle_bytes) for o in state["server"].prove_batch(state["requests"], raw=True)]
    length = ctypes.c_size_t()
    stream = state["stream"].cuda_stream if state["stream"] is not None else None
    rc = state["lib"].flock_gb300_commit_cap_noalloc(
        state["kind"], ctypes.c_void_p(state["records"].data_ptr()), state["n"],
        state["out"].ctypes.data_as(ctypes.c_char_p), state["out"].nbytes, ctypes.byref(length), ctypes.c_void_p(stream))
    if rc:
        raise flock_gb300.FlockError(rc, state["lib"].flock_gb300_last_error().decode())
    return state["out"][:32 * length.value].copy()


def _work_of(words, record_bytes, whole):
    """Records in, result out, and the GF(2^128) products (one operation each) of encoding
    `words` committed words at rate 1/2 and, for a whole proof, of the two sumchecks over
    them (three products of variables a word)."""
    layers = max(1, int(words).bit_length() - 6)
    products = words * layers + (3 * words if whole else 0)
    return {"bytes": record_bytes + (400e3 if whole else 8e3), "flops": products}


def work(case):
    form = case["form"]
    if form == "union":
        types, counts = case["types"].split(","), [int(c) for c in case["counts"].split(",")]
        parts = list(zip(types, counts))
        return _work_of(sum(USED_COLS[t] * c for t, c in parts), sum(_record_bytes(t) * c for t, c in parts), True)
    if form == "batch":
        each = [_work_of(USED_COLS[h] << n, _record_bytes(h) << n, True) for h, n in _requests(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    h, n = case["hash"], 1 << case["log_n"]
    return _work_of(USED_COLS[h] * n, _record_bytes(h) * n, form != "cap")


def _record_bytes(hash_name):
    return flock_gb300.SETUPS[KINDS[hash_name]].DTYPE.itemsize
