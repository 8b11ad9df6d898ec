"""Workloads of the MSM library over its real range, through its public entry
points: plain calls from host and from device buffers, partitioned calls, and
batched commitments over a resident table, on every curve, with integer and
Montgomery scalars, uniform and witness-like.

Paths (``case["path"]``):
  host    ``<Curve>MSM.msm`` / ``msmFr`` on host arrays (pinned or pageable)
  device  ``zkmsm_msm_device`` on buffers that already lie on the GPU
  parts   ``innerProductMSM`` over a partition of host arrays
  commit  ``CommitmentTable.batch_commit``: MSMs over prefixes of a resident
          table with its window shifts, scalars from pinned host memory
Outputs are the result points as bytes (affine coordinates in Montgomery form
with Z = 1), which every correct implementation gives alike.
"""
import ctypes
import math
import random

import numpy as np
import torch

from zkmetal_b200 import lib as zl
from zkmetal_b200 import msm as zm

CURVES = {"bn254": zl.BN254, "bls12_381": zl.BLS12_381, "bls12_377": zl.BLS12_377, "bn254_g2": zl.BN254_G2}
ENGINES = {"bn254": zm.MetalMSM, "bls12_381": zm.BLS12381MSM, "bls12_377": zm.BLS12377MSM, "bn254_g2": zm.BN254G2MSM}
# largest n of a drawn plain call: on every curve it costs less than 2^24
# points of BN254, the largest listed call
MAX_LOG2 = {"bn254": 23.9, "bls12_381": 22.0, "bls12_377": 22.0, "bn254_g2": 20.0}
_engines = {}


def engine(curve):
    """A program keeps one engine per curve for all its calls."""
    if curve not in _engines:
        _engines[curve] = ENGINES[curve]()
    return _engines[curve]


def listed():
    def plain(name, path, curve, n, fmt, dist="uniform", pinned=False):
        return {"name": name, "path": path, "curve": curve, "n": n, "fmt": fmt, "dist": dist, "pinned": pinned}

    return [
        # a verifier's handful of points, straight from arrays: latency alone
        plain("host_256", "host", "bn254", 256, "int"),
        # a small circuit's commitment from device buffers, odd length
        plain("device_1000", "device", "bn254", 1000, "mont"),
        # a round of an inner-product argument: eight uneven partitions
        {"name": "parts_8_of_2p14", "path": "parts", "curve": "bn254", "n": 1 << 14, "parts": 8, "sizes": 7,
         "fmt": "mont", "dist": "uniform", "pinned": False},
        # a mid-size prover, integer scalars
        plain("device_2p16_int", "device", "bn254", 1 << 16, "int"),
        # an odd-length prover call on the curve used under recursion
        plain("bls377_100003_int", "device", "bls12_377", 100003, "int"),
        # the second-group MSM of a pairing-based prover
        plain("g2_2p16", "device", "bn254_g2", 1 << 16, "mont"),
        # the size a prover's polynomial commitments are usually quoted at
        plain("device_2p20", "device", "bn254", 1 << 20, "mont"),
        # blob / polynomial commitments on BLS12-381
        plain("bls381_2p20", "device", "bls12_381", 1 << 20, "mont"),
        # a proof witness: mostly zeros, ones and short values, odd length
        plain("witness_3000001", "device", "bn254", 3000001, "mont", "witness"),
        # a drop-in call whose inputs lie in (pinned) host memory
        plain("host_2500000", "host", "bn254", 2500000, "mont", pinned=True),
        # the commitments of one proof over a resident key of 2^20 points
        {"name": "commit_24_of_2p20", "path": "commit", "curve": "bn254", "n": 1 << 20, "parts": 24, "sizes": 3,
         "fmt": "mont", "dist": "uniform", "pinned": True},
        # the largest proving systems
        plain("device_2p24", "device", "bn254", 1 << 24, "mont"),
    ]


def draw(rng):
    path = rng.choice(["device", "device", "device", "device", "host", "host", "parts", "commit"])
    curve = rng.choice(["bn254", "bn254", "bn254", "bls12_381", "bls12_381", "bls12_377", "bn254_g2"])
    fmt, dist = rng.choice(["mont", "mont", "int"]), rng.choice(["uniform", "uniform", "witness"])
    top = MAX_LOG2[curve]
    if path in ("device", "host"):
        n = int(2 ** rng.uniform(8, min(top, 22) if path == "host" else top)) | rng.randint(0, 1)
        return {"path": path, "curve": curve, "n": n, "fmt": fmt, "dist": dist,
                "pinned": path == "host" and rng.random() < 0.5}
    if path == "parts":
        n = int(2 ** rng.uniform(9, min(top, 20)))
        return {"path": path, "curve": curve, "n": n, "parts": rng.randint(2, 16), "sizes": rng.randint(0, 1 << 20),
                "fmt": fmt, "dist": dist, "pinned": False}
    n = int(2 ** rng.uniform(12, 20))
    return {"path": path, "curve": rng.choice(["bn254", "bn254", "bls12_381"]), "n": n, "parts": rng.randint(1, 24),
            "sizes": rng.randint(0, 1 << 20), "fmt": "mont", "dist": dist, "pinned": True}


def counts_of(case):
    """Points of each MSM of the pass."""
    n, k = case["n"], case.get("parts", 0)
    if not k:
        return [n]
    r = random.Random(case["sizes"])
    if case["path"] == "parts":
        cuts = sorted(r.randint(0, n) for _ in range(k - 1))
        return [b - a for a, b in zip([0] + cuts, cuts + [n])]
    low = math.log2(min(n, 1024))  # commitments: prefixes, sizes spread over their logarithm
    return [min(n, int(2 ** r.uniform(low, math.log2(n)))) for _ in range(k)]


def to_host(t, pinned):
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=pinned)
    h.copy_(t)
    return h


def prepare(case, seed):
    e, cid = engine(case["curve"]), CURVES[case["curve"]]
    L, n = zl.lib(), case["n"]
    counts = counts_of(case)
    ns = sum(counts)
    fmt = zl.SCALAR_MONT if case["fmt"] == "mont" else zl.SCALAR_INT
    points = torch.empty(n * 2 * zl.FP_BYTES[cid], dtype=torch.uint8, device="cuda")
    scalars = torch.empty(max(ns, 1) * 32, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert L.zkmsm_gen_bases(e.handle, cid, seed, 0, n, points.data_ptr()) == zl.SUCCESS, zl.last_error()
    assert L.zkmsm_gen_scalars(e.handle, cid, seed, 0, ns, 0 if case["dist"] == "uniform" else 1, fmt,
                               scalars.data_ptr()) == zl.SUCCESS, zl.last_error()
    st = {"path": case["path"], "engine": e, "curve": cid, "n": n, "counts": counts, "fmt": fmt}
    if case["path"] == "device":
        st.update(points=points, scalars=scalars, out=ctypes.create_string_buffer(3 * zl.FP_BYTES[cid]))
        return st
    st["hold"] = [to_host(scalars, case["pinned"])]
    st["scalars"] = st["hold"][0].numpy()
    if case["path"] == "commit":
        st["table"] = zm.CommitmentTable(e, points.data_ptr(), on_device=True, n=n)
        st["table"].precompute(4)
        return st
    st["hold"].append(to_host(points, case["pinned"]))
    st["points"] = st["hold"][1].numpy()
    st["bounds"] = [0]
    for c in counts:
        st["bounds"].append(st["bounds"][-1] + c)
    return st


def as_array(p):
    return np.frombuffer(p.x + p.y + p.z, dtype=np.uint8)


def run(st):
    e = st["engine"]
    if st["path"] == "device":
        if zl.lib().zkmsm_msm_device(e.handle, st["curve"], st["points"].data_ptr(), st["scalars"].data_ptr(),
                                     st["fmt"], st["n"], st["out"], None) != zl.SUCCESS:
            raise RuntimeError(zl.last_error())
        return np.frombuffer(st["out"].raw, dtype=np.uint8)
    if st["path"] == "host":
        call = e.msmFr if st["fmt"] == zl.SCALAR_MONT else e.msm
        return as_array(call(st["points"], st["scalars"]))
    if st["path"] == "parts":
        got = zm.innerProductMSM(e, st["points"], st["scalars"], st["bounds"], fr=st["fmt"] == zl.SCALAR_MONT)
    else:
        got = st["table"].batch_commit(st["scalars"], st["counts"], fmt=st["fmt"])
    return np.stack([as_array(p) for p in got])


def work(case):
    """Bytes: bases and scalars once.  Operations: each scalar's 256 digit
    bits in windows of about log2(n) bits, one affine addition (6 field
    products with a shared inversion) per window, a field product being
    2 N^2 + N multiply-adds of 32-bit words."""
    cid = CURVES[case["curve"]]
    fb = zl.FP_BYTES[cid]
    words, base = (8, 3) if case["curve"] == "bn254_g2" else (fb // 4, 1)
    adds = 0
    for c in counts_of(case):
        if c:
            adds += c * math.ceil(256 / max(4.0, math.log2(c) - 2))
    ns = sum(counts_of(case))
    return {"bytes": case["n"] * 2 * fb + ns * 32, "flops": 2.0 * adds * 6 * base * (2 * words * words + words)}


def tolerance(case):
    return "exact"


# ---- plain Python integers, for the small calls --------------------------

P = {"bn254": zl.FP_MODULUS[zl.BN254], "bls12_381": zl.FP_MODULUS[zl.BLS12_381],
     "bls12_377": zl.FP_MODULUS[zl.BLS12_377]}
R = {"bn254": 0x30644e72e131a029b85045b68181585d2833e84879b9709143e1f593f0000001,
     "bls12_381": 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001,
     "bls12_377": 0x12ab655e9a2ca55660b44d1e5c37b00159aa76fed00000010a11800000000001}


def add(a, b, p):
    """Affine addition on y^2 = x^3 + b; None is the identity."""
    if a is None or b is None:
        return b if a is None else a
    if a[0] == b[0]:
        if (a[1] + b[1]) % p == 0:
            return None
        lam = 3 * a[0] * a[0] * pow(2 * a[1], -1, p) % p
    else:
        lam = (b[1] - a[1]) * pow(b[0] - a[0], -1, p) % p
    x = (lam * lam - a[0] - b[0]) % p
    return x, (lam * (a[0] - x) - a[1]) % p


def exact(case, seed):
    """The sum by plain double-and-add over the bits of all scalars at once."""
    if case["n"] > 1024 or case["path"] not in ("host", "device") or case["curve"] not in P:
        return None
    st = prepare(case, seed)
    p, r, fb = P[case["curve"]], R[case["curve"]], zl.FP_BYTES[st["curve"]]
    raw = [st[k].cpu().numpy() if isinstance(st[k], torch.Tensor) else st[k] for k in ("points", "scalars")]
    words = [[int.from_bytes(a[i:i + w].tobytes(), "little") for i in range(0, a.size, w)]
             for a, w in ((raw[0], fb), (raw[1], 32))]
    down = pow(1 << (8 * fb), -1, p)
    pts = [(x * down % p, y * down % p) for x, y in zip(words[0][::2], words[0][1::2])]
    sc = [s * pow(1 << 256, -1, r) % r if case["fmt"] == "mont" else s % r for s in words[1]]
    acc = None
    for bit in range(256, -1, -1):
        acc = add(acc, acc, p)
        for s, q in zip(sc, pts):
            if s >> bit & 1:
                acc = add(acc, q, p)
    up = (1 << (8 * fb)) % p
    vals = [up, up, 0] if acc is None else [acc[0] * up % p, acc[1] * up % p, up]
    return np.frombuffer(b"".join(v.to_bytes(fb, "little") for v in vals), dtype=np.uint8)
