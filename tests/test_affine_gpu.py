"""Affine bucket accumulation (csrc/affine.cuh) on the curves and sizes that
take it, against the oracle and against the same MSM by k_acc_l1 (a forced
chunk length).  The special pairs are frequent here: few distinct bases, their
negatives and identities, with few distinct scalars, so that most buckets add
equal, opposite and identity points."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import pyref as R
from tests.gpu_helpers import check, gen_inputs, jac_to_affine_bytes, oracle_msm, to_host
from zkmetal_b200 import BLS12377MSM, BLS12381MSM, BN254G2MSM
from zkmetal_b200 import lib as zl

pytestmark = pytest.mark.gpu
ENGINES = {"bls12_381": BLS12381MSM, "bls12_377": BLS12377MSM, "bn254_g2": BN254G2MSM}


@pytest.fixture(scope="module")
def engines():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    e = {k: c() for k, c in ENGINES.items()}
    yield e
    for x in e.values():
        x.close()


def run(e, pts, sc, n, fmt, chunk):
    fb = zl.FP_BYTES[e.curve]
    out = ctypes.create_string_buffer(3 * fb)
    check(zl.lib().zkmsm_engine_set_tuning(e.handle, 0, chunk, -1))
    try:
        torch.cuda.synchronize()
        check(zl.lib().zkmsm_msm_device(e.handle, e.curve, pts.data_ptr(), sc.data_ptr(), fmt, n, out, None))
    finally:
        check(zl.lib().zkmsm_engine_set_tuning(e.handle, 0, 0, -1))
    return out.raw


def levels(curve_id, n):
    buf = ctypes.create_string_buffer(1 << 22)
    arr = (ctypes.c_uint32 * 1)(n)
    check(zl.lib().zkmsm_plan_describe(curve_id, arr, 1, 1, 0, 0, -1, 0, buf, len(buf)))
    import json
    return json.loads(buf.value.decode())["affine"][0]


def repeated(e, n, seed):
    """n bases drawn from 24 points, their negatives and the identity; n
    scalars from 6 values (0, 1, r - 1 and random)."""
    cid, fb = e.curve, zl.FP_BYTES[e.curve]
    pts = torch.empty(24 * 2 * fb, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    check(zl.lib().zkmsm_gen_bases(e.handle, cid, seed, 0, 24, pts.data_ptr()))
    host = pts.cpu().numpy().reshape(24, 2, fb)
    w = 32 if cid == zl.BN254_G2 else fb  # base-field elements of a coordinate
    p = zl.FP_MODULUS[zl.BN254 if cid == zl.BN254_G2 else cid]
    neg = host.copy()
    for row in neg:
        for o in range(0, fb, w):
            y = int.from_bytes(row[1, o:o + w].tobytes(), "little")
            row[1, o:o + w] = np.frombuffer(((p - y) % p).to_bytes(w, "little"), dtype=np.uint8)
    pool = np.concatenate([host, neg, np.zeros((2, 2, fb), np.uint8)])
    rng = np.random.default_rng(seed)
    r = R.CURVES["bn254" if cid == zl.BN254_G2 else {zl.BLS12_381: "bls12_381", zl.BLS12_377: "bls12_377"}[cid]].r
    vals = [0, 1, r - 1] + [int.from_bytes(rng.bytes(40), "little") % r for _ in range(3)]
    sv = np.frombuffer(b"".join(v.to_bytes(32, "little") for v in vals), dtype=np.uint8).reshape(6, 32)
    pts = torch.from_numpy(pool[rng.integers(0, len(pool), n)].reshape(-1)).cuda()
    return pts, torch.from_numpy(sv[rng.integers(0, 6, n)].reshape(-1)).cuda()


@pytest.mark.parametrize("curve", list(ENGINES))
@pytest.mark.parametrize("n,kind", [(1 << 18, "uniform"), ((1 << 18) + 77, "repeated"), (700001, "witness")])
def test_affine_levels(engines, oracles, curve, n, kind):
    e = engines[curve]
    assert levels(e.curve, n) > 0
    if kind == "repeated":
        fmt = zl.SCALAR_INT
        pts, sc = repeated(e, n, 90 + e.curve)
    else:
        fmt = zl.SCALAR_MONT
        L, fb = zl.lib(), zl.FP_BYTES[e.curve]
        pts = torch.empty(n * 2 * fb, dtype=torch.uint8, device="cuda")
        sc = torch.empty(n * 32, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        check(L.zkmsm_gen_bases(e.handle, e.curve, 91, 0, n, pts.data_ptr()))
        check(L.zkmsm_gen_scalars(e.handle, e.curve, 91, 0, n, kind == "witness", fmt, sc.data_ptr()))
    got = run(e, pts, sc, n, fmt, 0)
    assert got == run(e, pts, sc, n, fmt, 64)
    if curve != "bn254_g2":
        ref, cm = oracles
        C = R.CURVES[curve]
        want = oracle_msm(ref if ref is not None else cm, curve, to_host(pts), to_host(sc), n, fmt)
        assert jac_to_affine_bytes(C, got) == want


def test_affine_slabs_past_the_expected_entries(engines):
    """A sampled plan expects a third of the entries there are: two in three
    of the scalars the sample reads (every 512th of 2^21) are zero, no other.
    The chunks past its slabs take k_acc_l1."""
    e, L = engines["bls12_381"], zl.lib()
    n = 1 << 21
    pts, sc = gen_inputs(e, "bls12_381", 92, n, "uniform", zl.SCALAR_MONT)
    v = sc.view(n // 512, 512, 32)
    zero = torch.arange(n // 512, device="cuda") % 3 != 0
    v[zero, 0] = 0
    few = sc.clone()  # the same sample, and as few entries as it promises
    few.view(n // 512, 512, 32)[zero] = 0

    def counted(scalars, chunk):
        k = L.zkmsm_engine_launch_count(e.handle)
        out = run(e, pts, scalars, n, zl.SCALAR_MONT, chunk)
        return out, L.zkmsm_engine_launch_count(e.handle) - k, L.zkmsm_engine_last_entries(e.handle)

    got, launches, entries = counted(sc, 0)
    _, same, expected = counted(few, 0)
    # one plan for both, in affine levels (two and more launch six kernels);
    # its slabs hold the expected entries and at most a tenth more
    assert launches == same and launches >= counted(sc, 64)[1] + 6
    assert expected >= 1 << 22 and entries > 2 * expected
    check(L.zkmsm_engine_set_sampling(e.handle, 0))
    try:
        assert got == run(e, pts, sc, n, zl.SCALAR_MONT, 64)
    finally:
        check(L.zkmsm_engine_set_sampling(e.handle, 1))


@pytest.mark.parametrize("pct", [50, 200])
def test_affine_tuned_chunks(engines, tmp_path, pct):
    """Chunk lengths from a saved schedule: more slabs, or longer chunks."""
    n = (1 << 19) + 5
    path = tmp_path / "tuning"
    path.write_text("zkmsm-tuning 2\n" + "s %d 19 %d 0 0\n" % (zl.BLS12_381 * 2 + 1, pct))
    pts, sc = gen_inputs(engines["bls12_381"], "bls12_381", 93, n, "uniform", zl.SCALAR_MONT)
    e = BLS12381MSM()
    check(zl.lib().zkmsm_tuning_load(e.handle, str(path).encode()))
    got = run(e, pts, sc, n, zl.SCALAR_MONT, 0)
    e.close()
    assert got == run(engines["bls12_381"], pts, sc, n, zl.SCALAR_MONT, 64)
