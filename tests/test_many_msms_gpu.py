"""Batches of many small MSMs: windows of few nodes, whose reduction ends in
single-warp blocks of quads or in k_reduce_level itself, against the oracle
(BN254 G2: against the same MSMs one by one)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import pyref as R
from tests.gpu_helpers import check, jac_to_affine_bytes, oracle_msm
from zkmetal_b200 import BLS12377MSM, BLS12381MSM, BN254G2MSM, MetalMSM
from zkmetal_b200 import lib as zl

pytestmark = pytest.mark.gpu
ENGINES = {"bn254": MetalMSM, "bls12_381": BLS12381MSM, "bls12_377": BLS12377MSM, "bn254_g2": BN254G2MSM}


def batch(e, pts, sc, counts, window):
    fb = zl.FP_BYTES[e.curve]
    out = ctypes.create_string_buffer(len(counts) * 3 * fb)
    arr = np.asarray(counts, dtype=np.uint32)
    check(zl.lib().zkmsm_engine_set_tuning(e.handle, window, 0, -1))
    check(zl.lib().zkmsm_msm_batch(e.handle, e.curve, pts.ctypes.data, sc.ctypes.data, zl.SCALAR_MONT,
                                   arr.ctypes.data, len(counts), out))
    return [out.raw[3 * fb * m:3 * fb * (m + 1)] for m in range(len(counts))]


@pytest.mark.parametrize("curve", list(ENGINES))
@pytest.mark.parametrize("counts,window", [
    ([5, 0, 9] * 20, 0),                     # 8 nodes a window, one warp each
    ([7] * 300, 0),                          # a level leaves one node a window
    ([20] * 30 + [0, 2000], 6),              # 32 nodes: blocks of 32 quads
    ([30] * 40, 13),                         # 4096 nodes: a level, then several blocks
    ([30] * 40, 5 | 7 << 16),                # 16 and 32 nodes in one launch
])
def test_many_small_msms(oracles, curve, counts, window):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    e = ENGINES[curve]()
    fb, n = zl.FP_BYTES[e.curve], sum(counts)
    pts = torch.empty(n * 2 * fb, dtype=torch.uint8, device="cuda")
    sc = torch.empty(n * 32, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    check(zl.lib().zkmsm_gen_bases(e.handle, e.curve, 31, 0, n, pts.data_ptr()))
    check(zl.lib().zkmsm_gen_scalars(e.handle, e.curve, 31, 0, n, 0, zl.SCALAR_MONT, sc.data_ptr()))
    pts, sc = pts.cpu().numpy(), sc.cpu().numpy()
    got = batch(e, pts, sc, counts, window)
    ref, cm = oracles
    off = 0
    for m, k in enumerate(counts):
        p, s = pts[off * 2 * fb:(off + k) * 2 * fb], sc[off * 32:(off + k) * 32]
        off += k
        if k == 0:
            assert got[m] == bytes(3 * fb)
        elif curve == "bn254_g2":
            assert got[m] == batch(e, p, s, [k], 0)[0], m
        else:
            want = oracle_msm(ref if ref is not None else cm, curve, p.tobytes(), s.tobytes(), k, zl.SCALAR_MONT)
            assert jac_to_affine_bytes(R.CURVES[curve], got[m]) == want, m
    e.close()


def test_workspace_of_many_msms():
    """16384 MSMs of one point: 524288 windows of eight buckets.  Apart from
    the buckets (604 MB, an eighth of slack on every buffer) the largest parts
    are two terms per window (134 MB) and the entries and partial sums."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rt, pool, used = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(), ctypes.c_uint64()
    torch.cuda.synchronize()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

    def in_use():
        torch.cuda.synchronize()
        assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0  # UsedMemCurrent
        return used.value

    e, k = MetalMSM(), 16384
    pts = torch.empty(k * 64, dtype=torch.uint8, device="cuda")
    sc = torch.empty(k * 32, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    check(zl.lib().zkmsm_gen_bases(e.handle, e.curve, 32, 0, k, pts.data_ptr()))
    check(zl.lib().zkmsm_gen_scalars(e.handle, e.curve, 32, 0, k, 0, zl.SCALAR_MONT, sc.data_ptr()))
    pts, sc = pts.cpu().numpy(), sc.cpu().numpy()
    before = in_use()
    got = batch(e, pts, sc, [1] * k, 0)
    taken = in_use() - before
    assert taken < 1000 << 20, taken >> 20
    for m in (0, 1, 777, k - 1):
        assert got[m] == batch(e, pts[64 * m:64 * m + 64], sc[32 * m:32 * m + 32], [1], 0)[0]
    e.close()
