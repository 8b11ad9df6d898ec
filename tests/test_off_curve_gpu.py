"""Points that lie on y^2 = x^3 + b' rather than on the curve itself: XYZZ
doublings and additions never see b, so without the endomorphism (short
scalars, or GLV switched off) the sum is the one on that other curve.  And a
point of order two, which the projective doubling chain has to carry."""
import ctypes
import random

import numpy as np
import pytest
import torch

from oracle import pyref as R
from tests.gpu_helpers import check, np_bytes
from zkmetal_b200 import BLS12377MSM, BLS12381MSM, MetalMSM
from zkmetal_b200 import lib as zl
from zkmetal_b200.msm import _batch

pytestmark = pytest.mark.gpu
ENGINES = {"bn254": MetalMSM, "bls12_381": BLS12381MSM, "bls12_377": BLS12377MSM}


@pytest.fixture(scope="module")
def engines():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    e = {k: c() for k, c in ENGINES.items()}
    for x in e.values():
        x.useGLV = False
    yield e
    for x in e.values():
        x.close()


def off_curve(C, rng, n):
    """n multiples of one point of y^2 = x^3 + b', b' != b."""
    P = (rng.randrange(1, C.p), rng.randrange(1, C.p))
    assert not C.on_curve(P)
    return [R.scalar_mul(C, P, rng.randrange(1, 1 << 40)) for _ in range(n)]


def affine(C, p):
    return C.dec_jacobian(p.x + p.y + p.z)


@pytest.mark.parametrize("curve", list(ENGINES))
@pytest.mark.parametrize("n", [1, 2, 33, 1500])
def test_off_curve_points(engines, curve, n):
    C, rng = R.CURVES[curve], random.Random(n)
    pts = off_curve(C, rng, min(n, 16))
    pts = [pts[i % len(pts)] for i in range(n)]
    sc = [rng.randrange(C.r) for _ in range(n)]
    got = engines[curve].msm(np_bytes(R.pack_points(C, pts)), np_bytes(R.pack_scalars_int(sc)))
    sums = {}
    for P, k in zip(pts, sc):
        sums[P] = sums.get(P, 0) + k
    assert affine(C, got) == R.naive_msm(C, list(sums), list(sums.values()))


@pytest.mark.parametrize("curve", list(ENGINES))
def test_off_curve_beside_on_curve(engines, curve):
    """MSMs of one batch, some of whose points are on the curve and some not."""
    C, rng = R.CURVES[curve], random.Random(5)
    on = [R.scalar_mul(C, (C.gx, C.gy), rng.randrange(1, C.r)) for _ in range(6)]
    sets = [on[:3], off_curve(C, rng, 4), on[3:], off_curve(C, rng, 2)]
    sc = [[rng.randrange(C.r) for _ in s] for s in sets]
    got = _batch(engines[curve], np_bytes(R.pack_points(C, sum(sets, []))), np_bytes(R.pack_scalars_int(sum(sc, []))),
                 [len(s) for s in sets], zl.SCALAR_INT)
    assert [affine(C, g) for g in got] == [R.naive_msm(C, p, k) for p, k in zip(sets, sc)]


@pytest.mark.parametrize("width", [1, 2, 4])
def test_off_curve_short_scalars(engines, width):
    """The short-scalar entry points never split a scalar."""
    C, rng = R.CURVES["bn254"], random.Random(width)
    pts = off_curve(C, rng, 5)
    sc = [rng.getrandbits(8 * width) for _ in pts]
    fn = {1: "u8", 2: "u16", 4: "u32"}[width]
    out = [ctypes.create_string_buffer(32) for _ in range(3)]
    e = MetalMSM()
    check(getattr(zl.lib(), "zkmetal_bn254_msm_" + fn)(
        e.handle, R.pack_points(C, pts), b"".join(k.to_bytes(width, "little") for k in sc), len(pts), *out))
    e.close()
    assert C.dec_jacobian(b"".join(o.raw for o in out)) == R.naive_msm(C, pts, sc)


@pytest.mark.parametrize("k", [1, 2, 3 << 90, (1 << 200) + 1])
def test_order_two_point(engines, k):
    """(-1, 0) on BLS12-377."""
    C = R.CURVES["bls12_377"]
    T = (C.p - 1, 0)
    assert C.on_curve(T)
    got = engines["bls12_377"].msm(np_bytes(R.pack_points(C, [T])), np_bytes(R.pack_scalars_int([k])))
    assert affine(C, got) == (T if k & 1 else None)
