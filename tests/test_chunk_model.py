"""The chunk lengths the level-1 kernels take on the device (acc_chunk in
msm_kernels.cuh, aff_len in affine.cuh), over real plans and every share of
their entries: all entries are covered by chunks the buffers have slots for,
none longer than the plan's (an eighth longer, in k_acc_l1), and however few
the entries are, they fill whole waves of resident threads."""
import pytest

from tests.test_affine_model import describe_sampled
from tests.test_schedule_model import plan, plan_shift
from zkmetal_b200 import lib as zl

WAVE = 148 * 512  # the planner's, where no device is known


def ceil(a, b):
    return -(-a // b)


def acc_chunk(M, K, T, wave):
    if not wave or not M:
        return K
    per = K * wave
    parts = min(max((M + per - per // 8 - 1) // per, 1) * wave, T)
    return max(8, ceil(M, parts))


def aff_len(M, K, T, threads, slabs):
    per = K * threads
    if M == 0 or M > per * slabs:
        return K
    parts = min(ceil(M, per) * threads, T)
    return min(K, max(16, ceil(M, 4 * parts) * 4))


def shares(M):
    ms = {M, M - 1, 1, 2, 8, 9, 1000, WAVE, 8 * WAVE, 8 * WAVE + 1}
    ms |= {M * k // 97 for k in range(1, 97)} | {M * k // 1000 for k in (900, 950, 981, 990, 995, 999)}
    return sorted(m for m in ms if 0 < m <= M)


PLANS = [plan(c, n) for c in (zl.BN254, zl.BLS12_381, zl.BN254_G2)
         for n in ([5000], [1 << 14], [100003], [1 << 18], [600001], [1 << 20], [1 << 22], [64] * 1024, [1024] * 1024)]
PLANS += [plan_shift(zl.BN254, [8192] * 256, 4, 8192), plan_shift(zl.BLS12_381, [4096] * 256, 4, 4096),
          plan_shift(zl.BLS12_381, [1 << 18] * 4, 4, 1 << 18)]


@pytest.mark.parametrize("pl", PLANS, ids=range(len(PLANS)))
def test_level1_chunks(pl):
    K, T, bound = pl["acc"][0]
    for M in shares(bound):
        k = acc_chunk(M, K, T, WAVE)
        chunks = ceil(M, k)
        assert 8 <= k <= K * 9 // 8 + 1 and chunks <= T
        if k > 8:
            # whole waves (or all T chunks), but for rounding the length up
            parts = min(ceil(chunks, WAVE) * WAVE, T)
            assert chunks > parts - ceil(parts, k), (M, k)
    assert acc_chunk(0, K, T, WAVE) == K and acc_chunk(bound, K, T, 0) == K


AFF = [p for p in PLANS if p["affine"][0]]
AFF += [describe_sampled(zl.BLS12_381, n, 15, e) for n, e in ((1 << 21, 8390000), (1 << 22, 1 << 23), (1 << 20, 5000000))]
AFF += [describe_sampled(zl.BLS12_377, 1 << 20, pct=p) for p in (50, 99, 200)]


@pytest.mark.parametrize("pl", AFF, ids=range(len(AFF)))
def test_affine_chunks(pl):
    K, T, bound = pl["acc"][0]
    _, threads, slabs = pl["affine"]
    ends = [slabs * threads * K + d for d in (-1, 0, 1)]
    for M in shares(bound) + [m for m in ends if 0 < m <= bound]:
        k = aff_len(M, K, T, threads, slabs)
        chunks = ceil(M, k)
        assert 16 <= k <= K and k % 4 == 0 and chunks <= T
        if chunks > slabs * threads:  # the rest is k_acc_l1's, in chunks of K
            assert k == K
        else:  # and what is launched for chunks past the slabs starts after the last entry
            assert slabs * threads * K >= M
    assert len(AFF) >= 8
