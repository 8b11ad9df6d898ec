"""CPU replay of the quads' bucket reduction on real host plans.

The index logic of k_reduce_level (the plan's first levels), k_reduce_quads,
k_reduce_windows and k_combine's shifted sum is replayed with integers in
place of points, for window sizes at the edges of blocks and of the rules that
choose them, and compared with sum_w 2^bit(w) * sum_i (i + 1) * A_i.
"""
import random

import pytest

from tests.test_schedule_model import plan, plan_shift, win_bit, win_bucket, win_width
from zkmetal_b200 import lib as zl

QUADS, SLOTS1, SLOTS2 = 64, 8, 12


def tree(S, w, quads):
    """reduce_step over `quads` quads until one step covers `used` of them."""
    st = 1
    while st < quads:
        S0, w0 = list(S), list(w)
        for i in range(len(S)):
            low = i & (st - 1)
            j = i ^ st
            if i & st:
                if low == st - 1:
                    w[i] = w0[i] + w0[j]
            elif low & (low - 1) == 0 and j < len(S):
                S[i] = S0[i] + S0[j]
        st <<= 1
    return st


def reduce_model(pl, buckets):
    L, lg, Q = pl["red_L"], pl["red_log2L"], pl["quad"]
    inS, inW = buckets, None
    for lvl, tasks in enumerate(pl["red"][:Q["levels"]]):
        nout = sum(t[3] for t in tasks)
        oS, oW = [0] * nout, [0] * nout
        for in_off, n_in, out_off, n_out in tasks:
            for g in range(n_out):
                ch = range(in_off + g * L, in_off + min(n_in, (g + 1) * L))
                oS[out_off + g] = sum(inS[c] for c in ch)
                oW[out_off + g] = (sum((c - ch[0]) * inS[c] for c in ch) << (lvl * lg)) + \
                    (sum(inW[c] for c in ch) if inW else 0)
        inS, inW = oS, oW
    J, E, span = 1 << Q["log2J"], 1 << Q["log2E"], Q["levels"] * lg
    assert not (Q["direct"] and (Q["windows"] or any(t[1] != 1 for t in Q["tasks"])))
    out = [[0] * SLOTS1 for _ in range(Q["blocks"])]
    for in_off, n_in, out_off, n_out in Q["tasks"]:
        # what the block's quads (a power of two, a warp at least) reach
        assert min(QUADS * J, n_in) <= Q["quads"] * J and Q["quads"] in (8, 16, 32, 64)
        assert not Q["windows"] or Q["quads"] == QUADS
        assert n_out == -(-n_in // (QUADS * J))
        for b in range(n_out):
            n0 = b * QUADS * J
            cnt = min(QUADS * J, n_in - n0)
            S, w = [0] * QUADS, [0] * QUADS
            for i in range(QUADS):
                mine = range(i * J, min(cnt, (i + 1) * J))
                S[i] = sum(inS[in_off + n0 + k] for k in mine)
                w[i] = sum((k - i * J) * inS[in_off + n0 + k] for k in mine)
                if inW:
                    w[i] = (w[i] << span) + sum(inW[in_off + n0 + k] for k in mine)
            st = tree(S, w, -(-cnt // J))
            out[out_off + b] = [S[0]] + [S[1 << j] if 1 << j < st else 0 for j in range(6)] + [w[st - 1]]
    terms, bits = out, [0] + [span + Q["log2J"] + j for j in range(6)] + [0]
    if Q["windows"]:
        terms = []
        for _, _, out_off, n_out in Q["tasks"]:
            assert n_out <= 8 * E
            rows = [[out[out_off + i * E + s] if i * E + s < n_out else [0] * SLOTS1 for s in range(E)]
                    for i in range(8)]
            S = [sum(r[0] for r in row) for row in rows]
            x = [sum(s * r[0] for s, r in enumerate(row)) for row in rows]
            tree(S, x, 8)
            plain = [sum(r[a] for row in rows for r in row) for a in range(SLOTS1)]
            terms.append([S[0]] + plain[1:] + [x[7], S[1], S[2], S[4]])
        bx = bits[1] + 6
        bits = bits + [bx] + [bx + Q["log2E"] + j for j in range(3)]
    return [sum(t << b for t, b in zip(row, bits)) for row in terms]


def check(pl, seed):
    rng = random.Random(seed)
    A = [rng.getrandbits(40) for _ in range(pl["nbuckets"])]
    got = reduce_model(pl, A)
    k = 0
    for d in pl["descs"]:
        c, nwin, boff, nred, nlo = d[3], d[4], d[6], d[10], d[11]
        for w in range(nred):
            o = boff + win_bucket(c, nlo, w)
            B = 1 << (win_width(c, nlo, w) - 1)
            assert got[k] == sum((i + 1) * A[o + i] for i in range(B)), (c, w)
            k += 1
    assert k == len(pl["quad"]["tasks"]) == len(got)


@pytest.mark.parametrize("window", [2, 3, 4, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 5 | 3 << 16, 9 | 1 << 16, 12 | 4 << 16])
def test_quad_reduction(window):
    check(plan(zl.BN254, [5000], window=window), window)


def test_quad_reduction_batches():
    check(plan(zl.BLS12_381, [700, 0, 1 << 16, 3]), 1)
    check(plan_shift(zl.BN254, [1, 400, 1 << 17, 9000], 4, 1 << 17), 2)
    check(plan_shift(zl.BN254, [1 << 18], 4, 1 << 18), 3)


@pytest.mark.parametrize("counts", [[64] * 256, [16] * 400, [40] * 1024, [1000] * 300, [3000] * 200 + [0, 1 << 17]])
def test_quad_reduction_many_windows(counts):
    """Batches of many small MSMs: what the quads' warps add up follows the
    nodes there are, not 64 quads for each of thousands of windows."""
    pl = plan(zl.BN254, counts)
    Q = pl["quad"]
    nodes = [t[1] for t in Q["tasks"]]
    if max(nodes) == 1 and Q["levels"]:
        assert Q["direct"]
    else:
        # a block is no wider than the largest window needs
        assert Q["quads"] == 8 or Q["quads"] << Q["log2J"] < 2 * max(nodes)
        warps = sum(-(-min(n, 64 << Q["log2J"]) // (8 << Q["log2J"])) for n in nodes)
        assert 8 * warps <= 2 * (sum(nodes) >> Q["log2J"]) + 8 * len(nodes)
    check(pl, len(counts))


@pytest.mark.parametrize("counts", [[0], [0] * 3, [0, 1], [1]])
def test_plan_of_few_entries(counts):
    """A batch of empty MSMs has no entries: its one segmented-sum level is
    the shortest there is."""
    pl = plan(zl.BN254, counts)
    K, T, M = pl["acc"][0]
    assert M == pl["entry_bound"] and K == QUADS * 4 and T == 1 and len(pl["acc"]) == 1
