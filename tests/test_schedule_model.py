"""CPU model of the device schedule, driven by the library's real host plan.

The plan (window widths, bucket layout, segmented-sum chunking, reduction
tree) comes from the C++ planner through zkmsm_plan_describe.  The kernels'
index logic -- the entries in bucket order (shuffled within a bucket, as
atomics allow), k_acc_l1's chunks with their two fixed slots, k_acc_fold's
leaves, quads and merges on every level after it, the bucket reduction by
levels and quads, and the windows' shifted sum -- is replayed here with
integers mod r standing in for group elements (P_i -> p_i, phi(P) ->
lambda*p).  Every index is checked against the sizes the engine allocates from
the same plan, every bucket with entries must be written exactly once and no
other, and the result must equal sum s_i p_i mod r.  No GPU needed.
"""
import ctypes
import json
import random

import pytest

from oracle import pyref as R
from zkmetal_b200 import lib as zl


def plan(curve, counts, fmt=0, window=0, chunk=0, glv=-1, bits=0):
    L = zl.lib()
    arr = (ctypes.c_uint32 * len(counts))(*counts)
    buf = ctypes.create_string_buffer(1 << 22)
    st = L.zkmsm_plan_describe(curve, arr, len(counts), fmt, window, chunk, glv, bits, buf, len(buf))
    assert st == 0, zl.last_error()
    return json.loads(buf.value.decode())


def halves(C, s, glv):
    """Device prepare_scalar: integer mod r, then GLV split with signs."""
    s %= C.r
    if not glv:
        return [(s, 0)]
    k1, k2 = R.glv_split(C, s)
    return [(abs(k1), int(k1 < 0)), (abs(k2), int(k2 < 0))]


def win_width(c, nlo, w):
    return c + (1 if w >= nlo else 0)


def win_bit(c, nlo, w):
    return w * c + max(0, w - nlo)


def win_bucket(c, nlo, w):
    return (w + max(0, w - nlo)) << (c - 1)


def digits(k, c, nwin, nlo=None):
    """Signed digits; windows [0, nlo) are c bits, later ones c + 1 bits."""
    nlo = nwin if nlo is None else nlo
    carry = 0
    for w in range(nwin):
        cw = win_width(c, nlo, w)
        v = ((k >> win_bit(c, nlo, w)) & ((1 << cw) - 1)) + carry
        if v > (1 << (cw - 1)):
            yield w, (1 << cw) - v, 1
            carry = 1
        else:
            yield w, v, 0
            carry = 0


EMPTY = None  # ACC_EMPTY
FOLD_QUADS = 64


class Node:
    """FoldNode: the first and last run of a range (one run when `whole`)."""

    def __init__(self, kl=EMPTY, l=0):
        self.kl, self.l, self.kr, self.r, self.whole = kl, l, EMPTY, 0, True


def fold_merge(a, b, write):
    """a ++ b, runs that end inside written to their buckets."""
    if b.kl is EMPTY:
        return a
    if a.kl is EMPTY:
        return b
    ka, s = (a.kl, a.l) if a.whole else (a.kr, a.r)
    same = ka == b.kl
    if same:
        s = s + b.l
    o = Node(a.kl, a.l)
    o.kr, o.r, o.whole = a.kr, a.r, a.whole
    if not a.whole and not (same and b.whole):
        write(ka, s)
    if not same and not b.whole:
        write(b.kl, b.l)
    if same and a.whole:
        o.l = s
    if same and b.whole:
        if not a.whole:
            o.r = s
    else:
        o.kr, o.r = (b.kl, b.l) if b.whole else (b.kr, b.r)
        o.whole = False
    return o


def fold_block(leaves, J, write):
    """One block of k_acc_fold: `leaves` of its FOLD_QUADS * J places."""
    nodes = []
    for i in range(FOLD_QUADS):
        a = Node()
        for key, val in leaves[i * J:(i + 1) * J]:
            a = fold_merge(a, Node(key, val), write)
        nodes.append(a)
    st = 1
    while st < FOLD_QUADS:  # three steps inside the warps, three over them
        for i in range(0, FOLD_QUADS, 2 * st):
            nodes[i] = fold_merge(nodes[i], nodes[i + st], write)
        st *= 2
    return nodes[0]


def acc_l1(entries, K, write):
    """k_acc_l1: slots 2t and 2t + 1 take chunk t's first and last run."""
    slots = []
    for start in range(0, len(entries), K):
        chunk = entries[start:start + K]
        runs = []
        for k, v in chunk:
            if runs and runs[-1][0] == k:
                runs[-1] = (k, runs[-1][1] + v)
            else:
                runs.append((k, v))
        for k, v in runs[1:-1]:
            write(k, v)
        slots += [runs[0], runs[-1] if len(runs) > 1 else (EMPTY, 0)]
    return slots


def plan_shift(curve, counts, shift_bits, table_points, window=0):
    L = zl.lib()
    arr = (ctypes.c_uint32 * len(counts))(*counts)
    buf = ctypes.create_string_buffer(1 << 22)
    st = L.zkmsm_plan_describe_shift(curve, arr, len(counts), 0, window, shift_bits, table_points, buf, len(buf))
    assert st == 0, zl.last_error()
    return json.loads(buf.value.decode())


def run_model(C, pl, bases, scalars, seed=0, chunk=0):
    """`bases`: the base table as the entries index it (for a shift-table
    plan, copy k of the table at k * table_points + i)."""
    r = C.r
    lam = C.lam
    rng = random.Random(seed)
    descs = pl["descs"]
    G = pl["nbuckets"]
    # 1-3: digits, sort
    entries = []
    for d in descs:
        soff, n, boff, c, nwin, glv, bucket_off, fmt, win_off, wstep, nred, nlo = d
        for i in range(n):
            for j, (k, hneg) in enumerate(halves(C, scalars[soff + i], glv)):
                assert k < 1 << sum(win_width(c, nlo, w) for w in range(nwin)) - 1, "windows cover bits + 1"
                for w, a, dneg in digits(k, c, nwin, nlo):
                    if a:
                        if wstep:  # shift table: one bucket set, window w reads copy w*c/s
                            gb = bucket_off + (a - 1)
                            idx = boff + i + w * wstep
                            assert idx < len(bases) and idx <= 0x3FFFFFFF
                            entries.append((gb, idx | ((hneg ^ dneg) << 31)))
                        else:
                            gb = bucket_off + win_bucket(c, nlo, w) + (a - 1)
                            entries.append((gb, (boff + i) | (j << 30) | ((hneg ^ dneg) << 31)))
                        assert gb < G
    assert len(entries) <= pl["entry_bound"]
    rng.shuffle(entries)  # atomics give any order within a bucket
    entries.sort(key=lambda e: e[0])
    keys = [e[0] for e in entries]
    vals = [e[1] for e in entries]

    def point(v):
        idx = v & 0x3FFFFFFF
        x = bases[idx] * (lam if (v >> 30) & 1 else 1) % r
        return (-x) % r if v >> 31 else x

    buckets = [0] * G
    written = [False] * G

    def write_bucket(k, x):
        assert not written[k], "bucket %d written twice" % k
        written[k] = True
        buckets[k] = x % r

    # 4: segmented sums
    assert pl["affine"][0] == 0
    lst = [(k, point(v)) for k, v in zip(keys, vals)]
    fold = pl["entry_bound"] <= 1 << 16 and not chunk
    for lvl, (K, T, Mbound) in enumerate(pl["acc"]):
        M, last = len(lst), lvl + 1 == len(pl["acc"])
        assert M <= Mbound and T == max(1, -(-Mbound // K))
        if lvl == 0 and not fold:
            assert not last
            lst = acc_l1(lst, K, write_bucket)
        else:
            assert K % FOLD_QUADS == 0
            out = []
            for blk in range(0, M, K):
                a = fold_block(lst[blk:blk + K], K // FOLD_QUADS, write_bucket)
                if last:
                    assert a.kl is not EMPTY
                    write_bucket(a.kl, a.l)
                    if not a.whole:
                        write_bucket(a.kr, a.r)
                else:
                    out += [(a.kl, a.l), (EMPTY, 0) if a.whole else (a.kr, a.r)]
            lst = out
        assert len(lst) == (0 if last else 2 * -(-M // K))
        if last:
            assert T == 1
        else:
            assert len(lst) <= pl["acc"][lvl + 1][2]
    assert {k for k in range(G) if written[k]} == set(keys)
    # 5: bucket reduction and the windows' sum
    from tests.test_quad_reduce_model import reduce_model
    wins = reduce_model(pl, buckets)
    results = []
    for d in descs:
        soff, n, boff, c, nwin, glv, bucket_off, fmt, win_off, wstep, nred, nlo = d
        assert nred == (1 if wstep else nwin)
        acc = sum(wins[win_off + w] << (0 if wstep else win_bit(c, nlo, w)) for w in range(nred))
        results.append(acc % r if n else 0)
    return results


CASES = [
    # curve, counts, dist, window, chunk, glv, bits
    ("bn254", [700], "uniform", 0, 0, -1, 0),
    ("bn254", [700], "witness", 0, 8, -1, 0),
    ("bn254", [2000], "witness", 6, 8, -1, 0),        # hot buckets -> several partial levels
    ("bn254", [2000], "witness", 7, 0, -1, 0),        # entry sets above the fold threshold: k_acc_l1 first
    ("bn254", [900, 40] * 3, "uniform", 0, 0, -1, 0),
    ("bn254", [300, 0, 17, 1, 900], "uniform", 0, 0, -1, 0),
    ("bn254", [500], "uniform", 11, 33, 0, 0),          # no GLV: 255-bit scalars
    ("bn254", [400], "uniform", 0, 0, -1, 16),          # small-scalar plan
    ("bls12_381", [600], "uniform", 16, 16, -1, 0),     # 9 windows for 128-bit halves
    ("bls12_381", [250, 0, 40], "witness", 0, 0, -1, 0),
    ("bls12_381", [300], "uniform", 13, 64, 0, 0),
    ("bls12_377", [500], "uniform", 0, 0, -1, 0),       # 126-bit GLV halves
    ("bls12_377", [200, 0, 33], "witness", 9, 16, 0, 0),
]


@pytest.mark.parametrize("curve,counts,dist,window,chunk,glv,bits", CASES)
def test_schedule_model(curve, counts, dist, window, chunk, glv, bits):
    C = R.CURVES[curve]
    cid = {"bn254": zl.BN254, "bls12_381": zl.BLS12_381, "bls12_377": zl.BLS12_377}[curve]
    pl = plan(cid, counts, 0, window, chunk, glv, bits)
    rng = random.Random(sum(counts) + window)
    total = sum(counts)
    bases = [rng.randrange(1, C.r) for _ in range(total)]
    if bits:
        scalars = [rng.getrandbits(bits) for _ in range(total)]
    elif dist == "uniform":
        scalars = [rng.randrange(1 << 256) for _ in range(total)]
    else:
        scalars = []
        for _ in range(total):
            u = rng.randrange(100)
            scalars.append(0 if u < 40 else 1 if u < 60 else rng.getrandbits(32) if u < 85 else rng.randrange(C.r))
    got = run_model(C, pl, bases, scalars, seed=len(counts), chunk=chunk)
    off = 0
    for m, n in enumerate(counts):
        # the plan puts every MSM on a prefix of one base table (base_off = 0)
        want = sum(s * b for s, b in zip(scalars[off:off + n], bases[:n])) % C.r
        assert got[m] == want, m
        off += n


LAYOUT_CASES = [
    # curve, counts, dist, c, nlo (nlo windows of c bits, then c + 1-bit ones)
    ("bn254", [700], "uniform", 5, 10),
    ("bn254", [2000], "witness", 6, 1),
    ("bn254", [300, 0, 17, 1, 900], "uniform", 7, 4),
    ("bls12_381", [600], "uniform", 8, 3),
    ("bls12_381", [250, 0, 40], "witness", 4, 20),
]


@pytest.mark.parametrize("curve,counts,dist,c,nlo", LAYOUT_CASES)
def test_schedule_model_two_width(curve, counts, dist, c, nlo):
    """Forced two-width layouts (window setting c | nlo << 16): digits,
    bucket offsets, reduction tasks and the windows' shifts per window width."""
    C = R.CURVES[curve]
    cid = zl.BN254 if curve == "bn254" else zl.BLS12_381
    pl = plan(cid, counts, 0, c | (nlo << 16), 0, -1, 0)
    for d in pl["descs"]:
        if d[1]:
            assert d[3] == c and d[11] == nlo < d[4]
    rng = random.Random(sum(counts) + c)
    total = sum(counts)
    bases = [rng.randrange(1, C.r) for _ in range(total)]
    if dist == "uniform":
        scalars = [rng.randrange(1 << 256) for _ in range(total)]
    else:
        scalars = [0 if u < 40 else 1 if u < 60 else rng.getrandbits(32) if u < 85 else rng.randrange(C.r)
                   for u in (rng.randrange(100) for _ in range(total))]
    got = run_model(C, pl, bases, scalars, seed=len(counts))
    off = 0
    for m, n in enumerate(counts):
        want = sum(sc * b for sc, b in zip(scalars[off:off + n], bases[:n])) % C.r
        assert got[m] == want, m
        off += n


SHIFT_CASES = [
    # curve, counts, dist, shift spacing, table points, window override
    ("bn254", [700], "uniform", 4, 700, 0),
    ("bn254", [700], "witness", 4, 1000, 0),
    ("bn254", [300, 0, 17, 1, 900], "uniform", 4, 1000, 0),
    ("bn254", [500], "uniform", 4, 600, 10),   # 10 rounds up to a multiple of 4
    ("bn254", [400], "witness", 8, 400, 16),
    ("bls12_381", [600], "uniform", 6, 600, 0),
    ("bls12_381", [250, 0, 40], "witness", 5, 300, 0),
]


@pytest.mark.parametrize("curve,counts,dist,s,tp,window", SHIFT_CASES)
def test_schedule_model_shift_table(curve, counts, dist, s, tp, window):
    """MSMs over a table with window shifts: every window's digits index
    copy w*c/s of the table and add into one bucket set; one window sum."""
    C = R.CURVES[curve]
    cid = zl.BN254 if curve == "bn254" else zl.BLS12_381
    pl = plan_shift(cid, counts, s, tp, window)
    for d in pl["descs"]:
        if d[1]:
            assert d[3] % s == 0 and d[5] == 0 and d[10] == 1 and d[9] == (d[3] // s) * tp
            if window:
                assert d[3] == -(-window // s) * s
    copies = -(-(C.r.bit_length() + 1) // s)
    rng = random.Random(sum(counts) + s)
    table = [rng.randrange(1, C.r) for _ in range(tp)]
    ext = [p * pow(2, s * k, C.r) % C.r for k in range(copies) for p in table]
    total = sum(counts)
    if dist == "uniform":
        scalars = [rng.randrange(1 << 256) for _ in range(total)]
    else:
        scalars = []
        for _ in range(total):
            u = rng.randrange(100)
            scalars.append(0 if u < 40 else 1 if u < 60 else rng.getrandbits(32) if u < 85 else rng.randrange(C.r))
    got = run_model(C, pl, ext, scalars, seed=len(counts))
    off = 0
    for m, n in enumerate(counts):
        want = sum(sc * b for sc, b in zip(scalars[off:off + n], table[:n])) % C.r
        assert got[m] == want, m
        off += n


def test_shift_plan_falls_back_outside_table():
    """An MSM longer than the shift table's prefix uses ordinary windows."""
    pl = plan_shift(zl.BN254, [100, 5000], 4, 1000)
    assert pl["descs"][0][9] > 0 and pl["descs"][0][10] == 1
    assert pl["descs"][1][9] == 0 and pl["descs"][1][10] == pl["descs"][1][4]


def test_plan_sizes_2_24():
    """The full-size plan: entry and bucket counts fit 32-bit indices and the
    window choice is the cost model's."""
    pl = plan(zl.BN254, [1 << 24])
    d = pl["descs"][0]
    c, nwin, nlo = d[3], d[4], d[11]
    assert win_bucket(c, nlo, nwin) == pl["nbuckets"]
    assert pl["entry_bound"] == 2 * (1 << 24) * nwin < (1 << 32)
    assert 14 <= c <= 22
    # GLV halves of 127 bits: the windows cover exactly the 128 bits of the
    # signed recoding, the wider ones on top
    assert sum(win_width(c, nlo, w) for w in range(nwin)) == 128 and nlo <= nwin


@pytest.mark.parametrize("curve,n", [("bn254", 1 << 20), ("bn254", 1 << 22), ("bn254", 1 << 24),
                                     ("bls12_381", 1 << 22)])
def test_two_width_layout_covers_scalar(curve, n):
    """Large plans split the signed recoding's bits + 1 bits into windows
    whose widths differ by at most one."""
    cid = zl.BN254 if curve == "bn254" else zl.BLS12_381
    d = plan(cid, [n])["descs"][0]
    c, nwin, nlo = d[3], d[4], d[11]
    widths = [win_width(c, nlo, w) for w in range(nwin)]
    assert max(widths) - min(widths) <= 1 and widths == sorted(widths)
    assert sum(widths) - widths[-1] < 128 <= sum(widths)


def _types_const(name):
    import os
    import re
    text = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zkmetal_b200", "csrc",
                             "types.cuh")).read()
    m = re.search(r"constexpr\s+\w+\s+%s\s*=\s*([^;]+);" % name, text)
    return int(m.group(1))


@pytest.mark.parametrize("curve,counts,window,glv", [
    (0, [1 << 24], 0, -1), (0, [1 << 20], 0, -1), (0, [1 << 12], 0, -1), (0, [3000], 6, -1), (0, [5000], 2, 0),
    (1, [1 << 22], 0, -1), (2, [1 << 16], 0, -1), (3, [1 << 14], 0, -1), (0, [4096, 1 << 20, 333, 1 << 18], 0, -1),
    (0, [1 << 10] * 64, 0, 0), (0, [100], 3 | 1 << 16, -1)])
def test_digit_block_slices_fit(curve, counts, window, glv):
    """k_radix_digits gives each warp a slice of SORT_DBUF / 8 entries and runs
    min(32, spb / 8) lanes per warp in rounds of 8 * lanes scalars: for the
    plan's scalars per block (spb) and digits per scalar (maxd), a warp's
    digits of all its rounds must fit its slice."""
    dbuf, threads = _types_const("SORT_DBUF"), _types_const("SORT_DTHREADS")
    warps = threads // 32
    pl = plan(curve, counts, window=window, glv=glv)
    maxd, spb = pl["sort"][0], pl["sort"][1]
    assert maxd >= 1 and spb >= warps
    lanes = min(32, spb // warps)
    rounds = -(-spb // (warps * lanes))
    assert lanes >= 1 and rounds * lanes * maxd <= dbuf // warps, (maxd, spb, lanes, rounds)
    # the same number of scalars per block as the kernel's rounds cover
    assert spb <= rounds * warps * lanes
