"""CPU replay of one thread's affine levels (k_aff_pair, k_aff_add,
k_aff_finish) with integers in place of points: the pairs of each run, the
list of references rewritten behind its reader, sums written over their left
element.  Checked for every run pattern that matters: references stay inside
the places, a level leaves ceil(run / 2) elements of each run, a partner
always exists where one is read, and every key's sum is kept.  Also the plans'
rule: which calls take affine levels, and their chunks."""
import ctypes
import json
import random

import pytest

from zkmetal_b200 import lib as zl

ENTRY, LAST, INDEX = 0x8000, 0x4000, 0x3FFF


class Words:
    """AffList: four references a word, the reader's word and the next one
    cached, the writer's words stored when full."""

    def __init__(self, mem, n):
        self.mem, self.word, self.words = mem, 0, -(-n // 4)
        self.cur = mem[0:4] if self.words else None
        self.next = mem[4:8] if self.words > 1 else None
        self.out = [0] * 4

    def get(self, i):
        if i >> 2 != self.word:
            assert i >> 2 == self.word + 1
            self.word += 1
            self.cur = self.next
            if self.word + 1 < self.words:
                self.next = self.mem[4 * self.word + 4:4 * self.word + 8]
        return self.cur[i & 3]

    def put(self, k, ref):
        self.out[k & 3] = ref
        if k & 3 == 3:
            self.mem[k - 3:k + 1] = self.out

    def close(self, k):
        if k & 3:
            self.mem[k & ~3:(k & ~3) + 4] = self.out


def pair_first(ents, mem, runs):
    n, i, k, run, info = len(ents), 0, 0, 0, []
    w = Words(mem, 0)
    at = lambda x: ents[x] if x < n else (None, 0)
    while i < n:
        if at(i + 1)[0] != at(i)[0]:
            w.put(k, ENTRY | LAST)
            runs[run] = at(i)
            run += 1
            i += 1
        else:
            end = at(i + 2)[0] != at(i)[0]
            w.put(k, len(info) | (LAST if end else 0))
            if end:
                runs[run] = (at(i)[0], 0)
                run += 1
            info.append((len(info), at(i)[1], at(i + 1)[1]))
            i += 2
        k += 1
    w.close(k)
    return k, info, run


def pair_next(mem, n, runs, places):
    i, k, run, info = 0, 0, 0, []
    w = Words(mem, n)
    sval = runs[0][1]
    while i < n:
        r0 = w.get(i)
        last = r0
        if r0 & LAST:
            w.put(k, r0)
            i += 1
        else:
            assert not r0 & ENTRY, "only a run's last element lacks a place"
            r1 = w.get(i + 1)
            w.put(k, r0 | (r1 & LAST))
            info.append((r0 & INDEX, places[r0 & INDEX], sval if r1 & ENTRY else places[r1 & INDEX]))
            last = r1
            i += 2
        k += 1
        if last & LAST and i < n:
            run += 1
            sval = runs[run][1]
    w.close(k)
    return k, info


def add(info, places, cap):
    for place, a, b in reversed(info):
        assert place < cap
        places[place] = a + b


@pytest.mark.parametrize("pattern", [
    [1], [2], [3], [1, 1], [2, 2], [1, 2], [2, 1], [3, 3, 3], [1, 4, 1], [5, 1, 1, 6], [64], [63], [7] * 9,
    [1] * 10, [16, 1, 15, 2, 14], [31, 33], [8] * 8, [9, 8, 7, 6, 5, 4, 3, 2, 1], [1] * 33 + [40]])
def test_levels_keep_sums(pattern):
    rng = random.Random(len(pattern) * 100 + sum(pattern))
    ents = [(k, rng.getrandbits(60)) for k, r in enumerate(pattern) for _ in range(r)]
    K = -(-len(ents) // 4) * 4
    cap = K // 2
    mem, runs, places = [None] * K, [None] * K, [None] * max(cap, 1)
    want = [sum(v for q, v in ents if q == k) for k in range(len(pattern))]
    n, info, nrun = pair_first(ents, mem, runs)
    assert nrun == len(pattern) and len(info) <= cap
    add(info, places, cap)
    expect = list(pattern)
    for _ in range(8):
        expect = [-(-r // 2) for r in expect]
        assert n == sum(expect)
        # k_aff_finish: the elements of each run, its key from the table
        got, run, count, acc = [], 0, [], 0
        c = 0
        for i in range(n):
            r = mem[i]
            acc += runs[run][1] if r & ENTRY else places[r & INDEX]
            c += 1
            if r & LAST:
                assert runs[run][0] == run
                got.append(acc)
                count.append(c)
                acc, c, run = 0, 0, run + 1
        assert got == want and count == expect
        n, info = pair_next(mem, n, runs, places)
        add(info, places, cap)
    assert n == len(pattern)


def describe(curve, n, window=0, chunk=0):
    buf = ctypes.create_string_buffer(1 << 22)
    arr = (ctypes.c_uint32 * 1)(n)
    assert zl.lib().zkmsm_plan_describe(curve, arr, 1, 1, window, chunk, -1, 0, buf, len(buf)) == 0
    return json.loads(buf.value.decode())


@pytest.mark.parametrize("curve", [zl.BN254, zl.BLS12_381, zl.BLS12_377, zl.BN254_G2])
@pytest.mark.parametrize("n", [1 << 10, 1 << 16, 1 << 18, 1 << 20, 3000001, 1 << 22, 1 << 24])
def test_plan_rule(curve, n):
    pl = describe(curve, n)
    levels, threads, slabs = pl["affine"]
    K, T, M = pl["acc"][0]
    run = M // pl["nbuckets"]
    assert (levels > 0) == (curve != zl.BN254 and M >= 1 << 22 and run >= 8)
    if levels:
        assert 16 <= K <= 512 and K % 4 == 0 and threads % 512 == 0 and T == -(-M // K)
        assert slabs * threads >= T > (slabs - 1) * threads
        # a thread keeps several elements at the last level, and runs are
        # halved while more than one and a half long
        assert K >> levels >= 4 and 2 * run >= 3 << (levels - 1)
    assert describe(curve, n, chunk=64)["affine"] == [0, 0, 0]


def describe_sampled(curve, n, window=0, entries=0, pct=0):
    buf = ctypes.create_string_buffer(1 << 22)
    assert zl.lib().zkmsm_plan_describe_sampled(curve, n, 1, window, entries, pct, buf, len(buf)) == 0
    return json.loads(buf.value.decode())


@pytest.mark.parametrize("curve", [zl.BLS12_381, zl.BLS12_377, zl.BN254_G2])
@pytest.mark.parametrize("n", [1 << 18, 1 << 20, 3000001, 1 << 22])
@pytest.mark.parametrize("pct", [10, 50, 99, 100, 200, 1000])
def test_plan_rule_with_tuned_chunks(curve, n, pct):
    """An autotuned chunk length changes the affine chunks, and the slabs
    still hold all of them."""
    rule, pl = describe_sampled(curve, n), describe_sampled(curve, n, pct=pct)
    levels, threads, slabs = pl["affine"]
    K, T, M = pl["acc"][0]
    assert levels and rule == describe(curve, n)
    assert 16 <= K <= 512 and K % 4 == 0
    want = min(512, max(16, rule["acc"][0][0] * pct // 100))
    assert abs(K - want) <= 4 + 3 * pct // 100
    assert slabs * threads >= T > (slabs - 1) * threads, "chunks outside the slabs are none of the affine levels"


@pytest.mark.parametrize("n,entries", [(1 << 21, 8390000), (1 << 22, 1 << 23), (1 << 20, 5000000)])
def test_plan_rule_with_few_expected_entries(n, entries):
    """A sample that expects fewer entries than the bound: slabs for those,
    and chunks past them for k_acc_l1."""
    pl = describe_sampled(zl.BLS12_381, n, 15, entries)
    levels, threads, slabs = pl["affine"]
    K, T, M = pl["acc"][0]
    assert levels and M > entries
    assert slabs * threads * K >= entries > (slabs - 1) * threads * K
    assert T == -(-M // K) > slabs * threads
    assert describe_sampled(zl.BLS12_381, n, 15, (1 << 22) - 1)["affine"] == [0, 0, 0]
