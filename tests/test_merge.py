"""Deals played together (csrc/war_merge.cuh): the first floor(n/2) turns of a deal forget how the two players'
wins alternated, so C(f, a) deals share the state after them.  On the CPU, a restatement of the enumeration
(aligned blocks, ordered lists of unordered pairs, the number of them that player 1 wins) against every deal
of a range played turn by turn; on the GPU, the merged kernels against the oracle and the plain kernel at the
edges of blocks, units and piles.  Counts are whole numbers: every comparison is equality."""
import itertools
import math
import random
from collections import Counter

import pytest


def unrank(r, n):
    cards, out = list(range(n)), []
    for i in range(n):
        d, r = divmod(r, math.factorial(n - 1 - i))
        out.append(cards.pop(d))
    return out


def after_first_turns(deck, rule):
    """Both piles after floor(n/2) turns."""
    a, b = deck[0::2], deck[1::2]
    for _ in range(len(deck) // 2):
        x, y = a.pop(0), b.pop(0)
        pair = [min(x, y), max(x, y)] if rule else [max(x, y), min(x, y)]
        (a if x > y else b).extend(pair)
    return tuple(a), tuple(b)


def blocks(lo, hi, n):
    while lo < hi:
        j = n
        while lo % math.factorial(j) or lo + math.factorial(j) > hi:
            j -= 1
        yield lo, j
        lo += math.factorial(j)


def pair_lists(cards, f):
    if f == 0:
        yield []
        return
    for x, y in itertools.combinations(sorted(cards), 2):
        for rest in pair_lists([c for c in cards if c not in (x, y)], f - 1):
            yield [(y, x)] + rest


def merged(lo, hi, n, rule, half=False):
    """{state after the first turns: deals of the range in it}, by blocks."""
    out = Counter()
    h = n // 2
    for r, j in blocks(lo, hi, n):
        b = n - j
        deck = unrank(r, n)
        free = deck[b:]
        f = max(0, (2 * h - (b + b % 2)) // 2)
        singles = (1 if b % 2 and b < n else 0) + (1 if n % 2 and b < n else 0)
        for pick in itertools.permutations(free, singles):
            rest = [c for c in free if c not in pick]
            pick = list(pick)
            fixed = deck[:b] + ([pick.pop(0)] if b % 2 and b < n else [])
            top = [pick.pop(0) if b < n else deck[n - 1]] if n % 2 else []
            wins = [[], []]
            for t in range(0, min(len(fixed), 2 * h) - 1, 2):
                x, y = fixed[t], fixed[t + 1]
                wins[0 if x > y else 1] += [min(x, y), max(x, y)] if rule else [max(x, y), min(x, y)]
            for pairs in pair_lists(rest, f):
                cards = [list(reversed(p)) if rule else list(p) for p in pairs]
                for a in range(f + 1):
                    one = tuple(top + wins[0] + sum(cards[:a], []))
                    two = tuple(wins[1] + sum(cards[a:], []))
                    if not half or n - 1 in one:
                        out[one, two] += math.comb(f, a)
    return out


@pytest.mark.parametrize("n,rule", [(2, 0), (3, 1), (4, 0), (5, 0), (6, 1), (7, 0), (8, 1)])
def test_merged_enumeration_is_every_deal(n, rule):
    rnd = random.Random(100 * n + rule)
    total = math.factorial(n)
    ranges = [(0, total)] if n <= 7 else []
    for _ in range(5):
        lo = rnd.randrange(0, total)
        ranges.append((lo, min(total, lo + rnd.choice([1, 2, 25, 800]))))
    for lo, hi in ranges:
        for half in ((False, True) if n % 2 == 0 else (False,)):
            want = Counter()
            for r in range(lo, hi):
                deck = unrank(r, n)
                if not half or deck.index(n - 1) % 2 == 0:
                    want[after_first_turns(deck, rule)] += 1
            assert merged(lo, hi, n, rule, half) == want, (n, rule, lo, hi, half)


def memo_tune(wl, **kw):
    t = dict(variant=31, games=1, threads=256, defer=8, window=32, memo_bits=20)
    t.update(kw)
    return wl.make_tune(**t)


KEYS = ("cyc", "done", "maxfin", "hist", "endhist")


def same(wl, got, want, what):
    g, w = wl.to_dict(got), wl.to_dict(want)
    for k in KEYS:
        assert g[k] == w[k], (what, k)


@pytest.mark.gpu
@pytest.mark.parametrize("n", range(4, 17))
def test_merged_ranges(wl, n):
    """Ranges that begin and end at, before and after block ends, the first and the last deals, one deal, odd
    lengths; --half; both rules; a table of 2^12 words; several launch shapes."""
    rnd = random.Random(n)
    total = math.factorial(n)
    ranges = [(0, 1), (total - 1, total), (0, min(total, 362880)), (max(0, total - 362881), total)]
    for j in range(1, min(n, 10)):
        f = math.factorial(j)
        k = rnd.randrange(1, total // f) if total // f > 1 else 0
        ranges.append((k * f, min(total, (k + 1) * f)))
        ranges.append((max(0, k * f - 1), min(total, k * f + rnd.choice([1, f, 2 * f + 1]))))
    for _ in range(4):
        lo = rnd.randrange(0, total)
        ranges.append((lo, min(total, lo + rnd.choice([3, 1001, 1000003]))))
    shapes = [dict(), dict(threads=64, defer=4), dict(threads=1024, memo_bits=12), dict(window=1, defer=32),
              dict(blocks_per_sm=1, threads=128, variant=30)]
    for i, (lo, hi) in enumerate(ranges):
        for flags in ([0, wl.F_HALF] if n % 2 == 0 else [0]):
            job = wl.make_job(n, rule=i % 2, lo=lo, hi=hi, flags=flags, hbins=rnd.choice([0, 64, 256]))
            same(wl, wl.enumerate_job(job, memo_tune(wl, **shapes[i % len(shapes)])), wl.enumerate_plain(job),
                 (n, lo, hi, flags, i))


@pytest.mark.gpu
@pytest.mark.parametrize("n,rule", [(10, 0), (11, 1), (12, 0)])
def test_merged_whole_spaces(wl, n, rule):
    """Every deal (even n: mirror images played once, counted twice), and --half."""
    for flags in ([0, wl.F_HALF] if n % 2 == 0 else [0]):
        job = wl.make_job(n, rule=rule, flags=flags, hbins=256)
        want = wl.enumerate_plain(job)
        for kw in (dict(), dict(memo_bits=12, defer=4)):
            same(wl, wl.enumerate_job(job, memo_tune(wl, **kw)), want, (n, rule, flags, kw))


@pytest.mark.gpu
def test_merged_table_kept_between_ranges_of_different_sizes(wl):
    """A job smaller than the one before it with WAR_F_MEMO_KEEP, and one without: the part of the table in use
    follows the first job, or the job's own size."""
    t = memo_tune(wl, memo_bits=26)
    jobs = [(0, 0, 3 * 10 ** 7), (wl.F_MEMO_KEEP, 10 ** 9, 10 ** 9 + 12345), (0, 10 ** 9, 10 ** 9 + 54321),
            (wl.F_MEMO_KEEP, 5 * 10 ** 8, 5 * 10 ** 8 + 10 ** 7)]
    for flags, lo, hi in jobs:
        job = wl.make_job(13, flags=flags, lo=lo, hi=hi, hbins=128)
        same(wl, wl.enumerate_job(job, t), wl.enumerate_plain(wl.make_job(13, lo=lo, hi=hi, hbins=128)), (lo, hi))


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
def test_held_merged_games_and_turns(wl, rule):
    """The held-out-card engine's default turn (merged games) against its turn that plays every deal (variant 8):
    counts, lengths and the turns that playing every deal takes, with windows around the merged turns and around
    the cycle lengths of small decks (a deal on its own cycle is decided earlier than the rest of its game)."""
    keys = KEYS + ("turns",)
    rnd = random.Random(rule)
    for n in list(range(2, 12)) + [13, 14, 16, 17, 17]:
        total = math.factorial(n)
        lo = 0 if n < 10 else rnd.randrange(0, total - 300000)
        job = wl.make_job(n, rule=rule, lo=lo, hi=total if n < 10 else lo + 300000, hbins=128)
        for kw in (dict(), dict(window=16, defer=16, threads=128), dict(window=8, defer=4), dict(window=4, defer=4),
                   dict(window=64, defer=32, threads=1024)):
            got = wl.to_dict(wl.enumerate_held(job, wl.make_tune(**kw)))
            want = wl.to_dict(wl.enumerate_held(job, wl.make_tune(variant=8, **kw)))
            for k in keys:
                assert got[k] == want[k], (n, kw, k)


def ojob(oracle, job):
    return oracle.make_job(job.n, 0, job.rule, 0, job.lo, job.hi, job.hbins)


WIDE_KEYS = KEYS + ("turns", "undetermined")


def same_wide(wl, oracle, job, det, window, cap, kw):
    got = wl.to_dict(wl.enumerate_wide(job, det, cap=cap, **kw))
    want = oracle.to_dict(oracle.war24(ojob(oracle, job), det, window, cap or 1 << 22))
    for k in WIDE_KEYS:
        assert got[k] == want[k], (job.n, job.rule, det, window, cap, kw, k, got[k], want[k])


@pytest.mark.gpu
@pytest.mark.parametrize("n", range(2, 12))
def test_wide_merged_small(wl, oracle, n):
    """The 5-bit engine's merged games, every deal of n <= 11: counts, turns and undetermined games equal the
    oracle's under every detector, with windows, service periods and step caps at the edges of the rule."""
    for rule in (0, 1):
        job = wl.make_job(n, rule=rule, hbins=256)
        for window, cap, kw in ((32, 0, {}), (16, 0, dict(window=16, defer=4)), (32, 64, {}), (32, 63, {}),
                                (8, 0, dict(window=8, defer=8, threads=128)), (4, 0, dict(window=4, defer=4)),
                                (64, 0, dict(window=64, defer=64, threads=1024))):
            same_wide(wl, oracle, job, wl.DET_BRENT, window, cap, kw)
        job = wl.make_job(n, rule=rule)
        for cap, kw in ((0, {}), (0, dict(defer=4)), (2 * n, {}), (n + 2, dict(defer=64)), (n + 1, {})):
            same_wide(wl, oracle, job, wl.DET_FLOYD, 32, cap, kw)
        if n % 2 and not rule:
            for cap, kw in ((0, {}), (0, dict(defer=64, threads=128)), (200, dict(defer=4)), (90, {}), (2 * n, {}),
                            (n, {})):
                same_wide(wl, oracle, job, wl.DET_STREAK, 32, cap, kw)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [13, 14, 16, 17, 18, 19, 20])
def test_wide_merged_ranges(wl, oracle, n):
    rnd = random.Random(n)
    total = math.factorial(n)
    for i in range(3):
        lo = rnd.randrange(0, total) if i else total - 5041
        hi = min(total, lo + rnd.choice([1, 5041, 60001]))
        for det in (0, 1, 2) if n % 2 and i != 1 else (0, 1):
            job = wl.make_job(n, rule=0 if det == 2 else i % 2, lo=lo, hi=hi, hbins=0 if det else 256)
            same_wide(wl, oracle, job, det, 32, 0, {})


@pytest.mark.gpu
def test_merged_table_kept_after_a_much_smaller_job(wl):
    """WAR_F_MEMO_KEEP after a job of a few deals: the job takes the table that it would take by itself, so that it
    looks its games up as often and finds as many (to a few in a thousand: lanes race for what to store)."""
    t = memo_tune(wl, memo_bits=26)
    lo, hi = 10 ** 9, 10 ** 9 + 3 * 10 ** 7
    alone = wl.to_dict(wl.enumerate_job(wl.make_job(13, lo=lo, hi=hi, hbins=128), t))
    wl.enumerate_job(wl.make_job(13, lo=0, hi=1000, hbins=128), t)
    kept = wl.to_dict(wl.enumerate_job(wl.make_job(13, flags=wl.F_MEMO_KEEP, lo=lo, hi=hi, hbins=128), t))
    for k in KEYS:
        assert kept[k] == alone[k], k
    assert kept["turns"] < 1.05 * alone["turns"]


@pytest.mark.gpu
@pytest.mark.parametrize("det", [0, 1, 2])
def test_wide_merged_largest_launch_shape(wl, det):
    """Blocks of 1024 threads with the most histogram bins: more shared memory than a launch has unasked."""
    lo = 10 ** 13
    job = wl.make_job(17, lo=lo, hi=lo + 5041, hbins=wl.WAR_HBINS_MAX)
    got = wl.to_dict(wl.enumerate_wide(job, det, threads=1024))
    want = wl.to_dict(wl.enumerate_wide(job, det))
    for k in WIDE_KEYS:
        assert got[k] == want[k], (det, k)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 5, 6, 8, 11, 13, 16])
def test_canonical_units(wl, n):
    """Canonical scans with the path memo at the edges of orders, blocks and units: one position, part of an order,
    ranges that begin and end inside orders, the last positions; every output, both rules."""
    rnd = random.Random(n)
    total, s = wl.space_size(n, wl.CANON), n - 1
    ranges = [(0, 1), (total - 1, total), (total - min(total, 720 * s + 3), total), (0, min(total, 721 * s - 1))]
    for _ in range(4):
        lo = rnd.randrange(0, total)
        ranges.append((lo, min(total, lo + rnd.choice([1, s, 2 * s + 1, 100003]))))
    shapes = [dict(), dict(threads=64, defer=4), dict(threads=1024, memo_bits=12), dict(blocks_per_sm=1, variant=30)]
    keys = KEYS + ("dhist", "oncycle", "distinct_min", "shape_nonstd", "shape_unchecked", "s_count", "s_cyc",
                   "s_lamsum", "s_lensum", "s_maxfin")
    for i, (lo, hi) in enumerate(ranges):
        for flags in (0, wl.F_SHAPE, wl.F_DISTINCT, wl.F_DISTINCT | wl.F_SHAPE | wl.F_SAMPLE):
            job = wl.make_job(n, wl.CANON, i % 2, flags, lo, hi, hbins=128, dbins=64 if flags & wl.F_DISTINCT else 0,
                              sample_ppm=100000, seed=n)
            got = wl.to_dict(wl.enumerate_job(job, memo_tune(wl, window=128, **shapes[i % len(shapes)])))
            want = wl.to_dict(wl.enumerate_plain(job))
            for k in keys:
                assert got[k] == want[k], (n, lo, hi, flags, k)
