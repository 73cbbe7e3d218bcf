"""WAR_F_MEMO_KEEP between jobs that use different parts of one table, and between jobs whose entries mean different
things (csrc/war_capi.cu, prepare_memo): every count equals the plain kernel's.  Counts are whole numbers: every
comparison is equality."""
import math

import pytest

KEYS = ("cyc", "done", "maxfin", "hist", "endhist", "s_count", "s_cyc", "s_lamsum", "s_lensum", "s_maxfin", "oncycle",
        "distinct_min", "shape_nonstd", "shape_unchecked")


def tune(wl, canon, memo_bits):
    return wl.make_tune(variant=31, games=1, threads=256, defer=4, window=128 if canon else 32, memo_bits=memo_bits)


def check(wl, memo_bits, n, mode=0, rule=0, flags=0, **kw):
    if flags & wl.F_SAMPLE:
        kw.update(sample_ppm=100000, seed=n)
    got = wl.to_dict(wl.enumerate_job(wl.make_job(n, mode, rule, flags, hbins=128, **kw), tune(wl, mode, memo_bits)))
    want = wl.to_dict(wl.enumerate_plain(wl.make_job(n, mode, rule, flags & ~wl.F_MEMO_KEEP, hbins=128, **kw)))
    for k in KEYS:
        assert got[k] == want[k], (n, mode, rule, flags, k)


def words(useful):
    """log2 of the table that a job of so many useful words takes."""
    return max(12, math.ceil(math.log2(useful)))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [9, 11])
@pytest.mark.parametrize("canon", [False, True])
def test_sampled_deals_after_a_job_that_used_half_of_the_table(wl, n, canon):
    """Jobs of the other rule fill the whole table, canonical positions among them: their starts are states that
    games of both rules can reach (after a turn the pair under the winner's pile tells the rules apart).  A merged
    (or canonical) job clears and uses half of the table, a sampled job keeps that, a merged and a canonical one
    what the sampled one left.  (Sampled deals are played by another kernel than the others, in the same table.)"""
    if canon:
        games = 2 * math.factorial(n - 1) * (n - 1)
    else:
        f = n // 2
        games = math.factorial(n) // 2 ** f * (f + 1) // 4 * 3 + 1
    bits = words(games) + 1
    check(wl, bits, n, rule=1, flags=wl.F_SAMPLE)
    check(wl, bits, n, mode=1, rule=1, flags=wl.F_MEMO_KEEP)
    check(wl, bits, n, mode=1 if canon else 0)
    check(wl, bits, n, flags=wl.F_SAMPLE | wl.F_MEMO_KEEP)
    check(wl, bits, n, flags=wl.F_MEMO_KEEP)
    check(wl, bits, n, mode=1, flags=wl.F_MEMO_KEEP)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [9, 11])
def test_shape_scans_of_different_block_lengths(wl, n):
    """The loop-shape codes in a table are those of one block length: a job with another one does not read them."""
    bits = words(2 * math.factorial(n - 1) * (n - 1))
    for i, blk in enumerate((2, 1, 1, 4, 0)):
        check(wl, bits, n, mode=1, flags=wl.F_SHAPE | (wl.F_MEMO_KEEP if i else 0), blk=blk)
