"""The drain of the merged kernels' 32-bit bins and totals (csrc/war_merge.cuh, DRAIN_DEALS): a warp empties them when it
has dealt out games for 2^26 deals.  The default grids are too wide for that in any job of a second, so these jobs run on
one block of 64 threads per SM, where every warp passes it, and must give what the default grid gives.  Counts are whole
numbers: every comparison is equality."""
import math

import pytest

F13, F14 = math.factorial(13), math.factorial(14)
KEYS = ("cyc", "done", "maxfin", "hist", "endhist")
SMALL = dict(threads=64, blocks_per_sm=1)


def passes_the_drain(wl, deals):
    """Every warp deals out at least 2^26 deals (they share the units evenly to far less than a part in ten)."""
    return deals > 1.1 * 2 ** 26 * 2 * wl.device_info().sm_count


def equal(wl, got, want, keys, what):
    got, want = wl.to_dict(got), wl.to_dict(want)
    for k in keys:
        assert got[k] == want[k], (what, k)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [0, 1])
def test_main_engine(wl, rule):
    assert passes_the_drain(wl, F14)
    job = wl.make_job(16, rule=rule, lo=F14, hi=2 * F14, hbins=128)
    kw = dict(variant=31, games=1, window=32, defer=16, memo_bits=31)
    equal(wl, wl.enumerate_job(job, wl.make_tune(**kw, **SMALL)), wl.enumerate_job(job, wl.make_tune(threads=256, **kw)),
          KEYS, rule)


@pytest.mark.gpu
@pytest.mark.parametrize("n,rule", [(17, 0), (17, 1), (16, 0)])
def test_held_out_engine(wl, n, rule):
    """With the run test (17 cards, winner's card first) and without."""
    assert passes_the_drain(wl, 4 * F13)
    job = wl.make_job(n, rule=rule, lo=4 * F13, hi=8 * F13, hbins=128)
    equal(wl, wl.enumerate_held(job, wl.make_tune(**SMALL)), wl.enumerate_held(job), KEYS + ("turns",), (n, rule))


@pytest.mark.gpu
@pytest.mark.parametrize("det", [0, 1, 2])
def test_5_bit_engine(wl, det):
    assert passes_the_drain(wl, 4 * F13)
    job = wl.make_job(17, lo=4 * F13, hi=8 * F13, hbins=0 if det else 128)
    equal(wl, wl.enumerate_wide(job, det, **SMALL), wl.enumerate_wide(job, det), KEYS + ("turns", "undetermined"), det)
