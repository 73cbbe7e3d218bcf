"""The ranges that war_gpu.run hands to the engine, one call each: 14! deals where the engine plays them merged, and
just under 2^32 ranks, a second or so of work, where every game is played, so that progress is written as often."""
import math

import pytest


def spans(monkeypatch, n, tune, **kw):
    import warlib
    import war_gpu
    calls = []

    def enum(job, tune=None):
        calls.append((job.lo, job.hi))
        return warlib.Result()
    monkeypatch.setattr(warlib, "enumerate_job", enum)
    monkeypatch.setattr(warlib, "enumerate_plain", enum)
    monkeypatch.setattr(war_gpu, "_tune_for", lambda *a: None)
    war_gpu.run(n, quiet=True, tune=tune, **kw)
    assert all(a[1] == b[0] for a, b in zip(calls, calls[1:]))
    return [hi - lo for lo, hi in calls]


@pytest.mark.parametrize("variant,merged", [(31, True), (30, True), (28, False), (15, False), (7, False), (3, False), (None, False)])
def test_deals_per_call(monkeypatch, variant, merged):
    import warlib
    import war_gpu
    tune = None if variant is None else warlib.make_tune(variant=variant)
    got = spans(monkeypatch, 14, tune)
    assert got[0] == (math.factorial(14) if merged else war_gpu.CALL_RANKS), variant
    # the reference's launch geometry, where that is more
    got = spans(monkeypatch, 14, tune, per=1 << 16, batch_threads=1 << 20)
    assert got[0] == (math.factorial(14) if merged else 1 << 36), variant
    assert spans(monkeypatch, 14, tune, plain=True)[0] == war_gpu.CALL_RANKS
    assert spans(monkeypatch, 13, tune, canon=True)[0] == war_gpu.CALL_RANKS // 12 * 12
