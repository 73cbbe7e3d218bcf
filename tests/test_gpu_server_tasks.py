"""Tasks of the jobs that the server does not play merged (csrc/war_server.cu, RefillTask): more of them than a tick takes,
beside merged ones, and ranges whose ends are units of their own."""
import pytest

KEYS = ("cyc", "done", "maxfin", "hist", "endhist", "s_count", "s_cyc", "s_lamsum", "s_lensum", "s_maxfin", "shape_nonstd",
        "shape_unchecked")


@pytest.mark.gpu
@pytest.mark.parametrize("memo_bits", [0, -1])
def test_more_refill_tasks_than_a_tick_takes(wl, memo_bits):
    """Two sampled jobs of 1.5e8 deals are 4578 tasks of 2^16 ranks, a tick takes 2560; the loop-shape scan and the merged
    job wait with them and run beside them."""
    import serve
    S = dict(sample_ppm=10000, seed=5, hbins=64)
    jobs = [wl.make_job(12, 0, 0, wl.F_SAMPLE, 1, 150000000, **S),
            wl.make_job(12, 0, 1, wl.F_SAMPLE, 150000007, 300000007, **S),
            wl.make_job(10, wl.CANON, 0, wl.F_SHAPE, 3, 3000001, hbins=64),
            wl.make_job(12, 0, 0, 0, 12345, 9999999, hbins=64)]
    with serve.Server(tick_ranks=1 << 30, memo_bits=memo_bits) as s:
        got = [r for r, _ in s.wait_all([s.submit(j) for j in jobs])]
    for j, g in zip(jobs, got):
        g, want = wl.to_dict(g), wl.to_dict(wl.enumerate_plain(j))
        for k in KEYS:
            assert g[k] == want[k], (j.n, j.rule, j.flags, k)
