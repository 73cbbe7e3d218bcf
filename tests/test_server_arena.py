"""How much of a server's memo arena a class of jobs takes (csrc/war_server.cu, set_args), on the CPU with a fake CUDA
runtime."""
import pytest

from test_first_use import PKG, play  # noqa: F401  (the fixture)

CODE = """
import sys
sys.path.insert(0, %r)
import warlib as w, serve
with serve.Server(max_jobs=16, mem_budget=8 * %d + 16 * serve.SIZEOF_DEVACC) as s:
    for n, flags in %r:
        s.wait_all([s.submit(w.make_job(n, 0, 0, flags, 0, 1000, sample_ppm=1000))])
        print(s.memo_info()["used_bytes"] // 8)
"""


@pytest.mark.parametrize("words,jobs,used", [
    # deals of 13 and 14 cards would take 2^28 words; those played merged take half of what is left
    (1 << 25, [(13, 0)], [1 << 24]),
    (1 << 25, [(13, 0), (14, 0)], [1 << 24, 3 << 23]),
    # sampled deals (flag 8) take all of it, as both do of a small arena
    (1 << 25, [(13, 8)], [1 << 25]),
    (1 << 25, [(13, 0), (14, 8)], [1 << 24, 1 << 25]),
    (1 << 23, [(13, 0)], [1 << 23]),
])
def test_words_taken(play, words, jobs, used):  # noqa: F811
    assert play(CODE % (PKG, words, jobs)) == used
