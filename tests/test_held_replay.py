"""The held-out-card engine plays odd decks under the winner's card first with the run test, and again without it if
that left a game open (csrc/war_capi.cu, war_enumerate_held).  No deck is known to leave one, so the second pass is
tested on the CPU, with a CUDA runtime whose launches leave given accumulators."""
import pytest

from test_first_use import PKG, play  # noqa: F401  (the fixture)

WORD = {"cyc": 0, "done": 1, "maxfin": 2, "turns": 3, "undetermined": 19, "hist0": 20}
CODE = """
import sys
sys.path.insert(0, %r)
import warlib
job = warlib.make_job(%d, rule=%d, lo=1000, hi=2000, hbins=4)
r = warlib.Result()
for launch, word, v in %r: fake.fake_set_word(launch, word, ctypes.c_ulonglong(v))
st = war.war_enumerate_held(ctypes.byref(job), None, ctypes.byref(r))
print(st, fake.fake_launches(), fake.fake_same_kernel(0, 1), r.cyc, r.done, r.maxfin, r.turns, r.undetermined, r.hist[0])
"""


def run(play, n, rule, first, second):  # noqa: F811
    words = [(i, WORD[k], v) for i, d in enumerate((first, second)) for k, v in d.items()]
    return play(CODE % (PKG, n, rule, words))


FIRST = dict(cyc=7, done=900, maxfin=65537, turns=11, hist0=3)
SECOND = dict(cyc=8, done=1000, maxfin=99, turns=12, hist0=2)


def test_a_job_that_left_a_game_open_is_played_again_from_nothing(play):  # noqa: F811
    """Nothing of the first pass is left in the result, and the second is another kernel."""
    got = run(play, 17, 0, dict(FIRST, undetermined=1), SECOND)
    assert got == [0, 2, 0, 8, 1000, 99, 12, 0, 2]


@pytest.mark.parametrize("n,rule", [(17, 0), (17, 1), (16, 0), (13, 0)])
def test_a_job_that_decided_every_game_is_played_once(play, n, rule):  # noqa: F811
    got = run(play, n, rule, FIRST, SECOND)
    assert got[:2] + got[3:] == [0, 1, 7, 900, 65537, 11, 0, 3]
