"""What the library does on its first use (csrc/war_capi.cu, ensure_ready; csrc/war_server.cu, war_server_create), on
the CPU with a fake CUDA runtime (fake_cudart.c) loaded before the real one, in a process of its own."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "endless-games-of-war_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def play(tmp_path_factory):
    """Runs Python code with `war` (libwar.so) and `fake` (the runtime's counters); returns what it printed."""
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I" + os.path.join(CUDA, "include"), "-o", so,
                    os.path.join(HERE, "fake_cudart.c")], check=True)
    head = ("import ctypes, threading\n"
            "fake = ctypes.CDLL(%r)\n"
            "war = ctypes.CDLL(%r)\n" % (so, os.path.join(PKG, "libwar.so")))

    def run(code):
        p = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=60,
                           env=dict(os.environ, LD_PRELOAD=so))
        assert p.returncode == 0, p.stderr
        return [int(x) for x in p.stdout.split()]
    return run


def test_tables_are_on_the_device_before_the_first_launch(play):
    """The pair lists are read on a non-blocking stream, which waits for no other: the upload is waited for."""
    assert play("print(war.war_set_stream(None), fake.fake_unsynced())") == [0, 0]


def test_server_tables_are_on_the_device_before_the_first_launch(play):
    assert play("h = ctypes.c_void_p()\n"
                "print(war.war_server_create(None, ctypes.byref(h)), fake.fake_unsynced())\n"
                "war.war_server_destroy(h)\n") == [0, 0]


def test_first_use_by_several_threads(play):
    """The context is made once: a thread that came second would replace its buffers under the first one's job."""
    one = play("print(war.war_set_stream(None), fake.fake_streams_made(), fake.fake_live())")
    two = play("t = [threading.Thread(target=war.war_set_stream, args=(None,)) for _ in range(4)]\n"
               "[x.start() for x in t]\n[x.join() for x in t]\n"
               "print(war.war_set_stream(None), fake.fake_streams_made(), fake.fake_live())")
    assert one[:2] == [0, 1] and two == one


def test_first_use_that_fails_gives_back_what_it_had(play):
    """The upload of the pair lists fails twice: nothing is left, and the third call makes one whole context."""
    one = play("print(war.war_set_stream(None), fake.fake_live())")
    got = play("fake.fake_fail_copies(2)\n"
               "for i in range(3): print(war.war_set_stream(None), fake.fake_live())")
    ecuda = -2
    assert got == [ecuda, 0, ecuda, 0] + one
