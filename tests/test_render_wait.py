"""CPU tests of dbmp_render_wait: it returns when every candidate's flag is there, and
behind a long queue it does not hold a core."""
import ctypes
import threading
import time

from diffbmp_b200._lib import DBMP_ERR_INVALID, lib


def wait(delays):
    """(wall, processor) seconds of a wait whose candidates report after `delays`."""
    flags = (ctypes.c_int32 * (2 * len(delays)))(*[0, -1] * len(delays))

    def report():
        t0 = time.monotonic()
        for d, b in sorted((d, b) for b, d in enumerate(delays)):
            time.sleep(max(0.0, d - (time.monotonic() - t0)))
            flags[2 * b] = 10 + b
            flags[2 * b + 1] = b % 2
    t = threading.Thread(target=report)
    t.start()
    wall, busy = time.monotonic(), time.thread_time()
    assert lib.dbmp_render_wait(flags, len(delays), None) == 0
    wall, busy = time.monotonic() - wall, time.thread_time() - busy
    t.join()
    assert [flags[2 * b] for b in range(len(delays))] == [10 + b for b in range(len(delays))]
    return wall, busy


def test_wait_returns_with_the_last_flag():
    assert wait([0.0])[0] < 0.5
    assert 0.05 <= wait([0.05, 0.0, 0.02])[0] + 0.005


def test_a_long_wait_sleeps():
    wall, busy = wait([0.0, 0.6])
    assert wall >= 0.55
    assert busy < 0.25 * wall       # the sleeps themselves take a few per cent


def test_no_flags_is_an_error():
    assert lib.dbmp_render_wait(None, 1, None) == DBMP_ERR_INVALID
