"""Which batches share the result of a strategy race (csrc/batch_choice.h), on the
CPU: only those whose race would time the same launches."""
import ctypes

import pytest

import fft3d_b200 as fb

BASE = 1 << 40  # addresses are never touched


def segments(n_mb=15, offset_in=0, offset_out=0, **change):
    """Four 16^3 complex64 segments of n_mb MB of input and output each."""
    batch = n_mb * 1048576 // (2 * 8 * 16 ** 3)
    segs = [{"shape": (16, 16, 16), "batch": batch, "direction": fb.FORWARD, "precision": fb.C64,
             "in": BASE + (k << 32) + offset_in, "out": BASE + (k << 32) + (1 << 31) + offset_out} for k in range(4)]
    segs[2].update(change)
    return segs


@pytest.fixture()
def same(hostcheck):
    def f(a, b):
        return bool(hostcheck.hostcheck_same_choice(fb._segments(a), len(a), fb._segments(b), len(b)))
    return f


def test_other_buffers_share(same):
    a, b = segments(), segments()
    for s in b:
        s["in"] += 1 << 24
        s["out"] += 16
    assert same(a, b)
    # off 16 bytes alike
    assert same(segments(offset_in=8, offset_out=24), segments(offset_in=40, offset_out=8))


@pytest.mark.parametrize("a,b", [
    # one size class of counts, on either side of the 16 MB from which widths are timed, and on one side of it
    (segments(15), segments(17)), (segments(17), segments(25)),
    (segments(), segments(batch=1)), (segments(), segments(batch=0)),
    (segments(), segments(offset_in=8)), (segments(), segments(offset_out=8)),
    (segments(offset_in=8), segments(offset_out=8)),
    (segments(), segments(direction=fb.BACKWARD)), (segments(), segments(precision=fb.C128)),
    (segments(), segments(shape=(16, 16, 32))), (segments(), segments()[:3]),
    (segments(batch=7), segments(batch=7)[::-1])])
def test_others_race_for_themselves(same, a, b):
    assert not same(a, b)
    assert same(a, list(a)) and same(b, list(b))


@pytest.mark.parametrize("t_seg,t_persist,kept", [(0.1, 0.2, True), (0.0, 0.2, False), (0.1, 0.0, False), (1e30, 0.2, False),
                                                  (0.1, 1e30, False), (float("nan"), 0.2, False), (-1.0, 0.2, False)])
def test_only_measured_times_are_kept(hostcheck, t_seg, t_persist, kept):
    f = hostcheck.hostcheck_race_measured
    f.argtypes = [ctypes.c_float, ctypes.c_float]
    assert bool(f(t_seg, t_persist)) == kept
