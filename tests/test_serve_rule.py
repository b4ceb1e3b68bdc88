"""How the server runs the 36^3 volumes of a batch (csrc/serve_rule.h), on the CPU: of
the four ways (each precision's by a list launch or as items) the shortest by the
estimate that its comment states, written down here once more."""
import ctypes
import math
import random

import pytest


@pytest.fixture()
def rule(hostcheck):
    f = hostcheck.hostcheck_cubes_by_list
    f.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong, ctypes.c_double]
    return f


def estimate(way, n, other_bytes, sms):
    lists = sum(12 + us * k for bit, us, k in ((1, 0.48, n[0]), (2, 0.26, n[1])) if way & bit)
    a, b = (0 if way & bit else k for bit, k in ((1, n[0]), (2, n[1])))
    # items of 98 and 49 us on `sms` SMs, those with one of 98 taking part in the second round
    last = 49 * (math.ceil(a / sms) + math.ceil((a + b) / sms))
    return lists + max(last, other_bytes / 2.3e6 + (98 * a + 49 * b) / sms)


def test_shortest_of_the_four(rule):
    r = random.Random(36)
    for _ in range(20000):
        n = [int(math.exp(r.uniform(0, 6.5))) if r.random() < 0.8 else 0 for _ in range(2)]
        other, sms = math.exp(r.uniform(10, 21)), r.choice([148, 148, 132, 20])
        way = rule(sms, *n, other)
        times = [estimate(w, n, other, sms) for w in range(4)]
        assert times[way] <= min(times) + 1e-9
        assert all(n[k] > 0 for k in range(2) if way >> k & 1)


@pytest.mark.parametrize("sms,n128,n64,other_mb,way", [
    (148, 0, 0, 0, 0), (148, 1, 0, 0, 1), (148, 0, 1, 0, 2), (148, 64, 64, 0, 3), (148, 2, 3, 500, 0),
    # the precisions together: 7 alone would take a list, and so would 82; 13 and 145 are more than one round
    (148, 7, 81, 157, 0), (148, 82, 7, 82, 0), (148, 13, 145, 94, 1), (148, 12, 191, 167, 0),
    # the device's own SMs: 30 volumes are two rounds of 20
    (148, 30, 0, 150, 1), (20, 30, 0, 150, 1), (148, 30, 0, 300, 0), (20, 30, 0, 300, 1)])
def test_examples(rule, sms, n128, n64, other_mb, way):
    assert rule(sms, n128, n64, other_mb * 1e6) == way
