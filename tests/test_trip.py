"""TRIP kernel (csrc/trip.cuh, csrc/trip_kernels.cu): lines split over tasks.

The three trips of a plane item and the two of a row item run on the CPU
(hostcheck, alg = 800 + G) in ticket order against the oracle; the GPU kernel is
a variant of its extent and is run with all others by test_gpu_parity.py.  Its
control warp's bounded wait is tested here."""
import ctypes

import numpy as np
import pytest

import oracle
from conftest import field
from test_hostcheck import C64_TOL, C128_TOL, run

CASES = [(64, 0, 1, 1), (64, 0, 1, 3)]  # (N, precision, G, batch)


@pytest.mark.parametrize("n,prec,g,nvol", CASES, ids=[f"{c[0]}-c{64 if c[1] else 128}-g{c[2]}-b{c[3]}" for c in CASES])
@pytest.mark.parametrize("sign", [-1, +1])
def test_trip_items(hostcheck, n, prec, g, nvol, sign):
    """Same tolerances as the one-thread-per-line passes: the split changes the
    order of the sums, not their length (log2 N stages of rounding)."""
    hostcheck.hostcheck_twopass_violations.restype = ctypes.c_longlong
    hostcheck.hostcheck_twopass_violations()
    rng = np.random.default_rng(11000 + n + 10 * g + nvol + prec)
    x = field(rng, (nvol, n, n, n), dist="normal", dtype=np.complex128 if prec == 0 else np.complex64)
    got = run(hostcheck, x, (n, n, n), prec, sign, 800 + g, 1)
    assert hostcheck.hostcheck_twopass_violations() == 0
    x64 = x.astype(np.complex128)
    want = oracle.fft3d(x64) if sign < 0 else oracle.ifft3d(x64)
    assert oracle.rel_error_per_volume(got, want).max() < (C128_TOL if prec == 0 else C64_TOL)


@pytest.mark.gpu
def test_control_warp_gives_up_and_recovers():
    """The first volume's plane items are skipped, so a row item's planes never
    come: the launch ends by itself, the wait is reported, and the next launch is
    whole."""
    torch = pytest.importorskip("torch")
    import fft3d_b200 as fb
    rng = np.random.default_rng(64)
    x = field(rng, (20, 64, 64, 64), dist="normal")
    a = torch.from_numpy(x).cuda()
    b = torch.empty_like(a)
    plan = fb.Plan((64, 64, 64), len(x), fb.FORWARD, fb.C128, variant="twopass 64x64x64 double g1 trip nt256 minb2")
    assert fb.lib().fft3d_b200_debug_stall_next_execute(plan.handle) == fb.OK
    plan.execute(a.data_ptr(), b.data_ptr())
    with pytest.raises(fb.Fft3dError) as e:
        plan.check()
    assert e.value.status == fb.ERR_TIMEOUT
    plan.execute(a.data_ptr(), b.data_ptr())
    plan.check()
    assert oracle.rel_error_per_volume(b.cpu().numpy()[::7], oracle.fft3d(x[::7])).max() < C128_TOL
