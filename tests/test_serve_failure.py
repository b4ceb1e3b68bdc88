"""A server launch whose bounded wait runs out, without a GPU fault (needs a B200).

The list launch over 36^3 volumes is started at its first row item's ticket, so the
planes of its first volume never come and it ends after the wait's bound with outputs
missing.  Its requests must not be reported as completed; the next ones are served."""
import numpy as np
import pytest

import oracle
from conftest import field

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402


def requests(shape, n, prec):
    x = field(np.random.default_rng(n), (n,) + shape, dtype=np.complex128 if prec == fb.C128 else np.complex64)
    a = torch.from_numpy(x).cuda()
    b = torch.zeros_like(a)
    return x, a, b, {"shape": shape, "batch": n, "precision": prec, "in": a.data_ptr(), "out": b.data_ptr()}


@pytest.mark.parametrize("prec", [fb.C128, fb.C64])
def test_missing_outputs_are_not_completed(prec):
    x, a, b, cubes = requests((36, 36, 36), 40, prec)
    x2, a2, b2, others = requests((17, 17, 17), 9, prec)
    srv = fb.Server(4 << 30, max_inflight=1)
    lib = fb.lib()
    assert lib.fft3d_b200_debug_stall_next_list(srv._h) == fb.OK
    srv.submit(cubes)
    with pytest.raises(fb.Fft3dError) as e:
        srv.drain(30)
    assert e.value.status == fb.ERR_TIMEOUT
    with pytest.raises(fb.Fft3dError) as e:  # no ticket, and not "nothing yet"
        srv.poll()
    assert e.value.status == fb.ERR_TIMEOUT
    # served again: the counters and the error word are clear
    later = [srv.submit(cubes), srv.submit(others)]
    with pytest.raises(fb.Fft3dError):
        srv.drain(30)
    assert sorted(srv.poll()) == later
    srv.close()
    torch.cuda.synchronize()
    tol = 1e-13 if prec == fb.C128 else 1e-6  # as for every other request
    for got, want in ((b, x[::7]), (b2, x2)):
        got = got.cpu().numpy()[::7] if len(got) == 40 else got.cpu().numpy()
        assert oracle.rel_error_per_volume(got.astype(np.complex128), oracle.fft3d(want.astype(np.complex128))).max() < tol


def test_hook_refuses_a_server_without_lists():
    srv = fb.Server(1 << 30, max_inflight=1, flags=fb.SERVE_PLAIN)
    assert fb.lib().fft3d_b200_debug_stall_next_list(srv._h) == fb.ERR_UNSUPPORTED
    srv.close()
