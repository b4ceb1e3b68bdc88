"""The server's 36^3 volumes: a list launch of their own, or items of the persistent
kernel beside a large batch (csrc/serve_rule.h).  Either way every
volume matches the oracle and is the same, bit for bit, as alone in a pinned
persistent batch."""
import numpy as np
import pytest

import oracle
from conftest import field

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402

C128_TOL, C64_TOL = 1e-13, 1e-6


def request(side, n, direction, prec, offset=0):
    """`offset`: bytes past a 16-byte boundary (complex64 needs only 8)."""
    dt = np.complex128 if prec == fb.C128 else np.complex64
    x = field(np.random.default_rng(side + n + direction), (n, side, side, side), dtype=dt)
    eb = x.itemsize
    raw = [torch.zeros(x.nbytes + 16, dtype=torch.uint8, device="cuda") for _ in range(2)]
    view = [r[offset:offset + x.nbytes].view(torch.complex128 if eb == 16 else torch.complex64).view(x.shape) for r in raw]
    view[0].copy_(torch.from_numpy(x))
    seg = {"shape": (side,) * 3, "batch": n, "direction": direction, "precision": prec,
           "in": view[0].data_ptr(), "out": view[1].data_ptr()}
    return seg, x, view[1], raw


# cubes (volumes, direction, precision, offset) and volumes of 17^3 beside them: one, fewer and more than the SMs;
# both directions and precisions in one launch; an input off 16 bytes; few beside 0.5 GB, which stay in the batch;
# list launches
CASES = [([(1, fb.FORWARD, fb.C128, 0)], 0, 1),
         ([(64, fb.BACKWARD, fb.C128, 0), (37, fb.FORWARD, fb.C128, 0), (5, fb.BACKWARD, fb.C64, 0)], 3, 2),
         ([(50, fb.FORWARD, fb.C64, 0), (3, fb.FORWARD, fb.C64, 8), (64, fb.BACKWARD, fb.C64, 0)], 20, 1),
         ([(2, fb.FORWARD, fb.C128, 0), (3, fb.BACKWARD, fb.C64, 0)], 3500, 0)]


@pytest.fixture(scope="module")
def ahead():
    """About a millisecond of work: what is submitted behind it on the one slot becomes one batch."""
    x = torch.zeros((16000, 17, 17, 17), dtype=torch.complex128, device="cuda")
    y = torch.empty_like(x)
    yield {"shape": (17, 17, 17), "batch": len(x), "in": x.data_ptr(), "out": y.data_ptr()}, x, y


@pytest.mark.parametrize("cubes,others,lists", CASES)
def test_cubes(ahead, cubes, others, lists):
    work = [request(36, *c) for c in cubes]
    if others:
        work.append(request(17, others, fb.FORWARD, fb.C128))
    torch.cuda.synchronize()
    srv = fb.Server(8 << 30, max_inflight=1)
    for _ in range(2):  # the second time with the workspace there
        launches = srv.stats()["launches"]
        srv.submit(ahead[0])
        while srv.stats()["launches"] == launches:
            pass
        srv.submit_many([w[0] for w in work])
        srv.drain(60)
    assert srv.list_launches() == 2 * lists
    srv.close()
    torch.cuda.synchronize()
    for seg, x, out, raw in work:
        alone = torch.empty_like(out)
        b = fb.Batch([dict(seg, out=alone.data_ptr())], flags=fb.BATCH_PERSISTENT)
        b.execute()
        torch.cuda.synchronize()
        assert torch.equal(alone, out), seg
        b.close()
        pick = slice(0, len(x), max(1, len(x) // 4))
        x64 = x[pick].astype(np.complex128)
        want = oracle.fft3d(x64) if seg["direction"] == fb.FORWARD else oracle.ifft3d(x64)
        err = oracle.rel_error_per_volume(out[pick].cpu().numpy().astype(np.complex128), want).max()
        assert err < (C128_TOL if seg["precision"] == fb.C128 else C64_TOL), seg


def test_requests_of_their_own_hide_no_items(ahead):
    """45^3 has no kind in the persistent kernel: launched before the batch, 0.3 GB of it
    leaves the cubes' items as exposed as without it."""
    work = [request(36, 20, fb.FORWARD, fb.C128), request(45, 100, fb.FORWARD, fb.C128)]
    torch.cuda.synchronize()
    srv = fb.Server(8 << 30, max_inflight=1)
    srv.submit(ahead[0])
    while srv.stats()["launches"] == 0:
        pass
    srv.submit_many([w[0] for w in work])
    srv.drain(60)
    assert srv.list_launches() == 1
    srv.close()
    for _, x, out, _ in work:
        assert oracle.rel_error_per_volume(out[::19].cpu().numpy(), oracle.fft3d(x[::19])).max() < C128_TOL
