"""complex64 buffers need 8-byte alignment only, and bulk copies 16: every variant
that moves its input in bulk takes inputs and outputs off a 16-byte boundary."""
import numpy as np
import pytest

import oracle
from conftest import field

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402

C64_TOL = 1e-6
# the extents whose volumes are copied row by row, and odd volumes copied whole; volumes enough that a CTA takes several
CASES = [((30, 30, 30), 300), ((36, 36, 36), 60), ((45, 45, 45), 9), ((64, 64, 64), 5), ((9, 25, 7), 1500), ((15, 15, 15), 700)]


@pytest.mark.parametrize("shape,n", CASES, ids=[str(c[0]) for c in CASES])
@pytest.mark.parametrize("offset_in,offset_out", [(8, 0), (8, 8)])
def test_complex64_off_16_bytes(shape, n, offset_in, offset_out):
    x = field(np.random.default_rng(sum(shape)), (n,) + shape, dtype=np.complex64)
    raw = [torch.zeros(x.nbytes + 16, dtype=torch.uint8, device="cuda") for _ in range(2)]
    a, b = (r[o:o + x.nbytes].view(torch.complex64).view(x.shape) for r, o in zip(raw, (offset_in, offset_out)))
    a.copy_(torch.from_numpy(x))
    pick = slice(0, n, max(1, n // 6))
    want = oracle.fft3d(x[pick].astype(np.complex128))
    for v in fb.variants(shape, fb.C64):
        b.zero_()
        plan = fb.Plan(shape, n, fb.FORWARD, fb.C64, variant=v)
        plan.execute(a.data_ptr(), b.data_ptr())
        plan.check()
        err = oracle.rel_error_per_volume(b[pick].cpu().numpy().astype(np.complex128), want).max()
        assert err < C64_TOL, (v, err)
        plan.close()


def microseconds(plan, a, b):
    best = float("inf")
    for _ in range(4):
        t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        t[0].record()
        for _ in range(10):
            plan.execute(a.data_ptr(), b.data_ptr())
        t[1].record()
        torch.cuda.synchronize()
        best = min(best, t[0].elapsed_time(t[1]) * 100)
    return best


# a plan is tuned on aligned buffers and takes any: (shape, volumes, what is slowest allowed against VOLUME)
SLOWEST = [((30, 30, 30), 300, 1.25),    # 0.98 measured; 1.7 when one thread copied a chunk of rows
           ((15, 15, 15), 1864, 1.1),    # 0.88; 1.23 when an item's threads waited for their copies
           ((3, 5, 7), 59918, 1.1)]      # 0.99; 1.2 likewise


@pytest.mark.parametrize("shape,n,most", SLOWEST, ids=[str(c[0]) for c in SLOWEST])
def test_plans_off_16_bytes_keep_their_speed(shape, n, most):
    raw = [torch.zeros(8 * n * int(np.prod(shape)) + 16, dtype=torch.uint8, device="cuda")[8:] for _ in range(2)]
    names = fb.variants(shape, fb.C64)
    plans = [fb.Plan(shape, n, fb.FORWARD, fb.C64), fb.Plan(shape, n, fb.FORWARD, fb.C64, variant=next(
        v for v in names if v.startswith("volume")))]
    tuned, volume = [microseconds(p, *raw) for p in plans]
    assert tuned < most * volume, (plans[0].describe(), tuned, volume)
