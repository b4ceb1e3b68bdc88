"""TWOPASS with planes and rows copied in bulk at 30^3 complex128: one volume, fewer
volumes than the ring has slots, and more, so that slots are taken again."""
import numpy as np
import pytest

import oracle
from conftest import field
from test_hostcheck import C128_TOL

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402

NAMES = ["twopass 30x30x30 double g2 bulkqh nt64 minb6", "twopass 30x30x30 double g3 bulkqh nt96 minb4"]


@pytest.mark.parametrize("variant", NAMES)
@pytest.mark.parametrize("n", [1, 7, 700])
@pytest.mark.parametrize("direction", [fb.FORWARD, fb.BACKWARD])
def test_30_cubed(variant, n, direction):
    """The lines are the one-thread codelets that the CPU check runs: its tolerance."""
    x = field(np.random.default_rng(3000 + n), (min(n, 7), 30, 30, 30), dist="normal")
    a = torch.from_numpy(x).cuda().repeat((n + 6) // 7, 1, 1, 1)[:n].contiguous()
    b = torch.empty_like(a)
    plan = fb.Plan((30, 30, 30), n, direction, fb.C128, variant=variant)
    for _ in range(2):  # the second finds the counters of the first
        b.zero_()
        plan.execute(a.data_ptr(), b.data_ptr())
        plan.check()
        want = oracle.fft3d(x) if direction == fb.FORWARD else oracle.ifft3d(x)
        assert oracle.rel_error_per_volume(b[:len(x)].cpu().numpy(), want).max() < C128_TOL
        # every repetition of a volume holds the same bits
        k = len(x)
        for v in range(k, n, k):
            assert torch.equal(b[v:v + k], b[:min(k, n - v)])
