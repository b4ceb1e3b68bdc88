"""Order on the legacy default stream.

Plans launch there with programmatic stream serialization too (a kernel's CTAs may
be placed while the one before it drains).  The stream's own order, and its implicit
order with blocking streams in both directions, must hold: each round writes a
buffer on one stream and reads it on the other without any event between them, as
the legacy semantics allow."""
import ctypes

import numpy as np
import pytest

import oracle
from conftest import field

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402

# a long kernel first, then a short one that reads its output: 2048 volumes of 17^3 take about 65 us
CASES = [((17, 17, 17), 2048, fb.C128), ((8, 8, 8), 4096, fb.C128), ((9, 25, 7), 700, fb.C128), ((64, 64, 64), 6, fb.C128)]


def cudart():
    name = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart.so" in line)
    return ctypes.CDLL(name)


@pytest.fixture()
def blocking_stream():
    rt, s = cudart(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(s)) == 0  # flags 0: synchronises with the legacy default stream
    yield s.value
    torch.cuda.synchronize()
    assert rt.cudaStreamDestroy(s) == 0


def buffers(shape, n):
    x = torch.from_numpy(field(np.random.default_rng(n), (n,) + shape)).cuda()
    return x, torch.empty_like(x), torch.empty_like(x)


def same_as_expected(z, x, shape):
    pick = slice(0, len(x), max(1, len(x) // 5))
    want = oracle.fft3d(oracle.fft3d(x[pick].cpu().numpy()))
    return oracle.rel_error_per_volume(z[pick].cpu().numpy(), want).max() < 2e-13  # two transforms of 1e-13


@pytest.mark.parametrize("shape,n,prec", CASES, ids=[str(c[0]) for c in CASES])
@pytest.mark.parametrize("first,second", [("default", "default"), ("default", "blocking"), ("blocking", "default")])
def test_output_of_one_stream_read_on_the_next(blocking_stream, shape, n, prec, first, second):
    stream = {"default": 0, "blocking": blocking_stream}
    x, y, z = buffers(shape, n)
    p = fb.Plan(shape, n, fb.FORWARD, prec)
    good = None
    for _ in range(30):
        y.zero_()
        z.zero_()
        p.execute(x.data_ptr(), y.data_ptr(), stream[first])
        p.execute(y.data_ptr(), z.data_ptr(), stream[second])
        torch.cuda.synchronize()
        if good is None:
            assert same_as_expected(z, x, shape)
            good = z.clone()
        assert torch.equal(z, good)
    p.close()


def test_torch_kernels_before_and_after():
    """torch's kernels carry no such attribute: one before a plan is waited for whole, and one after it waits."""
    x, y, z = buffers((17, 17, 17), 1024)
    p = fb.Plan((17, 17, 17), 1024)
    p.execute(x.data_ptr(), y.data_ptr())
    want = (2 * y).clone()
    src = torch.empty_like(x)
    for _ in range(30):
        y.zero_()
        src.zero_()
        torch.add(x, x, out=src)
        p.execute(src.data_ptr(), y.data_ptr())
        torch.mul(y, 1, out=z)
        torch.cuda.synchronize()
        assert torch.equal(z, want)  # doubling is exact
    p.close()
