"""Batches whose segments fill the GPU: several widths of branches are timed, and a
second batch of the same segments takes over what the first found."""
import numpy as np
import pytest

import oracle
from conftest import field
from test_hostcheck import C64_TOL

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402

SHAPES = [(8, 8, 8), (12, 12, 12), (16, 16, 16), (24, 24, 24)]
SIZES = [9 << 20, 0]  # input bytes a segment; 0: three volumes, where widths are not timed


@pytest.mark.parametrize("bytes_in", SIZES)
@pytest.mark.parametrize("flags", [0, fb.FLAG_NO_GRAPH])
@pytest.mark.parametrize("nseg", [4, 7])
def test_second_batch_of_the_same_segments(bytes_in, flags, nseg):
    rng = np.random.default_rng(nseg)
    x8 = [field(rng, (3,) + SHAPES[k % 4], "uniform", np.complex64) for k in range(nseg)]
    ns = [max(3, bytes_in // (8 * int(np.prod(SHAPES[k % 4])))) for k in range(nseg)]
    ins = [torch.from_numpy(x).cuda().repeat((n + 2) // 3, 1, 1, 1)[:n].contiguous() for x, n in zip(x8, ns)]
    wants = [oracle.fft3d(x.astype(np.complex128)) for x in x8]
    notes = []
    for _ in range(2):
        outs = [torch.zeros_like(a) for a in ins]
        batch = fb.Batch([dict(shape=SHAPES[k % 4], batch=ns[k], direction=fb.FORWARD, precision=fb.C64,
                               **{"in": ins[k].data_ptr()}, out=outs[k].data_ptr()) for k in range(nseg)], flags=flags)
        notes.append(batch.describe())
        for o in outs:
            o.zero_()
        batch.execute()
        torch.cuda.synchronize()
        for k in range(nseg):
            got = outs[k][[0, 1, 2, ns[k] - 1]].cpu().numpy().astype(np.complex128)
            want = np.concatenate([wants[k], wants[k][(ns[k] - 1) % 3:][:1]])
            assert oracle.rel_error_per_volume(got, want).max() < C64_TOL, k
    # the second raced nothing: the first's choice, and its times as an earlier batch's
    assert notes[1] == notes[0].replace(" us)", " us; by an earlier batch)")
    assert "by an earlier batch" in notes[1]


def test_forgotten_with_the_plans_choices(tmp_path):
    """A batch's choice was timed with the kernels that the plans' choices name."""
    a = torch.zeros((500, 12, 12, 12), dtype=torch.complex128, device="cuda")
    b = torch.zeros_like(a)

    def remembered():
        batch = fb.Batch([dict(shape=(12, 12, 12), batch=250, **{"in": a[k:].data_ptr()}, out=b[k:].data_ptr())
                          for k in (0, 250)])
        note = batch.describe()
        batch.close()
        assert "timed" in note
        return "by an earlier batch" in note

    fb.wisdom_forget()
    assert [remembered(), remembered()] == [False, True]
    fb.wisdom_forget()
    assert [remembered(), remembered()] == [False, True]
    fb.wisdom_export(tmp_path / "w.txt")
    assert remembered()
    assert fb.wisdom_import(tmp_path / "w.txt") > 0
    assert [remembered(), remembered()] == [False, True]
    fb.wisdom_forget()
