"""Chains of 17^3 and 24^3 on clusters of four CTAs (csrc/chain_kernels.cu
k_chain_cluster) and, beyond what fits the device at once, on one CTA a volume: both
sides of the line, uneven slabs (17 planes on four CTAs), no step at all."""
import numpy as np
import pytest

import oracle
from conftest import field

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fft3d_b200 as fb  # noqa: E402

TOL = {fb.C128: 1e-13, fb.C64: 1e-6}  # a transform; errors add up linearly at most


def steps_of(x, c, m):
    for _ in range(m):
        y = oracle.fft3d(x)
        if c is None:
            x = y / np.sqrt(np.prod(x.shape[1:]))
        else:
            y = y + c
            x = y / (1 + np.abs(y))
    return x


def clusters_at_once(chain):
    return int(chain.describe().split("up to ")[1].split()[0])


@pytest.mark.parametrize("side,batch", [(17, 1), (17, 30), (17, 37), (24, 2), (24, 33), (24, 38)])
@pytest.mark.parametrize("prec", [fb.C128, fb.C64])
@pytest.mark.parametrize("kind", [fb.CHAIN_UNITARY, fb.CHAIN_MAP])
def test_chain(side, batch, prec, kind):
    dt = np.complex128 if prec == fb.C128 else np.complex64
    rng = np.random.default_rng(side + batch)
    x = field(rng, (batch, side, side, side), dtype=dt)
    c = field(rng, x.shape, dtype=dt) if kind == fb.CHAIN_MAP else None
    a = torch.from_numpy(x).cuda()
    dc = torch.from_numpy(c).cuda() if c is not None else None
    out = torch.empty_like(a)
    chain = fb.Chain((side,) * 3, batch, kind, prec, dc.data_ptr() if dc is not None else 0)
    most = clusters_at_once(chain)
    assert most >= 30  # of the B200's 37 groups of four SMs
    assert ("a cluster of 4 CTAs a volume" in chain.describe()) == (batch <= most), chain.describe()
    pick = sorted({0, batch // 2, batch - 1})
    for m in (0, 1, 3):
        out.zero_()
        chain.run(a.data_ptr(), out.data_ptr(), m)
        torch.cuda.synchronize()
        want = steps_of(x[pick].astype(np.complex128), None if c is None else c[pick].astype(np.complex128), m)
        err = oracle.rel_error_per_volume(out.cpu().numpy()[pick].astype(np.complex128), want).max()
        assert err <= TOL[prec] * max(m, 1), (m, err)
    chain.close()


@pytest.mark.parametrize("side,prec", [(17, fb.C128), (17, fb.C64), (24, fb.C128), (24, fb.C64)])
def test_both_sides_of_the_line(side, prec):
    """As many volumes as have a cluster each, and one more; the smaller cubes have none."""
    dt = np.complex128 if prec == fb.C128 else np.complex64
    chain = fb.Chain((side,) * 3, 1, fb.CHAIN_UNITARY, prec)
    most = clusters_at_once(chain)
    for batch, cluster in ((most, True), (most + 1, False)):
        x = field(np.random.default_rng(batch), (batch, side, side, side), dtype=dt)
        a = torch.from_numpy(x).cuda()
        out = torch.zeros_like(a)
        chain = fb.Chain((side,) * 3, batch, fb.CHAIN_UNITARY, prec)
        assert ("cluster of 4" in chain.describe()) == cluster
        chain.run(a.data_ptr(), out.data_ptr(), 2)
        torch.cuda.synchronize()
        err = oracle.rel_error_per_volume(out.cpu().numpy()[-2:].astype(np.complex128),
                                          steps_of(x[-2:].astype(np.complex128), None, 2)).max()
        assert err <= 2 * TOL[prec], err
    assert "one CTA a volume" in fb.Chain((16, 16, 16), 1, fb.CHAIN_UNITARY, prec).describe()
