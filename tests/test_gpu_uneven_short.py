"""Uneven runs of fewer steps than the strip-width tuner times, on shapes that it has not met."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [1, 2, 3])
@pytest.mark.parametrize("order", [4, 8, 10])
def test_short_runs(fomo, nt, order):
    rng = np.random.default_rng(10 * order + nt)
    sizes = [(201 + nt, 34 + order), (60 + order, 40 + nt)]
    vps = [rng.uniform(2000, 3000, s).astype(np.float32, order="F") for s in sizes]
    rhos = [rng.uniform(1500, 2500, s).astype(np.float32, order="F") for s in sizes]
    rx = [np.arange(1, s[0] + 1) for s in sizes]
    kw = dict(sx=[[s[0] // 2, 3] for s in sizes], sz=[[9, 20]] * 2, rx=rx,
              rz=[np.full(r.size, 9) for r in rx], nbc=11, fd_order=order,
              wavelet=np.full(nt, 50.0, np.float32))
    out = [fomo.acoustic2d_uneven(vps, rhos, 10.0, 1e-3, nt, 15.0, kernel=k, **kw).shots
           for k in (0, 1, 2)]
    for s in range(2):
        assert np.abs(out[0][s][0]).max() > 0
        for a, b, c in zip(*(o[s] for o in out)):
            assert np.array_equal(a, b) and np.array_equal(b, c)
