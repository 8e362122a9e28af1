"""fomo_min_positive against numpy, and the staged model upload against the direct one."""
import numpy as np
import pytest


@pytest.mark.parametrize("n", [1, 15, 16, 17, 1000, 2 ** 21 + 3, 3 * 2 ** 21 - 1, 2 ** 23 + 5])
def test_min_positive(fomo, n):
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 4000, n).astype(np.float32)
    a[rng.integers(0, n, 3)] = [0.0, np.nan, -np.inf]
    a[n // 2] = 1e-42  # subnormal
    if n > 1:
        a[-1] = np.inf
    assert fomo.api._min_pos(a) == a[a > 0].min()
    a[a < 1.0] = 0.0
    if np.isfinite(a[a > 0]).any():
        assert fomo.api._min_pos(a) == a[a > 0].min()


def test_min_positive_none(fomo):
    for a in (np.zeros(40, np.float32), np.full(3, np.nan, np.float32), np.empty(0, np.float32)):
        with pytest.raises(fomo.ArgumentError):
            fomo.api._min_pos(a)


@pytest.mark.gpu
def test_staged_upload_equals_pinned(fomo):
    """A pageable model of over 16 MB goes through the pinned slots (several rounds of
    them, an odd tail), a pinned one directly."""
    import torch

    nx, nz = 4201, 2603
    vp = np.random.default_rng(0).uniform(2000, 3000, (nx, nz)).astype(np.float32, order="F")
    pin = torch.from_numpy(vp.T).pin_memory().numpy().T
    assert np.array_equal(pin, vp)
    rx = np.linspace(1, nx, 400).astype(int)
    kw = dict(sx=rx, sz=np.full(400, nz // 2), rx=rx, rz=np.full(400, nz // 2 + 1), nbc=4, fd_order=2)
    a = fomo.scalar2d(vp, 10.0, 1e-3, 6, 15.0, **kw)
    b = fomo.scalar2d(pin, 10.0, 1e-3, 6, 15.0, **kw)
    assert np.array_equal(a.seis_u, b.seis_u)
    assert np.abs(a.seis_u).max() > 0
