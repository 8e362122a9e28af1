"""Small uneven batches cut their strips in z to have work for every SM; the cut
changes no result (the velocity / pressure kernels have no strips)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one shot of one strip, tall thin shots, flat wide ones, heights near the cuts
@pytest.mark.parametrize("sizes", [[(30, 40)], [(20, 700), (33, 511)], [(500, 20), (260, 70)],
                                   [(90, 96), (91, 193), (140, 31)],
                                   [(700, 300), (1, 1), (300, 9)]])
@pytest.mark.parametrize("fd_order", [4, 8, 10])
def test_uneven_cuts_equal_two_kernels(fomo, sizes, fd_order):
    rng = np.random.default_rng(fd_order)
    vps = [np.asfortranarray(rng.uniform(2000, 4000, s).astype(np.float32)) for s in sizes]
    rhos = [np.full(s, 2000.0, np.float32, order="F") for s in sizes]
    rx = [np.arange(1, nx + 1, 3) for nx, _ in sizes]
    kw = dict(sx=[(nx + 1) // 2 for nx, _ in sizes], sz=[max(nz - 3, 1) for _, nz in sizes], rx=rx,
              rz=[np.full(r.size, max(nz - 4, 1)) for r, (_, nz) in zip(rx, sizes)], nbc=7, fd_order=fd_order)
    a = fomo.acoustic2d_uneven(vps, rhos, 10.0, 1e-3, 90, 20.0, kernel=2, **kw)
    assert fomo.api.last_stats.kernel == 2
    d = fomo.acoustic2d_uneven(vps, rhos, 10.0, 1e-3, 90, 20.0, **kw)  # blocks per thread
    assert d.stats.tile == (128, 16)
    b = fomo.acoustic2d_uneven(vps, rhos, 10.0, 1e-3, 90, 20.0, kernel=1, **kw)
    for x, y, z in zip(a.shots, b.shots, d.shots):
        for p, q, r in zip(x, y, z):
            assert np.array_equal(p, q)
            assert np.array_equal(p, r)
            assert np.abs(p).max() > 0
