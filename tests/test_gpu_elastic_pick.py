"""AUTO's form for one large elastic shot: two-phase steps in blocks per thread where they
measured faster than the single sweep, the sweep elsewhere; same results either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,nbc,order,kernel", [
    (1950, 1900, 20, 10, 1), (300, 10000, 50, 10, 2), (8000, 420, 50, 10, 2), (2700, 2600, 20, 10, 2),
    (2700, 2600, 20, 8, 1), (2300, 2200, 100, 8, 2), (300, 10000, 50, 4, 2), (2400, 2300, 20, 2, 1),
])
def test_pick(fomo, nx, nz, nbc, order, kernel):
    rng = np.random.default_rng(order)
    vp = rng.uniform(2000, 3000, (nx, nz)).astype(np.float32, order="F")
    vs, rho = np.asfortranarray(vp / np.float32(1.8)), np.full((nx, nz), 2000, np.float32, order="F")
    rx = np.arange(1, nx + 1, 7)
    kw = dict(sx=rx, sz=np.full(rx.size, 3), rx=rx, rz=np.full(rx.size, 6), nbc=nbc, fd_order=order)
    a = fomo.elastic2d(vp, vs, rho, 10.0, 1e-3, 12, 15.0, **kw)
    assert fomo.api.last_stats.kernel == kernel
    b = fomo.elastic2d(vp, vs, rho, 10.0, 1e-3, 12, 15.0, kernel=3 - kernel, **kw)
    assert fomo.api.last_stats.kernel == 3 - kernel
    assert np.array_equal(a.seis_vx, b.seis_vx) and np.array_equal(a.seis_vz, b.seis_vz)
    assert np.abs(a.seis_vz).max() > 0
