"""Binary16 batches whose absorbing layers leave the shot-pair sweep no room for its ramps run
the one-shot binary16 sweep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbc,pair", [(2900, True), (2940, False)])
def test_thick_layers(fomo, nbc, pair):
    rng = np.random.default_rng(nbc)
    nx, nz = 24, 17
    vp = rng.uniform(2000, 3000, (nx, nz)).astype(np.float32, order="F")
    vs = np.asfortranarray(vp / np.float32(1.8))
    rho = rng.uniform(1500, 2500, (nx, nz)).astype(np.float32, order="F")
    kw = dict(sx=[6, 20], sz=[5, 9], rx=[3, 9, 21], rz=[8, 6, 11], nbc=nbc, fd_order=10,
              precision="fp16")
    out = []
    for kernel in (0, 1):
        out.append(fomo.elastic2d_batch(vp, vs, rho, 10.0, 1e-3, 30, 40.0, kernel=kernel, **kw))
        st = fomo.api.last_stats
        assert st.kernel == (1 if kernel else 2)
        if not kernel:
            assert (st.sweep_config // 1000000 == 24) == pair
    for a, b in zip(out[0][:2], out[1][:2]):
        assert np.array_equal(a, b)
        assert np.abs(a).max() > 0
