"""Device memory of the uneven batch (nine padded planes a shot and its acquisition) and the
launches it counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_models_are_staged_in_the_state(fomo, monkeypatch, kernel):
    import torch

    from fomo_b200 import _lib as L

    rng = np.random.default_rng(4)
    sizes = [(901, 700), (700, 903), (1100, 650), (640, 1201), (955, 777), (1201, 601)]
    vps = [rng.uniform(2000, 3000, s).astype(np.float32, order="F") for s in sizes]
    rhos = [rng.uniform(1500, 2500, s).astype(np.float32, order="F") for s in sizes]
    n, nbc, order = len(sizes), 5, 8
    kw = dict(sx=[[s[0] // 2] for s in sizes], sz=[[9]] * n, rx=[[s[0] // 2 + 3, s[0] // 2 - 6] for s in sizes],
              rz=[[12, 5]] * n,
              nbc=nbc, fd_order=order, kernel=kernel)
    call = lambda: fomo.acoustic2d_uneven(vps, rhos, 10.0, 1e-3, 40, 15.0, **kw)  # noqa: E731
    ref = call()  # the kernels are loaded
    fresh = L.Context(0)
    monkeypatch.setattr(L, "context", lambda device=0: fresh)
    before = torch.cuda.mem_get_info(0)[0]
    r = call()
    used = before - torch.cuda.mem_get_info(0)[0]
    pad = nbc + order // 2
    planes = sum(((a + 2 * pad + 31) // 32 * 32) * (b + 2 * pad) for a, b in sizes)
    # the workspace takes 1/16 more than it is asked for; 6 MB for tables and rounding
    assert used <= 4 * 9 * planes * 17 / 16 + 6e6, used
    for x, y in zip(r.shots, ref.shots):
        for a, b in zip(x, y):
            assert np.array_equal(a, b)
            assert np.abs(a).max() > 0


@pytest.mark.parametrize("nt,chunks", [(63, 0), (64, 2), (100, 3)])
def test_launches_counted(fomo, nt, chunks):
    """Three launches a step, and a step counter per replayed chunk of 32 steps."""
    vp = np.full((40, 31), 2500, np.float32, order="F")
    fomo.acoustic2d_uneven([vp, vp], [vp, vp], 10.0, 1e-3, nt, 15.0, sx=[[9]] * 2, sz=[[9]] * 2,
                           rx=[[3]] * 2, rz=[[4]] * 2, nbc=5)
    assert fomo.api.last_stats.gpu_launches == 3 * nt + chunks
