"""Runs that keep their state on the chip (resident2d.cuh) equal the same run
launched step by step, bit for bit: seismograms, snapshots and final fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT = 310  # over the 300 steps from which a run is kept on the chip


@pytest.fixture
def both(monkeypatch, fomo):
    """(on-chip result, launches, step-by-step result) of one call."""
    from fomo_b200 import _lib as L

    orig = fomo.api._opts

    def step_opts(*a, **kw):
        o = orig(*a, **kw)
        o.flags |= L.FOMO_F_STEP_LAUNCH
        return o

    def run(fn, *a, final=None, **kw):
        out = []
        for f in (orig, step_opts):
            monkeypatch.setattr(fomo.api, "_opts", f)
            fin = np.zeros(final, np.float32, order="F") if final else None
            r = fn(*a, **kw, **({"final_state": fin} if final else {}))
            out.append((r, fin, fomo.api.last_stats.gpu_launches))
        monkeypatch.setattr(fomo.api, "_opts", orig)
        assert out[0][2] <= 16 < out[1][2]
        return out[0][:2], out[1][:2]

    return run


def _same(a, b):
    for x, y in zip(a, b):
        if isinstance(x, np.ndarray):
            assert np.array_equal(x, y)
            assert np.isfinite(x).all()
        elif isinstance(x, list):
            assert len(x) == len(y)
            for p, q in zip(x, y):
                assert np.array_equal(p, q)


def _layers(nx, nz, seed):
    rng = np.random.default_rng(seed)
    vp = np.empty((nx, nz), np.float32, order="F")
    cuts = np.linspace(0, nz, 5).astype(int)
    for k in range(4):
        vp[:, cuts[k]:cuts[k + 1]] = rng.uniform(2000, 4000)
    rho = np.asfortranarray((310 * vp ** 0.25).astype(np.float32))
    return vp, rho


# one tile's width and height, ragged tiles, a grid too flat or too narrow for
# many tiles, no absorbing layer beyond the stencil, larger blocks per thread,
# materials off the chip
SIZES = [(33, 29, 10), (171, 90, 12), (401, 7, 3), (5, 260, 6), (120, 100, 1), (640, 470, 20),
         (910, 760, 20)]


@pytest.mark.parametrize("nx,nz,nbc", SIZES)
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
def test_acoustic2d_on_chip(fomo, both, nx, nz, nbc, order):
    vp, rho = _layers(nx, nz, nx + order)
    vp[:, 0] = rho[:, 0] = 0.0
    vp[: nx // 3, 0] = 1800.0
    rho[: nx // 3, 0] = 1900.0
    pad = nbc + order // 2
    rx = np.arange(1, nx + 1, 3)
    kw = dict(sx=[nx // 2 + 1, 1, nx], sz=[nz // 2 + 1, 1, nz], rx=rx,
              rz=np.full(rx.size, min(3, nz)), nbc=nbc, fd_order=order, snap_interval=35)
    a, b = both(fomo.acoustic2d, vp, rho, 10.0, 1e-3, NT, 15.0,
                final=(nx + 2 * pad, nz + 2 * pad, 3), **kw)
    _same(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert np.abs(a[0].seis_p).max() > 0


@pytest.mark.parametrize("nx,nz,nbc", SIZES[:-2] + [(430, 330, 20), (620, 540, 9)])
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
def test_elastic2d_on_chip(fomo, both, nx, nz, nbc, order):
    vp, rho = _layers(nx, nz, nx + order)
    vs = np.asfortranarray((vp / 1.8).astype(np.float32))
    vs[:, : nz // 4] = 0.0  # water
    vp[: nx // 3, 0] = rho[: nx // 3, 0] = 0.0
    pad = nbc + order // 2
    rx = np.arange(1, nx + 1, 3)
    kw = dict(sx=[nx // 2 + 1, 1, nx], sz=[nz // 2 + 1, 1, nz], rx=rx,
              rz=np.full(rx.size, min(3, nz)), nbc=nbc, fd_order=order, snap_interval=35)
    a, b = both(fomo.elastic2d, vp, vs, rho, 10.0, 1e-3, NT, 15.0,
                final=(nx + 2 * pad, nz + 2 * pad, 5), **kw)
    _same(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert np.abs(a[0].seis_vz).max() > 0


@pytest.mark.parametrize("order", [2, 8, 10])
def test_elastic2d_sponge_and_batch_on_chip(fomo, both, order):
    vp, rho = _layers(150, 111, 4)
    vs = np.asfortranarray((vp / 1.8).astype(np.float32))
    kw = dict(rx=np.arange(1, 151, 4), rz=np.full(38, 9), nbc=20, fd_order=order)
    a, b = both(fomo.elastic2d, vp, vs, rho, 10.0, 1e-3, NT, 15.0, sx=[70], sz=[9],
                boundary="sponge", snap_interval=100, **kw)
    _same(a[0], b[0])
    a, b = both(fomo.elastic2d_batch, vp, vs, rho, 10.0, 1e-3, NT, 15.0, sx=[20, 75, 140],
                sz=[4, 9, 100], **kw)
    _same(a[0], b[0])


@pytest.mark.parametrize("nx,nz,nbc", SIZES)
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
def test_scalar2d_on_chip(fomo, both, nx, nz, nbc, order):
    vp, _ = _layers(nx, nz, nx + order)
    pad = nbc + order // 2
    rx = np.arange(1, nx + 1, 3)
    kw = dict(sx=[nx // 2 + 1, 1, nx], sz=[nz // 2 + 1, 1, nz], rx=rx,
              rz=np.full(rx.size, min(3, nz)), nbc=nbc, fd_order=order)
    a, b = both(fomo.scalar2d, vp, 10.0, 1e-3, NT, 15.0,
                final=(nx + 2 * pad, nz + 2 * pad, 2), **kw)
    _same(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert np.abs(a[0].seis_u).max() > 0


@pytest.mark.parametrize("nx,nz,nbc", SIZES[:-2] + [(410, 310, 15), (590, 560, 9)])
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
def test_coupled2d_on_chip(fomo, both, nx, nz, nbc, order):
    vp, _ = _layers(nx, nz, nx + order)
    vp = np.minimum(vp, np.float32(3000.0))
    vs = np.asfortranarray((vp / 1.8).astype(np.float32))
    rx = np.arange(1, nx + 1, 3)
    kw = dict(sx=[nx // 2 + 1, 1, nx], sz=[nz // 2 + 1, 1, nz], rx=rx,
              rz=np.full(rx.size, min(3, nz)), nbc=nbc, fd_order=order, snap_interval=35)
    a, b = both(fomo.coupled2d, vp, vs, 10.0, 1e-3, NT, 15.0, **kw)
    _same(a[0], b[0])
    assert np.abs(a[0].seis_P).max() > 0


@pytest.mark.parametrize("order", [2, 8, 10])
def test_acoustic2d_sponge_on_chip(fomo, both, order):
    vp, rho = _layers(150, 111, 4)
    kw = dict(sx=[70], sz=[9], rx=np.arange(1, 151, 4), rz=np.full(38, 9), nbc=20,
              fd_order=order, boundary="sponge", snap_interval=100)
    a, b = both(fomo.acoustic2d, vp, rho, 10.0, 1e-3, NT, 15.0, **kw)
    _same(a[0], b[0])


@pytest.mark.parametrize("shots", [2, 5, 37])
def test_acoustic2d_batch_on_chip(fomo, both, shots):
    vp, rho = _layers(61, 47, 9)
    sx = np.linspace(1, 61, shots).astype(int)
    sx = np.stack([sx, np.roll(sx, 1) // 2 + 1], 1)  # two sources a shot, some coincident
    rx = np.array([1, 5, 5, 30, 61])
    kw = dict(sx=sx, sz=np.full(sx.shape, 4), rx=rx, rz=np.array([4, 4, 4, 47, 1]), nbc=9,
              fd_order=8)
    a, b = both(fomo.acoustic2d_batch, vp, rho, 10.0, 1e-3, NT, 15.0, **kw)
    _same(a[0], b[0])
    assert not np.array_equal(a[0].seis_p[..., 0], a[0].seis_p[..., 1])


def test_on_the_default_stream(fomo):
    """A run on chip launched on torch's current (legacy default) stream."""
    import torch

    from fomo_b200 import _lib as L

    rng = np.random.default_rng(3)
    vp = rng.uniform(2000, 3500, (90, 60)).astype(np.float32, order="F")
    rho = rng.uniform(1500, 2500, (90, 60)).astype(np.float32, order="F")
    kw = dict(sx=[45], sz=[10], rx=np.arange(1, 91, 5), rz=np.full(18, 8), nbc=10, fd_order=8)
    ctx = L.context(0)
    ctx.use_torch_stream(torch.cuda.current_stream())
    try:
        a = fomo.acoustic2d(vp, rho, 10.0, 1e-3, 400, 15.0, **kw)
        assert fomo.api.last_stats.gpu_launches < 400
    finally:
        ctx.set_stream(None)
    b = fomo.acoustic2d(vp, rho, 10.0, 1e-3, 400, 15.0, **kw)
    assert np.array_equal(a.seis_p, b.seis_p)
    assert np.array_equal(a.seis_vz, b.seis_vz)
    assert np.abs(a.seis_p).max() > 0
