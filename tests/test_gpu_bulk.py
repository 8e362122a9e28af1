"""Two-phase runs of large grids in blocks per thread (bulk2d.cuh) against the oracle, bit
for bit: seismograms, snapshots and final fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# inner rectangles of whole and ragged tiles, one tile wide or high, thin and thick edges
SIZES = [(900, 260, 10), (523, 411, 3), (131, 1601, 1), (4001, 57, 12)]


def _model(nx, nz, seed):
    rng = np.random.default_rng(seed)
    vp = rng.uniform(2000, 4000, (nx, nz)).astype(np.float32, order="F")
    rho = rng.uniform(1500, 2500, (nx, nz)).astype(np.float32, order="F")
    vp[: nx // 2, 0] = rho[: nx // 2, 0] = 0.0
    return vp, rho


def _acq(nx, nz):
    rx = np.concatenate([np.linspace(1, nx, 9).astype(int), [1, nx, nx // 2]])
    rz = np.concatenate([np.full(9, nz // 2), [1, nz, 2]])
    return dict(sx=[nx // 2, 1, nx], sz=[nz // 2, 1, nz], rx=rx, rz=rz)


@pytest.mark.parametrize("nx,nz,nbc", SIZES)
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
@pytest.mark.parametrize("boundary", ["habc", "sponge"])
def test_acoustic2d_bulk(fomo, oracle, nx, nz, nbc, order, boundary):
    vp, rho = _model(nx, nz, order)
    nt, pad = 26, nbc + order // 2
    fin = np.zeros((nx + 2 * pad, nz + 2 * pad, 3), np.float32, order="F")
    w = 100.0 * fomo.ricker_wavelet(60.0, 1e-3, nt)
    kw = dict(nbc=nbc, fd_order=order, snap_interval=13, **_acq(nx, nz))
    r = fomo.acoustic2d(vp, rho, 10.0, 1e-3, nt, 15.0, wavelet=w, kernel=1, boundary=boundary,
                        final_state=fin, **kw)
    sp = dict(sponge_factor=0.015) if boundary == "sponge" else {}
    o = oracle.acoustic2d(vp, rho, 10.0, 1e-3, nt, wavelet=np.repeat(w[None], 3, 0), final=True,
                          **sp, **kw)
    for k in ("seis_p", "seis_vx", "seis_vz"):
        assert np.array_equal(getattr(r, k), o[k][:, :, 0])
    for k in range(2):
        assert np.array_equal(r.snaps[k], o["snaps"][:, :, k, 0])
    assert np.array_equal(fin, o["final"][..., 0])
    assert np.abs(fin).max() > 0


def test_acoustic2d_bulk_without_tags(fomo, oracle):
    """Over 2 M shot-cells injection and recording are a launch of their own."""
    vp, rho = _model(1201, 301, 5)
    nt = 20
    w = fomo.ricker_wavelet(60.0, 1e-3, nt)
    a = _acq(1201, 301)
    kw = dict(rx=a["rx"], rz=a["rz"], nbc=20, fd_order=8)
    sx, sz = np.array([[600], [1], [1201], [30], [90], [700]]), np.array([[9], [1], [301], [7], [100], [200]])
    r = fomo.acoustic2d_batch(vp, rho, 10.0, 1e-3, nt, 15.0, wavelet=w, kernel=1, sx=sx, sz=sz, **kw)
    o = oracle.acoustic2d(vp, rho, 10.0, 1e-3, nt, wavelet=w[None], sx=sx.T, sz=sz.T, n_shots=6, **kw)
    for k in ("seis_p", "seis_vx", "seis_vz"):
        assert np.array_equal(getattr(r, k), o[k])


@pytest.mark.parametrize("nx,nz,nbc", SIZES)
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
@pytest.mark.parametrize("boundary", ["habc", "sponge"])
def test_elastic2d_bulk(fomo, oracle, nx, nz, nbc, order, boundary):
    vp, rho = _model(nx, nz, order)
    vs = np.asfortranarray((vp / 1.8).astype(np.float32))
    vs[nx // 3: nx // 2] = 0.0
    nt, pad = 22, nbc + order // 2
    fin = np.zeros((nx + 2 * pad, nz + 2 * pad, 5), np.float32, order="F")
    w = 100.0 * fomo.ricker_wavelet(60.0, 1e-3, nt)
    kw = dict(nbc=nbc, fd_order=order, snap_interval=11, **_acq(nx, nz))
    r = fomo.elastic2d(vp, vs, rho, 10.0, 1e-3, nt, 15.0, wavelet=w, kernel=1, boundary=boundary,
                       final_state=fin, **kw)
    sp = dict(sponge_factor=0.015) if boundary == "sponge" else {}
    o = oracle.elastic2d(vp, vs, rho, 10.0, 1e-3, nt, wavelet=np.repeat(w[None], 3, 0), final=True,
                         **sp, **kw)
    for k in ("seis_vx", "seis_vz"):
        assert np.array_equal(getattr(r, k), o[k][:, :, 0])
    for k in range(2):
        assert np.array_equal(r.snaps[k], o["snaps"][:, :, k, 0])
    assert np.array_equal(fin, o["final"][..., 0])
    assert np.abs(fin).max() > 0


@pytest.mark.parametrize("nx,nz,nbc", SIZES + [(2101, 1003, 5)])
@pytest.mark.parametrize("order", [2, 4, 6, 8, 10])
def test_scalar2d_bulk(fomo, oracle, nx, nz, nbc, order):
    vp, _ = _model(nx, nz, order)
    nt, pad = 20, nbc + order // 2
    fin = np.zeros((nx + 2 * pad, nz + 2 * pad, 2), np.float32, order="F")
    w = 100.0 * fomo.ricker_wavelet(60.0, 1e-3, nt)
    kw = dict(nbc=nbc, fd_order=order, **_acq(nx, nz))
    r = fomo.scalar2d(vp, 10.0, 1e-3, nt, 15.0, wavelet=w, source_scale="none", kernel=1,
                      final_state=fin, **kw)
    o = oracle.scalar2d(vp, 10.0, 1e-3, nt, wavelet=np.repeat(w[None], 3, 0), final=True, **kw)
    assert np.array_equal(r.seis_u, np.squeeze(o["seis_u"]))
    assert np.array_equal(fin, o["final"])
    assert np.abs(fin).max() > 0
