"""A 2D run that cannot finish on the chip is launched instead, with the same results.  The
failures are injected on the host; the kernels run as always."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT = 310  # over the 300 steps from which a run is kept on the chip


def _model(nx, nz, seed):
    rng = np.random.default_rng(seed)
    vp = np.minimum(rng.uniform(2000, 3000, (nx, nz)), 3000).astype(np.float32, order="F")
    vs = np.asfortranarray((vp / 1.8).astype(np.float32))
    rho = rng.uniform(1500, 2500, (nx, nz)).astype(np.float32, order="F")
    return vp, vs, rho


def _calls(fomo):
    vp, vs, rho = _model(150, 111, 1)
    rx = np.arange(1, 151, 4)
    geo = dict(rx=rx, rz=np.full(rx.size, 9), nbc=20, fd_order=8)
    one = dict(sx=[70, 1], sz=[9, 111], **geo)
    fin = lambda nf: dict(final_state=np.zeros((198, 159, nf), np.float32, order="F"))  # noqa: E731
    t = (10.0, 1e-3, NT, 15.0)
    return {
        "acoustic2d": lambda: (fin(3), lambda **k: fomo.acoustic2d(vp, rho, *t, snap_interval=35, **one, **k)),
        "sponge": lambda: (fin(3), lambda **k: fomo.acoustic2d(vp, rho, *t, boundary="sponge", **one, **k)),
        "elastic2d": lambda: (fin(5), lambda **k: fomo.elastic2d(vp, vs, rho, *t, snap_interval=50, **one, **k)),
        "scalar2d": lambda: (fin(2), lambda **k: fomo.scalar2d(vp, *t, **one, **k)),
        "coupled2d": lambda: ({}, lambda **k: fomo.coupled2d(vp, vs, *t, snap_interval=35, **one, **k)),
        "batch": lambda: ({}, lambda **k: fomo.acoustic2d_batch(
            vp, rho, *t, sx=[20, 75, 140], sz=[4, 9, 100], **geo, **k)),
    }


def _flat(r, fin):
    out = [x for x in r if isinstance(x, np.ndarray)] + [fin.get("final_state", np.ones(1))]
    for x in r:
        if isinstance(x, list):
            out += x
    return out


@pytest.mark.parametrize("flag", ["FOMO_F_ONCHIP_LATE", "FOMO_F_ONCHIP_REFUSED"])
@pytest.mark.parametrize("name", ["acoustic2d", "sponge", "elastic2d", "scalar2d", "coupled2d", "batch"])
def test_failed_run_on_chip_is_launched(fomo, monkeypatch, name, flag):
    from fomo_b200 import _lib as L

    orig, got = fomo.api._opts, []
    for f in (0, L.FOMO_F_STEP_LAUNCH, getattr(L, flag)):
        def opts(*a, f=f, **kw):
            o = orig(*a, **kw)
            o.flags |= f
            return o

        monkeypatch.setattr(fomo.api, "_opts", opts)
        fin, fn = _calls(fomo)[name]()
        got.append((_flat(fn(**fin), fin), fomo.api.last_stats.gpu_launches))
    assert got[0][1] <= 16  # the plain call does run on the chip
    assert got[2][1] > NT   # the failed one was launched
    for a, b, c in zip(*(g[0] for g in got)):
        assert np.array_equal(a, b) and np.array_equal(b, c)
        assert np.isfinite(a).all() and np.abs(a).max() > 0


@pytest.mark.parametrize("name", ["acoustic2d", "elastic2d", "scalar2d", "coupled2d"])
def test_two_phase_is_launched(fomo, monkeypatch, name):
    """FOMO_KERNEL_TWO_PHASE asks for launched steps; only AUTO keeps a run on the chip."""
    from fomo_b200 import _lib as L

    orig, got = fomo.api._opts, []
    for kernel in (L.FOMO_KERNEL_AUTO, L.FOMO_KERNEL_TWO_PHASE):
        def opts(*a, kernel=kernel, **kw):
            o = orig(*a, **kw)
            o.kernel = kernel
            return o

        monkeypatch.setattr(fomo.api, "_opts", opts)
        fin, fn = _calls(fomo)[name]()
        got.append((_flat(fn(**fin), fin), fomo.api.last_stats.gpu_launches))
    assert got[0][1] <= 16 and got[1][1] > NT
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)


def test_two_contexts_on_chip_at_once(fomo, monkeypatch):
    """Two threads with a context each: every run wants one CTA per SM."""
    from fomo_b200 import _lib as L

    vp, _, rho = _model(260, 190, 2)
    kw = dict(sx=[130], sz=[9], rx=np.arange(1, 261, 3), rz=np.full(87, 5), nbc=30, fd_order=8)
    call = lambda: fomo.acoustic2d(vp, rho, 10.0, 1e-3, 600, 15.0, **kw)  # noqa: E731
    ref = call()
    assert fomo.api.last_stats.gpu_launches == 1
    local = threading.local()

    def context(device=0):
        if not hasattr(local, "ctx"):
            local.ctx = L.Context(device)
        return local.ctx

    monkeypatch.setattr(L, "context", context)
    out = [[], []]

    def work(k):
        for _ in range(6):
            out[k].append(call())

    th = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for r in out[0] + out[1]:
        for a, b in zip(r[:3], ref[:3]):
            assert np.array_equal(a, b)
    assert [len(o) for o in out] == [6, 6]
