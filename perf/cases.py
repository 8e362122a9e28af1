"""Timed cases of the public solvers: what a user of the framework has it run.

Every case is one whole public call on host arrays (models in, seismograms and
snapshots out), or, for the learned corrector, the gradient call of a training
step on device tensors.  Sizes come from the repository's own workloads: the
throughput grids (240x200 .. 2000x1600), the 400x300 acoustic and coupled P-S
runs, the 32-shot 1000x500 elastic batch, the uneven batch and the 400x400x300
elastic model.  ``exact`` restates each scheme in float64 with plain torch.

A case is a dict of plain values:
  kind      which entry point (see ``_KINDS``)
  nx ny nz  interior grid;  nt time steps;  nbc absorbing cells;  order FD order
  shots     shots of a batch;  snap snapshot interval (0 none)
  boundary  "habc" or "sponge";  precision "fp32" or "fp16" storage
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "fomo.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fomo_b200 as F  # noqa: E402
from fomo_b200 import corrector as CR  # noqa: E402


def _case(name, kind, nx, nz, nt, *, ny=0, nbc=50, order=8, shots=1, snap=0, boundary="habc",
          precision="fp32"):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, nbc=nbc, order=order,
                shots=shots, snap=snap, boundary=boundary, precision=precision)


def listed():
    return [
        # the smallest call: one scalar shot on the smallest throughput grid, bound by
        # launches (the inner loop of constant-density migration or a source scan)
        _case("scalar2d_240x200", "scalar2d", 240, 200, 1000),
        # the plain single-shot acoustic run: small grid, thick absorbing layer, vacuum
        # surface, a snapshot every 50 steps for a movie
        _case("acoustic2d_400x300_snaps", "acoustic2d", 400, 300, 2000, nbc=100, snap=50),
        # the largest throughput grid: one acoustic shot over a regional section
        _case("acoustic2d_2000x1600", "acoustic2d", 2000, 1600, 400),
        # a handful of shots on a small shared model (inversion of a small survey)
        _case("acoustic2d_batch_8x240x200", "acoustic2d_batch", 240, 200, 1000, shots=8),
        # one elastic shot on an odd mid-size grid with snapshots
        _case("elastic2d_501x397_snaps", "elastic2d", 501, 397, 1000, snap=100),
        # the headline batch: 32 elastic shots, order 10
        _case("elastic2d_batch_32x1000x500", "elastic2d_batch", 1000, 500, 500, nbc=80, order=10,
              shots=32),
        # the same survey in binary16 storage, half the shots
        _case("elastic2d_batch_fp16_16x1000x500", "elastic2d_batch", 1000, 500, 250, nbc=80,
              order=10, shots=16, precision="fp16"),
        # shots on models of different sizes stepped together
        _case("acoustic2d_uneven_16", "acoustic2d_uneven", 2000, 800, 500, shots=16),
        # a small 3D acoustic model with odd sizes
        _case("acoustic3d_161x150x121", "acoustic3d", 161, 121, 200, ny=150, nbc=40, snap=50),
        # the large 3D elastic model (a stretch of its time loop)
        _case("elastic3d_400x400x300", "elastic3d", 400, 300, 60, ny=400, nbc=40),
        # coupled P-S potentials on the 400x300 demo grid, both wavefields kept as movies
        _case("coupled2d_400x300_snaps", "coupled2d", 400, 300, 2000, nbc=100, snap=100),
        # one training step of the learned corrector: loss and gradients of 32 windows of 64x64
        _case("corrector_step_32x64x64", "corrector", 64, 64, 1, shots=32),
    ]


def draw(rng):
    """A case of the same ranges, at most as costly as the largest listed one."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["scalar2d", "acoustic2d", "acoustic2d", "acoustic2d_batch", "elastic2d",
                       "elastic2d_batch", "elastic2d_batch", "acoustic2d_uneven", "acoustic3d",
                       "elastic3d", "coupled2d", "corrector"])
    order = rng.choice([2, 4, 6, 8, 8, 8, 10, 10])
    nbc = rng.randint(20, 100)
    boundary, precision, shots, snap, ny = "habc", "fp32", 1, 0, 0
    if kind == "corrector":
        return dict(kind=kind, nx=16 * rng.randint(1, 6), ny=0, nz=rng.randint(16, 96), nt=1,
                    nbc=50, order=8, shots=rng.randint(4, 48), snap=0, boundary="habc",
                    precision="fp32")
    if kind in ("acoustic3d", "elastic3d"):
        nx, ny, nz = size(60, 240), size(60, 240), size(60, 180)
        nbc = rng.randint(10, 40)
        nt = rng.randint(40, 120)
        snap = rng.choice([0, 20])
    elif kind == "acoustic2d_uneven":
        nx, nz, shots, nt = size(400, 2000), size(300, 800), rng.randint(4, 16), rng.randint(200, 500)
        order = max(order, 4)
    elif kind == "elastic2d_batch":
        precision = rng.choice(["fp32", "fp32", "fp16"])
        nx, nz, shots, nt = size(240, 1000), size(200, 500), rng.randint(2, 32), rng.randint(150, 500)
        nbc = max(nbc, 33)
    elif kind == "acoustic2d_batch":
        nx, nz, shots, nt = size(200, 800), size(200, 600), rng.randint(2, 16), rng.randint(300, 1000)
    elif kind == "coupled2d":
        nx, nz, nt = size(200, 700), size(200, 700), rng.randint(500, 2000)
        snap = rng.choice([0, 100])
    else:  # one 2D shot
        nx, nz, nt = size(200, 2000), size(200, 1600), rng.randint(300, 1000)
        if kind != "scalar2d":
            boundary = rng.choice(["habc", "habc", "sponge"])
            snap = rng.choice([0, 50, 100])
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, nbc=nbc, order=order, shots=shots,
                snap=snap, boundary=boundary, precision=precision)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _ricker(f0, dt, nt):
    """A Ricker wavelet delayed by 1.5 / f0, evaluated in float64."""
    x = np.pi * f0 * (np.arange(nt) * dt - 1.5 / f0)
    return ((1.0 - 2.0 * x * x) * np.exp(-x * x)).astype(np.float32)


def _gardner(vp):
    return np.asfortranarray((310.0 * vp.astype(np.float64) ** 0.25).astype(np.float32))


def _layers(rng, nx, nz, n, vmin, vmax):
    """Flat layers, velocities uniform in [vmin, vmax], (nx, nz)."""
    edges = np.sort(rng.choice(np.arange(1, nz), size=n - 1, replace=False))
    v = rng.uniform(vmin, vmax, n).astype(np.float32)
    row = v[np.searchsorted(edges, np.arange(nz), side="right")]
    return np.asfortranarray(np.broadcast_to(row[None, :], (nx, nz)))


def _field(seed, shape, corr, mean, std, vmin, vmax):
    """Gaussian random field on the GPU, returned as a (nx[, ny], nz) host array,
    x fastest; shape is (nz[, ny], nx), corr in cells."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(int(seed))
    w = torch.randn(shape, generator=g, device=dev)
    f = torch.fft.rfftn(w)
    for ax, n in enumerate(shape):
        k = (torch.fft.rfftfreq(n, device=dev) if ax == len(shape) - 1
             else torch.fft.fftfreq(n, device=dev)) * (2 * math.pi)
        f *= torch.exp(-(k * corr) ** 2 / 8.0).reshape([-1 if a == ax else 1 for a in range(len(shape))])
    f = torch.fft.irfftn(f, s=shape)
    f = (f - f.mean()) / (f.std() + 1e-30)
    return (mean + std * f).clamp_(vmin, vmax).cpu().numpy().T


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    kind, nx, nz, nt = c["kind"], c["nx"], c["nz"], c["nt"]
    rx = np.arange(1, nx + 1, 2)
    rz = np.full(rx.size, 10)
    kw = dict(nbc=c["nbc"], fd_order=c["order"])
    s = dict(kind=kind)
    if kind == "corrector":
        # one batch of training windows and the parameters, resident on the GPU
        K = CR.Kernels(0)
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        n = c["shots"]
        feat = torch.zeros(n, nz, nx, 16, device="cuda", dtype=torch.bfloat16)
        feat[..., :6] = torch.randn(n, nz, nx, 6, device="cuda", generator=g).to(torch.bfloat16)
        target = torch.randn(n, nz, nx, device="cuda", generator=g)
        mask = torch.zeros_like(target)
        mask[:, 4:-4, 4:-4] = 1.0
        fan = torch.cat([torch.full((864,), 54.0), torch.full((2304,), 144.0),
                         torch.full((144,), 144.0)]).cuda()
        params = torch.randn(CR.param_count(), device="cuda", generator=g) * (2.0 / fan).sqrt()
        s.update(K=K, feat=feat, target=target, mask=mask, params=params,
                 y=torch.empty_like(target))
        return s
    if kind in ("acoustic3d", "elastic3d"):
        ny = c["ny"]
        dh, dt, f0 = 10.0, 8e-4, 12.0
        vp = _field(seed, (nz, ny, nx), 25.0, 3200.0, 500.0, 1500.0, 5000.0)
        rho = (310.0 * vp.T ** np.float32(0.25)).T
        gx, gy = np.meshgrid(np.arange(1, nx + 1, 2), np.arange(1, ny + 1, 2), indexing="ij")
        geo = dict(sx=[nx // 2], sy=[ny // 2], sz=[10], rx=gx.ravel(order="F"),
                   ry=gy.ravel(order="F"), rz=np.full(gx.size, 10))
        models = [vp, rho]
        if kind == "elastic3d":
            models.insert(1, (vp.T / np.float32(1.8)).T)
        for m in models:
            m[:, :, 0] = 0.0  # vacuum surface
        s.update(models=models, geo=geo)
        kw.update(snap_interval=c["snap"])
    elif kind == "acoustic2d_uneven":
        dh, dt, f0 = 10.0, 1e-3, 15.0
        # the sizes belong to the case, the models to the seed
        sizes = np.random.default_rng(nx + 7 * nz + 131 * c["shots"])
        n = c["shots"]
        nxs = np.rint(np.exp(sizes.uniform(np.log(200), np.log(nx), n))).astype(int)
        nzs = np.rint(np.exp(sizes.uniform(np.log(200), np.log(nz), n))).astype(int)
        vps = [_field(seed + 1000 * k, (int(b), int(a)), 30.0, 3000.0, 600.0, 1500.0, 5000.0)
               for k, (a, b) in enumerate(zip(nxs, nzs))]
        rhos = [np.full(v.shape, 2000.0, np.float32, order="F") for v in vps]
        geo = dict(sx=[int(a) // 2 for a in nxs], sz=[10] * n,
                   rx=[np.arange(1, a + 1, 2) for a in nxs],
                   rz=[np.full((a + 1) // 2, 10) for a in nxs])
        s.update(models=[vps, rhos], geo=geo)
    else:
        vp_vs = 1.73
        if kind in ("elastic2d", "elastic2d_batch"):
            dh, dt, f0 = 5.0, 5e-4, 20.0
            vp = _layers(rng, nx, nz, 12, 1500.0, 4500.0)
        else:
            dh, dt, f0 = 10.0, 1e-3, 15.0
            vp = _layers(rng, nx, nz, 6, 2500.0, 4500.0 if kind != "coupled2d" else 3800.0)
        rho = _gardner(vp)
        vs = np.asfortranarray((vp / np.float32(vp_vs)).astype(np.float32))
        if kind == "acoustic2d":  # vacuum surface row
            vp = vp.copy(order="F")
            vp[:, 0] = 0.0
            rho[:, 0] = 0.0
        if kind.endswith("_batch"):
            n = c["shots"]
            sx = np.clip(np.rint((np.arange(n) + rng.uniform(0.2, 0.8)) * nx / n), 1, nx).astype(int)
            geo = dict(sx=sx, sz=np.full(n, 5), rx=rx, rz=rz)
        else:
            geo = dict(sx=[int(rng.integers(nx // 4, 3 * nx // 4))], sz=[10], rx=rx, rz=rz)
        s.update(models={"scalar2d": [vp], "coupled2d": [vp, vs]}.get(
            kind, [vp, vs, rho] if kind.startswith("elastic") else [vp, rho]), geo=geo)
        if kind in ("acoustic2d", "elastic2d"):
            kw.update(snap_interval=c["snap"], boundary=c["boundary"])
        elif kind == "coupled2d":
            kw.update(snap_interval=c["snap"])
        elif kind == "elastic2d_batch":
            kw.update(precision=c["precision"])
    s.update(args=(dh, dt, nt, f0), kw=kw, wavelet=_ricker(f0, dt, nt))
    return s


def run(s):
    kind = s["kind"]
    if kind == "corrector":
        loss, grad = s["K"].gradients(s["feat"], s["target"], s["mask"], s["params"], s["y"])
        return dict(loss=loss, grad=grad, y=s["y"])
    r = getattr(F, kind)(*s["models"], *s["args"], wavelet=s["wavelet"], **s["geo"], **s["kw"])
    if kind == "acoustic2d":
        return dict(p=r.seis_p, vx=r.seis_vx, vz=r.seis_vz, snaps=r.snaps)
    if kind == "acoustic2d_batch":
        return dict(p=r.seis_p, vx=r.seis_vx, vz=r.seis_vz)
    if kind in ("elastic2d", "elastic2d_batch"):
        return dict(vx=r.seis_vx, vz=r.seis_vz, snaps=getattr(r, "snaps", []))
    if kind == "scalar2d":
        return dict(u=r.seis_u)
    if kind == "coupled2d":
        return dict(P=r.seis_P, S=r.seis_S, snaps_P=r.snaps_P, snaps_S=r.snaps_S)
    if kind == "acoustic2d_uneven":
        return [list(x) for x in r.shots]
    return dict(vx=r[0], vy=r[1], vz=r[2], snaps=r[3])


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
# per cell and step: (wavefield words, material words, floating point operations with
# one stencil term of a first difference counted as subtract, multiply, add)
_KINDS = {
    "scalar2d": (2, 1, lambda N: 6 * N + 5),
    "acoustic2d": (3, 3, lambda N: 12 * N + 11),
    "elastic2d": (5, 5, lambda N: 24 * N + 25),
    "coupled2d": (4, 8, lambda N: 24 * N + 50),
    "acoustic3d": (4, 4, lambda N: 18 * N + 16),
    "elastic3d": (9, 8, lambda N: 54 * N + 55),
}
_L2 = 126e6  # bytes the chip keeps close to the SMs


def _shapes(case):
    """Interior grids of a case, one per model."""
    if case["kind"] == "acoustic2d_uneven":
        sizes = np.random.default_rng(case["nx"] + 7 * case["nz"] + 131 * case["shots"])
        n = case["shots"]
        a = np.rint(np.exp(sizes.uniform(np.log(200), np.log(case["nx"]), n))).astype(int)
        b = np.rint(np.exp(sizes.uniform(np.log(200), np.log(case["nz"]), n))).astype(int)
        return [(int(x), int(z)) for x, z in zip(a, b)]
    if case["ny"]:
        return [(case["nx"], case["ny"], case["nz"])]
    return [(case["nx"], case["nz"])]


def work(case):
    """Models, seismograms and snapshots once; the wavefields (and materials) once in and
    once out per step only where they cannot all stay in L2."""
    if case["kind"] == "corrector":
        pix = case["shots"] * case["nx"] * case["nz"]
        macs = 9 * (6 * 16 + 16 * 16 + 16)
        return dict(bytes=pix * (32 + 4 + 4 + 4) + 2 * 4 * 3312, flops=pix * macs * 2 * 3)
    base = case["kind"].replace("_batch", "").replace("_uneven", "")
    fields, mats, ops = _KINDS[base]
    N = case["order"] // 2
    pad = case["nbc"] + N
    word = 2 if case["precision"] == "fp16" else 4
    per_model = case["shots"] if case["kind"].endswith("_batch") else 1
    byts = flops = live = 0.0
    nseis = {"scalar2d": 1, "elastic2d": 2, "coupled2d": 2}.get(base, 3)
    nmodel = {"scalar2d": 1, "acoustic2d": 2, "coupled2d": 2, "acoustic3d": 2}.get(base, 3)
    for shape in _shapes(case):
        cells = math.prod(n + 2 * pad for n in shape)
        inner = math.prod(shape)
        nrec = math.prod((n + 1) // 2 for n in shape[:-1])
        byts += 4.0 * nmodel * inner + 4.0 * nseis * nrec * case["nt"] * per_model
        if case["snap"]:
            frame = shape[0] * shape[-1]
            byts += 4.0 * frame * (case["nt"] // case["snap"]) * (2 if base == "coupled2d" else 1)
        flops += float(ops(N)) * cells * per_model * case["nt"]
        live += cells * (word * fields * per_model + 4.0 * mats)
    if live > _L2:
        for shape in _shapes(case):
            cells = math.prod(n + 2 * pad for n in shape)
            byts += case["nt"] * cells * (2.0 * word * fields * per_model + 4.0 * mats)
    return dict(bytes=byts, flops=flops)


# ---------------------------------------------------------------------------
# float64 restatement
# ---------------------------------------------------------------------------
_FD = {2: [1.0], 4: [1.125, -0.041666667], 6: [1.171875, -0.065104167, 0.0046875],
       8: [1.1962890625, -0.079752604167, 0.0095703125, -0.000697544643],
       10: [1.2115478515625, -0.089721679687, 0.0138427734375, -0.00176565987723, 0.0001186795166]}
_D1 = {2: [1 / 2], 4: [2 / 3, -1 / 12], 6: [3 / 4, -3 / 20, 1 / 60],
       8: [4 / 5, -1 / 5, 4 / 105, -1 / 280], 10: [5 / 6, -5 / 21, 5 / 84, -5 / 504, 1 / 1260]}
_D2 = {2: [1.0], 4: [4 / 3, -1 / 12], 6: [3 / 2, -3 / 20, 1 / 90],
       8: [8 / 5, -1 / 5, 8 / 315, -1 / 560], 10: [5 / 3, -5 / 21, 5 / 126, -5 / 1008, 1 / 3150]}
_C0 = {2: -2.0, 4: -5 / 2, 6: -49 / 18, 8: -205 / 72, 10: -5269 / 1800}


def _f32(v):
    return [float(np.float32(x)) for x in v]


class _Grid:
    """Padded grid in float64: arrays are (shots, nz[, ny], nx)."""

    def __init__(self, shape, case, dh, dt, v_ref):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.order, self.M = case["order"], case["order"] // 2
        self.nbc, self.pad = case["nbc"], case["nbc"] + case["order"] // 2
        self.dims = len(shape)
        self.n = [m + 2 * self.pad for m in shape[::-1]]  # z[, y], x
        self.c = _f32(_FD[self.order])
        self.dh, self.dt = float(np.float32(dh)), float(np.float32(dt))
        self.r = self.dt / self.dh
        self.sponge = case["boundary"] == "sponge"
        edge = None  # distance to the nearest edge
        for ax, n in enumerate(self.n):
            i = torch.arange(n, device=self.dev)
            d = torch.minimum(i, n - 1 - i).reshape([-1 if a == ax else 1 for a in range(self.dims)])
            edge = d if edge is None else torch.minimum(edge, d)
        self.edge = edge
        if self.sponge:
            k = np.float32(0.015) * (self.nbc - np.arange(self.nbc)).astype(np.float32)
            damp = np.exp(-(k * k).astype(np.float64)).astype(np.float32).astype(np.float64)
            damp = torch.cat([torch.from_numpy(damp), torch.ones(1, dtype=torch.float64)]).to(self.dev)
            self.damp = damp[edge.clamp(max=self.nbc)]
            return
        zone = self.zone = self.pad - 1
        count = torch.zeros_like(edge)
        inside = edge >= 1
        for ax, n in enumerate(self.n):
            i = torch.arange(n, device=self.dev)
            d = torch.minimum(i, n - 1 - i).reshape([-1 if a == ax else 1 for a in range(self.dims)])
            count = count + ((d <= zone) & inside)
        self.frame, self.count = count > 0, count.clamp(min=1)
        self.set_vref(v_ref)

    def set_vref(self, v_ref):
        r = float(np.float32(v_ref)) * self.r
        b = float(np.float32(0.45))
        self.q = (b * (1 + r) - r) / ((1 + r) * (1 - b))
        self.qt = (b * (1 + r) - 1) / ((1 + r) * (1 - b))
        self.qxt = b / (b - 1)

    def weights(self, off):
        w = ((self.edge.double() - off) / (self.pad - 1)).clamp(0.0, 1.0)
        w = torch.where(self.frame, w, torch.ones_like(w))
        return w, torch.where(self.frame, (1.0 - w) / self.count, torch.zeros_like(w))

    def padded(self, m):
        t = torch.from_numpy(np.ascontiguousarray(m.T)).to(self.dev).double()
        for ax, n in enumerate(self.n):
            i = (torch.arange(n, device=self.dev) - self.pad).clamp(0, t.shape[ax] - 1)
            t = t.index_select(ax, i)
        return t

    def zeros(self, shots=1):
        return torch.zeros([shots] + self.n, dtype=torch.float64, device=self.dev)

    def inner(self, f, ax=None, shift=0):
        """Cells at least M from every edge, shifted along axis ax (negative, from x)."""
        M = self.M
        s = [slice(M, n - M) for n in self.n]
        if ax is not None:
            n = self.n[ax]
            s[ax] = slice(M + shift, n - M + shift)
        return f[(Ellipsis, *s)]

    def back(self, f, ax):
        return sum(a * (self.inner(f, ax, l) - self.inner(f, ax, -l - 1)) for l, a in enumerate(self.c))

    def fwd(self, f, ax):
        return sum(a * (self.inner(f, ax, l + 1) - self.inner(f, ax, -l)) for l, a in enumerate(self.c))

    def absorb(self, f, old, w):
        """The boundary applied to the updated field f (old: the field before the update)."""
        if self.sponge:
            return f.mul_(self.damp)
        W, A = w
        out = f * W
        for ax in range(-self.dims, 0):
            n = self.n[ax]
            for lo, hi, step in ((1, self.zone + 1, 1), (n - 1 - self.zone, n - 1, -1)):
                s = [slice(1, m - 1) for m in self.n]
                t = list(s)
                s[ax] = slice(lo, hi)
                t[ax] = slice(lo + step, hi + step)
                s, t = (Ellipsis, *s), (Ellipsis, *t)
                out[s] += A[s] * (-self.q * f[t] - self.qt * old[s] - self.qxt * old[t])
        return out

    def at(self, *ix):
        """Flat index of 1-based interior cells given as x[, y], z."""
        k = torch.zeros(len(np.atleast_1d(ix[0])), dtype=torch.int64)
        for i, n in zip(ix[::-1], self.n):
            k = k * n + torch.as_tensor(np.atleast_1d(i).astype(np.int64)) - 1 + self.pad
        return k.to(self.dev)

    def crop(self, f):
        p = self.pad
        return f[(Ellipsis, *[slice(p, n - p) for n in self.n])]


def _harm2(a, b):
    s = torch.where(a == 0, b, torch.where(b == 0, a, a + b))
    return torch.where(s == 0, torch.zeros_like(s), 2.0 / torch.where(s == 0, torch.ones_like(s), s))


def _mean_pair(f, ax, up, fn):
    """fn(cell - 1, cell) along ax (up: fn(cell, cell + 1)); the edge copies its neighbour."""
    n = f.shape[ax]
    v = fn(f.narrow(ax, 0, n - 1), f.narrow(ax, 1, n - 1))
    e = v.narrow(ax, n - 2, 1) if up else v.narrow(ax, 0, 1)
    return torch.cat([v, e] if up else [e, v], ax)


def _harm4(mu, axes):
    """4 over the sum of 1/mu of four cells; 0 where one is 0; axes: [(axis, up)]."""
    inv = torch.where(mu == 0, torch.full_like(mu, float("inf")), 1.0 / mu)
    for ax, up in axes:
        inv = _mean_pair(inv, ax, up, torch.add)
    return torch.where(torch.isinf(inv), torch.zeros_like(inv), 4.0 / inv)


def _staggered(base, case, models, s, shape, src, rec):
    """acoustic / elastic runs in 2D and 3D, shots stacked: {name: (n_rec, nt[, shots])}."""
    dh, dt, nt, _ = s["args"]
    vp = models[0]
    g = _Grid(shape, case, dh, dt, vp[vp > 0].min())
    el = base.startswith("elastic")
    three = g.dims == 3
    X, Y, Z = -1, -2, -g.dims
    rho, vpp = g.padded(models[-1]), g.padded(vp)
    b = {X: _mean_pair(rho, X, False, _harm2), Z: _mean_pair(rho, Z, True, _harm2)}
    if three:
        b[Y] = _mean_pair(rho, Y, False, _harm2)
    b = {a: g.inner(v).clone() for a, v in b.items()}
    kap = g.inner(rho * vpp * vpp).clone()
    if el:
        vs = g.padded(models[1])
        mu = rho * vs * vs
        lam = kap - 2 * g.inner(mu)
        mm = {(X, Z): _harm4(mu, [(X, False), (Z, True)])}
        if three:
            mm[(X, Y)] = _harm4(mu, [(X, False), (Y, False)])
            mm[(Y, Z)] = _harm4(mu, [(Y, False), (Z, True)])
        mm = {a: g.inner(v).clone() for a, v in mm.items()}
        del mu, vs
    del rho, vpp
    axes = [X, Y, Z] if three else [X, Z]
    offs = {X: 0.0, Y: 0.25, Z: 0.5}
    if not three:
        offs[Z] = 0.5
    wv = None if g.sponge else {a: g.weights(offs[a]) for a in axes}
    wp = None if g.sponge else g.weights(0.75)
    ns = src.shape[0]
    v = {a: g.zeros(ns) for a in axes}
    if el:
        T = {(a, a): g.zeros(ns) for a in axes}
        T.update({a: g.zeros(ns) for a in mm})
    else:
        T = {0: g.zeros(ns)}
    # which side a difference looks to: velocities sit half a cell back in x and y, ahead in z
    def dv(f, of, ax):  # difference of field f along ax for the velocity component `of`
        ahead = (ax == Z) == (of == ax)
        return g.fwd(f, ax) if ahead else g.back(f, ax)
    key = (lambda a, c: (a, c) if (a, c) in T else (c, a))
    names = {X: "vx", Y: "vy", Z: "vz"}
    out = {k: torch.zeros(nt, ns, rec.numel(), dtype=torch.float64, device=g.dev)
           for k in ([] if el or three else ["p"]) + [names[a] for a in axes]}
    snaps = []
    wav = torch.from_numpy(s["wavelet"]).double().to(g.dev)
    rows = torch.arange(ns, device=g.dev)
    for it in range(nt):
        for a in axes:
            old = v[a].clone()
            d = sum(dv(T[key(a, c)] if el else T[0], a, c) for c in (axes if el else [a]))
            g.inner(v[a]).add_(b[a] * g.r * d)
            v[a] = g.absorb(v[a], old, wv and wv[a])
        dd = {a: (g.back(v[a], a) if a == Z else g.fwd(v[a], a)) for a in axes}
        div = sum(dd.values())
        if el:
            upd = {(a, a): g.r * (lam * div + (kap - lam) * dd[a]) for a in axes}
            for a, c in mm:
                e = (g.fwd(v[a], c) if c == Z else g.back(v[a], c)) + g.back(v[c], a)
                upd[(a, c)] = g.r * mm[(a, c)] * e
        else:
            upd = {0: kap * g.r * div}
        for k, du in upd.items():
            old = T[k].clone()
            g.inner(T[k]).add_(du)
            T[k] = g.absorb(T[k], old, wp)
        for k in [(a, a) for a in axes] if el else [0]:
            T[k].view(ns, -1).index_put_((rows, src), wav[it].expand(ns), accumulate=True)
        for a in axes:
            out[names[a]][it] = v[a].reshape(ns, -1)[:, rec]
        if "p" in out:
            out["p"][it] = T[0].reshape(ns, -1)[:, rec]
        if case["snap"] and (it + 1) % case["snap"] == 0:
            f = g.crop(v[Z] if el else T[0])[0]
            if three:
                f = f[:, shape[1] // 2 - 1, :]
            snaps.append(f.T.cpu().numpy())
    res = {k: o.permute(2, 0, 1).cpu().numpy() for k, o in out.items()}  # (n_rec, nt, shots)
    return res, snaps


def _exact_scalar(case, s):
    dh, dt, nt, _ = s["args"]
    vp, geo = s["models"][0], s["geo"]
    g = _Grid(vp.shape, case, dh, dt, vp[vp > 0].min())
    c2 = g.inner((g.padded(vp) * g.r) ** 2).clone()
    d, w = _f32(_D2[g.order]), g.weights(0.75)
    c0 = 2 * float(np.float32(_C0[g.order]))
    u0, u1 = g.zeros(), g.zeros()
    src, rec = g.at(geo["sx"], geo["sz"]), g.at(geo["rx"], geo["rz"])
    v = np.float64(vp[geo["sx"][0] - 1, geo["sz"][0] - 1])
    wav = s["wavelet"].astype(np.float64) * (v * g.dt) ** 2
    out = torch.zeros(nt, rec.numel(), dtype=torch.float64, device=g.dev)
    for it in range(nt):
        lap = c0 * g.inner(u1)
        for l, a in enumerate(d, 1):
            lap += a * (g.inner(u1, -1, l) + g.inner(u1, -1, -l) + g.inner(u1, -2, l) + g.inner(u1, -2, -l))
        u2 = u1.clone()
        g.inner(u2).copy_(c2 * lap + 2 * g.inner(u1) - g.inner(u0))
        u2 = g.absorb(u2, u1, w)
        u2.view(-1)[src] += wav[it]
        out[it] = u2.view(-1)[rec]
        u0, u1 = u1, u2
    return dict(u=out.T.cpu().numpy())


def _exact_coupled(case, s):
    dh, dt, nt, _ = s["args"]
    (vp, vs), geo = s["models"], s["geo"]
    g = _Grid(vp.shape, case, dh, dt, vp[vp > 0].min())
    d1, d2, c0 = _f32(_D1[g.order]), _f32(_D2[g.order]), float(np.float32(_C0[g.order]))
    ih = 1.0 / g.dh

    def smooth(f):  # Gaussian of 3 grid points, 9 taps each side, edges clamped
        k = torch.exp(-0.5 * (torch.arange(-9, 10, device=g.dev).double() / 3.0) ** 2)
        k /= k.sum()
        for ax in (-1, -2):
            n = f.shape[ax]
            i = torch.arange(n, device=g.dev)
            f = sum(k[q + 9] * f.index_select(ax, (i + q).clamp(0, n - 1)) for q in range(-9, 10))
        return f

    def grad(f, ax):
        return ih * sum(a * (g.inner(f, ax, l) - g.inner(f, ax, -l)) for l, a in enumerate(d1, 1))

    def lap(f):
        return ih * ih * (2 * c0 * g.inner(f) + sum(
            a * (g.inner(f, -1, l) + g.inner(f, -1, -l) + g.inner(f, -2, l) + g.inner(f, -2, -l))
            for l, a in enumerate(d2, 1)))

    al, be = g.padded(vp) ** 2, g.padded(vs) ** 2
    sa, sb = smooth(al), smooth(be)
    ax_, az, bx, bz, la, lb = grad(sa, -1), grad(sa, -2), grad(sb, -1), grad(sb, -2), lap(sa), lap(sb)
    al, be = g.inner(al).clone(), g.inner(be).clone()
    P, S, dP, dS = (g.zeros() for _ in range(4))
    src, rec = g.at(geo["sx"], geo["sz"]), g.at(geo["rx"], geo["rz"])
    wv, wp = g.weights(0.0), g.weights(0.75)
    vrp, vrs = vp[vp > 0].min(), vs[vs > 0].min()

    def both(p, op, s_, os, w):
        g.set_vref(vrp)
        p = g.absorb(p, op, w)
        g.set_vref(vrs)
        return p, g.absorb(s_, os, w)

    o = torch.zeros(2, nt, rec.numel(), dtype=torch.float64, device=g.dev)
    snaps = ([], [])
    for it in range(nt):
        Px, Pz, Sx, Sz = grad(P, -1), grad(P, -2), grad(S, -1), grad(S, -2)
        Pc = g.inner(P)
        rP = Pc * (la - 2 * lb) + 2 * (ax_ * Px + az * Pz + bx * Sz - bz * Sx) + al * lap(P)
        rS = 2 * (bx * Sx + bz * Sz + bz * Px - bx * Pz) + be * lap(S)
        o1, o2 = dP.clone(), dS.clone()
        g.inner(dP).add_(g.dt * rP)
        g.inner(dS).add_(g.dt * rS)
        dP, dS = both(dP, o1, dS, o2, wv)
        o1, o2 = P.clone(), S.clone()
        g.inner(P).add_(g.dt * g.inner(dP))
        g.inner(S).add_(g.dt * g.inner(dS))
        P, S = both(P, o1, S, o2, wp)
        P.view(-1)[src] += float(s["wavelet"][it])
        o[0, it], o[1, it] = P.view(-1)[rec], S.view(-1)[rec]
        if case["snap"] and (it + 1) % case["snap"] == 0:
            for k, f in enumerate((P, S)):
                snaps[k].append(g.crop(f)[0].T.cpu().numpy())
    o = o.cpu().numpy()
    return dict(P=o[0].T, S=o[1].T, snaps_P=snaps[0], snaps_S=snaps[1])


def _exact_corrector(s):
    """Loss, parameter gradients and output of the three convolutions in float64."""
    p = s["params"].double().requires_grad_()
    x = s["feat"].double()[..., :6].permute(0, 3, 1, 2)
    w = [p[:864].reshape(3, 3, 6, 16), p[864:3168].reshape(3, 3, 16, 16), p[3168:].reshape(3, 3, 16, 1)]
    for k, t in enumerate(w):
        x = torch.nn.functional.conv2d(x, t.permute(3, 2, 0, 1), padding=1)
        x = torch.relu(x) if k < 2 else x
    y = x[:, 0]
    loss = ((s["mask"].double() * (y - s["target"].double())) ** 2).mean()
    loss.backward()
    return dict(loss=loss.detach().reshape(1), grad=p.grad, y=y.detach())


def exact(case, seed):
    kind = case["kind"]
    base = kind.replace("_batch", "").replace("_uneven", "")
    if kind != "corrector":
        N = case["order"] // 2
        cells = sum(math.prod(n + 2 * (case["nbc"] + N) for n in sh) for sh in _shapes(case))
        if kind.endswith("_batch"):
            cells *= case["shots"]
        if cells * case["nt"] * _KINDS[base][2](N) > 3e12:  # over about 20 seconds in float64
            return None
    s = prepare(case, seed)
    if kind == "corrector":
        return _exact_corrector(s)
    if kind == "scalar2d":
        return _exact_scalar(case, s)
    if kind == "coupled2d":
        return _exact_coupled(case, s)
    geo = s["geo"]
    if kind == "acoustic2d_uneven":
        res = []
        for k, (vp, rho) in enumerate(zip(*s["models"])):
            g = _Grid(vp.shape, case, *s["args"][:2], 1.0)
            o, _ = _staggered(base, case, [vp, rho], s, vp.shape, g.at(geo["sx"][k], geo["sz"][k]),
                              g.at(geo["rx"][k], geo["rz"][k]))
            res.append([o["p"][..., 0], o["vx"][..., 0], o["vz"][..., 0]])
        return res
    shape = s["models"][0].shape
    g = _Grid(shape, case, *s["args"][:2], 1.0)
    ax = ("x", "y", "z") if len(shape) == 3 else ("x", "z")
    src, rec = g.at(*[geo["s" + a] for a in ax]), g.at(*[geo["r" + a] for a in ax])
    res, snaps = _staggered(base, case, s["models"], s, shape, src, rec)
    if not kind.endswith("_batch"):
        res = {k: v[..., 0] for k, v in res.items()}
    if kind != "acoustic2d_batch":
        res["snaps"] = snaps
    return res
