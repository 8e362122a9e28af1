"""The z cuts of the fused 3D half steps (every tile in up to ten chunks, or whole columns
with the last wave in four) against the per-cell kernels, bit for bit, wavefields included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# few planes, tiles in five to ten chunks, tiles just below and above the lines of the rule
SIZES = [("acoustic", 20, 10, 5, 1), ("acoustic", 20, 10, 23, 1), ("acoustic", 25, 9, 41, 1),
         ("acoustic", 61, 30, 57, 3), ("acoustic", 430, 180, 32, 1), ("acoustic", 450, 190, 32, 1),
         ("acoustic", 780, 270, 122, 1), ("acoustic", 780, 255, 116, 1), ("acoustic", 780, 255, 122, 1),
         ("elastic", 20, 10, 5, 1), ("elastic", 20, 10, 23, 1), ("elastic", 61, 30, 57, 3),
         ("elastic", 230, 100, 40, 2), ("elastic", 260, 110, 40, 2), ("elastic", 350, 166, 122, 1),
         ("elastic", 350, 166, 112, 1), ("elastic", 380, 170, 122, 1)]


@pytest.mark.parametrize("order", [2, 8])
@pytest.mark.parametrize("kind,nx,ny,nz,nbc", SIZES)
def test_cuts_equal_per_cell(fomo, kind, nx, ny, nz, nbc, order):
    rng = np.random.default_rng(nx + nz + order)
    vp = rng.uniform(2000, 3500, (nx, ny, nz)).astype(np.float32, order="F")
    rho = rng.uniform(1500, 2500, (nx, ny, nz)).astype(np.float32, order="F")
    vs = (vp / 1.9).astype(np.float32, order="F")
    kw = dict(sx=[nx // 2, 2], sy=[ny // 2, 2], sz=[nz // 2, 2], rx=[nx // 2 + 2, 3, nx],
              ry=[ny // 2, 4, ny], rz=[nz // 2, 3, nz], nbc=nbc, fd_order=order)
    pad = 2 * (nbc + order // 2)
    out = []
    for kernel in (0, 1):
        fin = np.zeros((nx + pad, ny + pad, nz + pad, 4 if kind == "acoustic" else 9), np.float32,
                       order="F")
        if kind == "acoustic":
            r = fomo.acoustic3d(vp, rho, 10.0, 1e-3, 12, 40.0, kernel=kernel, final_state=fin, **kw)
        else:
            r = fomo.elastic3d(vp, vs, rho, 10.0, 8e-4, 12, 40.0, kernel=kernel, final_state=fin,
                               **kw)
        assert fomo.api.last_stats.kernel == (1 if kernel else 2)
        out.append((r[0], r[1], r[2], fin))
    assert np.abs(out[1][3]).max() > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
