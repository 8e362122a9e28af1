"""Binary16 batches on the shot-pair sweep (binary16 values in FP32 words) against
the oracle's storage emulation, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# odd batches (a zero shot rides along), a zone inside and outside the FP32 band,
# sources inside and outside the band, a grid that is all band
@pytest.mark.parametrize("nx,nz,nbc,order,shots", [(130, 75, 40, 10, 3), (70, 60, 12, 8, 2),
                                                   (26, 20, 9, 4, 5), (240, 31, 60, 2, 3)])
def test_fp16_pairs_bitwise(fomo, oracle, nx, nz, nbc, order, shots):
    from fomo_b200.synthetic import layered_elastic

    vp, vs, rho = layered_elastic(nx, nz, n_layers=4, seed=nx)
    nt, pad = 220, nbc + order // 2
    sx = np.linspace(1, nx, shots).astype(int)[:, None]
    sz = np.linspace(1, nz, shots).astype(int)[:, None]
    rx = np.arange(1, nx + 1, 3)
    rz = np.full(rx.size, nz // 2)
    fin = np.zeros((nx + 2 * pad, nz + 2 * pad, 5, shots), np.float32, order="F")
    r = fomo.elastic2d_batch(vp, vs, rho, 5.0, 5e-4, nt, 20.0, sx=sx, sz=sz, rx=rx, rz=rz,
                             nbc=nbc, fd_order=order, precision="fp16", kernel=2, final_state=fin)
    assert fomo.api.last_stats.sweep_config // 1000000 == 24
    w = fomo.ricker_wavelet(20.0, 5e-4, nt).reshape(1, -1)
    o = oracle.elastic2d(vp, vs, rho, 5.0, 5e-4, nt, sx=sx.T, sz=sz.T, rx=rx, rz=rz, wavelet=w,
                         nbc=nbc, fd_order=order, n_shots=shots, final=True, store="fp16",
                         sv=2.0 ** 22, st=1.0, fp32_band=32)
    assert np.array_equal(r.seis_vx, o["seis_vx"])
    assert np.array_equal(r.seis_vz, o["seis_vz"])
    assert np.array_equal(fin, o["final"])
