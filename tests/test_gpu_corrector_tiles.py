"""The corrector's convolutions in staged tiles and its weight gradients in twelve warps: edges
of tiles, few and many blocks, more than one chunk of partials, and features off a 16-byte
boundary.  Tolerances are those of the kernels' other oracle tests (BF16 storage, FP32 sums)
times ten for images of under 500 pixels, where a rounding of a stored activation that falls
the other way (2^-9 of it) is not averaged out."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _inputs(n, h, w, seed):
    import torch

    from fomo_b200 import corrector as CR
    from oracle import corrector_ref as R

    K = CR.Kernels(0)
    rng = np.random.default_rng(seed)
    f = torch.zeros(n, h, w, 16, dtype=torch.bfloat16, device=K.dev)
    f[..., :6] = torch.from_numpy(rng.standard_normal((n, h, w, 6)).astype(np.float32)).to(K.dev)
    params = CR.init_params(seed)
    params[-R.N3:] = 0.1 * rng.standard_normal(R.N3).astype(np.float32)
    return K, f, torch.from_numpy(params).to(K.dev), params, rng


# one row and column, widths around 16 and 64, heights around 4; blocks of one and of four rows
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (2, 5, 15), (1, 3, 17), (3, 4, 63), (2, 9, 65),
                                   (40, 7, 129), (75, 13, 66)])
def test_forward_tiles(n, h, w):
    from oracle import corrector_ref as R

    K, f, p, params, _ = _inputs(n, h, w, n + h + w)
    y = K.forward(f, p)
    want, _ = R.forward(f[..., :6].float().cpu().numpy(), params, bf16=True)
    assert rel_l2(y.cpu().numpy(), want) < 2e-3 * (10 if n * h * w < 500 else 1)
    # an image alone (blocks of one row) has the bits it has in the batch
    for k in {0, n - 1}:
        assert np.array_equal(K.forward(f[k:k + 1], p)[0].cpu().numpy(), y[k].cpu().numpy())


@pytest.mark.parametrize("n,h,w", [(1, 1, 16), (2, 5, 48), (5, 21, 80), (33, 64, 64)])
def test_gradient_tiles(n, h, w):
    import torch

    from oracle import corrector_ref as R

    K, f, p, params, rng = _inputs(n, h, w, 7 * n + h)
    target = torch.from_numpy(rng.standard_normal((n, h, w)).astype(np.float32)).to(K.dev)
    loss, grad = K.gradients(f, target, None, p)
    l_bf, g_bf, _ = R.loss_and_grad(f[..., :6].float().cpu().numpy(), target.cpu().numpy(), params,
                                    np.ones((n, h, w), np.float32), bf16=True)
    slack = 10 if n * h * w < 500 else 1
    assert abs(float(loss.item()) - l_bf) <= 2e-3 * slack * l_bf
    g = grad.cpu().numpy()
    for lo, hi in ((0, R.N1), (R.N1, R.N1 + R.N2), (R.N1 + R.N2, R.NPARAM)):
        assert rel_l2(g[lo:hi], g_bf[lo:hi]) < 5e-3 * slack, (lo, hi)
    # the same features four bytes past a 16-byte boundary
    flat = torch.empty(f.numel() + 2, dtype=torch.bfloat16, device=K.dev)
    f2 = flat[2:].view(f.shape)
    f2.copy_(f)
    assert f2.data_ptr() % 16 == 4
    loss2, grad2 = K.gradients(f2, target, None, p)
    assert torch.equal(loss, loss2) and torch.equal(grad, grad2)
