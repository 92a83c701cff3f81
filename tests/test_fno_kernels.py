"""FNO kernels at the edges of their tiles: mode counts from 1 (one chunk of
the mode lists, most of it padding) to 16, maps of 8 rows (less than one row
tile) to 256, and batches that leave the row runs, the mixing lists and the
pixel tiles with remainders.  Device against the FP64 network on the CPU.

Bounds, from BF16's unit roundoff 2^-9 = 2e-3 (grids of 128 on multiply BF16
operands, smaller ones FP32): an output passes two rounded activations per
layer and the projection, errors adding as root mean squares, about
sqrt(2 L + 3) x 2e-3 < 7e-3 of its norm; 2e-2 leaves the outputs' small mean.
A gradient passes the same chain twice: 5e-2, and 0.999 for the cosine, which
an angle of 5e-2 gives (1 - 0.05^2 / 2)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("S,M,L,batch", [(8, 1, 1, 1), (16, 5, 2, 17), (64, 12, 2, 3),
                                         (128, 1, 1, 3), (128, 16, 3, 1), (256, 5, 1, 1)])
def test_forward_and_gradients(S, M, L, batch):
    import torch
    from highuvlith_b200.fno import FnoSurrogate
    from oracle import fno_ref
    net = FnoSurrogate(grid=S, modes=M, layers=L, seed=11)
    rng = np.random.default_rng(S + M)
    masks = (rng.random((batch, S, S)) > 0.5).astype(np.float32)
    targets = rng.random((batch, S, S)).astype(np.float32)
    params = net.get_params()
    dm = torch.from_numpy(masks).cuda()
    out = net.forward(dm).cpu().numpy()
    ref, p, a = fno_ref.forward(params.astype(np.float64), masks, S, m=M, L=L, requires_grad=True)
    assert _rel(out, ref.detach().numpy()) < 2e-2
    loss_ref = ((ref - torch.tensor(targets, dtype=torch.float64)) ** 2).mean()
    loss_ref.backward()
    loss, pg, ig = net.backward(dm, targets=torch.from_numpy(targets).cuda(), want_input_grad=True)
    net.device_status()  # no bounded device-side wait gave up
    assert abs(loss - loss_ref.item()) < 2e-2 * loss_ref.item()
    for got, want in ((pg.cpu().numpy(), p.grad.numpy()), (ig.cpu().numpy(), a.grad.numpy())):
        got, want = got.ravel().astype(np.float64), want.ravel()
        assert _rel(got, want) < 5e-2
        assert np.dot(got, want) / (np.linalg.norm(got) * np.linalg.norm(want)) > 0.999
