"""Gradients of the boundary network at the edges of the training kernel's row
tiles, against float64, with a bound from the rounding errors of float32."""
import numpy as np
import pytest

import mlp_oracle

pytestmark = pytest.mark.gpu


def exact(p, x, t, batch):
    """float64 gradients, and the same sums over absolute values."""
    q = mlp_oracle.unpack(p)
    w1, w2, w3 = (mlp_oracle.bf16_round(q[k]).astype(np.float64) for k in ("w1", "w2", "w3"))
    b1, b2, b3 = (q[k].astype(np.float64) for k in ("b1", "b2", "b3"))
    x, t = x.astype(np.float64), t.astype(np.float64)

    def sums(a1, a2, a3, c1, c2, c3, xx, tt, absolute):
        z1 = xx @ a1.T + c1
        h1 = np.maximum(z1, 0)
        z2 = h1 @ a2.T + c2
        h2 = np.maximum(z2, 0)
        e = h2 @ a3 + c3 + (np.abs(tt) if absolute else -tt)
        dy = 2.0 * e / batch
        d2 = np.outer(dy, a3) * (z2 > 0)
        d1 = (d2 @ a2) * (z1 > 0)
        g = np.concatenate([(d1.T @ xx).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dy, [dy.sum()]])
        return g, (e * e).sum(), z1, z2

    g, loss, z1, z2 = sums(w1, w2, w3, b1, b2, b3[0], x, t, False)
    ga, la, _, _ = sums(*(np.abs(a) for a in (w1, w2, w3, b1, b2)), abs(b3[0]), np.abs(x), t, True)
    return g, ga, loss, la, z1, z2


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 1000, 148 * 64 + 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_gradient_at_tile_edges(rw, rows, offset):
    import torch
    rng = np.random.default_rng(rows)
    p = rng.normal(0, 0.3, rw.MLP_PARAMS).astype(np.float32)
    x = rng.normal(0, 1, (rows + 400 + rows // 2, 16)).astype(np.float32)
    t = rng.normal(0, 1, len(x)).astype(np.float32)
    # rows whose hidden units all stay off zero, so that float32 and float64
    # agree on which units are active (their errors are below 1e-4)
    _, _, _, _, z1, z2 = exact(p, x, t, rows)
    keep = np.flatnonzero((np.abs(z1).min(1) > 1e-4) & (np.abs(z2).min(1) > 1e-4))[:rows]
    assert len(keep) == rows
    x, t = x[keep], t[keep]
    want, size, loss, loss_size, _, _ = exact(p, x, t, rows)
    dp, dx, dt = (torch.from_numpy(a).cuda() for a in (p, x, t))
    grad = torch.zeros(rw.MLP_PARAMS + 1, device="cuda")[offset:][:rw.MLP_PARAMS]  # 16-byte aligned or not
    g, got_loss = rw.mlp_grad(dp, dx, dt, rows, grad=grad)
    # every value is a sum of products through three layers: at most
    # 16 + 64 + 64 + 64 roundings on a path and rows more in the last sum
    bound = (208 + rows) * 2.0 ** -24 * np.maximum(size, 1e-30)
    assert (np.abs(g.cpu().numpy() - want) <= bound).all()
    assert abs(float(got_loss.item()) - loss) <= (208 + rows) * 2.0 ** -23 * loss_size
