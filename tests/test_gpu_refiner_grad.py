"""Loss and gradient of the refinement network at the edges of its tiles: one to a few tiles, odd widths, the largest network."""
import numpy as np
import pytest

import curfil_b200 as cf

pytestmark = pytest.mark.gpu

U = 2.0 ** -24   # rounding of float32


@pytest.fixture(scope="module")
def ctx():
    from curfil_b200 import _build
    _build.build()
    c = cf.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("classes,hidden,n", [(2, 1, 1), (2, 128, 64), (3, 9, 65), (13, 64, 130), (33, 127, 63), (64, 128, 129)])
def test_gradient_within_the_rounding_bound(ctx, classes, hidden, n):
    """Against float64, each entry within the bound that float32 sums of these lengths have (first order)."""
    D = 3 * classes + 2
    r = cf.Refiner(ctx, classes, hidden=hidden, seed=5)
    rng = np.random.default_rng(classes * 1000 + n)
    params = (rng.standard_normal(r.params().size) * 0.2).astype(np.float32)
    r.params(params)
    X = rng.random((n, D)).astype(np.float32)
    Y = rng.integers(0, classes, n).astype(np.uint8)
    loss, g = r.loss_grad(X, Y)
    r.close()

    p, x = params.astype(np.float64), X.astype(np.float64)
    cut = np.cumsum([hidden * D, hidden, classes * hidden])
    W1, b1, W2, b2 = np.split(p, cut)
    W1, W2 = W1.reshape(hidden, D), W2.reshape(classes, hidden)
    a = x @ W1.T + b1
    ea = (D + 2) * U * (x @ np.abs(W1).T + np.abs(b1))
    h = np.maximum(a, 0)
    z = h @ W2.T + b2
    ez = ea @ np.abs(W2).T + (hidden + 2) * U * (h @ np.abs(W2).T + np.abs(b2))
    ez = ez.max(axis=1, keepdims=True)
    soft = np.exp(z - z.max(axis=1, keepdims=True))
    total = soft.sum(axis=1, keepdims=True)
    soft /= total
    onehot = np.eye(classes)[Y]
    dz = (soft - onehot) / n
    edz = (soft * (2 * ez + (classes + 32) * U) + 4 * U) / n
    G = (dz @ W2) * (a > 0)
    # where the sign of the pre-activation is within its rounding, the whole term may be there or not
    eG = edz @ np.abs(W2) + (classes + 2) * U * (np.abs(dz) @ np.abs(W2)) + (np.abs(a) <= ea) * np.abs(dz @ W2)
    steps = (n + 2) * U
    want = np.concatenate([(G.T @ x).ravel(), G.sum(0), (dz.T @ h).ravel(), dz.sum(0)])
    bound = np.concatenate([((eG + steps * np.abs(G)).T @ x).ravel(), (eG + steps * np.abs(G)).sum(0),
                            ((edz + steps * np.abs(dz)).T @ h + np.abs(dz).T @ ea).ravel(),
                            (edz + steps * np.abs(dz)).sum(0)])
    assert np.all(np.abs(g - want) <= bound), float((np.abs(g - want) / bound).max())
    want_loss = float(np.mean(np.log(total[:, 0]) + z.max(axis=1) - z[np.arange(n), Y]))
    assert abs(loss - want_loss) <= float(np.mean(2 * ez)) + (classes + 32 + n) * U * (1 + float(np.abs(z).max()))
