"""The training kernel's gradient and the scorer's logits at the edges of
their tiles (32 and 16 rows), with one tile per block and with several, against
the float64 restatement."""
import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu


def _case(lib, n):
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(n)
    s = g.Scorer(0, seed=3)
    w = s.weights()
    w[mlp.O_B1:mlp.O_W2] = rng.uniform(-0.2, 0.2, mlp.H)
    w[mlp.O_B2:mlp.O_W3] = rng.uniform(-0.2, 0.2, mlp.H)
    s.set_weights(w)
    x = rng.random((n, g.SCORER_FEATURES), dtype=np.float32)
    y = (rng.random(n) < 0.3).astype(np.float32)
    return s, w, x, y


@pytest.mark.parametrize("n", [1, 31, 32, 33, 152 * 32 - 1, 152 * 32, 152 * 32 + 1, 20011])
def test_gradient_at_tile_edges(lib, n):
    s, w, x, y = _case(lib, n)
    grad, loss = s.gradient(x, y)
    want_loss, want = mlp.loss_and_grad(w.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    # FP32 dot products of 64 terms and means over n rows: a few hundred units
    # in the last place of the largest entry. A ReLU whose input rounds to the
    # other side of zero moves one unit's 77 entries by a row's share, 1/n.
    off = np.abs(grad - want)
    tight = 512 * 2.0 ** -24 * np.abs(want).max()
    assert off.max() <= tight + 1.0 / n and (off > tight).mean() <= 0.02
    assert abs(loss - want_loss) <= 64 * 2.0 ** -24 * abs(want_loss)
    again, _ = s.gradient(x, y)
    np.testing.assert_array_equal(grad, again)
    s.train_step(x, y, lr=1e-3)
    assert np.isfinite(s.weights()).all()
    s.close()


@pytest.mark.parametrize("n", [1, 7, 8, 15, 16, 17, 40000, 70001])
def test_logits_at_tile_edges(lib, n):
    s, w, x, _ = _case(lib, n)
    got = s.infer(x)
    want = mlp.forward(w.astype(np.float64), x.astype(np.float64))[0]
    # BF16 operands: 8 bits, sums of 12 and 64 terms of size one
    assert np.abs(got - want).max() <= 0.1
    one = np.concatenate([s.infer(x[k:k + 1]) for k in range(0, n, max(1, n // 40))])
    np.testing.assert_array_equal(got[::max(1, n // 40)], one)
    s.close()
