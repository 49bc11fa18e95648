"""The training kernel's gradient and Adam step, entry by entry, at the edges
of its tiles: against the float64 restatement, with a bound for every entry
that is carried through the network from the sizes of the terms.

The bound. A sum of k terms in FP32 is off by at most k units (2^-24) of the
sum of their absolute values. Run with absolute values, the network gives the
sums behind every logit (64 + 64 + 12 terms deep), and the backward pass run
with them gives A, the sum of the absolute terms behind every entry of the
gradient (64 + 64 terms, then the rows: a block's tiles of 32, up to 5 of them,
and a quarter of 152 blocks). That is 500 units of A with the functions'
roundings, 512 here. Rows with a unit so close to zero that rounding could
move it across are left out, so no ReLU is allowed for.

That the bound can fail: a gradient with the entries of any one layer's
weights or biases left out breaks it, in every case, and so does one without
the last row (CPU test below)."""
import numpy as np
import pytest

from oracle import mlp

U = 2.0 ** -24
SIZES = [1, 31, 32, 33, 152 * 32 - 1, 152 * 32, 152 * 32 + 1, 20011]
GROUPS = {"W1": (mlp.O_W1, mlp.O_B1), "b1": (mlp.O_B1, mlp.O_W2), "W2": (mlp.O_W2, mlp.O_B2),
          "b2": (mlp.O_B2, mlp.O_W3), "w3": (mlp.O_W3, mlp.O_B3), "b3": (mlp.O_B3, mlp.P)}


def _absolute(w, x):
    """The sums of absolute terms behind z1, z2 and the logit."""
    W1, b1, W2, b2, w3, b3 = (np.abs(a) for a in mlp.unpack(w))
    a1 = np.abs(x) @ W1.T + b1
    a2 = a1 @ W2.T + b2
    return a1, a2, a2 @ w3 + b3


def _case(n):
    """Weights, and n rows whose units all stay clear of zero."""
    rng = np.random.default_rng(n)
    w = np.zeros(mlp.P, np.float32)
    for (a, b), r in zip(GROUPS.values(), (0.7, 0.2, 0.3, 0.2, 0.3, 0.5)):
        w[a:b] = rng.uniform(-r, r, b - a)
    x = rng.random((n + n // 2 + 400, mlp.F), dtype=np.float32)
    w64, x64 = w.astype(np.float64), x.astype(np.float64)
    W1, b1, W2, b2, _, _ = mlp.unpack(w64)
    z1 = x64 @ W1.T + b1
    z2 = np.maximum(z1, 0) @ W2.T + b2
    a1, a2, _ = _absolute(w64, x64)
    clear = (np.abs(z1) > 16 * U * a1).all(1) & (np.abs(z2) > 96 * U * a2).all(1)
    x = x[clear][:n]
    assert len(x) == n
    y = (rng.random(n) < 0.3).astype(np.float32)
    return w, x, y


def _bound(w, x, y):
    """512 units of the absolute terms behind every entry."""
    w, x, y = (np.asarray(a, np.float64) for a in (w, x, y))
    W1, b1, W2, b2, w3, b3 = mlp.unpack(w)
    z, (_, h1, h2) = mlp.forward(w, x)
    a1, a2, a3 = _absolute(w, x)
    p = 1 / (1 + np.exp(-z))
    dz = (np.abs(p - y) + p * (1 - p) * a3) / len(y)
    d2 = np.outer(dz, np.abs(w3)) * (h2 > 0)
    d1 = (d2 @ np.abs(W2)) * (h1 > 0)
    a1, a2 = a1 * (h1 > 0), a2 * (h2 > 0)
    A = np.concatenate([(d1.T @ np.abs(x)).ravel(), d1.sum(0), (d2.T @ a1).ravel(), d2.sum(0), dz @ a2, [dz.sum()]])
    return 512 * U * A


@pytest.mark.parametrize("n", SIZES)
def test_bound_tells_a_missing_group(n):
    w, x, y = _case(n)
    _, g = mlp.loss_and_grad(w, x, y)
    bound = _bound(w, x, y)
    for name, (a, b) in GROUPS.items():
        wrong = g.copy()
        wrong[a:b] = 0
        assert (np.abs(wrong - g) > bound).any(), name
    # and the last row of the batch left out, with a head of zeros
    w[mlp.O_W3:] = 0
    _, g = mlp.loss_and_grad(w, x, y)
    less = mlp.loss_and_grad(w, x[:-1], y[:-1])[1] * (n - 1) / n if n > 1 else np.zeros(mlp.P)
    assert (np.abs(less - g) > _bound(w, x, y)).any()


@pytest.mark.gpu
@pytest.mark.parametrize("head", [True, False])
@pytest.mark.parametrize("n", SIZES)
def test_gradient_entry_by_entry(lib, n, head):
    """head False: the last layer's weights are zero, every logit is too, and
    b3's entry tells a single row of 20011."""
    import gpusharesat_gb300 as g
    w, x, y = _case(n)
    if not head:
        w[mlp.O_W3:] = 0
    s = g.Scorer(0)
    s.set_weights(w)
    grad, loss = s.gradient(x, y)
    want_loss, want = mlp.loss_and_grad(w, x, y)
    bound = _bound(w, x, y)
    for name, (a, b) in GROUPS.items():
        assert (np.abs(grad - want)[a:b] <= bound[a:b]).all(), name
    a3 = _absolute(w.astype(np.float64), x.astype(np.float64))[2]
    assert abs(loss - want_loss) <= 192 * U * (want_loss + a3.mean())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_adam_step_entry_by_entry(lib, n):
    """From zero moments the step is lr g / (|g| + eps), which grows with g:
    the new weight lies between what the two ends of g's bound give, to the
    rounding of the step (64 units of lr) and of the sum."""
    import gpusharesat_gb300 as g
    w, x, y = _case(n)
    s = g.Scorer(0)
    s.set_weights(w)
    lr = 1e-3
    s.train_step(x, y, lr=lr)
    _, want = mlp.loss_and_grad(w, x, y)
    bound = _bound(w, x, y)
    new = s.weights().astype(np.float64)
    room = 64 * U * lr + U * np.abs(w)
    for name, (a, b) in GROUPS.items():
        ends = []
        for e in (want + bound, want - bound):
            zero = np.zeros(mlp.P)
            ends.append(mlp.adam_step(w.astype(np.float64), e, zero, zero, 1, lr)[0])
        assert (new >= ends[0] - room)[a:b].all() and (new <= ends[1] + room)[a:b].all(), name
        moved = np.abs(want[a:b]) > 0
        assert (new[a:b] != w[a:b])[moved].mean() > 0.9 or not moved.any(), name
    s.close()
