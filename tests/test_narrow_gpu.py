"""Passes of few words, checked a lane per clause: every word count of that
path and the next ones, clauses from one literal to hundreds, databases at the
edges of a warp's 32 clauses, fair-coin and trail-like states, deletions, and
the learned order's permutation, against the oracle."""
import numpy as np
import pytest

import oracle
from gpusharesat_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _same(rep, ref, alive=None):
    import gpusharesat_gb300 as g
    if alive is not None:
        ref = ref[alive[ref["clause"]]]
    rep = g.sort_reports(rep)
    assert len(rep) == len(ref)
    for f in ("clause", "word", "mask"):
        np.testing.assert_array_equal(rep[f], ref[f], err_msg=f)


@pytest.mark.parametrize("n_words", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n,n_vars", [(1, 40), (32, 40), (33, 700), (4000, 700), (70000, 5000)])
def test_narrow_pass_equals_oracle(lib, n_words, n, n_vars):
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(n_words * 7 + n)
    lengths = rng.integers(1, 14, n)
    if n > 1000:
        lengths[rng.choice(n, 12, replace=False)] = [31, 32, 33, 34, 63, 64, 65, 100, 255, 256, 257, 600]
    lits, offsets = W.distinct_var_clauses(rng, lengths, n_vars)
    state = W.random_state(rng, n_vars, n_words, rng.uniform(0.3, 0.99, 32 * n_words))
    if n > 1000:  # long clauses that report, in the last word
        for c in np.nonzero(lengths > 30)[0]:
            v = lits[offsets[c]:offsets[c + 1]] >> 1
            state[v, n_words - 1, 0] |= np.uint32(1 << 7)
            t = (state[v, n_words - 1, 1] >> np.uint32(7)) & 1
            lits[offsets[c]:offsets[c + 1]] = 2 * v + t.astype(np.int32)
    start = rng.integers(0, 2 ** 32, n_words, dtype=np.uint32)
    start[n_words - 1] |= np.uint32(1 << 7)
    ref = oracle.check(lits, offsets, state, start)
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_state(state, start)
    _same(eng.check(), ref)
    eng.set_start(np.zeros(n_words, np.uint32))
    assert len(eng.check()) == 0
    eng.set_start(start)
    alive = np.ones(n, bool)
    if n > 1000:
        dead = rng.choice(n, n // 3, replace=False)
        eng.delete(dead.astype(np.uint32))
        alive[dead] = False
        _same(eng.check(), ref, alive)
    eng.order_enable(head_fraction=0.4, retrain_interval=0)
    for _ in range(3):
        eng.launch()
        _same(np.concatenate([eng.wait_head(), eng.copy_tail()]), ref, alive)
    eng.close()
