"""Passes that do run behind the word-level filter, as its counter says: every
layout with more than one slot block, deletions, other start masks, graph
replay and new states, against the oracle; and what the density's sample and
the pause decide, with both sides' reports."""
import numpy as np
import pytest

import oracle
from test_filter_gpu import _database, _same, _trail_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_words", [5, 16, 31, 32, 33, 45, 64, 96, 130])
@pytest.mark.parametrize("graph", [False, True])
def test_every_pass_filtered(lib, n_words, graph):
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(100 + n_words)
    n_vars, n = 700, 3000
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, n, n_vars, model, (33, 64, 65, 257, 500))
    start = np.full(n_words, 0xFFFFFFFF, np.uint32)
    start[rng.integers(0, n_words, max(1, n_words // 8))] = rng.integers(0, 2 ** 32, max(1, n_words // 8))
    start[n_words // 2] = 0
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_graph(graph)
    alive = np.ones(n, bool)
    passes = 0
    for k in range(4):
        state = _trail_state(rng, n_vars, n_words, model, flips=6)
        eng.set_state(state, start)
        assert _same(eng, lits, offsets, state, start, alive) > 0
        eng.set_start(start ^ np.uint32(0x0F0F00FF))
        _same(eng, lits, offsets, state, start ^ np.uint32(0x0F0F00FF), alive)
        passes += 2
        dead = rng.choice(np.nonzero(alive)[0], n // 8, replace=False).astype(np.uint32)
        eng.delete(dead)
        alive[dead] = False
        _same(eng, lits, offsets, state, start ^ np.uint32(0x0F0F00FF), alive)
        passes += 1
    assert eng.filtered_passes == passes
    assert eng.graph_captures == (1 if graph else 0)
    eng.close()


@pytest.mark.parametrize("n_words", [8, 20, 32, 40])
def test_states_from_dense_to_sparse_and_back(lib, n_words):
    """Fair-coin states between trails: those run plain, the trails behind the
    filter at once, from host and device buffers."""
    import torch
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(n_words)
    n_vars, n = 600, 3000
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, n, n_vars, model)
    start = np.full(n_words, 0xFFFFFFFF, np.uint32)
    ds = torch.from_numpy(start.view(np.int32)).cuda()
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    for k, dense in enumerate((1, 1, 0, 1, 0, 0, 1)):
        state = _trail_state(rng, n_vars, n_words, model, flips=6, wild=n_words if dense else 0)
        for device in (False, True):
            if device:
                dev = torch.from_numpy(state.view(np.int32)).cuda()
                eng.set_state_device(dev.data_ptr(), n_vars, n_words, ds.data_ptr())
            else:
                eng.set_state(state, start)
            before = eng.filtered_passes
            for _ in range(3):
                _same(eng, lits, offsets, state, start)
            ran = eng.filtered_passes - before
            assert ran == 0 if dense else ran >= 2
    eng.close()


def test_table_filled_over_a_resident_state(lib):
    """A large state against a small database: the first passes run plain, the
    later ones behind a table filled in place."""
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(3)
    n_vars, n_words, n = 60_000, 40, 2000
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, n, n_vars, model, (40, 300))
    state = _trail_state(rng, n_vars, n_words, model, flips=200)
    start = rng.integers(0, 2 ** 32, n_words, dtype=np.uint32)
    ref = oracle.check(lits, offsets, state, start)
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_state(state, start)
    ran = []
    for _ in range(12):
        got = g.sort_reports(eng.check())
        ran.append(eng.filtered_passes)
        assert len(got) == len(ref)
        for f in ("clause", "word", "mask"):
            np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    assert ran[-1] > ran[0]
    eng.close()


def test_pause_is_short_for_one_bad_state(lib):
    """One state of which the filter keeps nearly everything between states of
    which it keeps little: reports as the oracle's throughout, and the good
    states are back behind the filter after four plain passes."""
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(8)
    n_vars, n, n_words = 600, 3000, 32
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, n, n_vars, model)
    start = np.full(n_words, 0xFFFFFFFF, np.uint32)
    good = _trail_state(rng, n_vars, n_words, model, flips=3)
    bad = good.copy()  # unassigned for the most part: short clauses report, and long ones may in some slot
    bad[:, :, 1] = ~bad[:, :, 1]
    bad[rng.random((n_vars, n_words)) < 0.1] = 0
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    ran = []
    for k in range(10):
        state = bad if k == 2 else good
        eng.set_state(state, start)
        before = eng.filtered_passes
        _same(eng, lits, offsets, state, start)
        ran.append(eng.filtered_passes - before)
    assert ran[:3] == [1, 1, 1] and ran[7:] == [1, 1, 1]
    eng.close()
