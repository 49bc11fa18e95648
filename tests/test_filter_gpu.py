"""The word-level filter in front of the exact check: passes on trail-like
states, where it is in use, equal the oracle's and the plain kernel's, for
every layout, odd word counts, ragged starts, deletions, graphs and the
learned order; and the table follows every state that is set."""
import numpy as np
import pytest

import oracle
from gpusharesat_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _trail_state(rng, n_vars, n_words, model, flips, wild=0):
    """Each word one solver's trail of model values, a few variables changed
    from slot to slot; the last `wild` words fair coins."""
    state = np.zeros((n_vars, n_words, 2), np.uint32)
    state[:, :, 0] = np.where(rng.random((n_vars, n_words)) < 0.5, np.uint32(0xFFFFFFFF), np.uint32(0))
    state[:, :, 1] = np.where(model[:, None] == 1, np.uint32(0xFFFFFFFF), np.uint32(0))
    k = flips * n_words
    v, w, b = rng.integers(0, n_vars, k), rng.integers(0, n_words, k), rng.integers(0, 32, k)
    np.bitwise_xor.at(state[:, :, 0], (v, w), (np.uint32(0xFFFFFFFF) << b.astype(np.uint32)))
    v, w, b = rng.integers(0, n_vars, k), rng.integers(0, n_words, k), rng.integers(0, 32, k)
    np.bitwise_xor.at(state[:, :, 1], (v, w), np.uint32(1) << b.astype(np.uint32))
    if wild:
        state[:, n_words - wild:] = rng.integers(0, 2 ** 32, (n_vars, wild, 2), dtype=np.uint32)
    return state


def _database(rng, n, n_vars, model, long=()):
    lengths = np.concatenate([rng.integers(1, 12, n - len(long)), np.array(long, np.int64)]).astype(np.int64)
    rng.shuffle(lengths)
    lits, offsets = W.model_clauses(rng, np.maximum(lengths, 2), n_vars, model)
    # one clause in 16 false under the model, so that trails report it
    bad = np.nonzero(rng.random(n) < 1 / 16)[0]
    for c in bad:
        b, e = offsets[c], offsets[c + 1]
        lits[b:e] = 2 * (lits[b:e] >> 1) + model[lits[b:e] >> 1]
    return lits, offsets


def _same(eng, lits, offsets, state, start, alive=None):
    import gpusharesat_gb300 as g
    ref = oracle.check(lits, offsets, state, start)
    if alive is not None:
        ref = ref[alive[ref["clause"]]]
    got = g.sort_reports(eng.check())
    assert len(got) == len(ref)
    for f in ("clause", "word", "mask"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    return len(got)


@pytest.mark.parametrize("n_words", [5, 7, 8, 9, 11, 15, 16, 17, 31, 32, 33, 45, 96])
@pytest.mark.parametrize("n", [1, 31, 33, 3000])
def test_filtered_pass_equals_oracle(lib, n_words, n):
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(n_words * 31 + n)
    n_vars = 700
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    long = (33, 64, 65, 257, 500) if n > 100 else ()
    lits, offsets = _database(rng, n, n_vars, model, long)
    state = _trail_state(rng, n_vars, n_words, model, flips=12, wild=n_words // 12)
    start = rng.integers(0, 2 ** 32, n_words, dtype=np.uint32)
    start[rng.integers(0, n_words)] = 0
    start[0] = 0xFFFFFFFF
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_state(state, start)
    found = _same(eng, lits, offsets, state, start)
    assert found > 0 or n < 100
    eng.set_start(start ^ np.uint32(0x00FF00FF))
    _same(eng, lits, offsets, state, start ^ np.uint32(0x00FF00FF))
    if n > 100:
        dead = rng.choice(n, n // 3, replace=False).astype(np.uint32)
        eng.delete(dead)
        eng.set_graph(True)
        alive = np.ones(n, bool)
        alive[dead] = False
        for _ in range(2):
            state = _trail_state(rng, n_vars, n_words, model, flips=30)
            eng.set_state(state, start)
            _same(eng, lits, offsets, state, start, alive)
    eng.close()


def test_states_from_device_and_host_agree(lib):
    """Device buffers, aligned to 8 bytes and not, and host buffers."""
    import torch
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(5)
    n_vars = 500
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, 2000, n_vars, model)
    for n_words in (1, 3, 8, 32, 40):
        state = _trail_state(rng, n_vars, n_words, model, flips=8)
        start = np.full(n_words, 0xFFFFFFFF, np.uint32)
        eng = g.Engine(0)
        eng.set_db(lits, offsets)
        flat = torch.zeros(state.size + 1, dtype=torch.int32, device="cuda")
        ds = torch.from_numpy(start.view(np.int32)).cuda()
        for shift in (0, 1):
            flat[shift:shift + state.size] = torch.from_numpy(state.reshape(-1).view(np.int32)).cuda()
            # no wait here: the call orders itself behind the default stream
            eng.set_state_device(flat.data_ptr() + 4 * shift, n_vars, n_words, ds.data_ptr())
            flat.zero_()
            _same(eng, lits, offsets, state, start)
        eng.close()


def test_filter_through_learned_order_and_host_passes(lib):
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(6)
    n_vars, n = 900, 4000
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, n, n_vars, model, (40, 300))
    start = np.full(40, 0xFFFFFFFF, np.uint32)
    states = [_trail_state(rng, n_vars, 40, model, flips=10 + 40 * k) for k in range(4)]
    states.append(_trail_state(rng, n_vars, 40, model, flips=10, wild=40))  # the filter keeps nearly all of these
    refs = [oracle.check(lits, offsets, s, start) for s in states]
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    for reps in (g.passes_host(eng, states, start), g.passes_host(eng, states[::-1], start)[::-1]):
        for rep, ref in zip(reps, refs):
            rep = g.sort_reports(rep)
            assert len(rep) == len(ref)
            for f in ("clause", "word", "mask"):
                np.testing.assert_array_equal(rep[f], ref[f], err_msg=f)
    eng.order_enable(head_fraction=0.3, retrain_interval=0)
    for state, ref in zip(states, refs):
        eng.set_state(state, start)
        eng.launch()
        rep = g.sort_reports(np.concatenate([eng.wait_head(), eng.copy_tail()]))
        assert len(rep) == len(ref)
        for f in ("clause", "word", "mask"):
            np.testing.assert_array_equal(rep[f], ref[f], err_msg=f)
    eng.close()


def test_reports_do_not_depend_on_the_pause(lib):
    """A state whose filter keeps most clauses (every clause reports) turns it
    off for some passes; the reports are the same with it, without, and after
    it is tried again."""
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(8)
    n_vars, n, n_words = 600, 3000, 32
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    var = rng.integers(0, n_vars, 2 * n)
    lits = (2 * var + model[var]).astype(np.int32)  # false under the model
    offsets = np.arange(0, 2 * n + 1, 2, dtype=np.int64)
    state = _trail_state(rng, n_vars, n_words, model, flips=3)
    start = np.full(n_words, 0xFFFFFFFF, np.uint32)
    ref = oracle.check(lits, offsets, state, start)
    assert len(ref) > n * n_words // 4
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_state(state, start)
    for _ in range(70):
        got = g.sort_reports(eng.check())
        assert len(got) == len(ref)
        for f in ("clause", "word", "mask"):
            np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    eng.close()


def test_masks_at_any_address(lib):
    """Device masks that start between words are read as they are."""
    import torch
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(9)
    n_vars, n_words = 400, 9
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, 1500, n_vars, model)
    state = _trail_state(rng, n_vars, n_words, model, flips=8)
    start = rng.integers(0, 2 ** 32, n_words, dtype=np.uint32)
    solver = rng.integers(0, 50, n_words).astype(np.int32)
    ref = oracle.check(lits, offsets, state, start)
    ds = torch.from_numpy(state.view(np.int32)).cuda()
    for shift in (0, 1, 2, 3):
        masks = [torch.zeros(4 * n_words + 4, dtype=torch.uint8, device="cuda") for _ in range(2)]
        for m, src in zip(masks, (start, solver)):
            m[shift:shift + 4 * n_words] = torch.from_numpy(src.view(np.uint8)).cuda()
        eng = g.Engine(0)
        eng.set_db(lits, offsets)
        eng.set_state_device(ds.data_ptr(), n_vars, n_words, masks[0].data_ptr() + shift, masks[1].data_ptr() + shift)
        got = g.sort_reports(eng.check())
        assert len(got) == len(ref)
        for f in ("clause", "word", "mask"):
            np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
        np.testing.assert_array_equal(got["solver"], solver[got["word"]])
        eng.close()


def test_tables_make_room(lib):
    """Without room for the queues the filter's table goes, not the pass."""
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(10)
    n_vars, n_words = 500, 40
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, 2000, n_vars, model)
    state = _trail_state(rng, n_vars, n_words, model, flips=8)
    start = np.full(n_words, 0xFFFFFFFF, np.uint32)
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_state(state, start)
    try:
        g.debug_fail_device_alloc(1 << 23, 1)  # the queues, 16 MB
        _same(eng, lits, offsets, state, start)
        eng.set_state(state, start)
        _same(eng, lits, offsets, state, start)
        g.debug_fail_device_alloc(1 << 23, 2)  # with the table gone there is still no room
        eng.set_capacity(1 << 22)
        with pytest.raises(g.GssError):
            eng.check()
    finally:
        g.debug_fail_device_alloc(0, 0)
    _same(eng, lits, offsets, state, start)
    eng.close()


@pytest.mark.parametrize("n_words,ok", [(16, False), (17, False), (31, False), (32, True), (33, True)])
def test_length_plan_wants_full_blocks(lib, n_words, ok):
    import gpusharesat_gb300 as g
    rng = np.random.default_rng(n_words)
    n_vars = 300
    model = rng.integers(0, 2, n_vars).astype(np.uint8)
    lits, offsets = _database(rng, 500, n_vars, model)
    state = _trail_state(rng, n_vars, n_words, model, flips=8)
    start = np.full(n_words, 0xFFFFFFFF, np.uint32)
    eng = g.Engine(0)
    eng.set_db(lits, offsets)
    eng.set_state(state, start)
    eng.set_length_plan((4, 1 << 30), [g.LAYOUT_4x8_G2, g.LAYOUT_4x8_G1])
    if ok:
        _same(eng, lits, offsets, state, start)
    else:
        with pytest.raises(g.GssError):
            eng.check()
    eng.close()
