"""Report records that come back with a pass's counters: passes with as many
records as that buffer holds, one fewer, one more and none, plain, replayed as
a graph and through the learned order's head and tail."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INLINE = 65520  # kEngineInline


def _unit_clauses(eng, n, n_words):
    """n unit clauses of unassigned variables: every word reports each."""
    eng.set_db(2 * np.arange(n, dtype=np.int32) % 2000, np.arange(n + 1, dtype=np.int64))
    eng.set_state(np.zeros((1000, n_words, 2), np.uint32), np.full(n_words, 0xF, np.uint32))


def _check(rep, n, n_words):
    import gpusharesat_gb300 as g
    rep = g.sort_reports(rep)
    assert len(rep) == n * n_words
    np.testing.assert_array_equal(rep["clause"], np.repeat(np.arange(n), n_words))
    np.testing.assert_array_equal(rep["word"], np.tile(np.arange(n_words), n))
    np.testing.assert_array_equal(rep["solver"], rep["word"])
    assert (rep["mask"] == 0xF).all()


@pytest.mark.parametrize("n_words,n", [(1, 1), (1, INLINE - 1), (1, INLINE), (1, INLINE + 1), (32, INLINE // 32),
                                       (32, INLINE // 32 + 1), (32, 0)])
@pytest.mark.parametrize("graph", [False, True])
def test_records_at_the_inline_limit(lib, n_words, n, graph):
    import gpusharesat_gb300 as g
    eng = g.Engine(0)
    eng.set_graph(graph)
    _unit_clauses(eng, n, n_words)
    for _ in range(2):
        _check(eng.check(), n, n_words)
    # fewer records after more, in the same buffer
    eng.set_start(np.zeros(n_words, np.uint32))
    assert len(eng.check()) == 0
    eng.close()


@pytest.mark.parametrize("n", [40, INLINE // 32, INLINE // 32 + 1, INLINE // 8])
def test_head_and_tail_records(lib, n):
    import gpusharesat_gb300 as g
    eng = g.Engine(0)
    _unit_clauses(eng, n, 32)
    eng.order_enable(head_fraction=0.25, retrain_interval=0)
    for _ in range(3):
        eng.launch()
        head = eng.wait_head()
        tail = eng.copy_tail()
        assert len(head) and len(tail)
        _check(np.concatenate([head, tail]), n, 32)
        _check(eng.reports(), n, 32)
    eng.close()
