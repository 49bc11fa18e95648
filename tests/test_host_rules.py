"""What the library's host code decides, over a CUDA runtime without a GPU
(fake_runtime.py)."""
import ctypes
import os
import subprocess

import pytest

from gpusharesat_gb300 import build

from fake_runtime import Fake, i64, vp


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return Fake(tmp_path_factory.mktemp("fake"))


@pytest.fixture(autouse=True)
def clean(fake):
    fake.reset()
    yield
    fake.reset()
    fake.lib.gss_debug_fail_device_alloc(i64(0), 0)


@pytest.mark.parametrize("what", ["malloc_host", "malloc"])
def test_engine_that_cannot_be_made_leaves_no_stream(fake, what):
    before = fake.lib.fake_streams()
    for after in range(3):
        fake.fail(what, after)
        rc, h = fake.engine()
        if rc == 0:  # fewer such allocations than that
            assert fake.lib.gss_engine_destroy(h) == 0
        else:
            assert h.value is None
        assert fake.lib.fake_streams() == before
    fake.fail(what)
    assert fake.engine()[0] != 0


def _noalloc(fake, lits=0, offsets=0, state=0, start=0, sow=0, out=0, counts=0, n=100):
    """One pass over buffers shifted by so many bytes; nothing is read."""
    room = ctypes.create_string_buffer(1 << 16)
    base = (ctypes.addressof(room) + 255) // 256 * 256
    p = [vp(base + 4096 * k + s) for k, s in enumerate((lits, offsets, state, start, sow, out, counts))]
    fake.reset()
    rc = fake.lib.gss_check_noalloc(p[0], p[1], n, p[2], 10, 1, p[3], p[4], p[5], 4, 16, p[6], None)
    return rc, [l.split()[1] for l in fake.log() if l.startswith("launch")], fake.log()


def test_noalloc_queue_address_picks_the_stores(fake):
    """A 16-byte store needs a queue on 16 bytes; a gss_report needs 4."""
    rc, wide, _ = _noalloc(fake)
    assert rc == 0 and len(wide) == 2 and "check_wide_persist" in wide[0]
    assert _noalloc(fake, out=16)[1] == wide and _noalloc(fake, out=32)[1] == wide
    by_word = set()
    for shift in (4, 8, 12, 20):
        rc, names, _ = _noalloc(fake, out=shift)
        assert rc == 0 and "check_wide_persist" in names[0]
        by_word.add(names[0])
    assert len(by_word) == 1 and wide[0] not in by_word


def test_noalloc_refuses_what_the_kernel_cannot_read(fake):
    for kw in ({"state": 8}, {"state": 16}, {"lits": 2}, {"offsets": 4}, {"start": 1}, {"sow": 2}, {"out": 2}):
        rc, names, _ = _noalloc(fake, **kw)
        assert rc == -1 and not names, kw
        assert _noalloc(fake, n=0, **kw)[0] == 0  # nothing to read
    rc, names, log = _noalloc(fake, counts=1)  # copied, not stored by a kernel
    assert rc == 0 and len(names) == 1 and any(l.startswith("copy2d") for l in log)


def _read_by_kernels(fake):
    """The buffers given to the kernels that load states and masks."""
    return {int(a, 16) for l in fake.log() if l.startswith("launch") and "load_" in l for a in l.split()[2:5]}


@pytest.mark.parametrize("n_words", [1, 3, 8, 32, 33, 64])
def test_buffers_of_another_gpu_are_copied(fake, n_words):
    """No kernel reads a buffer on another GPU, nor words that are none; the
    copies take them. On the engine's own GPU the kernels read them."""
    n_vars = 50
    room = ctypes.create_string_buffer(1 << 16)
    base = (ctypes.addressof(room) + 255) // 256 * 256
    at = [base, base + (1 << 15), base + (1 << 15) + 1024]  # state, start, solver words
    rc, eng = fake.engine()
    assert rc == 0

    def load(far=None, shift=(0, 0, 0)):
        fake.reset()
        p = [a + s for a, s in zip(at, shift)]
        if far is not None:
            fake.lib.fake_far(vp(p[far]), 512)
        assert fake.lib.gss_state_set(eng, vp(p[0]), i64(n_vars), n_words, vp(p[1]), vp(p[2]), 1) == 0, fake.error()
        copied = {int(l.split()[2], 16) for l in fake.log() if l.startswith("copy")}
        return p, _read_by_kernels(fake), copied

    for far, shift in ((0, (0, 0, 0)), (1, (0, 0, 0)), (2, (0, 0, 0)), (None, (4, 0, 0)), (None, (0, 1, 0)),
                       (None, (0, 0, 2))):
        k = far if far is not None else [i for i in range(3) if shift[i]][0]
        p, read, copied = load(far, shift)
        assert p[k] not in read and p[k] in copied, (far, shift)
    p, read, copied = load()
    assert p[1] in read and p[2] in read and (p[0] in read) != (p[0] in copied)
    assert fake.lib.gss_engine_destroy(eng) == 0


def _database(fake, eng, n=100, n_vars=50):
    lits = (ctypes.c_int32 * (2 * n))(*[2 * (k % n_vars) + k // n_vars % 2 for k in range(2 * n)])
    offsets = (i64 * (n + 1))(*range(0, 2 * n + 1, 2))
    assert fake.lib.gss_db_set(eng, lits, offsets, i64(n)) == 0, fake.error()


def _state(fake, eng, n_words, n_vars=50):
    state = (ctypes.c_uint32 * (2 * n_vars * n_words))()
    start = (ctypes.c_uint32 * n_words)(*[0xFFFFFFFF] * n_words)
    assert fake.lib.gss_state_set(eng, state, i64(n_vars), n_words, start, None, 0) == 0, fake.error()


@pytest.mark.parametrize("n_words", [2, 20])
def test_launcher_reports_the_runtime_error_and_asks_again(tmp_path, n_words):
    """A library of its own: the launchers keep what they learned."""
    fake = Fake(tmp_path)
    rc, eng = fake.engine()
    _database(fake, eng)
    _state(fake, eng, n_words)
    fake.fail("occupancy")
    assert fake.lib.gss_check_launch(eng) == -2 and "Occupancy" in fake.error()
    for _ in range(2):
        assert fake.lib.gss_check_launch(eng) == 0, fake.error()
        assert fake.lib.gss_check_wait(eng, None) == 0
    assert fake.log().count("occupancy") == 2  # refused, answered; not asked a third time
    checks = [l for l in fake.log() if "check_narrow_kernel" in l or "check_filtered_kernel" in l]
    assert len(checks) == 2
    assert fake.lib.gss_engine_destroy(eng) == 0


@pytest.mark.parametrize("n_words", [3, 20])
def test_no_pass_of_a_state_that_found_no_room(fake, n_words):
    """gss_state_set gives the old state's buffer up for a larger one; when that
    cannot be had, the next pass is refused instead of reading nothing."""
    rc, eng = fake.engine()
    fake.lib.gss_engine_set_variant(eng, 0, 0, 2, 0)  # (the direct kernel: no table that could make room)
    _database(fake, eng)
    _state(fake, eng, n_words)
    assert _passes(fake, eng, 1) == 0
    state = (ctypes.c_uint32 * (2 * 5000 * n_words))()
    start = (ctypes.c_uint32 * n_words)()
    fake.lib.gss_debug_fail_device_alloc(i64(0), 1)
    assert fake.lib.gss_state_set(eng, state, i64(5000), n_words, start, None, 0) == -3
    fake.reset()
    assert fake.lib.gss_check_launch(eng) < 0 and not any("check" in l for l in fake.log())
    _state(fake, eng, n_words)
    assert fake.lib.gss_check_launch(eng) == 0, fake.error()
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_database_that_found_no_room_is_empty(fake):
    """gss_db_set gives the old buffers up for larger ones; when those cannot be
    had the database is empty, and later batches start from there."""
    rc, eng = fake.engine()
    fake.lib.gss_engine_set_variant(eng, 0, 0, 2, 0)  # (the direct kernel: no table that could make room)
    fake.lib.gss_db_clause_count.restype = fake.lib.gss_db_live_count.restype = i64
    _database(fake, eng)
    _state(fake, eng, 3)
    n = 3000
    lits, offsets = (ctypes.c_int32 * (2 * n))(), (i64 * (n + 1))(*range(0, 2 * n + 1, 2))
    for after in range(3):
        fake.reset()
        fake.fail("malloc", after)
        assert fake.lib.gss_db_set(eng, lits, offsets, i64(n)) == -3
        assert fake.lib.gss_db_clause_count(eng) == 0 and fake.lib.gss_db_live_count(eng) == 0
        fake.reset()
        assert fake.lib.gss_check_launch(eng) == 0 and fake.lib.gss_check_wait(eng, None) == 0
        assert not any("check_kernel" in l for l in fake.log())
        assert fake.lib.gss_db_append(eng, lits, offsets, i64(10), None) == 0, fake.error()
        assert fake.lib.gss_db_clause_count(eng) == 10
        assert fake.lib.gss_engine_destroy(eng) == 0  # (small buffers again)
        rc, eng = fake.engine()
        fake.lib.gss_engine_set_variant(eng, 0, 0, 2, 0)
        _database(fake, eng)
        _state(fake, eng, 3)
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_batch_that_found_no_room_changes_nothing(fake):
    rc, eng = fake.engine()
    fake.lib.gss_engine_set_variant(eng, 0, 0, 2, 0)
    fake.lib.gss_db_clause_count.restype = fake.lib.gss_db_live_count.restype = i64
    _database(fake, eng)
    n = 3000
    lits, offsets = (ctypes.c_int32 * (2 * n))(), (i64 * (n + 1))(*range(0, 2 * n + 1, 2))
    ids = (ctypes.c_uint32 * n)(*range(200, 200 + n))
    for after in (0, 1, 1):  # literals, offsets, ids: what was had stays
        fake.fail("malloc", after)
        assert fake.lib.gss_db_append(eng, lits, offsets, i64(n), ids) == -3
        assert fake.lib.gss_db_clause_count(eng) == 100
        assert fake.lib.gss_db_delete(eng, ids, i64(1)) == -6
    fake.reset()
    assert fake.lib.gss_db_append(eng, lits, offsets, i64(n), ids) == 0, fake.error()
    assert fake.lib.gss_db_delete(eng, ids, i64(1)) == 0 and fake.lib.gss_db_live_count(eng) == 99 + n
    assert fake.lib.gss_engine_destroy(eng) == 0


def _append(fake, eng):
    n = 3000
    lits = (ctypes.c_int32 * (2 * n))(*[2 * (k % 50) for k in range(2 * n)])
    assert fake.lib.gss_db_append(eng, lits, (i64 * (n + 1))(*range(0, 2 * n + 1, 2)), i64(n), None) == 0, fake.error()


def _delete(fake, eng):
    ids = (ctypes.c_uint32 * 3)(5, 6, 7)
    assert fake.lib.gss_db_delete(eng, ids, i64(3)) == 0
    assert fake.lib.gss_check_launch(eng) == 0, fake.error()


def _launch(fake, eng):
    assert fake.lib.gss_check_launch(eng) == 0, fake.error()


def _order(fake, eng):
    assert fake.lib.gss_order_enable(eng, None) == 0, fake.error()


@pytest.mark.parametrize("n_words", [20, 40])
@pytest.mark.parametrize("grow", [lambda f, e: _database(f, e, 3000), _append, _delete, _launch, _order,
                                  lambda f, e: _state(f, e, 64)],
                         ids=["set", "append", "delete", "queues", "order", "state"])
def test_filter_table_makes_room_for_what_a_pass_needs(fake, n_words, grow):
    """Whatever the engine must have and cannot get, it gets once the filter's
    table is given back, as if there had been no table."""
    rc, eng = fake.engine()
    _database(fake, eng)
    _state(fake, eng, n_words)
    fake.lib.gss_debug_fail_device_alloc(i64(0), 1)
    grow(fake, eng)
    fake.lib.gss_debug_fail_device_alloc(i64(0), 0)
    fake.reset()
    assert fake.lib.gss_check_launch(eng) == 0, fake.error()
    assert fake.lib.gss_check_wait(eng, None) == 0
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_order_takes_the_table_before_the_pass_reads_it(fake):
    """A pass whose own scoring makes the table go does not run behind it."""
    rc, eng = fake.engine()
    _database(fake, eng)
    assert fake.lib.gss_order_enable(eng, None) == 0
    _state(fake, eng, 20)
    fake.lib.gss_debug_fail_device_alloc(i64(0), 1)  # the queues
    fake.reset()
    assert fake.lib.gss_check_launch(eng) == 0, fake.error()
    assert not any("check_filtered_kernel" in l for l in fake.log())
    assert fake.lib.gss_check_wait(eng, None) == 0
    _append(fake, eng)  # the scoring buffers have to grow
    _state(fake, eng, 20)
    fake.lib.gss_debug_fail_device_alloc(i64(0), 1)
    fake.reset()
    assert fake.lib.gss_check_launch(eng) == 0, fake.error()
    assert not any("check_filtered_kernel" in l for l in fake.log())
    assert any("check_wide_persist_kernel" in l for l in fake.log())
    assert fake.lib.gss_engine_destroy(eng) == 0


def _passes(fake, eng, n, kept=0, n_false=0):
    """n passes; how many of them ran behind the filter."""
    before = fake.lib.gss_engine_filtered_passes(eng)
    fake.lib.fake_filter(n_false, kept)
    for _ in range(n):
        assert fake.lib.gss_check_launch(eng) == 0, fake.error()
        assert fake.lib.gss_check_wait(eng, None) == 0, fake.error()
    return fake.lib.gss_engine_filtered_passes(eng) - before


@pytest.mark.parametrize("other", ["states", "database", "words", "variables"])
def test_pause_of_the_filter_ends_with_what_caused_it(fake, other):
    """One state of which the filter keeps too much: the states after it, or
    another database or layout, do not wait 64 passes for the filter."""
    rc, eng = fake.engine()
    _database(fake, eng)
    _state(fake, eng, 20)
    assert _passes(fake, eng, 1, kept=90) == 1
    assert _passes(fake, eng, 3) == 0  # it pauses
    if other == "states":
        assert _passes(fake, eng, 1) == 0
        for _ in range(10):
            _state(fake, eng, 20)
            assert _passes(fake, eng, 1) == 1
    else:
        if other == "database":
            _database(fake, eng, 200)
        elif other == "words":
            _state(fake, eng, 21)
        else:
            _state(fake, eng, 20, 51)
        assert _passes(fake, eng, 10) == 10
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_pause_of_the_filter_grows_while_it_keeps_too_much(fake):
    rc, eng = fake.engine()
    _database(fake, eng)
    _state(fake, eng, 20)
    ran = [_passes(fake, eng, 1, kept=90) for _ in range(1 + 4 + 1 + 8 + 1 + 16 + 1 + 32 + 1 + 64 + 1 + 64 + 1)]
    assert [k for k, r in enumerate(ran) if r] == [0, 5, 14, 31, 64, 129, 194]
    # one success, and the next failure pauses for as long as the first
    assert [_passes(fake, eng, 1) for _ in range(65)] == [0] * 64 + [1]
    assert [_passes(fake, eng, 1, kept=90) for _ in range(6)] == [1, 0, 0, 0, 0, 1]
    assert fake.lib.gss_engine_destroy(eng) == 0


def _tables(fake):
    return sum("load_state_kernel" in l and " table" in l for l in fake.log())


def _device_state(fake, eng, n_words, n_vars, n_false):
    """A state and masks in (the fake's) device memory; what its sample finds."""
    room = ctypes.create_string_buffer(8 * n_vars * n_words + 8 * n_words + 512)
    base = (ctypes.addressof(room) + 255) // 256 * 256
    fake.lib.fake_filter(n_false, 0)
    assert fake.lib.gss_state_set(eng, vp(base), i64(n_vars), n_words, vp(base + 8 * n_vars * n_words), None,
                                  1) == 0, fake.error()


@pytest.mark.parametrize("n_words,most", [(5, 10), (8, 10), (9, 20), (16, 20), (17, 33), (32, 33), (40, 66)])
def test_share_the_filter_may_keep(fake, n_words, most):
    """Of 100 clauses, a block each: narrow blocks pause earlier, whose plain
    scan is cheap."""
    rc, eng = fake.engine()
    _database(fake, eng)
    _state(fake, eng, n_words)
    _passes(fake, eng, 2)
    assert _passes(fake, eng, 3, kept=most) == 3
    assert _passes(fake, eng, 2, kept=most + 1) == 1
    assert fake.lib.gss_engine_destroy(eng) == 0


@pytest.mark.parametrize("share,behind", [(0.59, True), (0.61, False)])
def test_density_up_to_which_passes_are_filtered(fake, share, behind):
    rc, eng = fake.engine()
    _database(fake, eng)
    fake.lib.fake_filter(int(share * 2 * 50 * 20), 0)
    _state(fake, eng, 20)
    assert _passes(fake, eng, 1, n_false=int(share * 2 * 50 * 20)) == behind
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_one_capture_for_plain_and_one_for_filtered_passes(fake):
    rc, eng = fake.engine()
    _database(fake, eng)
    assert fake.lib.gss_engine_set_graph(eng, 1) == 0
    _state(fake, eng, 20)
    ran = [_passes(fake, eng, 1, kept=90) for _ in range(40)]
    assert 0 < sum(ran) < 40 and fake.lib.gss_engine_graph_captures(eng) == 2
    assert fake.log().count("graph") == 40
    assert fake.lib.gss_engine_destroy(eng) == 0


@pytest.mark.parametrize("n_words", [8, 20, 32, 40])
def test_no_table_for_states_that_do_not_run_behind_it(fake, n_words):
    """A dense state (fair-coin slots set nearly every bit) after a dense one
    gets no table, and is a plain copy where the layouts are the same; the
    first sparse one after them runs behind one."""
    n_vars = 50
    dense = min(4096, n_vars * n_words) * 2
    rc, eng = fake.engine()
    _database(fake, eng)
    _device_state(fake, eng, n_words, n_vars, dense)
    for _ in range(3):
        fake.reset()
        _device_state(fake, eng, n_words, n_vars, dense)
        assert _tables(fake) == 0
        assert any(l.startswith("copy") and int(l.split()[3]) == 8 * n_vars * n_words for l in fake.log()) == \
            (n_words in (8, 32))
        assert _passes(fake, eng, 2, n_false=dense) == 0 and _tables(fake) == 0
    _device_state(fake, eng, n_words, n_vars, dense // 10)
    assert _passes(fake, eng, 4) >= 3
    fake.reset()
    _device_state(fake, eng, n_words, n_vars, dense // 10)
    assert _tables(fake) == 1 and _passes(fake, eng, 1) == 1 and _tables(fake) == 1
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_no_table_during_a_pause(fake):
    rc, eng = fake.engine()
    _database(fake, eng)
    _device_state(fake, eng, 20, 50, 0)
    assert _passes(fake, eng, 1, kept=90) == 1
    fake.reset()
    for k in range(4):
        _device_state(fake, eng, 20, 50, 0)
        assert _passes(fake, eng, 1) == 0 and _tables(fake) == 0
    _device_state(fake, eng, 20, 50, 0)
    assert _passes(fake, eng, 1) == 1 and _tables(fake) == 1
    # a pause that ends over a state that was set during it
    assert _passes(fake, eng, 1, kept=90) == 1
    _device_state(fake, eng, 20, 50, 0)
    fake.reset()
    assert [_passes(fake, eng, 1) for _ in range(6)] == [0, 0, 0, 0, 1, 1] and _tables(fake) == 1
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_no_table_that_costs_more_than_it_saves(fake):
    """A hundred clauses against 2^19 variables: gss_state_set fills no table;
    passes over the same state fill it once they would have saved as much."""
    rc, eng = fake.engine()
    _database(fake, eng)
    fake.reset()
    _device_state(fake, eng, 8, 1 << 19, 0)
    assert _tables(fake) == 0
    ran = [_passes(fake, eng, 1) for _ in range(12)]
    assert ran[0] == 0 and ran[-1] == 1 and ran == sorted(ran) and _tables(fake) == 1
    _device_state(fake, eng, 8, 1 << 19, 0)
    assert _passes(fake, eng, 1) == 0 and _tables(fake) == 1
    assert fake.lib.gss_engine_destroy(eng) == 0


def test_host_passes_without_tables(fake):
    """Dense states through gss_check_passes_host: no pass gets a table."""
    n_vars, n_words = 50, 20
    rc, eng = fake.engine()
    _database(fake, eng)
    states = [(ctypes.c_uint32 * (2 * n_vars * n_words))() for _ in range(7)]
    start = (ctypes.c_uint32 * n_words)(*[0xFFFFFFFF] * n_words)
    outs = [(ctypes.c_uint32 * 64)() for _ in states]
    call = lambda: fake.lib.gss_check_passes_host(
        eng, len(states), (vp * 7)(*[ctypes.addressof(s) for s in states]), i64(n_vars), n_words, start, None,
        (vp * 7)(*[ctypes.addressof(o) for o in outs]), (i64 * 7)(*[16] * 7), (i64 * 7)())
    for n_false, kept, tables, filtered in ((0, 0, 7, 7), (2000, 0, 1, 0), (2000, 0, 0, 0), (0, 0, 7, 7)):
        fake.reset()
        fake.lib.fake_filter(n_false, kept)
        before = fake.lib.gss_engine_filtered_passes(eng)
        assert call() == 0, fake.error()
        assert (_tables(fake), fake.lib.gss_engine_filtered_passes(eng) - before) == (tables, filtered)
    assert fake.lib.gss_engine_destroy(eng) == 0


@pytest.fixture
def make_sharer(fake, monkeypatch):
    """The Python sharer over the library without a GPU: five solvers, one
    pass run with assignments and one without changes."""
    import gpusharesat_gb300 as g
    monkeypatch.setattr(g, "_lib", None)
    monkeypatch.setattr(g, "LIB_PATH", fake.path)
    made = []

    def make(filter_from):
        s = g.ClauseSharer(minGpuLatencyMicros=0, verbosity=0)
        made.append(s)
        s.setFilterFrom(filter_from)
        s.setVarCount(60)
        s.setCpuSolverCount(5)
        _some_clauses(s, 50)
        _some_passes(s)
        assert s.filteredPasses() == (2 if filter_from == 0 else 0)
        return s

    yield make
    for s in made:
        s.close()


def _some_clauses(s, n):
    for k in range(n):
        assert s.addClause(-1, [2 * (k % 20), 2 * (20 + k % 20), 2 * (40 + k % 20)]) >= 0


def _some_passes(s, n_vars=20):
    for solver in range(5):
        assert s.trySetSolverValues(solver, [2 * v for v in range(n_vars)])
        s.trySendAssignment(solver)
        s.unsetSolverValues(solver, [2 * v for v in range(n_vars)])
    s.gpuRun()
    for solver in range(5):
        s.trySendAssignment(solver)
    s.gpuRun()


@pytest.mark.parametrize("grow", ["clauses", "updates", "variables", "solvers"])
def test_sharer_drops_the_table_before_clauses(fake, make_sharer, grow):
    """An allocation that fails takes the filter's table, not the clauses: the
    database is not reduced and no out-of-memory is noted."""
    sharer = make_sharer(0)
    before = sharer.getGlobalStat("gpuReduceDbs")
    if grow == "clauses":
        _some_clauses(sharer, 5000)
    elif grow == "variables":
        sharer.setVarCount(5000)
    elif grow == "solvers":
        sharer.setCpuSolverCount(40)
    fake.lib.gss_debug_fail_device_alloc(i64(0), 1)
    if grow == "updates":
        sharer.setVarCount(60)
    for _ in range(3):
        _some_passes(sharer, 60)
    assert fake.lib.gss_debug_fail_device_alloc(i64(0), 0) == 0
    assert not sharer.hasRunOutOfGpuMemoryOnce()
    assert sharer.getGlobalStat("gpuReduceDbs") == before


@pytest.mark.parametrize("n_solvers,below,above", [(8, 200_000, 600_000), (40, 30_000, 45_000)])
def test_sharer_filters_where_it_pays(fake, make_sharer, n_solvers, below, above):
    """The default line, by clauses and solvers: a database of so many clauses
    is checked by the plain kernel, one of so many behind the filter."""
    sharer = make_sharer(1 << 60)
    sharer.setFilterFrom(-1)
    sharer.setCpuSolverCount(n_solvers)
    add, clause = sharer.lib.gss_sharer_add_clause, (ctypes.c_int * 3)(2, 5, 8)

    def grow_to(n):
        for _ in range(n - sharer.getAddedClauseCount()):
            add(sharer.h, -1, clause, 3)
        before = sharer.filteredPasses()
        _some_passes(sharer)
        return sharer.filteredPasses() - before

    assert grow_to(below) == 0
    assert grow_to(above) == 2


def test_sharer_keeps_no_table_up_during_a_pause(fake, make_sharer):
    """One pass of which the filter keeps too much, then passes without it: no
    launch fills or refreshes the table until it is used again."""
    sharer = make_sharer(0)
    upkeep = lambda: [l.split()[1] for l in fake.log() if "refresh_agg" in l or " table" in l]

    def one(kept):
        fake.reset()
        fake.lib.fake_filter(0, kept)
        before = sharer.filteredPasses()
        assert sharer.trySetSolverValues(1, [2, 5])
        sharer.trySendAssignment(1)
        sharer.unsetSolverValues(1, [2, 5])
        sharer.gpuRun()
        return sharer.filteredPasses() - before, len(upkeep())

    assert one(0)[0] == 1
    assert one(90) == (1, 2)  # refreshed after the pass before, and for its own updates
    assert [one(0) for _ in range(4)] == [(0, 0)] * 4
    assert one(0) == (1, 1) and one(0) == (1, 2)  # filled anew, then kept up


@pytest.mark.parametrize("after", [0, 1, 2])
def test_sharer_layout_that_ran_out_of_memory_is_made_again(fake, make_sharer, after):
    """The solvers' numbers of a new layout, 35 blocks of 32 words, reach the
    device whichever of its allocations failed."""
    sharer = make_sharer(1 << 60)  # (no table that could make room)
    sharer.setCpuSolverCount(1100)
    fake.reset()
    fake.fail("malloc", after)
    _some_passes(sharer)
    assert any(l.startswith("copy") and l.split()[3] == str(4 * 32 * 35) for l in fake.log())


def test_sharer_uploads_again_what_found_no_room(fake, make_sharer):
    """The database does not fit twice over: gpuRun fails, no kernel runs over
    buffers that are gone, and the next gpuRun brings all clauses back."""
    import gpusharesat_gb300 as g
    sharer = make_sharer(1 << 60)
    for k in range(4000):  # clauses that a reduction keeps
        assert sharer.addClause(-1, [2 * (k % 20), 2 * (20 + k % 20)]) >= 0
    fake.lib.gss_debug_fail_device_alloc(i64(0), 50)
    for _ in range(2):
        fake.reset()
        with pytest.raises(g.GssError):
            sharer.gpuRun()
        assert not any("check_" in l and "kernel" in l for l in fake.log() if l.startswith("launch"))
    fake.lib.gss_debug_fail_device_alloc(i64(0), 0)
    fake.reset()
    _some_passes(sharer)
    clauses = sharer.getGlobalStat("gpuClauses")
    assert clauses >= 4000
    assert any(l.startswith("copy") and l.split()[3] == str(8 * (clauses + 1)) for l in fake.log())  # the offsets
    assert sum("check_" in l for l in fake.log() if l.startswith("launch")) == 2


def test_sharer_keeps_its_state_when_the_variant_changes(fake, make_sharer):
    """The values that the solvers sent go over to the new layout, which runs
    the kernel that was asked for."""
    sharer = make_sharer(0)
    for kind, lanes, kernel in ((3, 16, "check_wide_kernel"), (2, 8, "check_wide_kernel"), (0, 4, "check_kernel"),
                                (-1, 0, "check_filtered_kernel")):
        sharer.setVariant(kind, lanes, 2)
        fake.reset()
        _some_passes(sharer)
        launched = [l.split()[1] for l in fake.log() if l.startswith("launch")]
        assert sum("copy_layout_kernel" in l for l in launched) == 1, kind
        assert sum(kernel in l for l in launched) == 2, (kind, launched)


def test_staged_records_lie_on_16_bytes_by_type(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-I", os.path.join(build.ROOT, "include"), "-I",
                    build.CSRC, "-c", os.path.join(here, "cpp", "stage_alignment.cu"), "-o",
                    str(tmp_path / "stage_alignment.o")], check=True)
