"""The sharer's passes behind the word-level filter, whose table follows the
state as variables change: the same calls to a sharer whose passes all run
behind it, to one whose passes never do, and to the plain-Python model, with
every report compared. Without the filter's keep-too-much pause in play: the
clauses are long and few of them report."""
import numpy as np
import pytest

from oracle.sharer_model import SharerModel

pytestmark = pytest.mark.gpu

NEVER = 1 << 60


def lit(v, neg=False):
    return 2 * v + (1 if neg else 0)


def _pair(n_vars, n_solvers):
    import gpusharesat_gb300 as g
    out = []
    for pairs in (0, NEVER):
        s = g.ClauseSharer(minGpuLatencyMicros=0, verbosity=0)
        s.setFilterFrom(pairs)
        s.setVarCount(n_vars)
        s.setCpuSolverCount(n_solvers)
        out.append(s)
    return out


class _Session:
    """Random calls to all of `every`: trails that grow and backtrack, clauses
    of 5 to 12 literals, some unit or false under a solver's trail."""

    def __init__(self, rng, every, n_vars, n_solvers):
        self.rng, self.every, self.n_vars = rng, every, n_vars
        self.trails = [[] for _ in range(n_solvers)]
        self.ids = []

    def add(self, n, planted=3):
        rng = self.rng
        for k in range(n):
            length = int(rng.integers(5, 13))
            trail = self.trails[int(rng.integers(len(self.trails)))]
            if k < planted and len(trail) > length:
                cl = [trail[i] ^ 1 for i in rng.choice(len(trail), length - 1, replace=False)]
                if rng.random() < 0.5:
                    used = {l >> 1 for l in trail}
                    free = [v for v in range(self.n_vars) if v not in used]
                    cl.append(lit(int(rng.choice(free)) if free else 0))
            else:
                cl = [lit(int(v), bool(rng.integers(0, 2)))
                      for v in rng.choice(self.n_vars, length, replace=False)]
            self.ids.append({s.addClause(-1, cl) for s in self.every})
            assert len(self.ids[-1]) == 1

    def move(self, solver, grow):
        """Backtracks a little, extends by `grow` and sends; an assignment of
        some variables of a full ring is refused by all alike."""
        rng, tr = self.rng, self.trails[solver]
        back = int(rng.integers(0, min(len(tr), 6) + 1))
        if back:
            gone = tr[len(tr) - back:]
            del tr[len(tr) - back:]
            for s in self.every:
                s.unsetSolverValues(solver, gone)
        used = {l >> 1 for l in tr}
        free = [v for v in range(self.n_vars) if v not in used]
        more = [lit(int(v), bool(rng.integers(0, 2))) for v in rng.choice(free, min(grow, len(free)), replace=False)]
        took = {bool(s.trySetSolverValues(solver, more)) for s in self.every}
        assert len(took) == 1
        if took.pop():
            tr.extend(more)
        assert len({s.trySendAssignment(solver) for s in self.every}) == 1

    def run(self):
        for s in self.every:
            s.gpuRun()

    def compare(self, what):
        n = 0
        for solver in range(len(self.trails)):
            got = [sorted((tuple(l), c) for l, c in s.popAll(solver)) for s in self.every]
            for other in got[1:]:
                assert got[0] == other, (what, solver)
            n += len(got[0])
            assert len({s.getLastAssigAllReported(solver) for s in self.every}) == 1
        return n


@pytest.mark.parametrize("n_solvers", [5, 9, 17, 33, 70])
def test_session_behind_the_filter_matches_model(lib, n_solvers):
    """Also: passes that change more words than the state has rows, several
    assignments a pass, more variables and more solvers on the way."""
    n_vars = 90
    rng = np.random.default_rng(n_solvers)
    s, plain = _pair(n_vars, n_solvers)
    m = SharerModel()
    m.setVarCount(n_vars)
    m.setCpuSolverCount(n_solvers)
    try:
        ses = _Session(rng, [s, plain, m], n_vars, n_solvers)
        reports = 0
        for step in range(24):
            if step == 12:  # the state is laid out again
                ses.n_vars += 35
                for x in ses.every:
                    x.setVarCount(ses.n_vars)
            if step == 16:
                for x in ses.every:
                    x.setCpuSolverCount(n_solvers + 4)
                ses.trails += [[] for _ in range(4)]
            ses.add(60)
            for solver in range(len(ses.trails)):
                if rng.random() < 0.8:
                    for _ in range(int(rng.integers(1, 4))):
                        ses.move(solver, 60 if step % 8 == 0 else 6)
            ses.run()
            if step % 3 != 1:  # two passes, the second with nothing new
                ses.run()
            reports += ses.compare(step)
        assert reports > 100
        assert s.filteredPasses() >= 20 and plain.filteredPasses() == 0
    finally:
        s.close()
        plain.close()


def test_filter_switched_on_and_off(lib):
    """Across the threshold in both directions: the table is built again from
    the state it finds."""
    n_vars, n_solvers = 80, 12
    rng = np.random.default_rng(1)
    s, plain = _pair(n_vars, n_solvers)
    try:
        ses = _Session(rng, [s, plain], n_vars, n_solvers)
        seen = []
        for step in range(40):
            s.setFilterFrom(NEVER if step // 5 % 2 else 0)
            ses.add(40)
            for solver in range(n_solvers):
                ses.move(solver, 8)
            ses.run()
            seen.append(s.filteredPasses())
            ses.compare(step)
        ses.run()
        ses.compare("end")
        assert seen[4] == 5 and seen[9] == 5 and seen[14] == 10 and seen[-1] == 20
    finally:
        s.close()
        plain.close()


def test_table_after_a_pause(lib):
    """Most clauses are false under some solver's trail for a while: the filter
    keeps them and pauses, the state moves on without its table, and the passes
    behind the table filled anew report what the plain ones do."""
    n_vars, n_solvers = 60, 9
    rng = np.random.default_rng(5)
    s, plain = _pair(n_vars, n_solvers)
    try:
        ses = _Session(rng, [s, plain], n_vars, n_solvers)
        filtered = []
        for step in range(60):
            if step in (0, 30):
                for x in ses.every:  # short clauses, half of them reporting in each of many words
                    for k in range(300):
                        x.addClause(-1, [lit(k % n_vars, k % 3 == 0), lit((k + 7) % n_vars, k % 2 == 0)])
            if step in (12, 42):  # and many more that do not
                ses.add(3000, planted=20)
            for solver in range(n_solvers):
                ses.move(solver, 40 if step % 10 == 0 else 5)
            ses.run()
            filtered.append(s.filteredPasses())
            ses.compare(step)
        ses.run()
        ses.compare("end")
        assert any(filtered[k] == filtered[k + 4] for k in range(10))  # it pauses
        assert filtered[-1] > 20
    finally:
        s.close()
        plain.close()


def test_variant_changed_between_passes(lib):
    """The state that the solvers sent goes over to the layout of another
    kernel, and back behind the filter."""
    n_vars, n_solvers = 80, 12
    rng = np.random.default_rng(4)
    s, plain = _pair(n_vars, n_solvers)
    try:
        ses = _Session(rng, [s, plain], n_vars, n_solvers)
        reports = 0
        for step, variant in enumerate(((-1, 0, 2), (0, 4, 2), (2, 8, 2), (-1, 0, 2), (3, 16, 2), (-1, 0, 2))):
            s.setVariant(*variant)
            for _ in range(3):
                ses.add(40, planted=8)
                for solver in range(n_solvers):
                    ses.move(solver, 30 if step == 0 else 4)
                ses.run()
                reports += ses.compare(step)
        ses.run()
        assert reports + ses.compare("end") > 50
        assert s.filteredPasses() == 9  # (the last call's pass had nothing to do)
    finally:
        s.close()
        plain.close()


def test_evictions_and_reductions_behind_the_filter(lib):
    """Evicted clauses stay on the device as tombstones until a compaction;
    reduceDb moves the rest."""
    n_vars, n_solvers = 100, 33
    rng = np.random.default_rng(2)
    s, plain = _pair(n_vars, n_solvers)
    try:
        ses = _Session(rng, [s, plain], n_vars, n_solvers)
        for x in ses.every:
            x.setClauseBudget(900)
        reports = 0
        for step in range(40):
            ses.add(70, planted=8)
            for solver in range(n_solvers):
                ses.move(solver, 30 if step == 0 else 5)
            ses.run()
            if step == 25:
                for x in ses.every:
                    x.reduceDb()
            reports += ses.compare(step)
        assert reports > 100 and s.evictedCount() > 500 and s.deviceCompactions() > 0
        # (after the reduction little but reported clauses is left, of which the filter keeps too much)
        assert s.filteredPasses() >= 25 and plain.filteredPasses() == 0
    finally:
        s.close()
        plain.close()


def test_default_threshold_session(lib):
    """The default line: a database that grows past it, and one slot block
    that becomes two; reports as without the filter."""
    n_vars, n_solvers = 5000, 20
    rng = np.random.default_rng(3)
    s, plain = _pair(n_vars, n_solvers)
    s.setFilterFrom(-1)
    try:
        ses = _Session(rng, [s, plain], n_vars, n_solvers)

        def bulk(n):
            cl = rng.integers(0, 2 * n_vars, (n, 8)).astype(np.int32)
            cl[:, 1:] += 2 * np.arange(1, 8, dtype=np.int32) * (n_vars // 8)  # (repeats are harmless)
            cl %= 2 * n_vars
            for row in cl:
                for x in ses.every:
                    x.addClause(-1, row)

        bulk(60_000)
        seen = []
        for size in (0, 60_000, 120_000, 0, 0):
            bulk(size)
            ses.add(40, planted=30)
            for solver in range(len(ses.trails)):
                ses.move(solver, 1200)
            ses.run()
            ses.run()
            ses.compare(size)
            seen.append(s.filteredPasses())
        assert seen[0] == 0 and seen[-1] > 0 and plain.filteredPasses() == 0
        before = s.filteredPasses()
        for x in ses.every:
            x.setCpuSolverCount(40)
        ses.trails += [[] for _ in range(20)]
        for _ in range(2):
            for solver in range(40):
                ses.move(solver, 300)
            ses.add(30, planted=30)
            ses.run()
            ses.run()
            assert ses.compare("wide") > 0
        assert s.filteredPasses() > before
    finally:
        s.close()
        plain.close()
