"""gss_check_noalloc with its output queues and counters at addresses between
16-byte boundaries, as a caller's pool may cut them: the same reports as the
oracle, and nothing written outside the queues."""
import numpy as np
import pytest

import oracle
from test_zz_no_alloc import _bind, _Inputs, _workload, vp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [4, 8, 12])
def test_noalloc_queues_at_any_word(lib, shift):
    import torch
    import gpusharesat_gb300 as g
    fn = _bind(lib)
    wl = _workload()
    ref = oracle.check(wl.lits, wl.offsets, wl.state, wl.start, n_threads=8)
    inp = _Inputs(wl)
    n_parts, cap = 5, len(ref) // 5 * 2 + 1024
    guard = 64  # words before and after the queues
    room = torch.full((guard + 4 * n_parts * cap + guard + 4,), -7, dtype=torch.int32, device="cuda")
    first = guard + shift // 4
    counts = torch.full((4 * n_parts + 4,), -1, dtype=torch.int8, device="cuda")
    rc = fn(vp(inp.lits.data_ptr()), vp(inp.offsets.data_ptr()), wl.n_clauses, vp(inp.state.data_ptr()), wl.n_vars,
            inp.n_blocks, vp(inp.start.data_ptr()), vp(inp.sow.data_ptr()), vp(room.data_ptr() + 4 * first), n_parts,
            cap, vp(counts.data_ptr() + shift // 4), vp(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, lib.gss_last_error()
    torch.cuda.synchronize()
    counts = counts.cpu().numpy()[shift // 4:][:4 * n_parts].copy().view(np.uint32).astype(np.int64)
    assert (counts <= cap).all() and counts.sum() == len(ref)
    room = room.cpu().numpy()
    end = first + 4 * n_parts * cap
    assert (room[:first] == -7).all() and (room[end:] == -7).all()
    recs = room[first:end].copy().view(g.REPORT_DTYPE).reshape(n_parts, cap)
    got = g.sort_reports(np.concatenate([recs[p, :counts[p]] for p in range(n_parts)]))
    for f in ("clause", "word", "mask"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    np.testing.assert_array_equal(got["solver"], wl.solver_of_word[got["word"]])
