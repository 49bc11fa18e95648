"""Timing cases: the work a user has this framework do, through its public
entry points, with inputs made on the GPU from a seed.

A case is a dict of plain values. listed() gives the fixed cases, draw(rng)
one more of the same ranges, prepare(case, seed) what a program holds before
the call, run(state) one pass with its whole outputs, work(case) the bytes
the pass cannot do without, and exact(case, seed) the 64-bit result where the
outputs are computed numbers.

Reports have no order (warps reserve room in the queues as they find them),
so a pass's records are returned sorted, after their count and with zeros
after the last one, or, where most cells have one, as the dense [clause][word]
array of slot masks they stand for.

Assignment states:
  uniform  every slot assigns 50-88% of the variables on its own, with
           fair-coin values (the plain check's generator)
  model    every slot assigns half of the variables on its own, always to the
           value of one hidden model, and every clause has two literals true
           under it, as clauses of one satisfiable formula have (the
           learned-order generator); clauses report where planted
  trail    the same, but the 32 slots of a word are one solver's trail: each
           differs from the one before by four variables set and four unset
           (the serving generator)
"""
import ctypes

import numpy as np
import torch

import gpusharesat_gb300 as g

MEAN_LEN = {"geo8": 8.0, "scale": 18.0, "zipf": 15.0}
# room for the report records of a clause against 1024 uniform slots
ROOM = {"geo8": 20, "scale": 8, "zipf": 22}


def listed():
    return [
        # one short pass through host buffers: a solver process that checks a
        # small database now and then; launches, copies and waits count most
        {"name": "host_small", "kind": "host", "n_vars": 2 ** 14, "n_clauses": 10_000, "n_words": 2,
         "lengths": "geo8", "state": "uniform"},
        # one solver's 32 assignments: the narrowest rows
        {"name": "engine_one_word", "kind": "engine", "n_vars": 250_007, "n_clauses": 600_000, "n_words": 1,
         "lengths": "scale", "state": "trail", "feed": "resident", "uneven": False, "churn": False, "graph": False},
        # an odd number of solvers, states from a program on the same GPU
        {"name": "engine_odd_words", "kind": "engine", "n_vars": 300_007, "n_clauses": 400_000, "n_words": 11,
         "lengths": "zipf", "state": "model", "feed": "device", "uneven": False, "churn": False, "graph": False},
        # the plain check's shape: 2^20 variables, 1024 assignments
        {"name": "engine_scale", "kind": "engine", "n_vars": 2 ** 20, "n_clauses": 2_000_000, "n_words": 32,
         "lengths": "scale", "state": "model", "feed": "resident", "uneven": False, "churn": False, "graph": False},
        # uneven batches of 48 solvers over a churned database, graph replay
        {"name": "engine_uneven", "kind": "engine", "n_vars": 2 ** 19, "n_clauses": 1_000_000, "n_words": 96,
         "lengths": "zipf", "state": "trail", "feed": "device", "uneven": True, "churn": True, "graph": True},
        # independent fair-coin assignments, everything in the caller's device
        # buffers, five reports a clause
        {"name": "noalloc_uniform", "kind": "noalloc", "n_vars": 2 ** 20, "n_clauses": 1_000_000, "n_words": 32,
         "lengths": "scale", "state": "uniform"},
        # passes streamed through pinned host buffers, 8-byte records
        {"name": "host_stream", "kind": "cells", "n_vars": 2 ** 18, "n_clauses": 400_000, "n_words": 32,
         "lengths": "scale", "state": "uniform", "passes": 3},
        # clause sharing between a few solver threads, and between many
        {"name": "sharer_small", "kind": "sharer", "n_vars": 30_011, "n_clauses": 50_000, "n_solvers": 7,
         "lengths": "geo8"},
        {"name": "sharer_serving", "kind": "sharer", "n_vars": 2 ** 18, "n_clauses": 1_200_000, "n_solvers": 64,
         "lengths": "zipf"},
        # the learned scan order: scoring, early head, tail
        {"name": "order", "kind": "order", "n_vars": 2 ** 18, "n_clauses": 1_000_000, "n_words": 64,
         "lengths": "zipf", "state": "model"},
        # the scorer on its own: a training step of the default batch, and
        # the logits of a database's clauses
        {"name": "scorer_train", "kind": "train", "rows": 4096},
        {"name": "scorer_infer", "kind": "infer", "rows": 200_000},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["engine"] * 8 + ["noalloc"] * 2 + ["host"] * 2 + ["cells", "sharer", "sharer", "order", "train",
                                                                        "infer"])
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 200, 30_000)}
    if kind == "infer":
        return {"kind": kind, "rows": _log(rng, 100, 200_000)}
    lengths = rng.choice(["geo8", "scale", "zipf"])
    n_vars = _log(rng, 10_000, 2 ** 20) | 1
    if kind == "host":
        return {"kind": kind, "n_vars": _log(rng, 5_000, 60_000) | 1, "n_clauses": _log(rng, 1_000, 10_000),
                "n_words": rng.randint(1, 4), "lengths": lengths, "state": "uniform"}
    if kind == "cells":
        return {"kind": kind, "n_vars": _log(rng, 20_000, 2 ** 18) | 1, "n_clauses": _log(rng, 20_000, 400_000),
                "n_words": rng.choice([8, 20, 32]), "lengths": lengths, "state": "uniform",
                "passes": rng.randint(2, 3)}
    if kind == "sharer":
        return {"kind": kind, "n_vars": _log(rng, 10_000, 2 ** 18) | 1, "n_clauses": _log(rng, 20_000, 500_000),
                "n_solvers": _log(rng, 1, 64), "lengths": lengths}
    if kind == "order":
        return {"kind": kind, "n_vars": min(n_vars, 2 ** 18 + 1), "n_clauses": _log(rng, 100_000, 1_000_000),
                "n_words": _log(rng, 16, 64), "lengths": lengths, "state": "model"}
    if kind == "noalloc":
        return {"kind": kind, "n_vars": n_vars, "n_clauses": _log(rng, 10_000, 1_000_000), "n_words": 32,
                "lengths": lengths, "state": "uniform"}
    n_words = _log(rng, 1, 96)
    if n_words > 32:
        n_vars = min(n_vars, 2 ** 19 + 1)
    return {"kind": kind, "n_vars": n_vars, "n_clauses": _log(rng, 20_000, 1_200_000), "n_words": n_words,
            "lengths": lengths, "state": rng.choice(["model", "trail"]), "feed": rng.choice(["resident", "device"]),
            "uneven": rng.random() < 0.5, "churn": rng.random() < 0.3, "graph": rng.random() < 0.3}


# ---- inputs ----

def _cdf(lengths):
    if lengths == "geo8":  # 2..30, geometric with mean 8
        k = np.arange(2, 31)
        p = (1 - 1 / 7.0) ** (k - 2)
    elif lengths == "scale":  # 60% uniform on 2..16, 40% a geometric tail on 17..100 with mean 32
        k = np.arange(2, 101)
        tail = (1 - 1 / 16.0) ** (k - 17) * (k > 16)
        p = 0.6 / 15 * (k <= 16) + 0.4 * tail / tail.sum()
    else:  # 1 + Zipf(1.2), at most 256
        k = np.arange(2, 257)
        p = (k - 1.0) ** -1.2
    return int(k[0]), np.cumsum(p / p.sum())


def _clauses(gen, n, n_vars, lengths, model=None):
    """n clauses on the GPU: lits int32, offsets int64; with a model, two
    literals of each are true under it and the others with probability 1/2."""
    lo, cdf = _cdf(lengths)
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    length = torch.searchsorted(torch.from_numpy(cdf).cuda(), u).clamp_(max=len(cdf) - 1) + lo
    offsets = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(length, 0, out=offsets[1:])
    total = int(offsets[-1])
    var = torch.randint(0, n_vars, (total,), generator=gen, device="cuda", dtype=torch.int32)
    coin = torch.randint(0, 2, (total,), generator=gen, device="cuda", dtype=torch.int32)
    if model is None:
        return 2 * var + coin, offsets
    first = (torch.rand(n, generator=gen, device="cuda") * length).long().clamp_(max=255) % length
    second = (first + 1 + (torch.rand(n, generator=gen, device="cuda") * (length - 1)).long()) % length
    second = torch.where(second == first, (first + 1) % length, second)
    coin[offsets[:-1] + first] = 1
    coin[offsets[:-1] + second] = 1
    return 2 * var + torch.where(coin == 1, 1 - model[var], model[var]), offsets


def _words(gen, *shape):
    return torch.randint(-2 ** 31, 2 ** 31, shape, generator=gen, device="cuda", dtype=torch.int32)


def _starts(gen, n_words, uneven):
    """The slots sent: all 32 of each word, or 4 to 64 for each two words."""
    if not uneven:
        return torch.full((n_words,), -1, dtype=torch.int32, device="cuda")
    size = torch.randint(4, 65, ((n_words + 1) // 2,), generator=gen, device="cuda")
    per = torch.stack([size.clamp(max=32), (size - 32).clamp(min=0)], 1).reshape(-1)[:n_words]
    mask = (torch.ones_like(per) << per) - 1
    return torch.where(mask >= 2 ** 31, mask - 2 ** 32, mask).to(torch.int32)


def _state(gen, kind, n_vars, n_words, model):
    """[n_vars][n_words][2] = {isDef, isTrue}."""
    state = torch.empty((n_vars, n_words, 2), dtype=torch.int32, device="cuda")
    if kind == "uniform":
        a, b, c = (_words(gen, n_vars, n_words) for _ in range(3))
        share = torch.randint(0, 4, (n_words,), generator=gen, device="cuda")
        for k, bits in enumerate((a, a | (b & c), a | b, a | b | c)):  # 50%, 62.5%, 75%, 87.5%
            state[:, share == k, 0] = bits[:, share == k]
        state[:, :, 1] = _words(gen, n_vars, n_words)
        return state
    if kind == "model":
        state[:, :, 0] = _words(gen, n_vars, n_words)
    else:
        state[:, :, 0] = -torch.randint(0, 2, (n_vars, n_words), generator=gen, device="cuda", dtype=torch.int32)
        # slot j differs from slot j - 1 in eight variables, from then on
        word = torch.arange(n_words, device="cuda").repeat_interleave(31 * 8)
        slot = torch.arange(1, 32, device="cuda").repeat_interleave(8).repeat(n_words)
        cell = torch.randint(0, n_vars, word.shape, generator=gen, device="cuda") * n_words + word
        key = torch.unique(cell * 32 + slot)
        last = torch.ones_like(key, dtype=torch.bool)
        last[:-1] = key[1:] // 32 != key[:-1] // 32
        key = key[last]
        change = (-(torch.ones_like(key) << (key % 32))).to(torch.int32)
        flat = state[:, :, 0].reshape(-1)
        flat[key // 32] ^= change
        state[:, :, 0] = flat.reshape(n_vars, n_words)
    state[:, :, 1] = -model[:, None]
    return state


def _plant(gen, state, lits, offsets, start, count):
    """Makes `count` clauses report, each in one sent slot: every literal
    false there, the last one unassigned in half of them."""
    n, n_words = offsets.shape[0] - 1, state.shape[1]
    if count < 1:
        return
    chosen = torch.randperm(n, generator=gen, device="cuda")[:count]
    sent = (start[:, None] >> torch.arange(32, device="cuda", dtype=torch.int32)) & 1
    slots = torch.nonzero(sent.reshape(-1)).reshape(-1)
    slot = slots[torch.randint(0, slots.shape[0], (count,), generator=gen, device="cuda")]
    undef = torch.randint(0, 2, (count,), generator=gen, device="cuda")
    length = offsets[chosen + 1] - offsets[chosen]
    which = torch.repeat_interleave(torch.arange(count, device="cuda"), length)
    ends = torch.cumsum(length, 0)
    rank = torch.arange(which.shape[0], device="cuda") - (ends - length)[which]
    lit = lits[offsets[chosen][which] + rank].long()
    want = torch.where((rank == length[which] - 1) & (undef[which] == 1), 2, lit & 1)  # 2 unassigned, else the value
    key = ((lit >> 1) * n_words + slot[which] // 32) * 32 + slot[which] % 32
    key = torch.unique(key * 4 + want)  # where two clauses differ, the first one's wish
    keep = torch.ones_like(key, dtype=torch.bool)
    keep[1:] = key[1:] // 4 != key[:-1] // 4
    key = key[keep]
    want, bit, cell = key % 4, torch.ones_like(key) << (key // 4 % 32), key // 128
    cells, inverse = torch.unique(cell, return_inverse=True)

    def mask(on):
        m = torch.zeros(cells.shape[0], dtype=torch.int64, device="cuda").index_add_(0, inverse, bit * on)
        return torch.where(m >= 2 ** 31, m - 2 ** 32, m).to(torch.int32)

    v, w = cells // n_words, cells % n_words
    d, t = state[v, w, 0], state[v, w, 1]
    false, true, none = mask(want == 0), mask(want == 1), mask(want == 2)
    state[v, w, 0] = (d | false | true) & ~none
    state[v, w, 1] = (t | true) & ~false


def _host(t, dtype=None):
    a = t.cpu().numpy()
    return a if dtype is None else a.view(dtype)


# ---- passes of the engine ----

def _engine_inputs(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    n, n_vars, n_words, kind = case["n_clauses"], case["n_vars"], case["n_words"], case["state"]
    model = None
    if kind != "uniform":
        model = torch.randint(0, 2, (n_vars,), generator=gen, device="cuda", dtype=torch.int32)
    lits, offsets = _clauses(gen, n, n_vars, case["lengths"], model)
    start = _starts(gen, n_words, case.get("uneven", False))
    state = _state(gen, kind, n_vars, n_words, model)
    if model is not None:
        _plant(gen, state, lits, offsets, start, n // 5000)
    return gen, model, lits, offsets, start, state


def _prepare_engine(case, seed):
    gen, model, lits, offsets, start, state = _engine_inputs(case, seed)
    n, n_words = case["n_clauses"], case["n_words"]
    eng = g.Engine(0)
    eng.set_db(_host(lits), _host(offsets))
    if case.get("churn"):
        ids = torch.randperm(n, generator=gen, device="cuda")[:n // 20]
        eng.delete(_host(ids.to(torch.int32), np.uint32))
        more, ends = _clauses(gen, n // 20, case["n_vars"], "geo8", model)
        eng.append_db(_host(more), _host(ends))
    eng.set_graph(bool(case.get("graph")))
    sow = (torch.arange(n_words, device="cuda", dtype=torch.int32) // 2).contiguous()
    s = {"case": case, "eng": eng, "state": state, "start": start, "sow": sow}
    torch.cuda.synchronize()
    if case["kind"] == "order":
        eng.order_enable()
        lbd = (offsets[1:] - offsets[:-1] + 1) // 2
        eng.set_lbd(np.arange(n, dtype=np.uint32), _host(lbd).astype(np.uint16))
        s["head"], s["tail"] = np.zeros(1 << 20, g.REPORT_DTYPE), np.zeros(1 << 20, g.REPORT_DTYPE)
    if case.get("feed") == "resident":
        _set_state(s)
    return s


def _set_state(s):
    st = s["state"]
    s["eng"].set_state_device(st.data_ptr(), st.shape[0], st.shape[1], s["start"].data_ptr(), s["sow"].data_ptr())


def _sorted(rep, case):
    """Reports in (clause, word) order, one word each: cell, mask and the
    solver's low bits. Against uniform slots, where most cells report, dense."""
    n, n_words, n_clauses = len(rep), case["n_words"], case["n_clauses"]
    cell = rep["clause"].astype(np.uint64) * np.uint64(n_words) + rep["word"]
    if case["state"] == "uniform":
        out = np.zeros((2, n_clauses * n_words), np.uint32)
        out[0, cell] = rep["mask"]
        out[1, cell] = rep["solver"]
        return [n, out.view(np.int32)]
    out = np.zeros(4096 + n_clauses // 40, np.uint64)
    mask, solver = rep["mask"].astype(np.uint64), rep["solver"] % np.uint32(32)
    out[:n] = np.sort(cell << np.uint64(37) | mask << np.uint64(5) | solver)
    return [n, out.view(np.int64)]


def _run_engine(s):
    if s["case"]["feed"] == "device":
        _set_state(s)
    return _sorted(s["eng"].check(), s["case"])


def _run_order(s):
    _set_state(s)
    s["eng"].launch()
    head = s["eng"].wait_head(out=s["head"])
    tail = s["eng"].copy_tail(out=s["tail"])
    return _sorted(np.concatenate([head, tail]), s["case"])


def _prepare_host(case, seed):
    _, _, lits, offsets, start, state = _engine_inputs(case, seed)
    eng = g.Engine(0)
    eng.set_db(_host(lits), _host(offsets))
    return {"case": case, "eng": eng, "state": _host(state, np.uint32), "start": _host(start, np.uint32),
            "out": np.zeros(1 << 17, g.REPORT_DTYPE)}


def _run_host(s):
    return _sorted(s["eng"].pass_host(s["state"], s["start"], out=s["out"]), s["case"])


def _dense(cells, valid, masks, n_cells):
    """The slot masks of all cells; a cell without a record stays 0."""
    dense = torch.zeros(n_cells + 1, dtype=torch.int32, device="cuda")
    index = cells if valid is None else torch.where(valid, cells, n_cells)
    dense.scatter_(0, index, masks)
    return dense[:n_cells]


def _prepare_cells(case, seed):
    gen, _, lits, offsets, start, state = _engine_inputs(case, seed)
    n_vars, n_words, passes = case["n_vars"], case["n_words"], case["passes"]
    eng = g.Engine(0)
    eng.set_db(_host(lits), _host(offsets))
    states = [torch.empty(state.shape, dtype=torch.int32, pin_memory=True) for _ in range(passes)]
    for k, st in enumerate(states):
        st.copy_(state if k == 0 else _state(gen, case["state"], n_vars, n_words, None))
    cap = ROOM[case["lengths"]] * case["n_clauses"] + 65536
    outs = [torch.empty((cap, 2), dtype=torch.int32, pin_memory=True) for _ in range(passes)]
    vp = ctypes.c_void_p
    return {"case": case, "eng": eng, "start": _host(start, np.uint32), "states": states, "outs": outs,
            "sp": (vp * passes)(*[t.data_ptr() for t in states]), "op": (vp * passes)(*[t.data_ptr() for t in outs]),
            "caps": np.full(passes, cap, np.int64), "got": np.zeros(passes, np.int64)}


def _run_cells(s):
    c, eng = s["case"], s["eng"]
    rc = eng.lib.gss_check_passes_host_cells(eng.h, c["passes"], s["sp"], c["n_vars"], c["n_words"],
                                             s["start"].ctypes.data, None, s["op"], s["caps"].ctypes.data,
                                             s["got"].ctypes.data)
    if rc != 0:
        raise g.GssError(rc, eng.lib.gss_last_error().decode())
    out = []
    for n, t in zip(s["got"], s["outs"]):
        rec = t[:int(n)].cuda(non_blocking=True)
        out.append(_dense(rec[:, 0].long(), None, rec[:, 1], c["n_clauses"] * c["n_words"]))
    return out


N_PARTS = 16


def _prepare_noalloc(case, seed):
    _, _, lits, offsets, start, state = _engine_inputs(case, seed)
    cap = 4096 + ROOM[case["lengths"]] * case["n_clauses"] // N_PARTS
    lib = g.load()
    vp, u32 = ctypes.c_void_p, ctypes.c_uint32
    lib.gss_check_noalloc.argtypes = [vp, vp, u32, vp, u32, u32, vp, vp, vp, u32, u32, vp, vp]
    return {"case": case, "fn": lib.gss_check_noalloc, "lits": lits, "offsets": offsets, "state": state,
            "start": start, "sow": torch.arange(32, dtype=torch.int32, device="cuda"), "cap": cap,
            "out": torch.zeros((N_PARTS, cap, 4), dtype=torch.int32, device="cuda"),
            "counts": torch.zeros(N_PARTS, dtype=torch.int32, device="cuda"),
            "rank": torch.arange(cap, dtype=torch.int32, device="cuda")}


def _run_noalloc(s):
    c = s["case"]
    rc = s["fn"](s["lits"].data_ptr(), s["offsets"].data_ptr(), c["n_clauses"], s["state"].data_ptr(), c["n_vars"], 1,
                 s["start"].data_ptr(), s["sow"].data_ptr(), s["out"].data_ptr(), N_PARTS, s["cap"],
                 s["counts"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise g.GssError(rc, g.load().gss_last_error().decode())
    valid = s["rank"][None, :] < s["counts"][:, None]
    cell = s["out"][:, :, 0].long() * 32 + s["out"][:, :, 1]
    return [_dense(cell.reshape(-1), valid.reshape(-1), s["out"][:, :, 2].reshape(-1), c["n_clauses"] * 32),
            s["counts"].sum()]


# ---- the clause sharer ----

BURST = 2  # assignments a solver sends between two passes
GROUPS, GROUP = 4, 4


def _prepare_sharer(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    n_vars, n_solvers = case["n_vars"], case["n_solvers"]
    model = torch.randint(0, 2, (n_vars,), generator=gen, device="cuda", dtype=torch.int32)
    lits, offsets = _clauses(gen, case["n_clauses"], n_vars, case["lengths"], model)
    lits, ends = _host(lits), _host(offsets).tolist()
    true_lit = _host(2 * torch.arange(n_vars, device="cuda", dtype=torch.int32) + 1 - model)
    sh = g.ClauseSharer(minGpuLatencyMicros=0)
    sh.setVarCount(n_vars)
    sh.setCpuSolverCount(n_solvers)
    sh.setMaxClauseLen(256)
    add, h, base = sh.lib.gss_sharer_add_clause, sh.h, lits.ctypes.data
    for a, b in zip(ends[:-1], ends[1:]):
        add(h, -1, base + 4 * a, b - a)
    rng = np.random.default_rng(seed)
    groups = []
    for k in range(n_solvers):
        on = rng.random(n_vars) < 0.5
        trail, off = rng.permutation(np.nonzero(on)[0]), np.nonzero(~on)[0]
        first = np.ascontiguousarray(true_lit[trail])
        if not sh.trySetSolverValues(k, first):
            raise RuntimeError("no room for the first assignment")
        sh.trySendAssignment(k)
        move = [np.ascontiguousarray(first[q * GROUP:(q + 1) * GROUP]) for q in range(GROUPS)]
        groups.append([(m, m.ctypes.data) for m in move])
        # a clause for two of the groups that is unit while the group is on the trail
        for q in (1, 3):
            rest = first[GROUPS * GROUP + 20 * q:][:int(rng.integers(10, 18))]
            lit = 2 * int(off[int(rng.integers(len(off)))])
            sh.addClause(-1, np.concatenate([move[q][:1] ^ 1, rest ^ 1, np.array([lit], np.int32)]))
    s = {"case": case, "sh": sh, "groups": groups, "step": 0, "on": [True] * GROUPS}
    _run_sharer(s)
    return s


def _run_sharer(s):
    """Each solver backtracks or extends its trail and sends it, twice; the
    GPU thread runs the pass and the next one, which delivers its reports."""
    sh = s["sh"]
    h, lib = sh.h, sh.lib
    for _ in range(BURST):
        q = s["step"] % GROUPS
        s["step"] += 1
        move = lib.gss_sharer_unset_solver_values if s["on"][q] else lib.gss_sharer_try_set_solver_values
        s["on"][q] = not s["on"][q]
        for k, gr in enumerate(s["groups"]):
            move(h, k, gr[q][1], GROUP)
            lib.gss_sharer_try_send_assignment(h, k)
    sh.gpuRun()
    sh.gpuRun()
    ids, lits, done = [], [], []
    for k in range(len(s["groups"])):
        for l, i in sorted(sh.popAll(k), key=lambda x: x[1]):
            ids += [k, i]
            lits += l
        done.append(sh.getLastAssigAllReported(k))
    out = np.zeros((2, 1 << 14), np.int64)
    out[0, :len(ids)] = ids
    out[1, :len(lits)] = lits
    return [len(ids), len(lits), out, np.array(done, np.int64)]


# ---- the scorer ----

def _scorer_inputs(case, seed):
    """Weights as the scorer starts with, features and labels as the passes log them."""
    rng = np.random.default_rng(seed)
    f, h = g.SCORER_FEATURES, g.SCORER_HIDDEN
    w = [rng.uniform(-1, 1, (h, f)) * (6 / f) ** 0.5, rng.uniform(-0.05, 0.05, h),
         rng.uniform(-1, 1, (h, h)) * (6 / h) ** 0.5, rng.uniform(-0.05, 0.05, h), rng.uniform(-1, 1, h) * (6 / h) ** 0.5,
         np.zeros(1)]
    w = [a.astype(np.float32) for a in w]
    x = rng.random((case["rows"], f), dtype=np.float32)
    y = (rng.random(case["rows"]) < 0.05 + 0.4 * x[:, 4]).astype(np.float32)
    return w, x, y


def _prepare_scorer(case, seed):
    w, x, y = _scorer_inputs(case, seed)
    sc = g.Scorer(0)
    sc.set_weights(np.concatenate([a.reshape(-1) for a in w]))
    return {"case": case, "sc": sc, "x": x, "y": y}


def _run_train(s):
    return [s["sc"].train_step(s["x"], s["y"], 1e-3), s["sc"].weights()]


def _run_infer(s):
    return s["sc"].infer(s["x"])


def exact(case, seed):
    if case["kind"] not in ("train", "infer"):
        return None
    w, x, y = _scorer_inputs(case, seed)
    w1, b1, w2, b2, w3, b3 = (a.astype(np.float64) for a in w)
    x, y = x.astype(np.float64), y.astype(np.float64)
    h1 = np.maximum(x @ w1.T + b1, 0)
    h2 = np.maximum(h1 @ w2.T + b2, 0)
    z = h2 @ w3 + b3
    if case["kind"] == "infer":
        return z
    loss = np.mean(np.maximum(z, 0) - z * y + np.log1p(np.exp(-np.abs(z))))
    dz = (1 / (1 + np.exp(-z)) - y) / len(y)
    d2 = dz[:, None] * w3 * (h2 > 0)
    d1 = d2 @ w2 * (h1 > 0)
    grad = np.concatenate([(d1.T @ x).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), dz @ h2, [dz.sum()]])
    # Adam's first step from zero moments
    return [loss, np.concatenate([a.reshape(-1).astype(np.float64) for a in w]) - 1e-3 * grad / (np.abs(grad) + 1e-8)]


PREPARE = {"engine": _prepare_engine, "order": _prepare_engine, "host": _prepare_host, "cells": _prepare_cells,
           "noalloc": _prepare_noalloc, "sharer": _prepare_sharer, "train": _prepare_scorer, "infer": _prepare_scorer}
RUN = {"engine": _run_engine, "order": _run_order, "host": _run_host, "cells": _run_cells, "noalloc": _run_noalloc,
       "sharer": _run_sharer, "train": _run_train, "infer": _run_infer}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def run(state):
    return RUN[state["case"]["kind"]](state)


def work(case):
    kind = case["kind"]
    if kind in ("train", "infer"):
        params, rows = g.SCORER_PARAMS, case["rows"]
        macs = g.SCORER_HIDDEN * (g.SCORER_FEATURES + g.SCORER_HIDDEN + 1)
        if kind == "infer":
            return {"bytes": 4 * (params + rows * (g.SCORER_FEATURES + 1)), "flops": 2 * rows * macs}
        return {"bytes": 4 * (6 * params + rows * (g.SCORER_FEATURES + 1)), "flops": 6 * rows * macs}
    n, lits = case["n_clauses"], case["n_clauses"] * MEAN_LEN[case["lengths"]]
    if kind == "sharer":
        return {"bytes": 4 * lits + 8 * n + 8 * case["n_vars"] * case["n_solvers"], "flops": 0}
    reports = 4 * n if case["state"] == "uniform" else n / 1000
    state, passes = 8 * case["n_vars"] * case["n_words"], case.get("passes", 1)
    return {"bytes": passes * (4 * lits + 8 * n + state + 16 * reports), "flops": 0}
