"""The workloads this framework is timed on: what a program that links
libpcagb.so (or imports pca_gb300) has it do, each through a public entry
point.

  solve     Engine.solve: the exhaustive proof of one task (the shortest
            program, or that there is none up to a kernel depth), one launch
            shape and split level stated, with or without the reference's
            per-level counters
  batch     Engine.solve_batch, first program per task: the mix of synthetic
            tasks a server or a label generator submits together
  complete  Engine.complete: the shortest completion of a partly written
            program (what the labels of the value network are checked by)
  branch    Engine.solve_branch: the reference solver's default search, by
            its counters or by its hybrid solver's stopping rule
  score     ValueNet.forward_fused: the network's logits for the states of a
            level (value-ordered search)
  train     ValueNet.train_step_graph: one optimiser step on labelled states

A case is a dict of plain values; `listed()` names the fixed ones and
`draw(rng)` gives another of the same ranges.
"""
import math
import random

import numpy as np
import torch

GIB = 1 << 30

# tasks: a 16-bit function of one or two 16-bit inputs
M = 0xFFFF
ONE_STEP = [lambda x: -x & M, lambda x: 2 * x & M, lambda x: x * x & M, lambda x: x - 3 & M]
FUNCTIONS = {
    "is_power2": (1, lambda x: int(x != 0 and x & (x - 1) == 0)),
    "popcount": (1, lambda x: bin(x).count("1")),
    "abs": (1, lambda x: -x & M if x & 0x8000 else x),
    "relu": (1, lambda x: 0 if x & 0x8000 else x),
    "max": (2, lambda x, y: max(x, y)),
    "saturating_add": (2, lambda x, y: min(x + y, M)),
    "hamming": (2, lambda x, y: bin(x ^ y).count("1")),
}


def listed():
    return [
        # the smallest call: a one-instruction function, proven at depth 1
        # (latency: host work, launches, one read of the answer)
        dict(name="solve_one_step", kind="solve", fn="one_step", tests=16, depth=4, split=3,
             counters=False),
        # the headline proof: no branchless is_power2 of kernel depth <= 4
        dict(name="solve_power2_d4", kind="solve", fn="is_power2", tests=32, depth=4, split=3,
             counters=False),
        # the request that sets a server's p99: a two-input function with no
        # program up to depth 4, an odd number of tests
        dict(name="solve_two_input_d4", kind="solve", fn="max", tests=27, depth=4, split=2,
             counters=False),
        # a proof one instruction deeper (what the workloads' open tasks take)
        dict(name="solve_power2_d5", kind="solve", fn="is_power2", tests=32, depth=5, split=3,
             counters=False),
        # the reference enumerator's counters: every level built and
        # leaf-checked, at the reference's own task size (11 tests)
        dict(name="counters_popcount_d3", kind="solve", fn="popcount", tests=11, depth=3, split=3,
             counters=True),
        # the batched workload's mix, one engine's share of it
        dict(name="batch_256", kind="batch", tasks=256, depth=4),
        # a handful of requests found in a server's queue together
        dict(name="batch_8", kind="batch", tasks=8, depth=3),
        # completing a program three instructions from its end
        dict(name="complete_d3", kind="complete", tests=19, done=1, depth=3),
        # branch mode: the enumerator's counters on a task of the reference's
        # size, and the hybrid solver's stopping rule on a two-input one
        dict(name="branch_relu_d3", kind="branch", fn="relu", tests=11, depth=3, first=False),
        dict(name="branch_max_first", kind="branch", fn="max", tests=11, depth=3, first=True),
        # ranking a level of states, and one training step
        dict(name="score_131072", kind="score", states=131072),
        dict(name="train_8192", kind="train", states=8192),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "complete", "branch", "score", "train"])
    if kind == "solve":
        which = rng.choice(["one_step", "one", "one", "two", "counters", "deep"])
        if which == "one_step":
            return dict(kind=kind, fn="one_step", tests=rng.randint(8, 32), depth=rng.randint(2, 4),
                        split=rng.randint(2, 3), counters=False)
        if which == "one":
            return dict(kind=kind, fn=rng.choice(["is_power2", "popcount", "abs"]),
                        tests=rng.randint(14, 32), depth=4, split=rng.randint(2, 3),
                        counters=False)
        if which == "two":
            return dict(kind=kind, fn=rng.choice(["max", "saturating_add", "hamming"]),
                        tests=rng.randint(16, 32), depth=rng.randint(3, 4), split=2,
                        counters=False)
        if which == "counters":
            return dict(kind=kind, fn=rng.choice(["is_power2", "popcount", "abs"]),
                        tests=rng.randint(8, 32), depth=rng.randint(2, 3), split=3, counters=True)
        return dict(kind=kind, fn=rng.choice(["is_power2", "popcount"]), tests=rng.randint(24, 32),
                    depth=5, split=3, counters=False)
    if kind == "batch":
        n = round(math.exp(rng.uniform(math.log(2), math.log(256))))
        return dict(kind=kind, tasks=n, depth=rng.randint(3, 4))
    if kind == "complete":
        return dict(kind=kind, tests=rng.randint(8, 32), done=rng.randint(1, 2),
                    depth=rng.randint(2, 3))
    if kind == "branch":
        fn, depth, first = rng.choice([("abs", 3, False), ("abs", 3, True), ("relu", 3, False),
                                       ("relu", 3, True), ("max", 3, False), ("max", 3, True)])
        return dict(kind=kind, fn=fn, tests=rng.randint(8, 16), depth=depth, first=first)
    if kind == "score":
        return dict(kind=kind, states=round(math.exp(rng.uniform(math.log(4096), math.log(131072)))))
    return dict(kind=kind, states=round(math.exp(rng.uniform(math.log(1024), math.log(8192)))))


# ---- inputs ------------------------------------------------------------------

EDGES = [0, 1, 0xFFFF, 0x7FFF, 0x8000]


def _values(rng, fn, n):
    """n distinct inputs of a task: edge values and uniform ones (half powers
    of two for is_power2, as its specs have them)."""
    arity = FUNCTIONS[fn][0] if fn in FUNCTIONS else 1
    rows = []
    if fn == "is_power2":
        rows += [(1 << k,) for k in rng.sample(range(15), min(12, n * 3 // 8))]
        rows += [(0,), (0x8000,)]
    elif arity == 1:
        rows += [(v,) for v in EDGES]
    while len(rows) < n:
        row = tuple(rng.randrange(1 << 16) for _ in range(arity))
        if arity == 2 and len(rows) < n // 4:
            row = tuple(v % 64 for v in row)  # small values among them
        if row not in rows:
            rows.append(row)
    rows = rows[:n]
    rng.shuffle(rows)
    return rows


def _task(case, seed):
    from pca_gb300.pcalib import make_task
    rng = random.Random(seed)
    f = ONE_STEP[seed % len(ONE_STEP)] if case["fn"] == "one_step" else FUNCTIONS[case["fn"]][1]
    rows = _values(rng, case["fn"], case["tests"])
    return make_task(case["fn"], [list(r) for r in rows], [f(*r) for r in rows])


def _completion(case, seed, eng, lib):
    """A state `done` instructions into a program and a task whose outputs the
    program reaches `depth` instructions later, each reading the one before."""
    from pca_gb300.pcalib import make_task
    rng = random.Random(seed)
    rows = [[rng.randrange(1 << 16) for _ in range(2)] for _ in range(case["tests"])]
    task = make_task("completion", rows, [0] * len(rows))
    ctx = lib.init_ctx(task)
    state = end = lib.init_root(ctx)
    last = 1
    for d in range(case["done"] + case["depth"]):
        # words are [op:5][rd:3][rs:3][rt:3][pad:2], ops up to 0x0C reading rs and rt
        alu = [c for c in lib.gen_candidates(end)
               if c >> 11 <= 0x0C and (c >> 5 & 7) == last and (c >> 2 & 7) not in (0, last)]
        insn = rng.choice(alu)
        last = insn >> 8 & 7
        end = lib.step(ctx, end, insn)
        if d + 1 == case["done"]:
            state = end
    task = make_task("completion", rows, [end.regs[t][last] for t in range(len(rows))])
    return dict(case=case, eng=eng, ctx=lib.init_ctx(task), state=state)


def _net_weights(seed):
    """The network's weights as they are initialised for training, by layer."""
    g = torch.Generator().manual_seed(seed)
    sd = {}
    for name, out, inp in (("E1", 256, 176), ("E2", 256, 256), ("T1", 256, 528), ("T2", 128, 256),
                           ("H", 16, 128)):
        bound = 1.0 / math.sqrt(inp)
        w = (torch.rand(out, inp, generator=g) * 2 - 1) * bound
        if name == "T1":
            w[:, 521:] = 0.0  # padding columns
        sd["W." + name] = w
        sd["b." + name] = (torch.rand(out, generator=g) * 2 - 1) * bound
    return sd


TASKS_OF_STATES = 24


def _states(n, seed):
    """n states of 24 tasks in the level layout (regs [n][8][32] with unused
    tests zero, r0 zero), made on the GPU; half the registers hold values as
    searches leave them (an input, zero, a small constant), half are
    uniform."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    ri = lambda lo, hi, shape: torch.randint(lo, hi, shape, generator=g, device="cuda",  # noqa: E731
                                             dtype=torch.int32)
    T = ri(16, 33, (TASKS_OF_STATES,))
    io = ri(0, 1 << 16, (TASKS_OF_STATES, 3, 32))
    io[::2, 1] = 0  # one-input tasks
    inside = torch.arange(32, device="cuda")[None, :] < T[:, None]
    io = io * inside[:, None, :]
    task = ri(0, TASKS_OF_STATES, (n,)).sort().values
    regs = ri(0, 1 << 16, (n, 8, 32))
    kind = ri(0, 6, (n, 8, 1))
    t = task.long()
    regs = torch.where(kind == 0, torch.zeros_like(regs), regs)
    regs = torch.where(kind == 1, regs[:, :, :1] % 256, regs)
    regs = torch.where(kind == 2, io[t][:, :1, :].expand(-1, 8, -1), regs)
    regs = regs * inside[t][:, None, :]
    regs[:, 0] = 0
    flags = ri(0, 16, (n, 32)) * inside[t]
    live = ri(0, 256, (n,)) & 0xFE
    depth = ri(1, 5, (n,))
    label = (ri(0, 17, (n,)) == 0).float()
    remaining = torch.where(label > 0.5, ri(1, 4, (n,)), torch.full((n,), -1, device="cuda",
                                                                     dtype=torch.int32))
    half = lambda x: x.to(torch.int16).contiguous()  # noqa: E731 - raw 16-bit words
    byte = lambda x: x.to(torch.uint8).contiguous()  # noqa: E731
    return dict(regs=half(regs), flags=byte(flags), live=byte(live), task=half(task),
                task_io=half(io), task_T=T, depth=byte(depth), label=label, remaining=remaining,
                TP=32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("score", "train"):
        from pca_gb300.valuenet import ValueNet
        net = ValueNet(seed=0)
        net.load_state_dict(_net_weights(seed))
        return dict(case=case, net=net, batch=_states(case["states"], seed))
    from pca_gb300 import taskgen
    from pca_gb300.pcalib import Engine, PCALib
    if kind == "batch":
        tasks = taskgen.synthetic_batch(case["tasks"], seed)
        return dict(case=case, eng=Engine(0, 24 * GIB), tasks=tasks)
    if kind == "complete":
        return _completion(case, seed, Engine(0, 8 * GIB), PCALib())
    budget = 16 if kind == "solve" and case["depth"] >= 5 else 8
    return dict(case=case, eng=Engine(0, budget * GIB), task=_task(case, seed))


# ---- one pass ----------------------------------------------------------------


def _programs(programs, most):
    """Programs as rows (length, words), `most` rows."""
    out = np.zeros((most, 17), dtype=np.int32)
    for i, p in enumerate(programs[:most]):
        out[i, 0] = len(p)
        out[i, 1:1 + len(p)] = p
    return out


def _counts(per_depth):
    """A per-depth counter as depths 0..16 (-1 past the searched ones)."""
    return np.array(list(per_depth) + [-1] * (17 - len(per_depth)), dtype=np.int64)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "solve":
        s = state["eng"].solve(state["task"], max_depth=case["depth"], split_depth=case["split"],
                               count_levels=case["counters"])
        return dict(depth=s.optimal_depth, solutions=s.total_solutions,
                    programs=_programs(s.programs, 4096),
                    candidates=_counts(s.candidates),
                    evaluations=_counts(s.evaluations),
                    tried=_counts(s.tried),
                    pruned=_counts(s.pruned_cum),
                    children=_counts(s.level_children),
                    survivors=_counts(s.level_survivors))
    if kind == "batch":
        sols = state["eng"].solve_batch(state["tasks"], max_depth=case["depth"], first_only=True,
                                        sol_cap=1)
        return dict(depth=np.array([s.optimal_depth for s in sols], dtype=np.int32),
                    programs=_programs([s.programs[0] if s.programs else [] for s in sols],
                                       len(sols)))
    if kind == "complete":
        found, n, insns, _ = state["eng"].complete(state["ctx"], state["state"],
                                                   case["done"] + case["depth"])
        return dict(found=found, length=n, program=_programs([insns], 1))
    if kind == "branch":
        s = state["eng"].solve_branch(state["task"], max_depth=case["depth"],
                                      first_only=case["first"])
        out = dict(depth=s.optimal_depth, programs=_programs(s.programs, 100))
        if not case["first"]:
            out.update(tried=_counts(s.tried), pruned=_counts(s.pruned_cum))
        return out
    net, b = state["net"], state["batch"]
    if kind == "score":
        return net.forward_fused(b["regs"], b["flags"], b["live"], b["task"], b["depth"], b["TP"],
                                 b["task_io"], b["task_T"])
    loss = net.train_step_graph(b)
    return dict(loss=loss, mW=dict(net.mW), mb=dict(net.mb), W=dict(net.W), b=dict(net.b))


# ---- work --------------------------------------------------------------------

# Distinct states of levels 0..3 by inputs (one- and two-input tasks of 16 or
# more tests; the counts vary by a few percent with the task), the mean
# children of a state and the value classes among them.
LEVELS = {1: (1, 159, 24.5e3, 5.3e6), 2: (1, 311, 100e3, 42e6)}
CHILDREN = {1: (214, 397, 631, 918), 2: (435, 650, 914, 1190)}
CLASSES = {1: (36, 67, 104, 150), 2: (73, 108, 149, 192)}
ENCODER_FLOPS = 2 * 32 * 256 * (176 + 256)
TRUNK_FLOPS = 2 * (528 * 256 + 256 * 128 + 128 * 16)
WEIGHT_BYTES = 281488 * 4


def work(case):
    """What one pass cannot do without. A search has to put every child of
    every level it builds into the exact state table (an ALU operation per
    test and an 8-byte slot) and to decide every value class of the last
    position (one operation each); a state written is its registers on every
    test. A network pass reads the states and the weights and does the
    network's products."""
    kind = case["kind"]
    if kind == "score":
        n = case["states"]
        return {"bytes": n * (8 * 64 + 32 + 4 + 64) + WEIGHT_BYTES,
                "flops": n * (ENCODER_FLOPS + TRUNK_FLOPS)}
    if kind == "train":
        n = case["states"]
        back = 2 * 32 * 256 * 256 + TRUNK_FLOPS          # input gradients (none for E1)
        return {"bytes": n * (8 * 64 + 32 + 4 + 8) + 7 * WEIGHT_BYTES,
                "flops": n * (2 * (ENCODER_FLOPS + TRUNK_FLOPS) + back)}
    if kind == "branch":
        # CMP, BR, DIV and MOD besides: about twice the candidates of a state
        two = FUNCTIONS[case["fn"]][0] == 2
        last = {2: 5e4, 3: 2e7}[case["depth"]] * (8 if two else 1)
        return {"bytes": last / 100 * 8, "flops": last}
    if kind == "batch":
        # most tasks end at depth 1 or 2; a seventh take the whole search
        per = 2e5 if case["depth"] == 3 else 1.6e8
        return {"bytes": case["tasks"] * per / 30 * 8, "flops": case["tasks"] * per}
    if kind == "complete":
        inputs, depth, tests = 2, case["depth"] + case["done"] - 1, case["tests"]
        built = case["depth"] - 2
    elif case["fn"] == "one_step":
        return {"bytes": 16 * 17 + case["tests"] * 8, "flops": CLASSES[1][0] * case["tests"]}
    else:
        inputs, depth, tests = FUNCTIONS[case["fn"]][0], case["depth"], case["tests"]
        built = depth if case["counters"] else min(case["split"], depth - 1)
    kids, states = 0.0, 0.0
    for d in range(min(built, 3)):
        kids += LEVELS[inputs][d] * CHILDREN[inputs][d]
        states += LEVELS[inputs][d + 1]
    # the last position: the states of the split level times the middles
    s = min(built, 3)
    last = LEVELS[inputs][s] * CLASSES[inputs][s]
    for k in range(depth - s - 1):
        last *= CHILDREN[inputs][min(s + k, 3)]
    if case.get("counters"):
        last = 0.0
    return {"bytes": kids * 8 + states * 16 * tests, "flops": kids * tests + last}


# ---- the same in 64 bits -----------------------------------------------------


def _net64(W, b, s):
    """Logits of the network in 64 bits (states in the level layout)."""
    T = s["task_T"][s["task"].long()].long()
    io = s["task_io"][s["task"].long()].long() & M                       # [n][3][32]
    regs = s["regs"].view(-1, 8, 32)[:, 1:].long() & M                   # [n][7][32]
    bits = torch.arange(16, device=io.device)
    words = torch.cat([io, regs], 1)                                      # [n][10][32]
    x = ((words[..., None] >> bits) & 1).permute(0, 2, 1, 3).reshape(len(T), 32, 160)
    fl = (s["flags"].view(-1, 32, 1).long() >> torch.arange(4, device=io.device)) & 1
    x = torch.cat([x, fl, torch.zeros(len(T), 32, 12, dtype=torch.long, device=io.device)], 2)
    mask = torch.arange(32, device=io.device)[None, :] < T[:, None]
    x = x.double() * mask[:, :, None]
    lin = lambda v, k: v @ W[k].t() + b[k]  # noqa: E731
    h = torch.relu(lin(torch.relu(lin(x, "E1")), "E2"))
    mean = (h * mask[:, :, None]).sum(1) / T[:, None]
    top = h.masked_fill(~mask[:, :, None], -1e30).max(1).values
    g = torch.zeros(len(T), 16, dtype=torch.float64, device=io.device)
    g[:, :8] = ((s["live"].long()[:, None] >> torch.arange(8, device=io.device)) & 1).double()
    g[:, 8] = s["depth"].double()
    z = torch.relu(lin(torch.relu(lin(torch.cat([mean, top, g], 1), "T1")), "T2"))
    return lin(z, "H")


def exact(case, seed):
    if case["kind"] not in ("score", "train"):
        return None  # whole numbers
    s = _states(case["states"], seed)
    sd = {k: v.cuda().double() for k, v in _net_weights(seed).items()}
    W = {k[2:]: v for k, v in sd.items() if k[0] == "W"}
    b = {k[2:]: v for k, v in sd.items() if k[0] == "b"}
    per_state = ("regs", "flags", "live", "task", "depth")
    part = lambda i, j: dict(s, **{k: s[k][i:j] for k in per_state})  # noqa: E731
    n, step = case["states"], 2048
    if case["kind"] == "score":
        return torch.cat([_net64(W, b, part(i, i + step)) for i in range(0, n, step)])
    params = list(W.values()) + list(b.values())
    for p in params:
        p.requires_grad_(True)
    npos = s["label"].sum().double().clamp(min=1.0)
    loss = 0.0
    for i in range(0, n, step):
        lg = _net64(W, b, part(i, i + step))
        y = s["label"][i:i + step].double()
        # BCE with pos_weight 50 on column 0 and half the cross entropy of the
        # remaining steps over the positives
        bce = 50.0 * y * torch.nn.functional.softplus(-lg[:, 0]) + \
            (1 - y) * torch.nn.functional.softplus(lg[:, 0])
        ce = -torch.log_softmax(lg[:, 1:10], 1).gather(
            1, s["remaining"][i:i + step].long().clamp(min=0)[:, None])[:, 0]
        part_loss = bce.sum() / n + 0.5 * (ce * (y > 0.5)).sum() / npos
        part_loss.backward()
        loss += float(part_loss.detach())
    moment = lambda d: {k: 0.1 * v.grad for k, v in d.items()}  # noqa: E731 - Adam's first step
    return dict(loss=torch.tensor(loss, dtype=torch.float64), mW=moment(W), mb=moment(b),
                W=None, b=None)
