"""Performance cases: calls that programs make through the public API, over its range.

A case is a dict of plain values with a ``kind``:

* ``solve``  one rate set, one x0 through ``solve``: the interactive call
* ``full``   ``solve`` with its default method and every output (R and L too)
* ``host``   ``solve_host``: host arrays in and out, symbolic data built in the call
* ``table``  the transition table of a knock-out (one rate zero) as CSC
* ``graph``  SCCs, levels and order of a knock-out: ``Net.build`` and ``Net.export``
* ``batch``  B rate sets x R initial distributions on a network that is kept
* ``step``   the same with the network built in the call, as a parameter scan over
             zero-rate patterns does
* ``many``   ``solve_many``: several networks over a pool of contexts
* ``warm``   learned warm start: ``Mlp.predict`` and the mixed-precision batch solve
* ``grad``   loss and gradient of the warm-start network on a batch of samples

The network is part of the case (family, size, seed); rates, x0 and samples come from
the seed that ``prepare`` is given.
"""
from __future__ import annotations

import numpy as np
import torch

import paraexastolog_b200 as esl
from paraexastolog_b200 import synth


def listed():
    return [
        # a user trying out one small model: latency of one call
        {"name": "solve_n10", "kind": "solve", "family": "small", "n": 10, "net_seed": 0},
        # the reference's full answer for a small model: x_inf, R and L
        {"name": "full_n11", "kind": "full", "family": "small", "n": 11, "net_seed": 5},
        # command-line use: a few rate sets from host memory, network built on the way
        {"name": "host_n13_b3_r2", "kind": "host", "family": "precision", "n": 13, "net_seed": 2, "B": 3, "R": 2},
        # transition table of a large network with one rate knocked out
        {"name": "table_n22", "kind": "table", "family": "scale", "n": 22, "net_seed": 1, "knockout": 7},
        # symbolic data of the benchmark's network with one rate knocked out
        {"name": "graph_n20", "kind": "graph", "family": "precision", "n": 20, "net_seed": 2, "knockout": 12},
        # a parameter scan of a small network
        {"name": "batch_n12_b64", "kind": "batch", "family": "batch", "n": 12, "net_seed": 3, "B": 64, "R": 1,
         "occupation": False},
        # training data for the warm start: ragged batch, several x0, occupation kept
        {"name": "batch_n17_b37_r5", "kind": "batch", "family": "precision", "n": 17, "net_seed": 2, "B": 37, "R": 5,
         "occupation": True},
        # the benchmark's step: a large network and 512 rate sets from scratch
        {"name": "step_n20_b512", "kind": "step", "family": "precision", "n": 20, "net_seed": 2, "B": 512, "R": 1},
        # one solve of the largest network: no batch to fill the GPU with
        {"name": "solve_n22", "kind": "solve", "family": "scale", "n": 22, "net_seed": 1},
        # an ensemble of networks, as in the many-network workload
        {"name": "many_8_n12_15", "kind": "many", "family": "batch", "count": 8, "n_lo": 12, "n_hi": 15, "net_seed": 3,
         "B": 16, "R": 4},
        # serving with the learned warm start and mixed precision
        {"name": "warm_n16_b64", "kind": "warm", "family": "precision", "n": 16, "net_seed": 2, "B": 64, "R": 1},
        # one training step's gradient of the warm-start network
        {"name": "grad_n16_s16384", "kind": "grad", "family": "precision", "n": 16, "net_seed": 2, "sets": 256,
         "samples": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["solve", "full", "host", "table", "graph", "batch", "batch", "step", "many", "warm", "grad"])
    # networks that solve within the default budgets at every size below
    c = {"kind": kind, "net_seed": rng.randint(10, 50)}
    if kind == "solve":
        c["family"] = rng.choice(["small", "precision", "scale"])
        c["n"] = rng.randint(8, 20)
    elif kind == "full":
        c["family"], c["n"] = "small", rng.randint(7, 12)
    elif kind == "host":
        c["family"], c["n"] = rng.choice(["precision", "batch"]), rng.randint(9, 14)
        c["B"], c["R"] = _log_int(rng, 1, 8), rng.randint(1, 3)
    elif kind == "table":
        c["family"], c["n"] = rng.choice(["scale", "precision", "batch"]), rng.randint(10, 22)
        c["knockout"] = rng.randrange(2 * c["n"])
    elif kind == "graph":
        c["family"], c["n"] = rng.choice(["precision", "scale", "batch"]), rng.randint(10, 20)
        c["knockout"] = rng.randrange(2 * c["n"])
    elif kind in ("batch", "step"):
        c["family"], c["n"] = "precision", rng.randint(10, 18)
        c["B"], c["R"] = _log_int(rng, 1, min(512, 1 << (25 - c["n"]))), rng.randint(1, 3)
        if kind == "batch":
            c["occupation"] = rng.random() < 0.3
    elif kind == "many":
        c["family"], c["count"], c["n_lo"] = "batch", rng.randint(3, 12), rng.randint(10, 12)
        c["n_hi"] = c["n_lo"] + rng.randint(1, 3)
        c["B"], c["R"] = _log_int(rng, 1, 24), rng.randint(1, 5)
    elif kind == "warm":
        c["family"], c["n"] = "precision", rng.randint(14, 17)
        c["B"], c["R"] = 8 * _log_int(rng, 2, 12), 1
    else:
        c["family"], c["n"] = "precision", rng.randint(12, 17)
        c["sets"], c["samples"] = rng.randint(16, 512), _log_int(rng, 512, 32768)
    return c


# ---- networks and inputs ------------------------------------------------------------------


def _network(family, n, net_seed):
    if family == "precision":
        return synth.precision_network(net_seed, n)
    rng = np.random.default_rng(net_seed)
    if family == "small":
        return synth.random_table_network(rng, n, [2], 0.5)
    if family == "scale":
        return synth.nested_canalizing_network(rng, n, 3)
    return synth.random_table_network(rng, n, [3], 0.5)


def _networks(case):
    rng = np.random.default_rng(case["net_seed"])
    sizes = [int(rng.integers(case["n_lo"], case["n_hi"] + 1)) for _ in range(case["count"])]
    return [synth.random_table_network(rng, n, [3], 0.5) for n in sizes]


def _x0(rng, family, n, count):
    if family == "scale":
        nodes = rng.choice(n, size=4, replace=False)
        return np.stack([synth.fixed_nodes_x0(n, nodes, rng.integers(0, 2, size=4)) for _ in range(count)])
    free = min(8 if family == "precision" else 6, n)
    return np.stack([synth.dirichlet_subspace_x0(rng, n, rng.choice(n, size=free, replace=False))
                     for _ in range(count)])


def _inputs(case, seed):
    """(network, rates B x 2n, x0 R x N) of a case with one network, on the host."""
    n = case["n"]
    rng = np.random.default_rng(seed)
    return (_network(case["family"], n, case["net_seed"]), synth.log_uniform_rates(rng, n, case.get("B", 1)),
            _x0(rng, case["family"], n, case.get("R", 1)))


def _knockout(case, seed):
    """(network, rates) with one rate zero, the network's nodes listed in the seed's order."""
    net = _network(case["family"], case["n"], case["net_seed"])
    rng = np.random.default_rng(seed)
    order = [int(i) for i in rng.permutation(net.n)]
    place = {old: new for new, old in enumerate(order)}
    inputs = [[place[i] for i in net.inputs[old]] for old in order]
    tables = [net.tables[old] for old in order]
    names = [net.names[old] for old in order]
    rates = synth.log_uniform_rates(rng, net.n, 1)[0]
    rates[2 * place[case["knockout"] // 2] + case["knockout"] % 2] = 0.0
    return synth.Network(names, inputs, tables, synth.network_to_bnet(names, inputs, tables)), rates


def _samples(case, seed):
    """Parameters of the warm-start network and a batch of samples, on the host."""
    rng = np.random.default_rng(seed)
    rates = synth.log_uniform_rates(rng, case["n"], case["sets"])
    ks = rng.integers(0, case["sets"], size=case["samples"]).astype(np.int32)
    vs = rng.integers(0, 1 << case["n"], size=case["samples"]).astype(np.int32)
    target = rng.standard_normal(case["samples"]).astype(np.float32)
    parts = []
    for shape, fan in (((128, 77), 77), ((128,), 0), ((128, 128), 128), ((128,), 0), ((128,), 128), ((1,), 0)):
        bound = (6.0 / fan) ** 0.5 if fan else 0.05
        parts.append(rng.uniform(-bound, bound, size=shape).astype(np.float32).ravel())
    return rates, ks, vs, target, np.concatenate(parts)


_contexts = []


def _context(i=0):
    """A program's contexts live as long as it does, each on a stream of its own."""
    while len(_contexts) <= i:
        _contexts.append(esl.Context(0, torch.cuda.Stream()))
    return _contexts[i]


def _dev(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    s = {"kind": kind, "ctx": ctx}
    if kind == "many":
        rng = np.random.default_rng(seed)
        s["ctxs"] = [_context(i) for i in range(4)]
        s["jobs"] = []
        for net in _networks(case):
            rates, x0 = synth.log_uniform_rates(rng, net.n, case["B"]), _x0(rng, "batch", net.n, case["R"])
            s["jobs"].append((esl.Net.build(ctx, esl.Model.parse(net.bnet), rates[0]), _dev(rates), _dev(x0)))
        torch.cuda.synchronize()
        return s
    if kind in ("table", "graph"):
        net, s["rates"] = _knockout(case, seed)
        s["model"] = esl.Model.parse(net.bnet)
        return s
    if kind == "grad":
        net = _network(case["family"], case["n"], case["net_seed"])
        rates, ks, vs, target, params = _samples(case, seed)
        s["net"] = esl.Net.build(ctx, esl.Model.parse(net.bnet), rates[0])
        s["mlp"] = esl.Mlp(ctx, s["net"])
        s["mlp"].set_params(params, 0.0, 1.0)
        s["args"] = (_dev(rates), torch.as_tensor(ks, device="cuda"), torch.as_tensor(vs, device="cuda"),
                     torch.as_tensor(target, device="cuda"))
        torch.cuda.synchronize()
        return s
    net, rates, x0 = _inputs(case, seed)
    s["model"] = esl.Model.parse(net.bnet)
    if kind == "host":
        s["rates"], s["x0"] = rates, x0
        return s
    s["host_rates"], s["rates"], s["x0"] = rates, _dev(rates), _dev(x0)
    if kind != "step":
        s["net"] = esl.Net.build(ctx, s["model"], rates[0])
    if kind == "batch" and case["occupation"]:
        s["occupation"] = torch.empty((case["B"] * case["R"], 1 << case["n"]), dtype=torch.float64, device="cuda")
    if kind == "warm":
        # a short training on other rate sets of the same network
        train = synth.log_uniform_rates(np.random.default_rng(seed + 1), case["n"], 16)
        occ = torch.empty((16, 1 << case["n"]), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        esl.solve_batch(ctx, s["net"], train, s["x0"], method=esl.METHOD_DIRECT, occupation=occ)
        s["mlp"] = esl.Mlp(ctx, s["net"], seed=1)
        if s["mlp"].n_targets:
            s["mlp"].train(train, occ, steps=30, batch=4096)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "host":
        return esl.solve_host(ctx, s["model"], s["rates"], s["x0"], method=esl.METHOD_DIRECT)[:2]
    if kind == "grad":
        return s["mlp"].loss_grad(*s["args"])
    with torch.cuda.stream(ctx.stream):
        if kind == "solve":
            r = esl.solve(ctx, s["net"], s["rates"][0], s["x0"][0], method=esl.METHOD_DIRECT)
            return r.x_inf, r.marginals
        if kind == "full":
            r = esl.solve(ctx, s["net"], s["rates"][0], s["x0"][0], want_R=True, want_L=True)
            return r.x_inf, r.marginals, r.R, r.L
        if kind == "table":
            return esl.table(ctx, s["model"], s["rates"])
        if kind == "graph":
            return esl.Net.build(ctx, s["model"], s["rates"]).export()
        if kind == "many":
            return [(r.x_inf, r.marginals) for r in esl.solve_many(s["ctxs"], s["jobs"], method=esl.METHOD_DIRECT)]
        if kind == "warm":
            warm = s["mlp"].predict(s["rates"])
            r = esl.solve_batch(ctx, s["net"], s["rates"], s["x0"], method=esl.METHOD_MIXED, warm=warm)
            return r.x_inf, r.marginals
        net = s["net"] if kind == "batch" else esl.Net.build(ctx, s["model"], s["host_rates"][0])
        occ = s.get("occupation")
        r = esl.solve_batch(ctx, net, s["rates"], s["x0"], method=esl.METHOD_DIRECT, occupation=occ)
        return (r.x_inf, r.marginals) if occ is None else (r.x_inf, r.marginals, occ)


def work(case):
    """Inputs read once, outputs written once; one application of the generator (n
    multiply-adds per state and system) and one elimination for the operations."""
    kind = case["kind"]
    if kind == "many":
        each = [work(dict(case, kind="batch", n=net.n, occupation=False)) for net in _networks(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n = case["n"]
    N = 1 << n
    if kind in ("table", "graph"):
        # half of the n flips of a state, on average, are edges
        return {"bytes": 4 * N * (1 + n) if kind == "table" else 8 * N, "flops": N * n}
    if kind == "grad":
        macs = 77 * 128 + 128 * 128 + 128
        return {"bytes": 12 * case["samples"] + 16 * n * case["sets"] + 8 * 26625,
                "flops": 6 * macs * case["samples"]}
    B, R = case.get("B", 1), case.get("R", 1)
    K = B * R
    out = 2 if case.get("occupation") else 1
    w = {"bytes": 8 * (N * (R + K * out) + 2 * n * B + n * K), "flops": 2 * n * N * K}
    if kind == "full":
        w = {"bytes": 2 * w["bytes"], "flops": 2 * w["flops"]}
    if kind == "warm":
        w["bytes"] += 8 * N * K
    return w


# ---- the same results in 64 bits, from the networks' truth tables -------------------------


def _flips(net):
    """Bit i of F[v]: node i's rule differs from its value in state v."""
    v = np.arange(1 << net.n, dtype=np.int64)
    F = np.zeros(1 << net.n, dtype=np.int64)
    for i, (inputs, tab) in enumerate(zip(net.inputs, net.tables)):
        idx = np.zeros_like(v)
        for j, inp in enumerate(inputs):
            idx |= ((v >> inp) & 1) << j
        F |= (np.asarray(tab, dtype=np.int64)[idx] ^ ((v >> i) & 1)) << i
    return F


def _closure(F, n, start, backward=False):
    """States reachable from (backward: reaching) the start set."""
    v = np.arange(1 << n)
    seen = start.copy()
    while True:
        new = seen.copy()
        for i in range(n):
            u = v ^ (1 << i)
            if backward:
                new |= seen[u] & ((F >> i) & 1).astype(bool)
            else:
                new |= seen[u] & ((F[u] >> i) & 1).astype(bool)
        if np.array_equal(new, seen):
            return seen
        seen = new


def _terminals(F, n):
    """Terminal SCCs, by smallest state: state arrays, ascending."""
    found, left = [], np.ones(1 << n, dtype=bool)
    for v in np.flatnonzero(F == 0):
        found.append(np.array([v]))
    left &= ~_closure(F, n, F == 0, backward=True)
    while left.any():
        v = int(np.flatnonzero(left)[0])
        while True:
            start = np.zeros(1 << n, dtype=bool)
            start[v] = True
            ahead, behind = _closure(F, n, start), _closure(F, n, start, backward=True)
            rest = ahead & ~behind
            if not rest.any():
                break
            v = int(np.flatnonzero(rest)[0])
        found.append(np.flatnonzero(ahead))
        left &= ~behind
    return sorted(found, key=lambda c: int(c[0]))


def _generator(F, n, rates):
    """K (dest, source): rate of every flip, columns summing to zero; dense on the GPU."""
    N = 1 << n
    v = np.arange(N)
    K = torch.zeros((N, N), dtype=torch.float64, device="cuda")
    for i in range(n):
        src = v[((F >> i) & 1).astype(bool)]
        rate = torch.as_tensor(rates[2 * i + ((src >> i) & 1)], device="cuda")
        s, d = torch.as_tensor(src, device="cuda"), torch.as_tensor(src ^ (1 << i), device="cuda")
        K[d, s] = rate
        K[s, s] -= rate
    return K


def _stationary(net, rates, x0, outputs):
    """x_inf (B x R x N), marginals and, where asked for, R, L and the occupation."""
    n, N = net.n, 1 << net.n
    F = _flips(net)
    classes = _terminals(F, n)
    term = np.concatenate(classes)
    trans = torch.as_tensor(np.setdiff1d(np.arange(N), term), device="cuda")
    x0 = torch.as_tensor(x0, device="cuda")
    bits = torch.as_tensor(((np.arange(N)[:, None] >> np.arange(n)) & 1).astype(np.float64), device="cuda")
    xs, occs = [], []
    for r in rates:
        K = _generator(F, n, r)
        A = -K[trans][:, trans]
        z = torch.linalg.solve(A, x0[:, trans].T) if len(trans) else torch.zeros((0, len(x0)), device="cuda")
        occ = torch.zeros((len(x0), N), dtype=torch.float64, device="cuda")
        occ[:, trans] = z.T
        x = torch.zeros_like(occ)
        kernel, L = [], torch.zeros((len(classes), N), dtype=torch.float64, device="cuda")
        for t, c in enumerate(classes):
            c = torch.as_tensor(c, device="cuda")
            inflow = K[c][:, trans]
            B = K[c][:, c]
            B[-1] = 1.0
            e = torch.zeros(len(c), dtype=torch.float64, device="cuda")
            e[-1] = 1.0
            pi = torch.linalg.solve(B, e)
            kernel.append(pi)
            x[:, c] = (x0[:, c].sum(1) + (inflow @ z).sum(0))[:, None] * pi
            if "L" in outputs:
                L[t, c] = 1.0
                if len(trans):
                    L[t, trans] = torch.linalg.solve(A.T, inflow.sum(0))
        xs.append(x)
        occs.append(occ)
    x = torch.stack(xs)
    return {"x": x, "marg": x @ bits, "occ": torch.cat(occs), "R": torch.cat(kernel), "L": L}


def _exact_grad(case, seed):
    n = case["n"]
    net = _network(case["family"], n, case["net_seed"])
    rates, ks, vs, target, params = _samples(case, seed)
    F = _flips(net)
    reach = np.zeros((1 << n, 16))
    classes = _terminals(F, n)
    for t, c in enumerate(classes[:16]):
        start = np.zeros(1 << n, dtype=bool)
        start[c] = True
        reach[:, t] = np.where(_closure(F, n, start, backward=True), 1.0, -1.0)
    x = np.zeros((len(ks), 77))
    bit = (vs[:, None] >> np.arange(n)) & 1
    x[:, :n] = 2.0 * bit - 1.0
    r = rates[ks].reshape(len(ks), n, 2)
    out = np.take_along_axis(r, bit[:, :, None], 2)[:, :, 0] * ((F[vs][:, None] >> np.arange(n)) & 1)
    q = out.sum(1)
    x[:, 20] = np.where(q > 0, np.log(np.where(q > 0, q, 1.0)), 0.0)
    x[:, 21:37] = reach[vs]
    x[:, 37:37 + 2 * n] = np.log(rates[ks])
    p = torch.as_tensor(params)
    cut = np.cumsum([128 * 77, 128, 128 * 128, 128, 128, 1])
    parts = [p[a:b] for a, b in zip([0, *cut[:-1]], cut)]
    W1, b1, W2, b2, w3, b3 = [(w.bfloat16() if i % 2 == 0 else w).double().requires_grad_() for i, w in enumerate(parts)]
    h1 = torch.relu(torch.as_tensor(x) @ W1.reshape(128, 77).T + b1)
    h2 = torch.relu(h1 @ W2.reshape(128, 128).T + b2)
    loss = ((h2 @ w3 + b3 - torch.as_tensor(target).double()) ** 2).mean()
    loss.backward()
    return loss.item(), torch.cat([w.grad.ravel() for w in (W1, b1, W2, b2, w3, b3)])


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _exact_grad(case, seed)
    # dense elimination: up to 2^14 states, and rate sets as long as that takes seconds
    if kind not in ("solve", "full", "host", "batch", "step", "warm"):
        return None
    if case["n"] > 14 or case.get("B", 1) * 8 ** case["n"] > 64 * 8 ** 12:
        return None
    net, rates, x0 = _inputs(case, seed)
    e = _stationary(net, rates, x0, ("L",) if kind == "full" else ())
    if kind == "solve":
        return e["x"][0, 0], e["marg"][0, 0]
    if kind == "full":
        return e["x"][0, 0], e["marg"][0, 0], e["R"], e["L"]
    return (e["x"], e["marg"], e["occ"]) if case.get("occupation") else (e["x"], e["marg"])
