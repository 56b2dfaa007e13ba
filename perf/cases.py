"""What a user of this engine has it do, as cases that can be timed and compared.

A case is one call of the public Python API with everything a user's program reads from its result:
a simulation of one model (`Context.compile` + `Module.run`, in exact, fast or epoch mode), a
parameter sweep (`Batch`), or a differentiable evaluation (`autograd.window_probabilities` with its
backward pass). The models are the example models of the tests and the seeded benchmark networks.
"""
import os
import re

import numpy as np
import torch

import maboss.gpu_b200 as mb
from maboss.gpu_b200 import synth
from maboss.gpu_b200.autograd import window_probabilities

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MODELS = os.path.join(ROOT, "tests", "golden", "models")

# nodes, non-internal nodes, windows and transitions of one trajectory (its mean) of the models
FILES = {
    "cellcycle": (10, 4, 25, 25),
    "metastasis": (32, 5, 200, 34),
    "sizek": (87, 4, 20, 519),
    "Montagud2022_Prostate_Cancer": (133, 3, 500, 194),
}


def listed():
    return [
        # a first look at an example model with its own trajectory count: launch latency
        dict(name="metastasis exact 1e3", call="run", net="metastasis", mode="exact", trajectories=1000),
        # the example model in discrete time, 10 nodes: very short trajectories, default mode
        dict(name="cellcycle exact 1e6", call="run", net="cellcycle", mode="exact", trajectories=1_000_000),
        # the buffered mode (the one a program with statistics of its own runs), a mid-sized model
        dict(name="sizek epoch 1e5", call="run", net="sizek", mode="epoch", trajectories=100_000),
        # a published model as its authors configured it: 133 nodes, 500 windows, default mode
        dict(name="montagud exact 1e6", call="run", net="Montagud2022_Prostate_Cancer", mode="exact",
             trajectories=1_000_000),
        # the benchmark's 10-node network: a small histogram hit by everyone
        dict(name="10 nodes fast 1e5", call="run", net="c1", mode="fast", trajectories=100_000),
        # the benchmark's 50-node network, forward only
        dict(name="50 nodes fast 1e6", call="run", net="c4", mode="fast", trajectories=1_000_000),
        # the headline workload: 1000 nodes, fast mode
        dict(name="1000 nodes fast 1e6", call="run", net="c3", nodes=1000, outputs=10, max_time=50.0, mode="fast",
             trajectories=1_000_000),
        # the same network in the default mode, an odd trajectory count
        dict(name="1000 nodes exact 250001", call="run", net="c3", nodes=1000, outputs=10, max_time=50.0,
             mode="exact", trajectories=250_001),
        # a histogram of 100 x 2^20 cells of which few are filled
        dict(name="100 nodes 20 outputs fast", call="run", net="c2", outputs=20, discrete=False, mode="fast",
             trajectories=200_000),
        # more output nodes than a dense histogram takes: sparse window bins
        dict(name="100 nodes 77 outputs fast", call="run", net="c2", outputs=77, discrete=False, mode="fast",
             trajectories=20_000),
        # a parameter sweep over networks of 20 to 500 nodes
        dict(name="sweep 64 variants", call="sweep", variants=64, max_trajectories=100_000),
        # one step of a gradient-based fit: forward and backward, 40 rate parameters
        dict(name="50 nodes fit step 1e6", call="fit", trajectories=1_000_000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["file", "file", "small", "synthetic", "synthetic", "synthetic", "outputs", "sweep", "fit"])
    mode = rng.choice(["exact", "exact", "fast", "fast", "epoch"])
    if kind == "file":
        return dict(call="run", net=rng.choice(sorted(FILES)), mode=mode,
                    trajectories=_log_uniform(rng, 1000, 200_000 if mode == "epoch" else 1_000_000))
    if kind == "small":
        return dict(call="run", net=rng.choice(["c1", "c4"]), mode=mode, trajectories=_log_uniform(rng, 1000, 500_000))
    if kind == "synthetic":
        nodes = _log_uniform(rng, 16, 1000)
        case = dict(call="run", net="c3", nodes=nodes, outputs=rng.randint(2, 10),
                    max_time=float(rng.randint(5, 50)), mode=mode)
        # at most as many transitions as the largest listed case of the mode
        most = {"fast": 2.0e9, "exact": 5.0e8, "epoch": 2.0e8}[mode] / _steps(case)
        return dict(case, trajectories=_log_uniform(rng, 1000, min(1_000_000, int(most))))
    if kind == "outputs":
        discrete = rng.random() < 0.5
        outputs = rng.randint(8, 77)
        mode = rng.choice(["exact", "fast", "fast"])
        return dict(call="run", net="c2", outputs=outputs, discrete=discrete, mode=mode,
                    trajectories=_log_uniform(rng, 1000, 300_000 if outputs < 18 else 100_000 if outputs <= 20 else 20_000))
    if kind == "sweep":
        return dict(call="sweep", variants=rng.randint(3, 64), max_trajectories=_log_uniform(rng, 2000, 100_000))
    return dict(call="fit", trajectories=_log_uniform(rng, 1000, 1_000_000))


# ---------------------------------------------------------------- the models


def _texts(case):
    """(.bnd, .cfg) of a case's model."""
    net = case["net"]
    if net in FILES:
        return tuple(open(os.path.join(MODELS, net + ext)).read() for ext in (".bnd", ".cfg"))
    if net == "c1":
        return synth.c1()
    if net == "c2":
        return synth.c2(noninternal=case["outputs"], discrete=case["discrete"])
    if net == "c3":
        return synth.c3(n=case["nodes"], n_out=case["outputs"], max_time=case["max_time"])
    return synth.c4()


def _istate(case, n, seed):
    """Initial probabilities of a synthetic network's nodes: the experiment that the user varies."""
    base = 0.3 if case.get("net") == "c2" else 0.5
    return np.random.default_rng(seed).uniform(base - 0.2, base + 0.2, n).astype(np.float32)


def _theta(names, values, seed):
    """The parameters of a fit: the model's own, each off by some per cent."""
    rng = np.random.default_rng(seed)
    return [float(np.float32(values[k] * np.exp(rng.normal(0.0, 0.1)))) for k in names]


def _weights(seed, windows, bins):
    """The derivative of a loss by the window probabilities."""
    return np.random.default_rng(seed + 1).normal(0.0, 1.0, (windows, bins)).astype(np.float32)


FIXED_ROOM = 4096  # fixed points of one run that its buffers take (the example models have up to 2,300)


def prepare(case, seed):
    """Contexts, models, modules and batches are what a program keeps; so are the arrays that it collects
    lists of varying length in (fixed points, sparse entries), which have a fixed room here."""
    ctx = mb.Context(0)
    if case["call"] == "sweep":
        bases, variants = synth.c5_sweep(case["variants"])
        batch = mb.Batch(ctx)
        nets = [batch.add_model(mb.Model(*texts)) for texts in bases[: min(8, case["variants"])]]
        rng = np.random.default_rng(seed)
        ids = []
        for net, params, trajectories in variants:
            scaled = {k: float(np.float32(v * np.exp(rng.normal(0.0, 0.1)))) for k, v in params.items()}
            count = max(1000, trajectories * case["max_trajectories"] // 100_000)
            ids.append(batch.add_variant(nets[net], count, scaled))
        return dict(case, batch=batch, ids=ids, seed=seed, fixed_counts=np.zeros((len(ids), 64), np.int64))
    if case["call"] == "fit":
        model = mb.Model(*synth.c4())
        names = sorted(model.variables)
        theta = torch.tensor(_theta(names, model.variables, seed), device="cuda", requires_grad=True)
        weights = torch.from_numpy(_weights(seed, 40, 256)).cuda()
        return dict(case, ctx=ctx, model=model, names=names, theta=theta, weights=weights, seed=seed)
    model = mb.Model(*_texts(case))
    if case["net"] not in FILES:
        for i, p in enumerate(_istate(case, model.num_nodes, seed)):
            model.set_istate(i, float(p))
    nodes, outputs, windows = _shape(case)
    room = int(min(1.25 * case["trajectories"] * windows, windows * 2.0**outputs)) if outputs > 17 else 0
    lists = dict(fixed_states=np.zeros((FIXED_ROOM, (nodes + 31) // 32), np.uint32),
                 fixed_counts=np.zeros(FIXED_ROOM, np.int64), windows=np.zeros(room, np.int32),
                 states=np.zeros((room, 2), np.int64), probs=np.zeros(room, np.float64),
                 final_states=np.zeros((case["trajectories"] if outputs > 20 else 0, 2), np.int64),
                 final_counts=np.zeros(case["trajectories"] if outputs > 20 else 0, np.int64))
    return dict(case, module=ctx.compile(model), seed=seed, lists=lists, filled={})


def _collect(state, key, values):
    """`values` in the state's array for them, zeros behind (what an earlier pass left there is cleared)."""
    into, n, before = state["lists"][key], len(values), state["filled"].get(key, 0)
    if n:
        into[:n] = values
    if before > n:
        into[n:before] = 0
    state["filled"][key] = n
    return into


def run(state):
    if state["call"] == "sweep":
        state["batch"].run(state["seed"])
        results = [state["batch"].result(v) for v in state["ids"]]
        state["fixed_counts"][:] = 0
        for row, r in zip(state["fixed_counts"], results):
            counts = [c for _, c in r.fixed]
            row[: len(counts)] = counts
        return dict(probs=np.stack([r.window_probs for r in results]),
                    entropy=np.stack([r.window_entropy for r in results]),
                    final=np.stack([r.final_counts for r in results]).astype(np.int64),
                    fixed_counts=state["fixed_counts"],
                    transitions=np.array([r.transitions for r in results], np.int64))
    if state["call"] == "fit":
        state["theta"].grad = None
        probs = window_probabilities(state["theta"], state["ctx"], state["model"], state["names"],
                                     state["trajectories"], state["seed"])
        (probs * state["weights"]).sum().backward()
        return dict(probs=probs.detach(), grad=state["theta"].grad)
    res = state["module"].run(mode=state["mode"], sample_count=state["trajectories"], seed=state["seed"])
    fixed = res.fixed
    out = dict(transitions=res.transitions, entropy=res.window_entropy,
               fixed_states=_collect(state, "fixed_states", [x for x, _ in fixed]),
               fixed_counts=_collect(state, "fixed_counts", [c for _, c in fixed]))
    if res.windows_sparse:
        s = res.sparse()
        out.update(windows=_collect(state, "windows", s["windows"]),
                   states=_collect(state, "states", s["states"].view(np.int64)),
                   probs=_collect(state, "probs", s["probs"]))
    else:
        out.update(probs=res.window_probs)
    if res.is_sparse:
        out.update(final_states=_collect(state, "final_states", s["final_states"].view(np.int64)),
                   final_counts=_collect(state, "final_counts", s["final_counts"]))
    else:
        out.update(final_counts=res.final_counts)
    return out


# ---------------------------------------------------------------- what a pass cannot do without


def _steps(case):
    """Transitions of one trajectory (means, measured on the networks)."""
    net = case["net"]
    if net in FILES:
        return FILES[net][3]
    if net == "c3":
        return 2.5 * case["nodes"]
    return {"c1": 11, "c2": 100 if case.get("discrete") else 204, "c4": 131}[net]


def _shape(case):
    """nodes, non-internal nodes, windows"""
    net = case["net"]
    if net in FILES:
        return FILES[net][:3]
    if net == "c3":
        return case["nodes"], case["outputs"], int(np.ceil(case["max_time"] / 0.5))
    return {"c1": (10, 10, 25), "c2": (100, case.get("outputs"), 100), "c4": (50, 8, 40)}[net]


def work(case):
    """Operations: per transition the random numbers (about 60), the waiting time, the choice of the node,
    the two or three logic functions that read it and the window sum (about 60 together); per trajectory
    three for each node's initial value. Bytes: the filled cells of the histogram, 8 each, once."""
    if case["call"] == "sweep":
        transitions, nodes, cells = 0.0, 0.0, 0
        bases, variants = synth.c5_sweep(case["variants"])
        for net, _, count in variants:
            count = max(1000, count * case["max_trajectories"] // 100_000)
            transitions += count * (22, 160, 94, 90, 22, 30, 325, 1600)[net]
            nodes += count * bases[net][0].count("node ")
            cells += 40 * 256
        return {"bytes": 8.0 * cells, "flops": 120 * transitions + 3 * nodes}
    if case["call"] == "fit":
        # forward and backward; a transition of the backward pass moves the score of about 3 parameters
        n = case["trajectories"]
        return {"bytes": 8.0 * 40 * 256 * 3, "flops": n * (131 * (2 * 120 + 3 * 6) + 2 * 3 * 50.0)}
    n = case["trajectories"]
    nodes, outputs, windows = _shape(case)
    transitions = float(n) * _steps(case)
    cells = min(windows * 2.0**outputs, transitions)
    return {"bytes": 8.0 * cells, "flops": 120 * transitions + 3.0 * nodes * n}


# ---------------------------------------------------------------- the same trajectories in 64 bits


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _network(bnd, cfg):
    """Node names, logic as Python expressions over bool tensors n[i], rates, outputs and constants."""
    constants = {k: float(v) for k, v in re.findall(r"(?m)^(\$?\w+) = ([^;]+);$", cfg)}
    names, logic, up, down = [], [], [], []
    for name, expr, u, d in re.findall(
            r"node (\w+)\s*\{\s*logic = ([^;]+);\s*rate_up = @logic \? ([^ ]+) : 0;\s*"
            r"rate_down = @logic \? 0 : ([^;]+);", bnd):
        names.append(name)
        logic.append(expr.replace("!", "~"))
        up.append(u)
        down.append(d)
    logic = [compile(re.sub(r"\w+", lambda m: "n[%d]" % names.index(m.group()), e), "logic", "eval") for e in logic]
    internal = set(re.findall(r"(\w+)\.is_internal = 1;", cfg))
    return dict(names=names, logic=logic, up=up, down=down, constants=constants,
                outputs=[i for i, k in enumerate(names) if k not in internal])


def _philox(block, sequence, seed):
    """Philox4x32-10 (Salmon et al., 2011) at counter (block, 0, sequence, 0): four 32-bit words as int64."""
    mask = 0xFFFFFFFF
    c = [block & mask, block >> 32, sequence & mask, sequence >> 32]
    k0, k1 = seed & mask, seed >> 32
    for _ in range(10):
        # 32 x 32 bit products in two halves: an int64 holds no 64-bit unsigned product
        hi, lo = [], []
        for m, x in ((0xD2511F53, c[0]), (0xCD9E8D57, c[2])):
            a, b = m * (x & 0xFFFF), m * (x >> 16)
            s = (a >> 16) + b
            hi.append(s >> 16)
            lo.append((a & 0xFFFF) | ((s & 0xFFFF) << 16))
        c = [hi[1] ^ c[1] ^ k0, lo[1], hi[0] ^ c[3] ^ k1, lo[0]]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _simulate(net, values, istate, n, seed, weights=None):
    """Fast mode's process with every real number in 64 bits: the same random words, integer rates and
    choices, waiting times, window sums and entropies in float64. With `weights`, also the score-function
    estimate of d sum(weights * probabilities) / d parameter for the parameters in `values`."""
    dev = _device()
    const = net["constants"]
    max_time, tick = float(np.float32(const["max_time"])), float(np.float32(const["time_tick"]))
    discrete = const["discrete_time"] != 0
    windows = int(np.ceil(np.float32(max_time) / np.float32(tick)))
    N, k = len(net["names"]), len(net["outputs"])
    named = {**const, **values}
    rate = np.array([[float(np.float32(named[t] if t.startswith("$") else float(t))) for t in net[d]]
                     for d in ("up", "down")])  # [2, N]
    worst = max(rate.max(0)[i:i + 32].sum() for i in range(0, N, 32))
    shift = next(s for s in range(31, -1, -1) if worst * 2.0**s < 2.0**32)
    q = torch.tensor(np.rint(rate * 2.0**shift), dtype=torch.int64, device=dev)
    rate_t = torch.tensor(rate, device=dev)
    params = sorted(values)
    if weights is not None:
        weights = torch.as_tensor(weights, dtype=torch.float64, device=dev)
        grad = torch.zeros(len(params), dtype=torch.float64, device=dev)
        # d rate[direction, node] / d parameter is 0 or 1 here
        owner = torch.tensor([[params.index(t) if t in values else -1 for t in net[d]] for d in ("up", "down")],
                             device=dev)
    sequence = torch.arange(n, dtype=torch.int64, device=dev)
    node = []
    for i in range(N):
        if i % 4 == 0:
            words = _philox(torch.full_like(sequence, i // 4), sequence, seed)
        u = words[i % 4].to(torch.float32) * 2.0**-32 + 2.0**-33
        node.append(u <= float(istate[i]))
    state = torch.stack(node)  # [N, n]
    time = torch.zeros(n, dtype=torch.float64, device=dev)
    probs = torch.zeros(windows << k, dtype=torch.float64, device=dev)
    entropy = torch.zeros(windows, dtype=torch.float64, device=dev)
    if weights is not None:
        score = torch.zeros(n, len(params), dtype=torch.float64, device=dev)
    block = (N + 3) // 4
    while sequence.numel():
        words = _philox(torch.full_like(sequence, block), sequence, seed)
        block += 1
        logic = torch.stack([eval(e, {"n": state}) for e in net["logic"]])
        unstable = state != logic
        active = torch.where(unstable, torch.where(state, q[1][:, None], q[0][:, None]), 0)
        sums = active.cumsum(0)
        total = sums[-1]
        a0 = total.to(torch.float64) * 2.0**-shift
        if discrete:
            then = time + tick
            then = torch.where(then > max_time - tick, max_time, then)
        else:
            then = time - torch.log(((words[0] >> 8) + 1).to(torch.float64) * 2.0**-24) / a0
        then = torch.where(total == 0, max_time, then).clamp(max=max_time)
        r = torch.where(unstable, torch.where(state, rate_t[1][:, None], rate_t[0][:, None]), 0.0)[net["outputs"]]
        s = r.sum(0)
        h = torch.where(s > 0, torch.log2(s) - torch.special.xlogy(r, r).sum(0) / (np.log(2.0) * s), 0.0).clamp(min=0)
        index = sum(state[i].to(torch.int64) << j for j, i in enumerate(net["outputs"]))
        if weights is not None:
            drift = torch.zeros_like(score)
            for d in range(2):
                for i in range(N):
                    if int(owner[d, i]) >= 0:
                        drift[:, int(owner[d, i])] += (unstable[i] & (state[i] == bool(d))).to(torch.float64)
        if discrete:
            w = torch.round(time / tick).to(torch.int64)
            ok = w < windows
            probs.index_add_(0, ((w << k) + index)[ok], torch.ones_like(time)[ok])
            entropy.index_add_(0, w[ok], h[ok])
        else:
            at = torch.arange(len(time), device=dev)
            begin = time
            while at.numel():
                w = torch.floor(begin / tick).to(torch.int64)
                # (a begin that is itself the end of a window may fall on either side of it in floor)
                w = torch.where((w + 1).to(torch.float64) * tick <= begin, w + 1, w)
                end = torch.minimum(then[at], (w + 1).to(torch.float64) * tick)
                length = torch.where(w < windows, end - begin, 0.0)
                w = w.clamp(max=windows - 1)
                cell = (w << k) + index[at]
                probs.index_add_(0, cell, length)
                entropy.index_add_(0, w, h[at] * length)
                if weights is not None:
                    c = weights.reshape(-1)[cell] * length
                    grad += c @ score[at] - (c * (0.5 * (begin + end) - time[at])) @ drift[at]
                more = then[at] > end
                at, begin = at[more], end[more]
        keep = (then < max_time) & (total > 0)
        if weights is not None:
            score = (score - drift * (then - time)[:, None])[keep]
        state, time, sequence = state[:, keep], then[keep], sequence[keep]
        words = [w[keep] for w in words]
        sums, total = sums[:, keep], total[keep]
        # r = the top 64 bits of (64 random bits) * total, with total below 2^48 in 16-bit parts
        acc = torch.zeros_like(total)
        for part in (words[2] & 0xFFFF, words[2] >> 16, words[1] & 0xFFFF, words[1] >> 16):
            acc = (acc >> 16) + part * total
        r = acc >> 16
        flip = (sums <= r).sum(0)
        lane = torch.arange(flip.numel(), device=dev)
        was = state[flip, lane]
        if weights is not None:
            for d in range(2):
                own = torch.where(was == bool(d), owner[d][flip], -1)
                hit = own >= 0
                score[lane[hit], own[hit]] += 1.0 / rate_t[d][flip[hit]]
        state[flip, lane] = ~was
    scale = 1.0 / (n if discrete else n * tick)
    out = dict(probs=(probs * scale).reshape(windows, 1 << k), entropy=entropy * scale)
    if weights is not None:
        out["grad"] = grad * scale
    return out


def exact(case, seed):
    """Fast mode on the networks whose trajectories 64-bit tensors follow in some seconds. Exact and epoch
    mode draw from another generator and choose each node by sums in 32 bits, which is part of their
    definition; a sweep's and the large networks' trajectories take minutes."""
    if case["call"] == "fit":
        net = _network(*synth.c4())
        names = sorted(k for k in net["constants"] if k.startswith("$"))
        values = dict(zip(names, _theta(names, {k: float(np.float32(v)) for k, v in net["constants"].items()}, seed)))
        istate = np.full(len(net["names"]), 0.5, np.float32)
        out = _simulate(net, values, istate, case["trajectories"], seed, _weights(seed, 40, 256))
        return dict(probs=out["probs"], grad=out["grad"])
    if case["call"] != "run" or case["mode"] != "fast" or case["net"] in FILES:
        return None
    nodes, outputs, _ = _shape(case)
    if outputs > 10 or case["trajectories"] * _steps(case) * nodes > 1.0e10 or _steps(case) * nodes > 30_000:
        return None
    net = _network(*_texts(case))
    out = _simulate(net, {}, _istate(case, nodes, seed), case["trajectories"], seed)
    return dict(transitions=None, entropy=out["entropy"], fixed_states=None, fixed_counts=None, probs=out["probs"],
                final_counts=None)
