"""The calls that users of this framework make, as measurable cases.

Each case is one pass through the public entry points on a seeded graph:

* ``solve``      a single graph solved on an engine that the program keeps
                 (tolerance run, fixed sweeps with or without damping, FP32
                 or FP64, with evidence clamped before the engine is built);
* ``build``      host graph arrays to host beliefs: engine creation, a fixed
                 run, the beliefs, the engine released;
* ``labelling``  the alarm-ranking loop: an engine, then one label clamped
                 and a low-pass re-solve after each;
* ``batch``      many uneven graphs solved together, each to its tolerance;
* ``sets``       many evidence sets on one graph, each to its tolerance;
* ``gradient``   beliefs after unrolled sweeps and the gradient of a
                 cross-entropy with respect to every factor's probability;
* ``schedule``   a sequential (SEQFIX) schedule.

Sizes are those of this repository's workloads (fastlbp_b200.workloads) and
tests, between its smallest graph (2,000 tuples) and its largest (1 M).
"""

import math

import numpy as np
import torch

from fastlbp_b200 import BatchEngine, CausalFactorGraph, Engine, SetsEngine, api, autograd, workloads

# Edge slots, factors and variables per tuple of the three families of graphs:
# "bingo" (uniform small fan-ins), "zipf" (the large single graph's laws),
# "faultloc" (fan-in up to 4,096).
PER_TUPLE = {"bingo": (8.4, 2.4), "zipf": (6.3, 2.3), "faultloc": (9.8, 2.3)}


def listed():
    return [
        # a small derivation graph with labelled alarms: the shortest call, all latency
        dict(name="small-tol", kind="solve", family="bingo", tuples=2000, labels=10, precision=32, damping=0.0,
             tol=1e-6, sweeps=1000),
        # one mid-size graph re-solved to its tolerance on a kept engine (the interactive loop's graph)
        dict(name="medium-tol", kind="solve", family="bingo", tuples=50_000, labels=30, precision=32, damping=0.0,
             tol=1e-6, sweeps=500),
        # the large single graph: 1 M tuples, 200 damped sweeps
        dict(name="large-damped", kind="solve", family="zipf", tuples=1_000_000, labels=0, precision=32, damping=0.1,
             tol=0.0, sweeps=200),
        # double precision messages, an odd size
        dict(name="double-fixed", kind="solve", family="zipf", tuples=150_001, labels=0, precision=64, damping=0.0,
             tol=0.0, sweeps=100),
        # fault localisation: factors of up to 4,096 inputs, 2 % of the tuples clamped to test outcomes
        dict(name="faultloc-tol", kind="solve", family="faultloc", tuples=100_000, labels=-1, precision=32,
             damping=0.0, tol=1e-6, sweeps=500),
        # one-shot use: host arrays to host beliefs with a new engine
        dict(name="build-and-solve", kind="build", family="zipf", tuples=300_000, precision=32, damping=0.1,
             sweeps=50),
        # the alarm-ranking loop on a new engine: a label, then a low-pass run
        dict(name="labelling-loop", kind="labelling", family="bingo", tuples=20_000, labels=8, precision=32,
             tol=1e-6, min_iters=20, max_iters=200, hist=20),
        # batched serving of uneven graphs with their own evidence
        dict(name="batch-serving", kind="batch", family="bingo", graphs=48, lo=1000, hi=50_000, precision=32,
             damping=0.0, tol=1e-6, sweeps=500),
        # a few tiny graphs at once: batched, but latency-bound
        dict(name="batch-tiny", kind="batch", family="bingo", graphs=8, lo=500, hi=4000, precision=32, damping=0.0,
             tol=1e-6, sweeps=500),
        # many evidence sets on one graph
        dict(name="evidence-sets", kind="sets", family="bingo", tuples=20_000, sets=48, precision=32, damping=0.0,
             tol=1e-6, sweeps=500),
        # one learning step: beliefs and gradient through 100 unrolled sweeps, checkpoint every 10
        dict(name="gradient", kind="gradient", family="bingo", tuples=50_000, graphs=2, labels=200, precision=32,
             sweeps=100, every=10),
        # the reference's default sequential schedule on a small graph
        dict(name="seqfix", kind="schedule", family="bingo", tuples=4000, precision=32, damping=0.0, sweeps=10),
    ]


def _spread(rng, lo, hi):
    """An integer log-uniform in [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "build", "labelling", "batch", "sets", "gradient", "schedule"])
    precision = 64 if rng.random() < 0.2 else 32
    damping = rng.choice([0.0, 0.0, 0.1, 0.3])
    if kind == "solve":
        family = rng.choice(["bingo", "zipf", "faultloc"])
        tuples = _spread(rng, 1500, 100_000 if precision == 64 or family == "faultloc" else 500_000)
        if rng.random() < 0.6 or family == "faultloc":
            return dict(kind=kind, family=family, tuples=tuples, labels=-1 if family == "faultloc" else rng.randint(0, 40),
                        precision=precision, damping=0.0 if family == "faultloc" else damping, tol=1e-6, sweeps=500)
        return dict(kind=kind, family=family, tuples=tuples, labels=rng.randint(0, 40), precision=precision,
                    damping=damping, tol=0.0, sweeps=rng.randint(20, 200))
    if kind == "build":
        return dict(kind=kind, family=rng.choice(["bingo", "zipf"]), tuples=_spread(rng, 2000, 300_000),
                    precision=precision, damping=damping, sweeps=rng.randint(20, 100))
    if kind == "labelling":
        return dict(kind=kind, family=rng.choice(["bingo", "zipf"]), tuples=_spread(rng, 1500, 50_000),
                    labels=rng.randint(2, 10), precision=precision, tol=1e-6, min_iters=rng.randint(5, 30),
                    max_iters=200, hist=rng.randint(5, 40))
    if kind == "batch":
        return dict(kind=kind, family=rng.choice(["bingo", "zipf"]), graphs=_spread(rng, 2, 64), lo=500,
                    hi=_spread(rng, 1000, 30_000), precision=precision, damping=damping, tol=1e-6, sweeps=500)
    if kind == "sets":
        return dict(kind=kind, family=rng.choice(["bingo", "zipf"]), tuples=_spread(rng, 1500, 30_000),
                    sets=_spread(rng, 2, 64), precision=precision, damping=damping, tol=1e-6, sweeps=500)
    if kind == "gradient":
        return dict(kind=kind, family="bingo", tuples=_spread(rng, 1000, 50_000), graphs=rng.randint(1, 3),
                    labels=rng.randint(20, 200), precision=precision, sweeps=rng.randint(20, 100),
                    every=rng.randint(4, 12))
    return dict(kind=kind, family="bingo", tuples=_spread(rng, 1000, 10_000), precision=precision, damping=damping,
                sweeps=rng.randint(3, 10))


# ------------------------------------------------------------------ inputs


# rule probabilities of the families
P_RANGE = {"bingo": (0.85, 0.99), "zipf": (0.8, 0.999), "faultloc": (0.5, 0.99)}


def _factors(family, tuples, seed, alarms=50, graph=0):
    """(factor list, clamps) of one graph; clamps only for fault localisation.
    The structure belongs to the case (graph `graph` of it), so that results
    have one shape; the rule probabilities and the evidence come from the seed."""
    shape = 1 + 7 * tuples + 1009 * graph
    clamps = {}
    if family == "zipf":
        fl = workloads.config1(shape, scale=tuples / 1_000_000)
    elif family == "faultloc":
        fl, clamps = workloads.config2(shape, scale=tuples / 200_000)
    else:
        fl = workloads.bingo_graph(tuples, int(1.5 * tuples), max(10, tuples // 20), workloads.uniform_int(2, 4),
                                   workloads.uniform_int(1, 6), shape, n_alarms=alarms)
    rng = np.random.default_rng([seed, shape])
    rules = fl.kind == workloads.AND
    fl.p[rules] = rng.uniform(*P_RANGE[family], int(rules.sum()))
    return fl, {lab: int(rng.random() < 0.1) for lab in clamps}


def _labels(fl, n, seed):
    rng = np.random.default_rng([seed, 77])
    al = rng.permutation(fl.alarms)[:n]
    return dict(zip((int(a) for a in al), (int(x) for x in rng.integers(0, 2, al.size))))


def _inputs(case, seed):
    """The factor lists and clamps of a case, from the seed alone."""
    kind, family = case["kind"], case["family"]
    if kind == "batch":
        rng = np.random.default_rng([case["graphs"], case["lo"], case["hi"]])
        out = []
        for k in range(case["graphs"]):
            nt = int(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))
            fl, _ = _factors(family, nt, seed, graph=k)
            out.append((fl, _labels(fl, int(rng.integers(1, 51)), seed + k)))
        return out
    if kind == "gradient":
        return [(_factors(family, case["tuples"], seed, alarms=case["labels"], graph=k)[0], {})
                for k in range(case["graphs"])]
    fl, clamps = _factors(family, case["tuples"], seed)
    if kind == "solve" and case["labels"] > 0:
        clamps = _labels(fl, case["labels"], seed)
    return [(fl, clamps)]


def _arrays(fl, clamps):
    g = CausalFactorGraph.from_factors(fl)
    if clamps:
        g.clamp_labels(clamps)
        g = g.rebuild()
    return g.graph_arrays()


def _var_index(fl, labels):
    """Graph variable indices (ascending label order) of labels."""
    every = np.unique(np.concatenate([fl.head, fl.body]))
    return np.searchsorted(every, np.asarray(labels, np.int64))


def _sets(fl, n, seed):
    """Evidence sets as the labelling loop meets them: each adds a label to the one before."""
    rng = np.random.default_rng([seed, 9])
    al = _var_index(fl, fl.alarms)
    vals = rng.integers(0, 2, al.size)
    start = rng.integers(0, al.size)
    return [{int(al[(start + j) % al.size]): int(vals[(start + j) % al.size]) for j in range(1 + k % al.size)}
            for k in range(n)]


def _targets(lists, seed):
    """(variable indices over the graphs in order, 0/1 labels) of a learning step."""
    rng = np.random.default_rng([seed, 11])
    idx, off = [], 0
    for fl, _ in lists:
        idx.append(off + _var_index(fl, fl.alarms))
        off += np.unique(np.concatenate([fl.head, fl.body])).size
    idx = np.concatenate(idx)
    return idx, (rng.random(idx.size) < 0.3).astype(np.float64)


def prepare(case, seed):
    kind = case["kind"]
    lists = _inputs(case, seed)
    st = dict(case=case, kind=kind)
    if kind == "solve":
        fl, clamps = lists[0]
        st["engine"] = Engine(_arrays(fl, clamps), precision=case["precision"], damping=case["damping"])
    elif kind == "build":
        st["arrays"] = _arrays(*lists[0])
    elif kind == "labelling":
        fl = lists[0][0]
        st["arrays"] = _arrays(fl, {})
        lab = _labels(fl, case["labels"], seed)
        st["vars"], st["values"] = _var_index(fl, list(lab)), list(lab.values())
    elif kind == "batch":
        st["engine"] = BatchEngine([_arrays(fl, cl) for fl, cl in lists], precision=case["precision"],
                                   damping=case["damping"])
    elif kind == "sets":
        fl = lists[0][0]
        st["engine"] = SetsEngine(_arrays(fl, {}), _sets(fl, case["sets"], seed), precision=case["precision"],
                                  damping=case["damping"])
    elif kind == "gradient":
        graphs = [_arrays(fl, {}) for fl, _ in lists]
        st["engine"] = (Engine(graphs[0], precision=case["precision"]) if len(graphs) == 1 else
                        BatchEngine(graphs, precision=case["precision"]))
        dev = torch.device("cuda")
        st["p"] = torch.tensor(np.concatenate([a["factor_p"] for a in graphs]), device=dev, requires_grad=True)
        st["q"] = torch.tensor(np.concatenate([a["factor_q"] for a in graphs]), device=dev)
        idx, y = _targets(lists, seed)
        st["idx"], st["y"] = torch.tensor(idx, device=dev), torch.tensor(y, device=dev)
    else:
        fl = lists[0][0]
        arrays = _arrays(fl, {})
        st["engine"] = Engine(arrays, precision=case["precision"], damping=case["damping"])
        st["engine"].set_update_seq(api.update_seq(arrays, "SEQFIX", factor_order=_order(fl, seed)))
    return st


def _order(fl, seed):
    return np.random.default_rng([seed, 13]).permutation(fl.n).astype(np.int32)


# -------------------------------------------------------------------- a pass


def run(st):
    case, kind = st["case"], st["kind"]
    if kind == "solve":
        e = st["engine"]
        e.reset_counts()
        e.init()
        if case["tol"] > 0:
            info = e.run_tol(case["tol"], case["sweeps"], 1e9)
            return [e.beliefs(), info["sweeps"]]
        e.run_fixed(case["sweeps"])
        return [e.beliefs()]
    if kind == "build":
        e = Engine(st["arrays"], precision=case["precision"], damping=case["damping"])
        e.init()
        e.run_fixed(case["sweeps"])
        b = e.beliefs()
        e.close()
        return [b]
    if kind == "labelling":
        e = Engine(st["arrays"], precision=case["precision"])
        out, sweeps = [], []
        for v, x in zip(st["vars"], st["values"]):
            e.clamp(v, x)
            e.init()
            info = e.run_lowpass(case["tol"], case["min_iters"], case["max_iters"], case["hist"])
            out.append(e.lowpass())
            sweeps.append(info["sweeps"])
        e.close()
        return out + sweeps
    if kind == "batch":
        e = st["engine"]
        e.init()
        e.reset_counts()
        sweeps, reasons = e.run_batch_tol(case["tol"], case["sweeps"])
        return [e.beliefs(), sweeps, reasons]
    if kind == "sets":
        e = st["engine"]
        e.init()
        sweeps, reasons = e.run_sets_tol(case["tol"], case["sweeps"])
        return [e.beliefs(), sweeps, reasons]
    if kind == "gradient":
        b = autograd.unrolled_beliefs(st["p"], st["engine"], st["q"], case["sweeps"], case["every"])
        loss = torch.nn.functional.binary_cross_entropy(b[st["idx"]], st["y"], reduction="sum")
        (g,) = torch.autograd.grad(loss, st["p"])
        return [b.detach(), g]
    e = st["engine"]
    e.init()
    e.run_fixed(case["sweeps"])
    return [e.beliefs()]


def work(case):
    """Per sweep every message is read and written once in each direction with
    its 4-byte position (24 bytes a slot), every factor's and variable's
    constants once (16 and 12 bytes); a tolerance run takes about 35 sweeps."""
    e, v = PER_TUPLE[case["family"]]
    if case["kind"] == "batch":
        tuples = case["graphs"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    else:
        tuples = case["tuples"] * case.get("sets", 1) * case.get("graphs", 1)
    if case["kind"] == "labelling":
        sweeps = 35 * case["labels"]
    elif case.get("tol", 0) > 0:
        sweeps = 35 if case["family"] != "faultloc" else 250
    else:
        sweeps = case["sweeps"]
    size = 2 if case["precision"] == 64 else 1
    per = tuples * (size * 16 * e + 8 * e + 28 * v)
    passes = 3 if case["kind"] == "gradient" else 1
    return {"bytes": passes * sweeps * per, "flops": passes * sweeps * tuples * 30 * e}


# --------------------------------------------------------- 64-bit references


class _Exact:
    """Synchronous loopy belief propagation of one factor list in float64
    log-odds, plain torch (on the GPU where there is one)."""

    def __init__(self, fl, clamps=None):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        n = fl.n
        size = np.diff(fl.body_off)
        fac = np.repeat(np.arange(n), size)
        labels = np.unique(np.concatenate([fl.head, fl.body]))
        key = np.unique(fac * np.int64(labels[-1] + 1) + fl.body)  # a body names a variable once
        fac, body = key // (labels[-1] + 1), key % (labels[-1] + 1)
        self.V, self.F = labels.size, n
        put = lambda a, t=torch.int64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device=dev)  # noqa: E731
        self.bf, self.bv = put(fac), put(np.searchsorted(labels, body))
        self.hv = put(np.searchsorted(labels, fl.head))
        self.p, self.q = put(fl.p, torch.float64), put(fl.q, torch.float64)
        self.single = put(fl.kind == 0, torch.bool)
        self.sgn = put(np.where(fl.kind == 2, -1.0, 1.0), torch.float64)
        self.ev = torch.zeros(self.V, dtype=torch.float64, device=dev)  # +-inf where clamped
        for lab, x in (clamps or {}).items():
            at = int(np.searchsorted(labels, lab))
            if at < labels.size and labels[at] == lab:  # a label that is in no factor is passed over
                self.clamp(at, x)
        self.var = torch.cat([self.hv, self.bv])
        self.zeros = lambda k: torch.zeros(k, dtype=torch.float64, device=dev)  # noqa: E731

    def clamp(self, v, x):
        self.ev[v] = math.inf if x else -math.inf

    def factor(self, vf, p=None, smooth=False):
        """f->v messages, heads then bodies. smooth: without exact zeros, differentiable in p."""
        p, q, sgn = self.p if p is None else p, self.q, self.sgn
        y = sgn[self.bf] * vf[self.F:]
        ls = torch.nn.functional.logsigmoid(y)
        if smooth:
            lo_all = self.zeros(self.F).index_add(0, self.bf, ls)
            lo = lo_all[self.bf] - ls
            P, R = torch.exp(lo_all), -torch.expm1(lo_all)
            head = torch.log(p * P + q * R) - torch.log((1 - p) * P + (1 - q) * R)
            sh, th = torch.sigmoid(sgn * vf[:self.F]), torch.sigmoid(-sgn * vf[:self.F])
            P, R, pb, qb, shb, thb = torch.exp(lo), -torch.expm1(lo), p[self.bf], q[self.bf], sh[self.bf], th[self.bf]
            a, b = pb * P + qb * R, (1 - pb) * P + (1 - qb) * R
            body = torch.log(shb * a + thb * b) - torch.log(shb * qb + thb * (1 - qb))
            prior = torch.logit(torch.where(self.single, p, 0.5))
            return torch.cat([torch.where(self.single, prior, sgn * head), sgn[self.bf] * body])
        zero = ls == -math.inf
        fin = torch.where(zero, 0.0, ls)
        lo_all = self.zeros(self.F).index_add_(0, self.bf, fin)
        nz = self.zeros(self.F).index_add_(0, self.bf, zero.double())
        lo = torch.where((nz[self.bf] - zero.double()) > 0, -math.inf, lo_all[self.bf] - fin)
        lo_all = torch.where(nz > 0, -math.inf, lo_all)
        lp, lq, l1p, l1q = torch.log(p), torch.log(q), torch.log1p(-p), torch.log1p(-q)

        def weights(lo, f):
            lR = torch.log(-torch.expm1(lo))
            return torch.logaddexp(lp[f] + lo, lq[f] + lR), torch.logaddexp(l1p[f] + lo, l1q[f] + lR)

        a, b = weights(lo_all, slice(None))
        head = torch.where(self.single, lp - l1p, sgn * (a - b))
        lh = sgn * vf[:self.F]
        lh = torch.where(torch.isinf(self.ev[self.hv]), sgn * self.ev[self.hv], lh)
        s1, s0 = torch.nn.functional.logsigmoid(lh), torch.nn.functional.logsigmoid(-lh)
        den = torch.logaddexp(s1 + lq, s0 + l1q)
        a, b = weights(lo, self.bf)
        body = torch.logaddexp(s1[self.bf] + a, s0[self.bf] + b) - den[self.bf]
        # certain against the head's certain state: an exact zero, or no value
        sure = torch.where((p - q) * torch.sign(lh) > 0, math.inf, math.nan)
        body = torch.where(den[self.bf] == -math.inf, sure[self.bf], body)
        return torch.cat([head, sgn[self.bf] * body])

    def variable(self, fv):
        """(v->f messages, beliefs)."""
        fin = torch.where(torch.isinf(fv), 0.0, fv)
        pos, neg = (fv == math.inf).double(), (fv == -math.inf).double()
        S = self.zeros(self.V).index_add_(0, self.var, fin)
        npos = self.zeros(self.V).index_add_(0, self.var, pos)
        nneg = self.zeros(self.V).index_add_(0, self.var, neg)
        ev = self.ev[self.var]
        a, b = npos[self.var] - pos > 0, nneg[self.var] - neg > 0
        inf = torch.full_like(fv, math.inf)
        vf = torch.where(a & b, 0.0, torch.where(a, inf, torch.where(b, -inf, S[self.var] - fin)))
        vf = torch.where(torch.isinf(ev), ev, vf)
        bel = torch.sigmoid(S)
        bel = torch.where((npos > 0) & (nneg > 0), math.nan,
                          torch.where(npos > 0, 1.0, torch.where(nneg > 0, 0.0, bel)))
        return vf, torch.where(torch.isinf(self.ev), (self.ev > 0).double(), bel)

    def sweeps(self, damping=0.0):
        """Beliefs after each sweep from uniform messages."""
        n = self.var.numel()
        vf, old = self.zeros(n), self.zeros(n)
        vf = torch.where(torch.isinf(self.ev[self.var]), self.ev[self.var], vf)
        while True:
            fv = self.factor(vf)
            if damping:
                mix = (1 - damping) * fv + damping * old
                fv = torch.where(torch.isinf(fv), fv, torch.where(torch.isinf(old), old, mix))
                old = fv
            vf, b = self.variable(fv)
            yield b

    def fixed(self, n, damping):
        for k, b in enumerate(self.sweeps(damping)):
            if k + 1 == n:
                return b.cpu().numpy()

    def tol(self, tol, most, damping):
        last = self.zeros(self.V)
        for k, b in enumerate(self.sweeps(damping)):
            d = torch.nan_to_num((b - last).abs(), nan=0.0).max()
            last = b
            if float(d) <= tol or k + 1 >= most:
                return b.cpu().numpy()

    def lowpass(self, tol, lo, hi, hist):
        last, ring = self.zeros(self.V), []
        for k, b in enumerate(self.sweeps()):
            n = k + 1
            d = (b - last).abs()
            last = b
            ring = (ring + [b])[-hist:]
            if float(d.max()) <= tol:
                return b.cpu().numpy()
            frac = float((d > tol).double().mean())
            if n > hi or (n > lo and frac < (n - lo) / (hi - lo)):
                return torch.stack(ring).mean(0).cpu().numpy()

    def gradient(self, n, idx, y):
        p = self.p.clone().requires_grad_(True)
        vf = self.zeros(self.var.numel())
        for _ in range(n):
            fv = self.factor(vf, p, smooth=True)
            S = self.zeros(self.V).index_add(0, self.var, fv)
            vf = S[self.var] - fv
        b = torch.sigmoid(S)
        yt = torch.as_tensor(y, device=b.device)
        (g,) = torch.autograd.grad(torch.nn.functional.binary_cross_entropy(b[idx], yt, reduction="sum"), p)
        return b.detach(), g


def _sequential(fl, order, sweeps, damping):
    """Beliefs after `sweeps` sequential sweeps: the edges of each factor in
    `order`, variables in ascending label order, each update seen by the next."""
    labels = np.unique(np.concatenate([fl.head, fl.body]))
    at = {int(v): i for i, v in enumerate(labels)}
    rows = []
    for f in order:
        f = int(f)
        head = int(fl.head[f])
        vs = sorted({int(x) for x in fl.body[fl.body_off[f]:fl.body_off[f + 1]]} | {head})
        rows.append(([at[v] for v in vs], vs.index(head), int(fl.kind[f]), float(fl.p[f]), float(fl.q[f])))
    msg = [[0.0] * len(r[0]) for r in rows]
    S = [0.0] * labels.size
    sig = lambda x: 1 / (1 + math.exp(-x)) if x >= 0 else math.exp(x) / (1 + math.exp(x))  # noqa: E731
    for _ in range(sweeps):
        for (vs, h, kind, p, q), m in zip(rows, msg):
            s = -1.0 if kind == 2 else 1.0
            for k, v in enumerate(vs):
                if kind == 0:
                    new = math.log(p) - math.log1p(-p)
                else:
                    P, R = 1.0, 0.0  # product of the other body variables' weights, and its complement
                    for j, u in enumerate(vs):
                        if j != k and j != h:
                            y = s * (S[u] - m[j])
                            R += P * sig(-y)
                            P *= sig(y)
                    a, b = p * P + q * R, (1 - p) * P + (1 - q) * R
                    if k == h:
                        new = s * (math.log(a) - math.log(b))
                    else:
                        y = s * (S[vs[h]] - m[h])
                        t1, t0 = sig(y), sig(-y)
                        new = s * (math.log(t1 * a + t0 * b) - math.log(t1 * q + t0 * (1 - q)))
                if damping:
                    new = (1 - damping) * new + damping * m[k]
                S[v] += new - m[k]
                m[k] = new
    return np.array([sig(x) for x in S])


def exact(case, seed):
    kind = case["kind"]
    lists = _inputs(case, seed)
    if kind == "schedule":
        fl = lists[0][0]
        if (fl.n + fl.body.size) * case["sweeps"] > 1_000_000:
            return None
        return [_sequential(fl, _order(fl, seed), case["sweeps"], case["damping"])]
    if kind == "solve" and case["tol"] > 0:
        fl, clamps = lists[0]
        return [_Exact(fl, clamps).tol(case["tol"], case["sweeps"], case["damping"]), None]
    if kind in ("solve", "build"):
        fl, clamps = lists[0]
        return [_Exact(fl, clamps).fixed(case["sweeps"], case["damping"])]
    if kind == "labelling":
        fl = lists[0][0]
        bp, out = _Exact(fl), []
        lab = _labels(fl, case["labels"], seed)
        for v, x in zip(_var_index(fl, list(lab)), lab.values()):
            bp.clamp(int(v), x)
            out.append(bp.lowpass(case["tol"], case["min_iters"], case["max_iters"], case["hist"]))
        return out + [None] * len(out)
    if kind == "batch":
        return [np.concatenate([_Exact(fl, cl).tol(case["tol"], case["sweeps"], case["damping"])
                                for fl, cl in lists]), None, None]
    if kind == "sets":
        fl = lists[0][0]
        rows = []
        for cl in _sets(fl, case["sets"], seed):
            bp = _Exact(fl)
            for v, x in cl.items():
                bp.clamp(v, x)
            rows.append(bp.tol(case["tol"], case["sweeps"], case["damping"]))
        return [np.stack(rows), None, None]
    idx, y = _targets(lists, seed)  # gradient
    b, g, off, at = [], [], 0, 0
    for fl, _ in lists:
        bp = _Exact(fl)
        n = fl.alarms.size
        bk, gk = bp.gradient(case["sweeps"], torch.as_tensor(idx[at:at + n] - off, device=bp.p.device), y[at:at + n])
        b.append(bk)
        g.append(gk)
        at, off = at + n, off + bp.V
    return [torch.cat(b), torch.cat(g)]
