"""Timed cases: the simplification work that programs have this library do.

A pass is one whole request as a caller makes it: the formula goes in (from host
arrays, or from arrays already on the GPU), one sigmify round runs, the simplified
formula comes back into host buffers that the caller keeps, and the assigned literals
are set in the caller's assignment (host or GPU, where the formula came from). The
extension cases are the step after it: models of a batch's simplified formulas are
extended to the original ones.

The families are the repository's own workloads (random k-SAT, Tseitin-encoded AIGs,
unrolled AIGs of a model checker, community-structured CNFs, batches of mixed k-SAT),
each over the range of sizes that its tests, its benchmark and its server use. Large
formulas are drawn on the GPU so that making them stays quick. Every formula is
satisfiable by construction (a planted assignment, or a circuit without a property), as
most formulas that reach preprocessing are; a refuted formula has no simplified form to
compare.

All results are whole numbers: they are compared for equality.
"""
import math

import numpy as np
import torch

from parafrost_gb300 import cnfgen
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import ResultBuffers, Simplifier

DEV = "cuda"

OPTIONS = {
    "all": dict(all=1),                    # every elimination stage, the benchmark's setting
    "default": dict(),                     # the solver's default stages (no BCE)
    "lbound": dict(all=1, ve_lbound=1),    # elimination bounded by literals as well
}


# ---------------------------------------------------------------- cases
def listed():
    return [
        # a tiny instance, the smallest that the tests simplify: launch and host latency
        dict(name="ksat-tiny", family="ksat", vars=200, clauses=840, opts="all", resident=False),
        # the repository's 10k-variable random 3-SAT instance
        dict(name="ksat-10k", family="ksat", vars=10_000, clauses=42_600, opts="all", resident=False),
        # clauses of 2 to 5 literals at an odd size, elimination bounded by literals
        dict(name="mixed-odd", family="mixed", vars=266_689, clauses=1_000_083, opts="lbound", resident=False),
        # a model checker's request: 16k gates unrolled over 23 frames, reset units among the clauses
        dict(name="unrolled-1m", family="unrolled", gates=16_001, steps=23, opts="all", resident=False),
        # a large combinational circuit (2M AND, 200k XOR gates), already on the GPU
        dict(name="aig-2m", family="aig", inputs=50_000, ands=2_000_000, xors=200_000, opts="all", resident=True),
        # a middle-sized circuit with the solver's default stages, from host arrays
        dict(name="aig-100k-default", family="aig", inputs=5_003, ands=90_007, xors=9_001, opts="default",
             resident=False),
        # inprocessing: a structured formula whose last clauses were learnt by the search
        dict(name="inprocess-learnt", family="community", vars=30_011, clauses=120_007, communities=15,
             learnt=12_001, opts="all", resident=False),
        # structured industrial-like formulas, a tenth of the benchmark's size and the full size
        dict(name="community-2m", family="community", vars=2_000_000, clauses=8_000_000, communities=20, learnt=0,
             opts="all", resident=True),
        dict(name="community-20m", family="community", vars=20_000_000, clauses=80_000_000, communities=200,
             learnt=0, opts="all", resident=True),
        # many formulas of 1k to 200k clauses in one round, each from its own host arrays
        dict(name="batch-384", family="batch", formulas=384, cmin=1_000, cmax=200_000, opts="all"),
        # the answers of such a batch: every formula's model extended to its original variables
        dict(name="extend-384", family="extend", formulas=384, cmin=1_000, cmax=200_000, opts="all"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["ksat", "mixed", "unrolled", "aig", "community", "inprocess", "batch", "extend"])
    opts = rng.choice(["all", "all", "default", "lbound"])
    resident = rng.random() < 0.5
    if family == "ksat":
        n = _logint(rng, 200, 1_000_000)
        return dict(family="ksat", vars=n, clauses=int(n * rng.uniform(2.0, 4.26)), opts=opts, resident=resident)
    if family == "mixed":
        c = _logint(rng, 1_000, 5_000_000)
        return dict(family="mixed", vars=max(8, int(c / rng.uniform(3.0, 4.5))), clauses=c, opts=opts,
                    resident=resident)
    if family == "unrolled":
        return dict(family="unrolled", gates=_logint(rng, 1_000, 30_000), steps=_logint(rng, 5, 40), opts=opts,
                    resident=resident)
    if family == "aig":
        g = _logint(rng, 1_000, 2_200_000)
        x = int(g * rng.uniform(0.0, 0.2))
        return dict(family="aig", inputs=max(20, g // rng.randint(20, 60)), ands=g - x, xors=x, opts=opts,
                    resident=resident)
    if family in ("community", "inprocess"):
        n = _logint(rng, 3_000, 12_000_000 if family == "community" else 60_000)
        c = int(n * rng.uniform(3.4, 4.2))
        learnt = c // rng.randint(8, 40) if family == "inprocess" else 0
        return dict(family="community", vars=n, clauses=c, communities=max(2, n // rng.randint(2_000, 100_000)),
                    learnt=learnt, opts=opts, resident=resident)
    cmax = _logint(rng, 4_000, 200_000)
    return dict(family=family, formulas=rng.randint(2, 600), cmin=min(1_000, cmax), cmax=cmax, opts=opts)


# ---------------------------------------------------------------- formulas, drawn on the GPU
def _below(gen, bound, n):
    """n whole numbers, number i uniform below bound (or bound[i])."""
    u = torch.rand(n, device=DEV, generator=gen, dtype=torch.float64)
    return torch.minimum((u * bound).long(), torch.as_tensor(bound, device=DEV) - 1)


def _distinct(owner, var, redraw, num_vars):
    """Redraws repeated variables of a clause until it has none."""
    idx = None
    while True:
        o = owner if idx is None else owner[idx]
        key, order = torch.sort(o * (num_vars + 1) + (var if idx is None else var[idx]))
        dup = order[1:][key[1:] == key[:-1]]
        del key, order
        if idx is not None:
            dup = idx[dup]
        if dup.numel() == 0:
            return var
        var[dup] = redraw(dup)
        bad = torch.zeros(int(owner[-1]) + 1, dtype=torch.bool, device=DEV)
        bad[owner[dup]] = True
        idx = torch.nonzero(bad[owner]).squeeze(1)


def _planted(gen, num_vars, k, start, owner, var):
    """Literals with fair signs; one literal of every clause that a drawn assignment
    falsifies is flipped."""
    value = torch.randint(0, 2, (num_vars + 1,), device=DEV, generator=gen, dtype=torch.int8)
    sign = torch.randint(0, 2, (var.numel(),), device=DEV, generator=gen, dtype=torch.int8)
    sat = torch.zeros(k.numel(), dtype=torch.int32, device=DEV)
    sat.scatter_add_(0, owner, ((sign ^ 1) == value[var]).int())
    dead = torch.nonzero(sat == 0).squeeze(1)
    sign[start[dead] + _below(gen, k[dead], dead.numel())] ^= 1
    return (2 * var + sign).to(torch.int32)


def _offsets(k):
    off = torch.zeros(k.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(k, 0, out=off[1:])
    return off


def _uniform(gen, num_vars, k):
    """Clauses of k[i] distinct variables, uniform over all."""
    off = _offsets(k)
    owner = torch.repeat_interleave(torch.arange(k.numel(), device=DEV), k)
    var = 1 + _below(gen, num_vars, owner.numel())
    var = _distinct(owner, var, lambda d: 1 + _below(gen, num_vars, d.numel()), num_vars)
    return num_vars, _planted(gen, num_vars, k, off[:-1], owner, var), off


def _community(gen, num_vars, num_clauses, communities):
    """The benchmark's community-attachment formula: clause lengths geometric with mean
    3.5 in [2, 64], 0.8 of the clauses inside one community, variables of a community
    by a power law (exponent 2.5)."""
    per = num_vars // communities
    cdf = torch.cumsum(torch.arange(1, per + 1, device=DEV, dtype=torch.float64) ** (-1.0 / 1.5), 0)
    cdf = (cdf / cdf[-1]).float()
    place = torch.randperm(num_vars, device=DEV, generator=gen) + 1
    u = torch.rand(num_clauses, device=DEV, generator=gen, dtype=torch.float64)
    k = (1 + torch.ceil(torch.log1p(-u) / math.log1p(-1.0 / 2.5))).long().clamp_(2, min(64, max(2, per // 2)))
    del u
    off = _offsets(k)
    owner = torch.repeat_interleave(torch.arange(num_clauses, device=DEV), k)
    n = owner.numel()
    home = torch.randint(0, communities, (num_clauses,), device=DEV, generator=gen)
    inside = torch.rand(num_clauses, device=DEV, generator=gen) < 0.8
    comm = torch.where(inside[owner], home[owner], torch.randint(0, communities, (n,), device=DEV, generator=gen))

    def pick(at):
        c = comm if at is None else comm[at]
        r = torch.searchsorted(cdf, torch.rand(c.numel(), device=DEV, generator=gen), right=True)
        return place[c * per + r.clamp_(max=per - 1)]

    var = _distinct(owner, pick(None), pick, num_vars)
    return num_vars, _planted(gen, num_vars, k, off[:-1], owner, var), off


def _aig(gen, inputs, ands, xors):
    """Tseitin encoding of a random AIG: every gate takes two distinct nodes of the most
    recent tenth before it, with random polarities; `xors` of the gates are XORs."""
    gates = ands + xors
    g = torch.arange(inputs + 1, inputs + gates + 1, device=DEV)
    lo = torch.clamp(g - torch.clamp((0.1 * (g - 1)).long(), min=2), min=1)
    span = g - lo
    da = _below(gen, span, gates)
    a = lo + da
    b = lo + (da + 1 + _below(gen, span - 1, gates)) % span
    pol = torch.randint(0, 2, (2, gates), device=DEV, generator=gen)
    a, b, g = 2 * a + pol[0], 2 * b + pol[1], 2 * g
    xor = torch.zeros(gates, dtype=torch.bool, device=DEV)
    xor[torch.randperm(gates, device=DEV, generator=gen)[:xors]] = True
    z = torch.zeros_like(g)
    and_rows = torch.stack([g | 1, a, z, g | 1, b, z, g, a ^ 1, b ^ 1, z, z, z], 1)
    xor_rows = torch.stack([g | 1, a, b, g | 1, a ^ 1, b ^ 1, g, a ^ 1, b, g, a, b ^ 1], 1)
    rows = torch.where(xor[:, None], xor_rows, and_rows).reshape(-1, 3)
    k = (rows != 0).sum(1)
    k = k[k > 0]
    flat = rows.reshape(-1)
    return inputs + gates, flat[flat != 0].to(torch.int32), _offsets(k)


def _single(case, gen, seed):
    """(variables, literals, offsets) of a case's formula on the GPU."""
    f = case["family"]
    if f == "ksat":
        return _uniform(gen, case["vars"], torch.full((case["clauses"],), 3, device=DEV))
    if f == "mixed":
        return _uniform(gen, case["vars"], torch.randint(2, 6, (case["clauses"],), device=DEV, generator=gen))
    if f == "aig":
        return _aig(gen, case["inputs"], case["ands"], case["xors"])
    if f == "community":
        return _community(gen, case["vars"], case["clauses"], case["communities"])
    # the unrolled transition relation without its property (its last clause)
    nv, lits, off = cnfgen.aig_unrolled(case["gates"], case["steps"], seed=seed)
    lits, off = lits[:-1], off[:-1]
    return (nv, torch.from_numpy(lits.view(np.int32)).to(DEV), torch.from_numpy(off.view(np.int64)).to(DEV))


def _batch_sizes(case):
    """(clauses, variables) per formula: clause counts log-uniform in [cmin, cmax],
    clause/variable ratio in [3, 4.5], spread evenly over both ranges."""
    i = np.arange(case["formulas"])
    u, w = (i * 0.6180339887498949 + 0.5) % 1.0, (i * 0.7548776662466927 + 0.25) % 1.0
    ncls = np.exp(math.log(case["cmin"]) + u * math.log(case["cmax"] / case["cmin"])).astype(np.int64)
    return ncls, np.maximum((ncls / (3.0 + 1.5 * w)).astype(np.int64), 8)


def _batch(case, gen):
    """A batch of mixed k-SAT formulas as host arrays [(variables, literals, offsets)]."""
    nf = case["formulas"]
    ncls, nvar = (torch.from_numpy(x).to(DEV) for x in _batch_sizes(case))
    owner_f = torch.repeat_interleave(torch.arange(nf, device=DEV), ncls)
    k = torch.randint(2, 6, (owner_f.numel(),), device=DEV, generator=gen)
    off = _offsets(k)
    owner = torch.repeat_interleave(torch.arange(k.numel(), device=DEV), k)
    lit_f = owner_f[owner]
    bound, first = nvar[lit_f], (torch.cumsum(nvar, 0) - nvar)[lit_f]
    total = int(nvar.sum())

    def pick(at):
        b, o = (bound, first) if at is None else (bound[at], first[at])
        return 1 + o + _below(gen, b, b.numel())

    var = _distinct(owner, pick(None), pick, total)
    lits = _planted(gen, total, k, off[:-1], owner, var) - (2 * first).to(torch.int32)
    lits, off = lits.cpu().numpy().view(np.uint32), off.cpu().numpy().view(np.uint64)
    cb = np.concatenate([[0], np.cumsum(ncls.cpu().numpy())])
    out = []
    for f, nv in enumerate(nvar.tolist()):
        o = off[cb[f]:cb[f + 1] + 1]
        out.append((nv, lits[int(o[0]):int(o[-1])].copy(), o - o[0]))
    return out


# ---------------------------------------------------------------- passes
class _Buffers(ResultBuffers):
    """The caller's page-locked result buffers, of one size for all formulas of a case."""

    def __init__(self, num_vars, num_clauses, num_lits, formulas=1):
        super().__init__()
        room = dict(lits=(num_lits, torch.int32), offsets=(num_clauses + 1, torch.int64),
                    learnt=(num_clauses, torch.uint8), units=(num_vars, torch.int32),
                    resolved=(num_lits, torch.int32), eliminated=(num_vars + formulas, torch.uint8))
        self.whole = {k: torch.zeros(n, dtype=t, pin_memory=True).numpy() for k, (n, t) in room.items()}

    def take(self, name, count, dtype):
        return self.whole[name][:count].view(dtype)

    def outputs(self):
        """All buffers but the trail's, whose order is free."""
        return {k: v for k, v in self.whole.items() if k != "units"}


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    s = Simplifier(Options(**OPTIONS[case["opts"]]))
    nv, nc, nl = _shape(case)
    room = nl + nl // 8 + 4096  # the simplified clauses, or the witness stack, of the largest formula
    st = dict(case, s=s)
    if case["family"] in ("batch", "extend"):
        st["formulas"] = _batch(case, gen)
        if case["family"] == "batch":
            st["buf"] = _Buffers(nv, nc, room, case["formulas"])
        else:
            s.awaken_batch(st["formulas"])
            s.sigmify()
            rng = np.random.default_rng(seed)
            st["models"] = [rng.integers(0, 2, n + 1, dtype=np.uint8) for n, _, _ in st["formulas"]]
        return st
    st["buf"] = _Buffers(nv, nc + nc // 8 + 4096, room)
    nv, lits, off = _single(case, gen, seed)
    st["vars"], st["clauses"] = nv, off.numel() - 1
    learnt = case.get("learnt", 0)
    if case["resident"]:
        st["lits"], st["off"], st["learnt"] = lits, off, None
        if learnt:
            st["learnt"] = torch.zeros(st["clauses"], dtype=torch.uint8, device=DEV)
            st["learnt"][st["clauses"] - learnt:] = 1
    else:
        st["lits"] = lits.cpu().pin_memory().numpy().view(np.uint32)
        st["off"] = off.cpu().pin_memory().numpy().view(np.uint64)
        st["learnt"] = None
        if learnt:
            st["learnt"] = np.zeros(st["clauses"], dtype=np.uint8)
            st["learnt"][st["clauses"] - learnt:] = 1
    return st


def _run_batch(st):
    s, buf = st["s"], st["buf"]
    s.awaken_batch(st["formulas"])
    s.sigmify()
    results = s.batch_results(out=buf)
    res = [r[2] for r in results]
    # every formula's trail into one assignment (2: unassigned), formula after formula
    sizes = np.array([r.num_vars + 1 for r in res])
    counts = np.array([r.units.size for r in res])
    units = buf.take("units", int(counts.sum()), np.uint32)
    value = np.full(int(sizes.sum()), 2, dtype=np.uint8)
    value[np.repeat(np.cumsum(sizes) - sizes, counts) + (units >> 1)] = (units & 1) ^ 1
    return dict(buf.outputs(), value=value, status=np.array([r[0] for r in results], dtype=np.int32),
                phases=np.array([r[1] for r in results], dtype=np.int32),
                clauses=np.array([r.learnt.size for r in res]), words=np.array([r.resolved.size for r in res]))


def run(st):
    if st["family"] == "extend":
        return np.concatenate(st["s"].batch_extend(st["models"]))
    if st["family"] == "batch":
        return _run_batch(st)
    s, nv = st["s"], st["vars"]
    if st["resident"]:
        learnt = st["learnt"]
        s.awaken_device(nv, st["lits"].data_ptr(), st["off"].data_ptr(), st["clauses"],
                        None if learnt is None else learnt.data_ptr())
    else:
        s.awaken(nv, st["lits"], st["off"], st["learnt"])
    stats = s.sigmify()
    r = s.result(out=st["buf"])
    # the trail into the caller's assignment (2: unassigned)
    if st["resident"]:
        units = torch.from_numpy(r.units.view(np.int32)).to(DEV)
        value = torch.full((nv + 1,), 2, dtype=torch.uint8, device=DEV)
        value[units >> 1] = ((units & 1) ^ 1).to(torch.uint8)
    else:
        value = np.full(nv + 1, 2, dtype=np.uint8)
        value[r.units >> 1] = (r.units & 1) ^ 1
    return dict(st["buf"].outputs(), value=value, status=int(stats.status), clauses=r.learnt.size,
                words=r.resolved.size)


# ---------------------------------------------------------------- what a pass cannot do without
def _shape(case):
    """(variables, clauses, literals) of a case, in the mean over its seeds."""
    f = case["family"]
    if f == "ksat":
        return case["vars"], case["clauses"], 3 * case["clauses"]
    if f in ("mixed", "community"):
        return case["vars"], case["clauses"], int(3.5 * case["clauses"])
    if f == "aig":
        return (case["inputs"] + case["ands"] + case["xors"], 3 * case["ands"] + 4 * case["xors"],
                7 * case["ands"] + 12 * case["xors"])
    if f == "unrolled":
        g, t, tenth = case["gates"], case["steps"], max(2, case["gates"] // 10)
        return t * (g + tenth) + tenth, 3 * g * t + tenth, 7 * g * t + tenth
    ncls, nvar = _batch_sizes(case)
    return int(nvar.sum()), int(ncls.sum()), int(3.5 * ncls.sum())


def work(case):
    """The input's literals and clause ends once, and the output once: the literals of
    the simplified formula and the witness stack together are taken as the input's
    (an eliminated variable's clauses move from one to the other), with an eliminated
    flag and a value per variable. An extension reads the witness stack once and every
    variable's value before and after."""
    v, c, n = _shape(case)
    if case["family"] == "extend":
        return {"bytes": 2 * n + 2 * v, "flops": 0}
    return {"bytes": 4 * n + 8 * (c + 1) + 4 * n + 2 * v, "flops": 0}


def exact(case, seed):
    """No output is a computed number: all are whole numbers, held to equality."""
    return None
