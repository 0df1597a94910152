"""Propagation waves at the sizes where their form changes: a chain far deeper than the
walks of one wave, lists around the length where they are cut into parts (128), a wave
whose lists cover the store (a sweep), clauses that two walks make unit or false at the
same time, a conflict, and a batch in which one formula is refuted. Results equal the
oracle's, with sweeps chosen by size, always and never."""
import numpy as np
import pytest

import oracle_runner as orr
from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import PF_UNSAT, Simplifier
from test_emu import run_lib


def _pack(num_vars, clauses):
    sizes = np.array([len(c) for c in clauses], dtype=np.uint64)
    lits = np.array([2 * abs(x) + (x < 0) for c in clauses for x in c], dtype=np.uint32)
    return num_vars, lits, np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


def _rest(rng, lo, hi, n):
    """Random ternary clauses over variables lo..hi that set nothing."""
    return [[int(v) * int(s) for v, s in zip(rng.choice(np.arange(lo, hi), 3, replace=False), rng.choice([-1, 1], 3))]
            for _ in range(n)]


def chain(depth, conflict=False):
    """1 implies 2 implies ... implies depth; every link also strips a ternary clause."""
    rng = np.random.default_rng(depth)
    c = [[1]] + [[-i, i + 1] for i in range(1, depth)]
    c += [[-i, -(i + 1), depth + 1 + i % 50] if i % 3 else [-i, depth + 10 + i % 40, depth + 60] for i in range(1, depth)]
    c += _rest(rng, depth + 1, depth + 100, 150)
    if conflict:
        c.append([-depth])
    return _pack(depth + 100, c)


def hub(occurrences):
    """Literal 1 in `occurrences` clauses of each sign; its unit strips and deletes them."""
    rng = np.random.default_rng(occurrences)
    c = [[1]]
    for s in (-1, 1):
        c += [[s] + r for r in _rest(rng, 2, 400, occurrences)]
    return _pack(400, c + _rest(rng, 2, 400, 200))


def joins(n):
    """Clauses whose literals fall in the same wave: unit (a third variable) or false."""
    c = []
    for i in range(n):
        a, b, x, y = 4 * i + 1, 4 * i + 2, 4 * i + 3, 4 * i + 4
        c += [[a], [b], [-a, -b, x], [-a, -x, y], [-b, -y, x]]
    rng = np.random.default_rng(n)
    return _pack(4 * n + 60, c + _rest(rng, 4 * n + 1, 4 * n + 60, 90))


FORMS = {
    "chain-3": lambda: chain(3), "chain-5000": lambda: chain(5000), "conflict": lambda: chain(700, True),
    "hub-127": lambda: hub(127), "hub-128": lambda: hub(128), "hub-129": lambda: hub(129), "hub-9001": lambda: hub(9001),
    "joins": lambda: joins(3000),
    "units-community": lambda: cnfgen.with_units_of("community", 300, num_vars=20_000, num_clauses=80_000,
                                                    communities=10, seed=4),
}


def _check(lib, name, sweep_div):
    nv, lits, off = FORMS[name]()
    st, a, _ = orr.run_oracle(nv, lits, off, Options(all=1), level=1)
    stats, b, _ = run_lib(lib, nv, lits, off, Options(all=1, sweep_div=sweep_div), level=1)
    assert stats.status == st
    if st != PF_UNSAT:
        assert rd.canonical(a) == rd.canonical(b)


def _check_batch(lib):
    forms = [chain(40), chain(300, True), hub(300), joins(50)]
    with Simplifier(Options(all=1), library=lib) as s:
        s.awaken_batch(forms)
        s.sigmify()
        got = s.batch_results()
    for (nv, lits, off), (status, _, r) in zip(forms, got):
        st, a, _ = orr.run_oracle(nv, lits, off, Options(all=1), level=1)
        assert status == st
        if st != PF_UNSAT:
            assert rd.canonical(a) == rd.canonical_result(status, r)


@pytest.mark.parametrize("name", list(FORMS))
def test_prop_emu(built, name):
    _check(built["emu"], name, 0)


def test_prop_batch_emu(built):
    _check_batch(built["emu"])


@pytest.mark.gpu
@pytest.mark.parametrize("sweep_div", [0, 1_000_000, -1])
@pytest.mark.parametrize("name", list(FORMS))
def test_prop_gpu(cuda_lib, built, name, sweep_div):
    _check(cuda_lib, name, sweep_div)


@pytest.mark.gpu
def test_prop_batch_gpu(cuda_lib, built):
    _check_batch(cuda_lib)


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [1, 2, 9, 40])
def test_prop_loop_limit_gpu(cuda_lib, built, depth):
    """The loop bound that a propagation level by level (the serial waves) just keeps."""
    nv, lits, off = _pack(depth + 1, [[1]] + [[-i, i + 1] for i in range(1, depth)] + [[-depth, depth + 1]])
    stats, _, _ = run_lib(built["emu"], nv, lits, off, Options(all=1, sweep_div=-1), level=1)
    assert stats.status == 0 and stats.prop_waves >= depth
    opts = Options(all=1, sweep_div=-1, loop_limit=int(stats.prop_waves))
    assert run_lib(cuda_lib, nv, lits, off, opts, level=1)[0].status == 0
