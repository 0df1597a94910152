"""Redundancy elimination alone (no other stage), where a block's 256 pairs lie in few
positions, in many, and in more than its window holds: thousands of elected variables
without a pair beside a few with many, some of whose resolvents are clauses already. Every
stage equals the oracle's."""
import numpy as np
import pytest

import oracle_runner as orr
from parafrost_gb300 import rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib
from test_prop_waves import _pack


def _formula(pure, mixed, occ):
    """`pure` variables in two positive clauses each, `mixed` ones in `occ` clauses of each
    sign with every fourth resolvent added as a clause, over a pool of frequent variables."""
    rng = np.random.default_rng(pure + 7 * mixed + occ)
    pool = np.arange(pure + mixed + 1, pure + mixed + 81)

    def two():
        return [int(v) for v in rng.choice(pool, 2, replace=False) * rng.choice([-1, 1], 2)]

    c = []
    for v in range(1, pure + 1):
        c += [[v] + two(), [v] + two()]
    for v in range(pure + 1, pure + mixed + 1):
        pos, neg = [two() for _ in range(occ)], [two() for _ in range(occ)]
        c += [[v] + p for p in pos] + [[-v] + n for n in neg]
        for p in pos[::2]:
            for n in neg[::2]:
                if not {abs(x) for x in p} & {abs(x) for x in n}:
                    c.append(p + n)
    c += [[int(x) for x in rng.choice(pool, 3, replace=False) * rng.choice([-1, 1], 3)] for _ in range(3000)]
    return _pack(int(pool[-1]), [c[i] for i in rng.permutation(len(c))])


def _check(lib, pure, mixed, occ):
    nv, lits, off = _formula(pure, mixed, occ)
    opts = Options(ve=0, ve_plus=0, sub=0, bce=0, ere=1)
    st, a, _ = orr.run_oracle(nv, lits, off, opts, level=2)
    stats, b, _ = run_lib(lib, nv, lits, off, opts, level=2)
    assert stats.status == st
    assert rd.compare(rd.normalize(a), rd.normalize(b)) == []


CASES = [(0, 1, 1), (3, 5, 2), (0, 40, 16), (3000, 2, 3), (5000, 60, 9)]


@pytest.mark.parametrize("pure,mixed,occ", CASES[:3])
def test_ere_emu(built, pure, mixed, occ):
    _check(built["emu"], pure, mixed, occ)


@pytest.mark.gpu
@pytest.mark.parametrize("pure,mixed,occ", CASES)
def test_ere_gpu(cuda_lib, built, pure, mixed, occ):
    _check(cuda_lib, pure, mixed, occ)


def _learnt_formula(mixed, occ, seed):
    """As above, with learnt clauses: resolvents as original and as learnt clauses, some
    several times, of original and of learnt antecedents, so that who takes which clause
    depends on the order."""
    rng = np.random.default_rng(seed)
    pool = np.arange(mixed + 1, mixed + 31)

    def two():
        return [int(v) for v in rng.choice(pool, 2, replace=False) * rng.choice([-1, 1], 2)]

    orig, learnt = [], []
    for v in range(1, mixed + 1):
        pos, neg = [two() for _ in range(occ)], [two() for _ in range(occ)]
        pos, neg = pos + pos[:1], neg + neg[:1]  # equal antecedents: several resolvents of one literal set
        for x, side in ((v, pos), (-v, neg)):
            for c in side:
                (learnt if rng.random() < 0.3 else orig).append([x] + c)
        for p in pos[::2]:
            for n in neg[::2]:
                if not {abs(x) for x in p} & {abs(x) for x in n}:
                    for _ in range(rng.integers(1, 4)):
                        (learnt if rng.random() < 0.5 else orig).append(p + n)
    orig += [[int(x) for x in rng.choice(pool, 3, replace=False) * rng.choice([-1, 1], 3)] for _ in range(1500)]
    orig = [orig[i] for i in rng.permutation(len(orig))]
    learnt = [learnt[i] for i in rng.permutation(len(learnt))]
    nv, lits, off = _pack(int(pool[-1]), orig + learnt)
    flag = np.zeros(len(orig) + len(learnt), dtype=np.uint8)
    flag[len(orig):] = 1
    return nv, lits, off, flag


def _check_learnt(lib, mixed, occ, seed):
    nv, lits, off, flag = _learnt_formula(mixed, occ, seed)
    for opts in (Options(ve=0, ve_plus=0, sub=0, bce=0, ere=1), Options(all=1)):
        st, a, _ = orr.run_oracle(nv, lits, off, opts, level=2, learnt=flag)
        stats, b, _ = run_lib(lib, nv, lits, off, opts, level=2, learnt=flag)
        assert stats.status == st
        assert rd.compare(rd.normalize(a), rd.normalize(b)) == []


LEARNT = [(2, 2, 1), (12, 3, 2), (40, 6, 3), (150, 4, 4)]


@pytest.mark.parametrize("mixed,occ,seed", LEARNT)
def test_ere_learnt_emu(built, mixed, occ, seed):
    _check_learnt(built["emu"], mixed, occ, seed)


@pytest.mark.gpu
@pytest.mark.parametrize("mixed,occ,seed", LEARNT)
def test_ere_learnt_gpu(cuda_lib, built, mixed, occ, seed):
    _check_learnt(cuda_lib, mixed, occ, seed)
