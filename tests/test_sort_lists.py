"""Elected lists sorted by warps, at the lengths where the reference's sort changes (20) and
where a list is left to one lane (32): lists with all keys different, with equal keys
(same size, first and last literal and signature) and mixed. Every stage, the sorted
lists among them, equals the oracle's."""
import numpy as np
import pytest

import oracle_runner as orr
from parafrost_gb300 import rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib
from test_prop_waves import _pack


def _formula(n, ties):
    """Variable 50 in n clauses of each sign; `ties` of them (of each sign) share a key:
    they differ in a literal that leaves the signature's bits alone (16 variables apart)."""
    rng = np.random.default_rng(1000 * n + ties)
    mids = [51 + 16 * i for i in range(n)]
    last = 60 + 16 * n
    c = []
    for s in (1, -1):
        own = [[1, 50 * s, mids[i], last] for i in range(ties)]
        own += [[int(v) for v in (rng.choice(np.arange(2, 40), 2, replace=False) * rng.choice([-1, 1], 2))] + [50 * s, mids[i]]
                for i in range(ties, n)]
        c += [own[i] for i in rng.permutation(n)]
    others = np.concatenate([np.arange(1, 50), mids, [last]])
    for _ in range(90 * others.size // 3):
        c.append([int(v) * int(s) for v, s in zip(rng.choice(others, 3, replace=False), rng.choice([-1, 1], 3))])
    return _pack(last, [c[i] for i in rng.permutation(len(c))])


def _check(lib, n, ties):
    nv, lits, off = _formula(n, ties)
    opts = Options(all=1, phases=1, mu_pos=36, mu_neg=36)
    st, a, _ = orr.run_oracle(nv, lits, off, opts, level=2)
    assert any(k == "pvs" and 50 in list(d) for k, _, _, d in a)
    stats, b, _ = run_lib(lib, nv, lits, off, opts, level=2)
    assert stats.status == st
    assert rd.compare(rd.normalize(a), rd.normalize(b)) == []


CASES = [(n, t) for n in (2, 19, 20, 21, 31, 32, 33) for t in (0, n // 2, n)]


@pytest.mark.parametrize("n,ties", CASES[::4])
def test_sort_emu(built, n, ties):
    _check(built["emu"], n, ties)


@pytest.mark.gpu
@pytest.mark.parametrize("n,ties", CASES)
def test_sort_gpu(cuda_lib, built, n, ties):
    _check(cuda_lib, n, ties)
