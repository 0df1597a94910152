"""SUB's look at all pairs at once, around the 64 entries that a warp stages: one variable
with 62 to 66 clauses whose lists hold no hit, a clause that an earlier one subsumes, one
that the other list strengthens, or entries that propagation deleted. Every stage equals
the oracle's."""
import numpy as np
import pytest

import oracle_runner as orr
from parafrost_gb300 import rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib
from test_prop_waves import _pack


def _formula(entries, plant):
    rng = np.random.default_rng(entries)
    x, others = 1, np.arange(2, 62)
    npos = entries // 2
    seen, own = set(), []
    while len(own) < entries:
        a, b = sorted(rng.choice(others, 2, replace=False))
        if (a, b) in seen:
            continue
        seen.add((a, b))
        s = rng.choice([-1, 1], 2)
        own.append([x if len(own) < npos else -x, int(a * s[0]), int(b * s[1])])
    if plant == "subsume":
        own[1] = own[0] + [63]
    if plant == "strengthen":
        own[0] = [x, own[-1][1], own[-1][2], 63]
    rest = [[int(v) * int(s) for v, s in zip(rng.choice(others, 3, replace=False), rng.choice([-1, 1], 3))]
            for _ in range(2400)]
    rest += [[63, int(v), 64] for v in others[:40]] + [[-63, int(v), -64] for v in others[:40]]
    if plant == "deleted":
        own[2] = own[2] + [65]
        own[-3] = own[-3] + [65]
        rest.append([65])
    return _pack(66, own + rest)


def _check(lib, entries, plant):
    nv, lits, off = _formula(entries, plant)
    opts = Options(all=1, phases=1, mu_pos=34, mu_neg=34)
    st, a, _ = orr.run_oracle(nv, lits, off, opts, level=2)
    stats, b, _ = run_lib(lib, nv, lits, off, opts, level=2)
    assert stats.status == st
    assert rd.compare(rd.normalize(a), rd.normalize(b)) == []


PLANTS = ["none", "subsume", "strengthen", "deleted"]


@pytest.mark.parametrize("plant", PLANTS)
@pytest.mark.parametrize("entries", [62, 64, 65])
def test_sub_stage_emu(built, entries, plant):
    _check(built["emu"], entries, plant)


@pytest.mark.gpu
@pytest.mark.parametrize("plant", PLANTS)
@pytest.mark.parametrize("entries", [31, 32, 62, 63, 64, 65, 66])
def test_sub_stage_gpu(cuda_lib, built, entries, plant):
    _check(cuda_lib, entries, plant)
