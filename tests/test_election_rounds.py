"""The election's rounds at the sizes where their form changes: every vertex with its own
lanes, one thread a vertex (more undecided vertices than threads), more long-list
vertices than warps, lists of one variable only. The elected variables of every phase
equal the oracle's."""
import pytest

import oracle_runner as orr
from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib

FORMS = {
    "one-clause": lambda: cnfgen.random_ksat(3, 1, 3, seed=1),
    "33-vars": lambda: cnfgen.random_ksat(33, 120, 3, seed=2),
    "own-lanes": lambda: cnfgen.random_ksat(7000, 29_000, 3, seed=3),
    "thread-each": lambda: cnfgen.random_mixed_ksat(1_300_000, 4.0, seed=4),
    "long-lists": lambda: cnfgen.random_ksat(20_000, 240_000, 3, seed=5),
    "hubs": lambda: cnfgen.community(num_vars=60_000, num_clauses=240_000, communities=2, seed=6),
}


def _check(lib, name):
    nv, lits, off = FORMS[name]()
    st, a, _ = orr.run_oracle(nv, lits, off, Options(all=1), level=1)
    stats, b, _ = run_lib(lib, nv, lits, off, Options(all=1), level=1)
    assert stats.status == st
    assert rd.compare(a, b, kinds=("pvs", "counts", "elim")) == []


@pytest.mark.parametrize("name", ["one-clause", "33-vars", "own-lanes"])
def test_election_emu(built, name):
    _check(built["emu"], name)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(FORMS))
def test_election_gpu(cuda_lib, built, name):
    _check(cuda_lib, name)
