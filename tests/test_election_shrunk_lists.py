"""Elections over lists that have shrunk since the table was built (deleted clauses leave
them where they are, so a list can be empty in front of its variable's other one): units
and deletions of BVE with SUB off, binaries and AIGs. Every phase's elected variables and
the round equal the oracle's."""
import pytest

import oracle_runner as orr
from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib

FORMS = {
    "24-vars": lambda: [cnfgen.random_ksat(24, 19, 2, seed=1)],
    "21-vars": lambda: [cnfgen.random_ksat(21, 21, 2, seed=22)],
    "binaries": lambda: [cnfgen.random_ksat(20 + i, 18 + i + i % 5, 2, seed=i) for i in range(40)],
    "aigs": lambda: [cnfgen.aig_tseitin(num_inputs=8 + i, num_and=60 + 9 * i, num_xor=5, seed=i) for i in range(20)],
}


def _check(lib, name):
    opts = Options(sub=0, ve_plus=0)
    for nv, lits, off in FORMS[name]():
        st, a, _ = orr.run_oracle(nv, lits, off, opts, level=1)
        stats, b, _ = run_lib(lib, nv, lits, off, opts, level=1)
        assert stats.status == st
        assert rd.compare(a, b, kinds=("pvs", "counts", "elim")) == []


@pytest.mark.parametrize("name", list(FORMS))
def test_shrunk_emu(built, name):
    _check(built["emu"], name)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(FORMS))
def test_shrunk_gpu(cuda_lib, built, name):
    _check(cuda_lib, name)
