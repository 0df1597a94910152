"""Elections whose undecided vertices each have a group of lanes (32 down to one) while
other blocks decide the words that a group looks at: dense neighbourhoods, so that most
vertices are marked out during their tries. The elected variables of every phase equal
the oracle's, whatever the schedule of a run."""
import pytest

import oracle_runner as orr
from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib

SIZES = [60, 3_000, 12_000, 24_000, 48_000, 96_000, 180_000]


def _check(lib, n, runs):
    nv, lits, off = cnfgen.random_ksat(n, 3 * n, 5, seed=n)
    opts = Options(all=1, phases=2)
    st, a, _ = orr.run_oracle(nv, lits, off, opts, level=1)
    for _ in range(runs):
        stats, b, _ = run_lib(lib, nv, lits, off, opts, level=1)
        assert stats.status == st
        assert rd.compare(a, b, kinds=("pvs", "counts", "elim")) == []


@pytest.mark.parametrize("n", SIZES[:2])
def test_groups_emu(built, n):
    _check(built["emu"], n, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_groups_gpu(cuda_lib, built, n):
    _check(cuda_lib, n, 3)
