"""The radix sort of the election's order at its edges: one block for up to 4096 pairs, a
tile more and less, several tiles, keys of one to three bytes. The order of every phase
equals the oracle's (score, variable) order."""
import pytest

import oracle_runner as orr
from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib

SIZES = [3, 33, 4095, 4096, 4097, 8192, 8193, 20_481]


def _check(lib, nv, ratio):
    nv, lits, off = cnfgen.random_ksat(nv, max(1, int(nv * ratio)), 3, seed=nv)
    opts = Options(all=1, phases=1)
    st, a, _ = orr.run_oracle(nv, lits, off, opts, level=2)
    stats, b, _ = run_lib(lib, nv, lits, off, opts, level=2)
    assert stats.status == st
    assert rd.compare(rd.normalize(a), rd.normalize(b)) == []


@pytest.mark.parametrize("nv", SIZES[:4])
def test_order_emu(built, nv):
    _check(built["emu"], nv, 3.0)


@pytest.mark.gpu
@pytest.mark.parametrize("ratio", [1.5, 4.0, 14.0])
@pytest.mark.parametrize("nv", SIZES)
def test_order_gpu(cuda_lib, built, nv, ratio):
    _check(cuda_lib, nv, ratio)
