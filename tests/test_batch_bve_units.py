"""Batches whose units come from BVE with BCE off (SUB off or bounded, so that it leaves
them to BVE): the units of a phase are propagated before the next election, or by the
closing propagation, as in every formula's own round."""
import pytest

from parafrost_gb300 import cnfgen
from parafrost_gb300.options import Options
from test_batch import check_batch

OPTS = [dict(sub=0, ve_plus=0), dict(sub=0, ve_plus=0, phases=2), dict(sub_max=2), dict(sub_max=3),
        dict(sub=0, ve_plus=0, ere=0, phases=1)]

BATCHES = {
    "one": lambda: [cnfgen.random_ksat(120, 90, 2, seed=0)],
    "binaries": lambda: [cnfgen.random_ksat(40 + 9 * i, 34 + 8 * i + 5 * (i % 4), 2, seed=i) for i in range(24)],
    "aigs": lambda: [cnfgen.aig_tseitin(num_inputs=30, num_and=300, num_xor=40, seed=s) for s in range(10)],
    "families": lambda: [f(i) for i in range(4) for f in (
        lambda i: cnfgen.random_ksat(300, 340, 2, seed=i + 1),
        lambda i: cnfgen.random_mixed_ksat(200 + 50 * i, 2.5, seed=i),
        lambda i: cnfgen.aig_tseitin(num_inputs=20, num_and=150, num_xor=10, seed=i))],
}


@pytest.mark.parametrize("batch", list(BATCHES))
@pytest.mark.parametrize("opt", OPTS)
def test_bve_units_emu(built, opt, batch):
    check_batch(built["emu"], BATCHES[batch](), Options(**opt))


@pytest.mark.gpu
@pytest.mark.parametrize("batch", list(BATCHES))
@pytest.mark.parametrize("opt", OPTS)
def test_bve_units_gpu(cuda_lib, built, opt, batch):
    check_batch(cuda_lib, BATCHES[batch](), Options(**opt))
