"""Model extension by warps, at the sizes where a step of 32 records, the literals a
lane keeps and the words read ahead end: records of up to 13 literals, formulas with no
record, with a few and with thousands, stacks shorter and longer than the read-ahead.
Values are compared byte for byte with the oracle's host walk."""
import numpy as np
import pytest

from parafrost_gb300 import cnfgen
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import Simplifier
from test_model_extend import _check_batch, host_extend

FORMS = {
    "long-records": lambda: cnfgen.random_ksat(400, 120, 12, seed=3),
    "few-records": lambda: cnfgen.random_ksat(40, 60, 3, seed=5),
    "no-record": lambda: cnfgen.random_ksat(30, 900, 2, seed=7),
    "thousands": lambda: cnfgen.aig_tseitin(num_inputs=300, num_and=5000, num_xor=400, seed=9),
}


def _start(nv, seed):
    return np.random.default_rng(seed).integers(0, 2, nv + 1).astype(np.uint8)


def _single(lib, name):
    nv, lits, off = FORMS[name]()
    with Simplifier(Options(all=1), library=lib) as s:
        s.awaken(nv, lits, off)
        if s.sigmify().status != 0:
            return
        res = s.result()
        for seed in range(4):
            assert np.array_equal(s.extend(_start(nv, seed)), host_extend(res, _start(nv, seed)))


def _batch(lib, count):
    names = list(FORMS)
    forms = [FORMS[names[i % len(names)]]() for i in range(count)]
    _check_batch(lib, forms, [_start(f[0], i) for i, f in enumerate(forms)])


@pytest.mark.parametrize("name", list(FORMS))
def test_single_emu(built, name):
    _single(built["emu"], name)


@pytest.mark.parametrize("count", [1, 5])
def test_batch_emu(built, count):
    _batch(built["emu"], count)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(FORMS))
def test_single_gpu(cuda_lib, name):
    _single(cuda_lib, name)


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 3, 4, 5, 33])
def test_batch_gpu(cuda_lib, count):
    _batch(cuda_lib, count)
