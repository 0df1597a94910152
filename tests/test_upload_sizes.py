"""Upload of clauses around the length that is sorted in registers (8): every length from 1
to 9 and around 32, literals in any order, and an invalid literal (out of range, or of a
variable that is there already) at every place. Accepted formulas simplify as the oracle's."""
import numpy as np
import pytest

import oracle_runner as orr
from parafrost_gb300 import rounddump as rd
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import PF_EINVAL, SigmaError, Simplifier
from test_emu import run_lib

NV = 90


def _formula(size):
    rng = np.random.default_rng(size)
    sizes = np.concatenate([np.full(60, size), rng.integers(2, 6, 150)])
    lits = np.concatenate([2 * rng.choice(np.arange(1, NV + 1), n, replace=False) + (rng.random(n) < 0.3) for n in sizes])
    return lits.astype(np.uint32), np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


def _check(lib, size):
    lits, off = _formula(size)
    st, a, _ = orr.run_oracle(NV, lits, off, Options(all=1), level=1)
    stats, b, _ = run_lib(lib, NV, lits, off, Options(all=1), level=1)
    assert stats.status == st
    if st == 0:
        assert rd.canonical(a) == rd.canonical(b)
    with Simplifier(Options(all=1), library=lib) as s:
        for at in range(size):
            for bad in [0, 1, 2 * NV + 2, 0xFFFFFFFF] + ([int(lits[(at + 1) % size]) ^ 1] if size > 1 else []):
                l = lits.copy()
                l[at] = bad
                with pytest.raises(SigmaError) as e:
                    s.awaken(NV, l, off)
                assert e.value.status == PF_EINVAL


SIZES = [1, 2, 3, 4, 5, 6, 7, 8, 9, 31, 32, 33]


@pytest.mark.parametrize("size", [1, 4, 8, 9])
def test_upload_emu(built, size):
    _check(built["emu"], size)


@pytest.mark.gpu
@pytest.mark.parametrize("size", SIZES)
def test_upload_gpu(cuda_lib, built, size):
    _check(cuda_lib, size)
