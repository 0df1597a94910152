"""The per-variable kernels (SUB, BVE write, BCE count) around the number of elected
variables from which they run with more blocks per SM (48 warps per SM of the device):
copies of small formulas whose elected variables have clauses to subsume, to
strengthen, to resolve and blocked ones."""
import numpy as np
import pytest

import oracle_runner as orr
from parafrost_gb300 import rounddump as rd
from parafrost_gb300.options import Options
from test_emu import run_lib

KINDS = (
    [[1, 2, 3], [1, 2], [-1, 3, 4], [-1, -2, 4], [2, 3, 4, 5], [-3, -4, 5], [2, -5, 3]],  # subsumed, resolved
    [[1, 2, 3], [-1, 2], [1, -3, 4], [-1, 3, -4, 5], [-2, 4, 5], [3, -5, 2], [-3, 5, -2]],  # strengthened
    [[1, 2], [1, 3], [-1, -2, -3], [2, 3, 4], [-4, 5, 2], [4, -5, 3]],  # a gate; blocked clauses
)


ELECTED = (2, 1, 2)  # variables that the first phase elects in a copy of each


def _copies(n):
    """Copies with n elected variables in the first phase."""
    lits, off, i, left = [], [0], 0, n
    while left:
        k = i % len(KINDS) if left > 1 else ELECTED.index(1)
        for cl in KINDS[k]:
            lits.extend(2 * (5 * i + abs(x)) + (x < 0) for x in cl)
            off.append(len(lits))
        left -= ELECTED[k]
        i += 1
    return 5 * i, np.array(lits, np.uint32), np.array(off, np.uint64)


def _check(lib, n, phases):
    nv, lits, off = _copies(n)
    opts = Options(all=1, phases=phases)
    st, a, _ = orr.run_oracle(nv, lits, off, opts, level=1)
    stats, b, _ = run_lib(lib, nv, lits, off, opts, level=1)
    assert stats.status == st
    elected = stats.as_dict()["phases"][0]["elected"]
    assert elected == n
    assert rd.canonical(a) == rd.canonical(b)


def test_pv_emu(built):
    _check(built["emu"], 100, 5)


@pytest.mark.gpu
@pytest.mark.parametrize("phases", [1, 5])
@pytest.mark.parametrize("around", [-1, 0, 1, 7001])
def test_pv_gpu(cuda_lib, around, phases):
    import torch

    n = 48 * torch.cuda.get_device_properties(0).multi_processor_count + around
    _check(cuda_lib, n, phases)
