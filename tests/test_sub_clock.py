"""The SUB kernel's clock runs over every pass of a phase: where SUB can derive units, the
pass of the variables that can, their re-runs and the pass of all others (kernel figures
divide the bytes of all elected lists by it); one pass where it cannot."""
import pytest

from parafrost_gb300 import cnfgen
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import Simplifier


def _check(lib):
    opts = Options(all=1, phases=1)
    for f, passes in ((cnfgen.random_ksat(300, 340, 2, seed=1), 2), (cnfgen.random_ksat(2000, 8000, 3, seed=1), 1)):
        with Simplifier(opts, library=lib) as s:
            s.awaken(*f)
            d = s.sigmify().as_dict()
        k = d["kernels"]["sub"]
        assert k["launches"] >= passes if passes > 1 else k["launches"] == 1
        assert 0 < k["ms"] <= d["ms_stage"]["sub"] + 1e-3
        assert k["bytes"] > 0


def test_sub_clock_emu(built):
    _check(built["emu"])


@pytest.mark.gpu
def test_sub_clock_gpu(cuda_lib):
    _check(cuda_lib)
