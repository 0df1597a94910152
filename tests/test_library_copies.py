"""Two copies of the library in one process (a test's own build beside an installed one):
each asks for its kernels' shared memory itself, so rounds of both give the same."""
import shutil

import pytest

from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import Simplifier


def _check(lib, tmp_path):
    copy = str(tmp_path / "copy.so")
    shutil.copy(lib, copy)
    nv, lits, off = cnfgen.random_mixed_ksat(3000, 3.8, seed=1)
    got = []
    for path in (lib, copy, lib):
        for buckets in (1, -1):  # the bucket table build and the plain one
            with Simplifier(Options(all=1, ot_buckets=buckets), library=path) as s:
                s.awaken(nv, lits, off)
                st = s.sigmify()
                got.append(rd.canonical_result(st.status, s.result()))
    assert all(g == got[0] for g in got)


def test_copies_emu(built, tmp_path):
    _check(built["emu"], tmp_path)


@pytest.mark.gpu
def test_copies_gpu(cuda_lib, tmp_path):
    _check(cuda_lib, tmp_path)
