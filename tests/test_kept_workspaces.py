"""A context that repeats a request of the same size allocates nothing: rounds, batch
results and model extension keep their workspaces, and a destroyed context returns all
of them (the stage times of a round still add up to its phases')."""
import numpy as np
import pytest

from parafrost_gb300 import cnfgen
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import Simplifier


def _check(lib):
    forms = [cnfgen.random_mixed_ksat(300 + 50 * i, 3.2, seed=i) for i in range(7)]
    models = [np.zeros(f[0] + 1, dtype=np.uint8) for f in forms]
    with Simplifier(Options(all=1), library=lib) as s:
        counts = []
        for _ in range(4):
            s.awaken_batch(forms)
            st = s.sigmify()
            s.batch_results()
            s.batch_extend(models)
            counts.append((s.lib.pf_device_alloc_count(), s.footprint()))
        assert len(set(counts[1:])) == 1
    d = st.as_dict()
    phases = sum(p["ms"] for p in d["phases"])
    assert 0 < phases <= sum(d["ms_stage"].values()) + 1e-6


def test_kept_emu(built):
    _check(built["emu"])


@pytest.mark.gpu
def test_kept_gpu(cuda_lib):
    import gc
    import torch
    _check(cuda_lib)
    gc.collect()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        _check(cuda_lib)
    gc.collect()
    assert torch.cuda.mem_get_info()[0] >= free0 - (8 << 20)  # less than one context of this size
