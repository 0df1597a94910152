"""Batch upload from separate arrays: formulas without clauses, of one clause, around the
size of a piece (32,768 literals or offsets), offsets that start above 0, and arrays that
are not aligned to their words (which a kernel cannot read in place). Every result equals
that of the same formulas packed into one array."""
import numpy as np
import pytest

from parafrost_gb300 import cnfgen, rounddump as rd
from parafrost_gb300.options import Options
from parafrost_gb300.sigma import PF_EINVAL, SigmaError, Simplifier, lits_offsets_begin, pack_batch


def _shifted(a, by):
    """A copy of array a whose data starts `by` bytes past an aligned address."""
    raw = np.zeros(a.nbytes + 64, dtype=np.uint8)
    start = (-raw.ctypes.data) % 64 + by
    out = np.frombuffer(raw.data, dtype=a.dtype, count=a.size, offset=start)
    out[:] = a
    return out


def _forms():
    rng = np.random.default_rng(3)
    out = [(5, np.zeros(0, np.uint32), np.zeros(1, np.uint64)), cnfgen.random_ksat(3, 1, 3, seed=1)]
    for n in (10_921, 10_922, 10_923, 32_766, 32_767, 32_768):  # 3 n literals, n + 1 offsets
        out.append(cnfgen.random_ksat(12_000, n, 3, seed=n))
    nv, lits, off = cnfgen.random_mixed_ksat(4000, 3.3, seed=9)
    out.append((nv, np.concatenate([rng.integers(0, 9, 77).astype(np.uint32), lits]), off + np.uint64(77)))
    return out


def _results(s):
    s.sigmify()
    return [(st, rd.canonical_result(st, r if st == 0 else None)) for st, _, r in s.batch_results()]


def _check(lib, shift):
    forms = _forms()
    plain = [(nv, l[int(o[0]):], o - o[0]) for nv, l, o in forms]
    nv, lits, off = pack_batch(plain)
    cb, lits, off = lits_offsets_begin(plain, lits, off)
    with Simplifier(Options(all=1), library=lib) as s:
        s.upload_batch(nv, cb, lits, off)
        want = _results(s)
        moved = [(n, _shifted(l, shift), _shifted(o, shift)) for n, l, o in forms]
        s.awaken_batch(moved)
        assert _results(s) == want


@pytest.mark.parametrize("shift", [0, 1])
def test_parts_emu(built, shift):
    _check(built["emu"], shift)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 4, 8, 2, 1])
def test_parts_gpu(cuda_lib, shift):
    _check(cuda_lib, shift)


def test_parts_past_the_literals_emu(built):
    good = cnfgen.random_ksat(3, 4, 3, seed=1)
    bad = (3, good[1][:-1].copy(), good[2])  # the last clause's last literal is missing
    with Simplifier(Options(all=1), library=built["emu"]) as s:
        with pytest.raises(SigmaError) as e:
            s.awaken_batch([good, bad])
        assert e.value.status == PF_EINVAL
