"""Pass ranges applied again, or over one another: the first pass of a range
corrects by the norm record of the tensor-core pass that ran last, also where
the range is about to run that pass again (csrc/fused_tc.cu)."""
import ctypes as C

import numpy as np
import pytest

from quantumlab_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def norms(L, p, i):
    v = (C.c_double * 3)()
    assert L.lib.quest_gb300_planPassNorms(p, i, v) == 1
    return list(v)


@pytest.mark.parametrize("first,second", [((2, 99), (2, 99)), ((1, 4), (2, 99)), ((3, 2), (1, 5)), ((2, 1), (2, 3)), ((0, 99), (1, 3))])
def test_a_range_starts_from_the_last_record(gpulib, first, second):
    L = gpulib
    n = 20
    p = L.plan(n, 6, W.c2_circuit(n=n, layers=3, seed=6))
    passes = L.lib.quest_gb300_planCompile(p)
    tc = [i for i in range(passes) if L.lib.quest_gb300_planPassUsesTensorCores(p, i) >= 2]
    assert passes >= 6 and tc == list(range(passes))
    q = L.lib.quest_gb300_createQuregF32(n)
    r = np.random.default_rng(1)
    psi = r.normal(size=(2, 1 << n))
    psi /= np.linalg.norm(psi)
    D = C.POINTER(C.c_double)
    L.lib.quest_gb300_initStateFromAmpsF32(q, psi[0].ctypes.data_as(D), psi[1].ctypes.data_as(D))
    assert L.lib.quest_gb300_applyPlanF32Range(q, p, 0, 2) == 0
    assert L.lib.quest_gb300_applyPlanF32Range(q, p, *first) == 0
    last = min(passes, first[0] + first[1]) - 1
    into, out, scale = norms(L, p, last)
    want = into * scale / out                               # undoes that pass's drift
    assert L.lib.quest_gb300_applyPlanF32Range(q, p, *second) == 0
    got = norms(L, p, second[0])[2]
    assert abs(out / (into * scale) - 1) > 2e-8             # there is a drift to correct
    # the scale is held in FP32 as its distance from 1
    assert abs(got - want) <= 1e-6 * abs(want - 1), (got, want)
    L.lib.quest_gb300_destroyQuregF32(q)
    L.lib.quest_gb300_planDestroy(p)
