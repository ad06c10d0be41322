"""planPassUsesTensorCores tells what applyPlanF32 runs: its answer against the
norm records, which only tensor-core passes leave."""
import ctypes as C

import pytest

from quantumlab_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9, 10, 13, 16, 19, 20])
@pytest.mark.parametrize("mode", ["default", "kernel 5", "off", "split-FP16", "events"])
def test_reported_applier_is_the_one_that_ran(gpulib, n, mode):
    lib = gpulib.lib
    p = gpulib.plan(n, 6 if n >= 13 and mode != "off" else 5 if n >= 12 or mode == "off" else 4, W.c2_circuit(n=n, layers=2, seed=n))
    passes = lib.quest_gb300_planCompile(p)
    q = lib.quest_gb300_createQuregF32(n)
    lib.quest_gb300_setTensorCoreKernel(5 if mode == "kernel 5" else 0)
    lib.quest_gb300_setTensorCores(0 if mode == "off" else 1)
    lib.quest_gb300_setTensorCorePrecision(2 if mode == "split-FP16" else 0)
    lib.quest_gb300_setPassEvents(1 if mode == "events" else 0)
    try:
        assert lib.quest_gb300_applyPlanF32(q, p) == 0
        v = (C.c_double * 3)()
        for i in range(passes):
            assert (lib.quest_gb300_planPassUsesTensorCores(p, i) > 0) == (lib.quest_gb300_planPassNorms(p, i, v) == 1), (n, mode, i)
    finally:
        lib.quest_gb300_setTensorCoreKernel(0)
        lib.quest_gb300_setTensorCores(1)
        lib.quest_gb300_setTensorCorePrecision(0)
        lib.quest_gb300_setPassEvents(0)
        lib.quest_gb300_destroyQuregF32(q)
        lib.quest_gb300_planDestroy(p)
