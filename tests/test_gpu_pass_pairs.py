"""Six-qubit tensor-core passes on few tiles, which two CTAs share (csrc/fused_tc.cu):
each output is the same sum whether one CTA forms it or one of a pair does."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [13, 14, 17, 18])                     # 1, 2, 16 and 32 tiles; 38 are the most for pairs here
@pytest.mark.parametrize("targets", [[0, 1, 2, 3, 4, 5], [0, 1, 5, 8, 10, 12], [1, 3, 5, 7, 9, 11], [7, 8, 9, 10, 11, 12]])
@pytest.mark.parametrize("precision, staging", [(0, 0), (0, 1), (1, 0), (1, 1), (2, 0)])
def test_pairs_match_single_ctas(gpulib, n, targets, precision, staging):
    """The same amplitudes in the lower part of a 20-qubit register, whose
    128 tiles go to one CTA each: the same bits."""
    L = gpulib
    lib = L.lib
    rng = np.random.default_rng(n)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    u = np.linalg.qr(rng.normal(size=(64, 64)) + 1j * rng.normal(size=(64, 64)))[0]
    assert lib.quest_gb300_setTensorCorePrecision(precision) == 0
    assert lib.quest_gb300_setTensorCoreStaging(staging) == 0
    lib.quest_gb300_setTensorCoreKernel(5)
    out = []
    try:
        for m in (n, 20):
            q64 = L.create(m)
            full = np.zeros(1 << m, complex)
            full[: 1 << n] = psi
            L.set_amps(q64, full)
            q32 = lib.quest_gb300_createQuregF32(m)
            lib.quest_gb300_copyFromQureg(q32, q64)
            plan = lib.quest_gb300_planCreate(m, 6)
            re, im = np.ascontiguousarray(u.real.ravel()), np.ascontiguousarray(u.imag.ravel())
            double_p = C.POINTER(C.c_double)
            assert lib.quest_gb300_planAddGate(plan, (C.c_int * 6)(*targets), 6, re.ctypes.data_as(double_p),
                                               im.ctypes.data_as(double_p)) == 0
            lib.quest_gb300_planCompile(plan)
            assert lib.quest_gb300_applyPlanF32(q32, plan) == 0
            out.append(L.amps_f32(q32, m))
            lib.quest_gb300_planDestroy(plan)
            if m == n:
                L.multiQubitUnitary(q64, targets, u)
                err = C.c_double(0)
                lib.quest_gb300_compareF32(q32, q64, C.byref(err))
                assert err.value < 1e-5
            lib.quest_gb300_destroyQuregF32(q32)
            L.destroy(q64)
    finally:
        lib.quest_gb300_setTensorCoreKernel(0)
        lib.quest_gb300_setTensorCoreStaging(0)
        lib.quest_gb300_setTensorCorePrecision(0)
    assert np.array_equal(out[0], out[1][: 1 << n])
    assert not out[1][1 << n:].any()
