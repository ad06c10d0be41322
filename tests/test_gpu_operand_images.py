"""Operand images that the device forms (csrc/fused_build.cu) against the ones
that the host forms (csrc/fused_tc.cu, fused_small.cu): the same gates through
a captured flush and through a plan.  The matrices' entries are dyadic numbers
of 15 bits, so that a pass's product of up to three gates is exact on either
side and has more bits than an operand's parts hold: states of equal bits mean
images of equal bits, low parts and scales included."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
D = C.POINTER(C.c_double)


def gates(n, width, seed):
    """Pairs of gates on `width` qubits in all, one after another on sets that
    share a qubit with the last pair's, so that few gates come to a pass."""
    r = np.random.default_rng(seed)
    out, used = [], []
    for _ in range(6):
        fresh = [int(q) for q in r.permutation(n) if q not in used[-1:]]
        qs = used[-1:] + fresh[:width - len(used[-1:])]
        used = qs
        for ts in (qs[:width // 2], qs[width // 2:]):
            m = r.integers(-(1 << 14), 1 << 14, (2, 1 << len(ts), 1 << len(ts)))
            out.append((sorted(ts), (m[0] + 1j * m[1]) * 2.0 ** -15))
    return out


@pytest.mark.parametrize("n,precision", [(12, 0), (16, 0), (19, 0), (16, 2), (19, 2), (20, 0), (20, 1), (20, 2), (21, 0)])
@pytest.mark.parametrize("width", [4, 5, 6])
def test_device_and_host_images(gpulib, n, precision, width):
    L, lib = gpulib, gpulib.lib
    ops = gates(n, width, 10 * n + width)
    r = np.random.default_rng(n)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    assert lib.quest_gb300_setTensorCorePrecision(precision) == 0
    lib.quest_gb300_setCaptureFusion(width)
    cap, plain = L.create(n), L.create(n)
    q32 = lib.quest_gb300_createQuregF32(n)
    p = lib.quest_gb300_planCreate(n, min(width, 5) if n < 13 else width)
    try:
        L.set_amps(cap, psi)
        assert lib.quest_gb300_setCapture(cap, 1) == 0
        for ts, m in ops:
            L.applyMatrixN(cap, ts, m)
        a = L.amps(cap).copy()
        assert lib.quest_gb300_planSetMaxControls(p, 0) == 0 and lib.quest_gb300_planSetLookahead(p, 0) == 0
        for ts, m in ops:
            re, im = np.ascontiguousarray(m.real.ravel()), np.ascontiguousarray(m.imag.ravel())
            assert lib.quest_gb300_planAddGate(p, (C.c_int * len(ts))(*ts), len(ts), re.ctypes.data_as(D), im.ctypes.data_as(D)) == 0
        passes = lib.quest_gb300_planCompile(p)
        assert passes >= 4                                  # (12 gates: up to three a pass)
        L.set_amps(plain, psi)
        lib.quest_gb300_copyFromQureg(q32, plain)
        assert lib.quest_gb300_applyPlanF32(q32, p) == 0
        lib.quest_gb300_copyToQureg(q32, plain)
        b = L.amps(plain).copy()
        assert np.array_equal(a, b), np.max(np.abs(a - b)) / np.max(np.abs(b))
    finally:
        lib.quest_gb300_setTensorCorePrecision(0)
        lib.quest_gb300_setCaptureFusion(6)
        lib.quest_gb300_planDestroy(p)
        lib.quest_gb300_destroyQuregF32(q32)
        L.destroy(cap)
        L.destroy(plain)
