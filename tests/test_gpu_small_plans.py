"""Plans on small registers as one launch (csrc/fused_small.cu) against the
passes applied in complex128."""
import ctypes as C

import numpy as np
import pytest

from quantumlab_gb300 import workloads as W

pytestmark = pytest.mark.gpu
D = C.POINTER(C.c_double)


def apply(psi, targets, m, n):
    k = len(targets)
    t = psi.reshape((2,) * n)                               # axis a is qubit n - 1 - a
    axes = [n - 1 - q for q in reversed(targets)]           # matrix bit 0 is targets[0]
    t = np.moveaxis(t, axes, range(k))
    shape = t.shape
    t = (m @ t.reshape(1 << k, -1)).reshape(shape)
    return np.moveaxis(t, range(k), axes).reshape(-1)


@pytest.mark.parametrize("n", [10, 11, 13, 16, 17, 18, 19])
def test_dense_passes(gpulib, n):
    """Dense gates on 1 to 6 qubits: low, high, adjacent and spread sets, one
    of them not unitary.  A sum has 128 products in four runs, so its rounding
    is within 35 x 2^-24 of the pass's operands, entry by entry; entries round
    independently, and so does the norm of the error."""
    L = gpulib
    r = np.random.default_rng(n)
    sets = [[0], [n - 1], [0, 1], [1, n - 2], [0, 1, 2, 3, 4, 5], list(range(n - 6, n)), [1, 3, 5, 7, 9], [0, n - 1],
            sorted(r.permutation(n)[:6].tolist()), sorted(r.permutation(n)[:4].tolist()), [2, 3, 4, 5, 6, 7]]
    widest = 6 if n >= 13 else 5                            # what a plan takes at this size
    sets = [s[:widest] for s in sets]
    p = L.lib.quest_gb300_planCreate(n, 6)
    gates = []
    for i, ts in enumerate(sets):
        z = r.normal(size=(1 << len(ts),) * 2) + 1j * r.normal(size=(1 << len(ts),) * 2)
        m = np.linalg.qr(z)[0] * (0.5 if i == 3 else 1.0)
        gates.append((ts, m))
        re, im = np.ascontiguousarray(m.real.ravel()), np.ascontiguousarray(m.imag.ravel())
        assert L.lib.quest_gb300_planAddGate(p, (C.c_int * len(ts))(*ts), len(ts), re.ctypes.data_as(D), im.ctypes.data_as(D)) == 0
    passes = L.lib.quest_gb300_planCompile(p)
    psi = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    q32 = L.lib.quest_gb300_createQuregF32(n)
    re, im = np.ascontiguousarray(psi.real), np.ascontiguousarray(psi.imag)
    want = psi
    for ts, m in gates:
        want = apply(want, ts, m, n)
    for half in (False, True):                              # in one application, and in two ranges
        L.lib.quest_gb300_initStateFromAmpsF32(q32, re.ctypes.data_as(D), im.ctypes.data_as(D))
        before = L.lib.quest_gb300_launchCount()
        if half:
            assert L.lib.quest_gb300_applyPlanF32Range(q32, p, 0, passes // 2) == 0
            assert L.lib.quest_gb300_applyPlanF32Range(q32, p, passes // 2, passes) == 0
        else:
            assert L.lib.quest_gb300_applyPlanF32(q32, p) == 0
        assert L.lib.quest_gb300_launchCount() - before == (2 if half else 1)
        got = L.amps_f32(q32, n)
        err = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert err <= (passes + 1) * 35 * 2.0 ** -24, (n, err)
    L.lib.quest_gb300_planDestroy(p)
    L.lib.quest_gb300_destroyQuregF32(q32)


def test_replanned_circuit_takes_its_own_matrices(gpulib):
    """Recompiling a plan with further gates, and applying one plan to two
    registers: nothing of an earlier program is kept."""
    L = gpulib
    n = 12
    ops = W.c2_circuit(n=n, layers=2, seed=4)
    p = L.plan(n, 6, ops)
    regs = [L.lib.quest_gb300_createQuregF32(n) for _ in range(2)]
    for q in regs:
        assert L.lib.quest_gb300_applyPlanF32(q, p) == 0
    a, b = (L.amps_f32(q, n) for q in regs)
    assert np.array_equal(a, b)
    x = np.array([[0, 1], [1, 0]], dtype=float).ravel()
    zero = np.zeros(4)
    assert L.lib.quest_gb300_planAddGate(p, (C.c_int * 1)(n - 1), 1, x.ctypes.data_as(D), zero.ctypes.data_as(D)) == 0
    L.lib.quest_gb300_planCompile(p)
    L.lib.quest_gb300_initZeroStateF32(regs[0])
    assert L.lib.quest_gb300_applyPlanF32(regs[0], p) == 0
    flipped = L.amps_f32(regs[0], n)
    assert np.max(np.abs(flipped - a.reshape(2, -1)[::-1].reshape(-1))) < 1e-5
    for q in regs:
        L.lib.quest_gb300_destroyQuregF32(q)
    L.lib.quest_gb300_planDestroy(p)
