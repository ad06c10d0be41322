"""Capture flushes whose pass products and operand images the device forms
(csrc/fused_build.cu): every operand form and pass width, gates on 1 to 3
qubits, repeated flushes that reuse memory, against the same calls in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def calls(L, q, n, seed, gates):
    r = np.random.default_rng(seed)
    lib = L.lib
    for g in range(gates):
        a, b, c = (int(v) for v in r.permutation(n)[:3])
        kind, t = g % 6, float(r.uniform(-3, 3))
        if kind == 0:
            lib.rotateY(q, a, t)
        elif kind == 1:
            lib.controlledNot(q, a, b)
        elif kind == 2:
            lib.controlledPhaseShift(q, a, b, t)
        elif kind == 3:
            L.multiRotatePauli(q, sorted([a, b, c]), [1, 3, 2], t)
        elif kind == 4:
            lib.rotateX(q, a, t)
        else:
            z = r.normal(size=(4, 4)) + 1j * r.normal(size=(4, 4))
            L.multiQubitUnitary(q, [a, b], np.linalg.qr(z)[0])


@pytest.mark.parametrize("n", [6, 12, 14, 19, 20, 21])
@pytest.mark.parametrize("width", [4, 5, 6])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_flushes_match_fp64(gpulib, n, width, precision):
    L = gpulib
    lib = L.lib
    assert lib.quest_gb300_setTensorCorePrecision(precision) == 0
    lib.quest_gb300_setCaptureFusion(width)
    try:
        direct, cap = L.create(n), L.create(n)
        assert lib.quest_gb300_setCapture(cap, 1) == 0
        # two circuits of one shape, a longer one (memory grows), the first again
        for seed, gates in ((1, 24), (1, 24), (2, 90), (1, 24)):
            for q in (direct, cap):
                lib.initPlusState(q)
                calls(L, q, n, seed, gates)
            a, b = L.amps(direct).copy(), L.amps(cap).copy()
            # a pass (at most one a gate) rounds its input's parts to 2^-21 of
            # each (split-BF16 2^-17) and sums up to 64 of them: 2^3 of that
            # in norm, and in no entry more
            tol = (gates + 1) * 8 * (2.0 ** -17 if precision == 1 else 2.0 ** -21)
            assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)
            assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(a))
        L.destroy(cap)
        L.destroy(direct)
    finally:
        lib.quest_gb300_setTensorCorePrecision(0)
        lib.quest_gb300_setCaptureFusion(6)
