"""More one-launch plans alive than there are shared error words
(csrc/fused_small.cu), and words that are given back and out again; a flush of
one pass, which has no such plan."""
import numpy as np
import pytest

from quantumlab_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_many_plans(gpulib):
    L, n = gpulib, 10
    q = L.lib.quest_gb300_createQuregF32(n)
    ops = W.c2_circuit(n=n, layers=1, seed=1)
    want = None
    for _ in range(2):
        plans = []
        for i in range(1040):
            p = L.plan(n, 6, ops)
            plans.append(p)
            L.lib.quest_gb300_initZeroStateF32(q)
            assert L.lib.quest_gb300_applyPlanF32(q, p) == 0
            if i % 260 == 0 or i >= 1022:
                got = L.amps_f32(q, n)
                want = got if want is None else want
                assert np.array_equal(got, want)
        for p in plans:
            L.lib.quest_gb300_planDestroy(p)
    L.lib.quest_gb300_destroyQuregF32(q)


@pytest.mark.parametrize("n", [10, 13, 19])
def test_flush_of_one_pass(gpulib, n):
    L = gpulib
    r = np.random.default_rng(n)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    direct, cap = L.create(n), L.create(n)
    assert L.lib.quest_gb300_setCapture(cap, 1) == 0
    for targets in ([n - 1], [0, n - 1], [1, 2, 3, 4], list(range(n - 5, n))):
        u = np.linalg.qr(r.normal(size=(1 << len(targets),) * 2) + 1j * r.normal(size=(1 << len(targets),) * 2))[0]
        for q in (direct, cap):
            L.set_amps(q, psi)
            L.multiQubitUnitary(q, targets, u)
        a, b = L.amps(direct).copy(), L.amps(cap).copy()
        # as test_gpu_device_operands.py: parts of 2^-21, 2^3 of that in norm
        assert np.linalg.norm(a - b) <= 2 * 8 * 2.0 ** -21
    L.destroy(cap)
    L.destroy(direct)
