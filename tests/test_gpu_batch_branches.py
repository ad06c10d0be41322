"""A Trotter batch of more classes than branches of its graph: every run, the
first one in stream order, gives the same energies and states."""
import ctypes as C

import numpy as np
import pytest

from quantumlab_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes,qubits", [(2, 12), (17, 12), (70, 12), (3, 20)])
def test_runs_agree(gpulib, classes, qubits):
    L, lib = gpulib, gpulib.lib
    b = lib.quest_gb300_trotterBatchCreate(qubits, 2 * classes)
    for i in range(2 * classes):                            # two instances a class, of its own step count
        codes, coeffs, _ = W.hubbard_terms(qubits // 2, 1.0 + 0.1 * i, 1.0)
        h = L.pauli_hamil(codes, coeffs)
        assert lib.quest_gb300_trotterBatchSetInstance(b, i, h, 0.5, 1, 2 + i // 2, W.neel_index(qubits // 2)) == 0
        lib.destroyPauliHamil(h)
    runs = []
    q = L.create(qubits)
    for _ in range(3):
        e = np.zeros(2 * classes)
        assert lib.quest_gb300_trotterBatchRun(b, e.ctypes.data_as(C.POINTER(C.c_double))) == 0
        states = []
        for i in (0, classes, 2 * classes - 1):
            assert lib.quest_gb300_trotterBatchCopyState(b, i, q) == 0
            states.append(L.amps(q).copy())
        runs.append((e, states))
    assert lib.quest_gb300_trotterBatchNumClasses(b) == classes
    for e, states in runs[1:]:
        assert np.array_equal(e, runs[0][0])
        for x, y in zip(states, runs[0][1]):
            assert np.array_equal(x, y)
    L.destroy(q)
    lib.quest_gb300_trotterBatchDestroy(b)
