"""applyTrotterCircuit at its edges: orders with millions of rotations, angles
that are not finite, single rotations."""
import math
import resource

import numpy as np
import pytest

from test_gpu_pauli_tile import rotate, rotations

pytestmark = pytest.mark.gpu


def apply(L, n, codes, coeffs, psi, time, order, reps, density=False):
    q = L.create(n, density)
    L.set_amps(q, psi)
    h = L.pauli_hamil(np.array(codes, dtype=np.int32), np.array(coeffs, dtype=float))
    L.lib.applyTrotterCircuit(q, h, time, order, reps)
    got = L.amps(q).copy()
    L.lib.destroyPauliHamil(h)
    L.destroy(q)
    return got


def test_high_orders_in_bounded_memory(gpulib):
    """Order 18: 5^8 times the 4 rotations of order 2, 75 MB as one list."""
    n, codes, coeffs = 4, [[1, 0, 0, 0], [3, 3, 0, 0]], [0.3, 0.2]
    psi = np.ones(16, complex) / 4
    apply(gpulib, n, codes, coeffs, psi, 0.1, 4, 1)
    before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
    got = apply(gpulib, n, codes, coeffs, psi, 0.1, 18, 1)
    grown = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before          # KB
    assert grown < 40 << 10, grown
    # a high order is the evolution itself; 1.5 million rotations, each off by
    # at most 6 roundings
    H = np.zeros((16, 16))
    for c, w in zip(codes, coeffs):
        m = np.eye(1)
        for p in c[::-1]:
            m = np.kron(m, [np.eye(2), [[0, 1], [1, 0]], None, np.diag([1, -1])][p])
        H += w * m
    e, v = np.linalg.eigh(H)
    want = v @ (np.exp(-0.1j * e) * (v.T @ psi))
    assert np.linalg.norm(got - want) <= 6 * 2.0 ** -53 * 4 * 5 ** 8
