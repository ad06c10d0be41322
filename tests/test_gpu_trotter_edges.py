"""applyTrotterCircuit at its edges: orders with millions of rotations, angles
that are not finite or of many turns, single rotations."""
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


@pytest.mark.parametrize("n", [2, 6, 9, 13])
@pytest.mark.parametrize("time,weight", [(math.inf, 0.5), (math.nan, 0.5), (0.1, math.inf), (0.1, math.nan), (0.1, 1e200)])
def test_angles_that_are_not_finite_show(gpulib, n, time, weight):
    """Every amplitude that such a rotation acts on becomes NaN, zeros too."""
    z = np.zeros(1 << n, complex)
    z[0] = 1.0
    for codes in ([[3] + [0] * (n - 1), [0, 3] + [0] * (n - 2)], [[1] + [0] * (n - 1), [3, 1] + [0] * (n - 2)]):
        got = apply(gpulib, n, codes, [weight, 0.25], z, time, 1, 1)
        if math.isfinite(time * weight):
            assert np.isfinite(got).all() and abs(np.vdot(got, got) - 1) < 1e-12
        else:
            assert np.isnan(got.real).all() and np.isnan(got.imag).all()


@pytest.mark.parametrize("n", [4, 9, 13])
@pytest.mark.parametrize("scale", [50.0, 1e3, 1e7, 1e9, 1e15, 1e200])
def test_angles_of_many_turns(gpulib, n, scale):
    """Rotations of many turns next to ordinary ones that merge with them."""
    r = np.random.default_rng(n)
    codes, coeffs = [], []
    for _ in range(4):
        x = [int(v) for v in r.choice((0, 0, 1, 2), n)]
        for w in (scale * r.uniform(0.5, 1), 0.3, -0.2 * scale):
            codes.append([v if v else int(r.choice((0, 3))) for v in x])
            coeffs.append(w)
        for w in (scale * r.uniform(0.5, 1), 0.3):
            codes.append([int(v) for v in r.choice((0, 3), n)])
            coeffs.append(w)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    got = apply(gpulib, n, codes, coeffs, psi, 1.0, 1, 1)
    want = psi
    for t, phi in rotations(coeffs, 1.0, 1, 1):
        want = rotate(want, codes[t], phi)                  # by the cosine and sine of the whole angle
    assert np.linalg.norm(got - want) <= 2 * 6 * 2.0 ** -53 * len(codes) * 2


@pytest.mark.parametrize("n", [1, 2, 4, 9, 12, 13])
def test_single_and_wide_rotations(gpulib, n):
    """One rotation, and strings with more X/Y qubits than a tile: the same
    kernels as multiRotatePauli, so the same bits."""
    L = gpulib
    r = np.random.default_rng(n)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    wide = [[int(v) for v in r.integers(1, 3, n)] for _ in range(3)]
    for codes, coeffs in (([wide[0]], [0.7]), ([[3] * n], [0.7]), (wide, [0.3, -1.1, 0.6])):
        got = apply(L, n, codes, coeffs, psi, 0.4, 1, 1)
        want = psi
        for t, phi in rotations(coeffs, 0.4, 1, 1):
            want = rotate(want, codes[t], phi)
        assert np.linalg.norm(got - want) <= 12 * 2.0 ** -53 * len(codes) * 2
        if len(codes) == 1:
            q = L.create(n)
            L.set_amps(q, psi)
            L.multiRotatePauli(q, list(range(n)), codes[0], 2 * 0.4 * coeffs[0])
            assert np.array_equal(got, L.amps(q))
            L.destroy(q)
