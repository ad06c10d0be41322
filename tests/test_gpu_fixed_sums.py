"""Norms, outcome probabilities and inner products summed on the integer pipes
(csrc/fixed_sum.cuh) against numpy."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(N, seed):
    r = np.random.default_rng(seed)
    z = r.standard_normal(N) + 1j * r.standard_normal(N)
    yield z / np.linalg.norm(z)
    yield z * np.exp2(r.integers(-80, 4, N))
    w = np.zeros(N, complex)                              # mostly zeros, as after initClassicalState
    w[r.integers(0, N, 3)] = (0.6, 1e-9j, 0.8j)
    yield w
    yield z * 2.0 ** -515                                 # squares near the smallest numbers
    yield z * 2.0 ** 480


def close(got, want, scale, n):
    # products rounded to 2^-53 of the largest in their group of eight, sums at
    # most (n + 8)-deep; squares below 2^-1022 are subnormal
    return abs(got - want) <= 2 * (n + 8) * 2.0 ** -53 * scale + 2.0 ** -1060


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 9, 14])
def test_norms_probabilities_inner_products(gpulib, n):
    L, N = gpulib, 1 << n
    j = np.arange(N)
    for psi, phi in zip(states(N, n), list(states(N, n + 50))[::-1]):
        q, k = L.create(n), L.create(n)
        L.set_amps(q, psi)
        L.set_amps(k, phi)
        p = psi.real ** 2 + psi.imag ** 2
        total = math.fsum(p)
        assert close(L.lib.calcTotalProb(q), total, total, n)
        for t in range(n):
            zero = math.fsum(p[(j >> t) & 1 == 0])
            assert close(L.lib.calcProbOfOutcome(q, t, 0), zero, total, n), (n, t)
        got = L.lib.calcInnerProduct(k, q)
        prod = phi.conj() * psi
        scale = math.fsum(np.abs(psi)) * float(np.max(np.abs(phi)))
        scale = max(scale, math.fsum(np.abs(phi)) * float(np.max(np.abs(psi))))
        assert close(got.real, math.fsum(prod.real), scale, n) and close(got.imag, math.fsum(prod.imag), scale, n)
        L.destroy(q)
        L.destroy(k)


def test_infinities_and_nans_show(gpulib):
    L = gpulib
    for bad in (np.inf, np.nan):
        for at in (0, 5, 31):
            q = L.create(5)
            z = np.full(32, 0.1 + 0.1j)
            z[at] = complex(bad, 0.1)
            L.set_amps(q, z)
            assert not np.isfinite(L.lib.calcTotalProb(q))
            assert not np.isfinite(L.calcProbOfAllOutcomes(q, [0, 4])).all()
            L.destroy(q)


@pytest.mark.parametrize("n,qubits", [
    (1, [0]), (3, [2, 0]), (5, [0, 1, 2, 3, 4]), (8, [7, 0, 3]), (9, [8]), (9, [0, 8]), (11, list(range(10))), (12, [11, 10, 9]),
    (13, [5, 12, 0, 9]), (14, list(range(14))[::-1]), (16, [2, 3]), (16, [15, 14, 13, 12, 11, 10, 9, 8, 7, 6])])
def test_outcomes(gpulib, n, qubits):
    L, N = gpulib, 1 << n
    j = np.arange(N)
    o = sum(((j >> t) & 1) << b for b, t in enumerate(qubits))
    for psi in states(N, n):
        q = L.create(n)
        L.set_amps(q, psi)
        got = np.array(L.calcProbOfAllOutcomes(q, qubits))
        p = psi.real ** 2 + psi.imag ** 2
        want = np.zeros(1 << len(qubits))
        np.add.at(want, o, p)
        assert np.all(np.abs(got - want) <= 2 * (n + 8) * 2.0 ** -53 * np.sum(p) + 2.0 ** -1060)
        L.destroy(q)
    if n <= 9:
        q = L.create(n, True)
        r = np.random.default_rng(n)
        rho = r.standard_normal(N * N) + 1j * r.standard_normal(N * N)
        L.set_amps(q, rho)
        d = rho[j * (N + 1)].real
        want = np.zeros(1 << len(qubits))
        np.add.at(want, o, d)
        got = np.array(L.calcProbOfAllOutcomes(q, qubits))
        assert np.all(np.abs(got - want) <= 2 * (n + 8) * 2.0 ** -53 * np.sum(np.abs(d)))
        L.destroy(q)
