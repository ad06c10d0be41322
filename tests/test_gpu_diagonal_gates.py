"""Diagonal gates (fixed point where the coefficients allow it, FP64 otherwise)
against numpy, amplitude by amplitude, on amplitudes of every magnitude."""
import cmath
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ANGLES = [0.0, 1e-9, 0.05, 0.0626, 0.7, math.pi / 2, math.pi - 0.03, math.pi, 3.0, -2.2, 6.2, 12.0]


def state(N, seed):
    r = np.random.default_rng(seed)
    z = (r.standard_normal(N) + 1j * r.standard_normal(N)) * np.exp2(r.integers(-90, 3, N))
    z[r.integers(0, N, N // 8 + 1)] = 0
    z.real[r.integers(0, N, N // 8 + 1)] *= 2.0 ** -70          # one part far below the other
    z[r.integers(0, N, 2)] *= 2.0 ** -900
    return z


@pytest.mark.parametrize("n", [1, 2, 3, 5, 12])
def test_diagonal_gates(gpulib, n):
    L = gpulib
    N = 1 << n
    j = np.arange(N)
    bit = lambda q: (j >> q) & 1  # noqa: E731
    turn = lambda a, par: np.exp(1j * a * (par - 0.5))  # noqa: E731
    for a in ANGLES:
        cases = []
        for q in range(n):
            c, d = (q + 1) % n, (q + 2) % n
            cases.append(("phaseShift", lambda r, q=q: L.lib.phaseShift(r, q, a), np.where(bit(q) == 1, cmath.exp(1j * a), 1)))
            cases.append(("rotateZ", lambda r, q=q: L.lib.rotateZ(r, q, a), turn(a, bit(q))))
            if n > 1:
                cases.append(("controlledPhaseShift", lambda r, q=q, c=c: L.lib.controlledPhaseShift(r, c, q, a),
                              np.where(bit(q) & bit(c) == 1, cmath.exp(1j * a), 1)))
                cases.append(("controlledRotateZ", lambda r, q=q, c=c: L.lib.controlledRotateZ(r, c, q, a),
                              np.where(bit(c) == 1, turn(a, bit(q)), 1)))
                cases.append(("multiRotateZ", lambda r, q=q, c=c: L.multiRotateZ(r, [q, c], a), turn(a, bit(q) ^ bit(c))))
            if n > 2:
                cases.append(("multiControlledMultiRotateZ", lambda r, q=q, c=c, d=d: L.multiControlledMultiRotateZ(r, [d], [q, c], a),
                              np.where(bit(d) == 1, turn(a, bit(q) ^ bit(c)), 1)))
                m = np.diag([cmath.exp(1j * a), cmath.exp(0.4j - 2j * a)])
                cases.append(("multiControlledUnitary", lambda r, q=q, c=c, m=m: L.multiControlledUnitary(r, [c], q, m),
                              np.where(bit(c) == 1, np.where(bit(q) == 1, m[1, 1], m[0, 0]), 1)))
        for k, (name, call, factor) in enumerate(cases):
            z = state(N, 7 * k + n)
            reg = L.create(n)
            L.set_amps(reg, z)
            call(reg)
            got = L.amps(reg).copy()
            L.destroy(reg)
            # both sides: the factor's parts to half an ulp, two products and a
            # sum: (1 + 2) x 2^-53 of |z| each, and the smallest subnormal
            tol = 6 * 2.0 ** -53 * np.abs(z) + 2.0 ** -1073
            assert np.all(np.abs(got - factor * z) <= tol), (name, a, n)
