"""applyTrotterCircuit's passes of many rotations (csrc/pauli_tile.cu) against
the rotations applied one by one in complex128."""
import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def hamiltonian(n, seed):
    """Strings of every kind that the planner tells apart: weights 1 to n,
    neighbours with one X/Y mask (equal, opposite and other weights, commuting
    and not), runs of diagonal terms short and wide, angles beyond a turn."""
    r = random.Random(seed)
    codes, coeffs = [], []

    def add(c, w):
        codes.append(c)
        coeffs.append(w)
    for _ in range(14):
        kind = r.randrange(5)
        w = r.choice((0.3, 1.0, 5.0)) * r.uniform(-1, 1)
        if kind == 0:
            add([r.randrange(4) for _ in range(n)], w)
        elif kind == 1:
            for _ in range(r.randint(1, 6)):
                add([r.choice((0, 0, 3)) for _ in range(n)], r.uniform(-1, 1))
        elif kind == 2:
            a, b = sorted(r.sample(range(n), 2)) if n > 1 else (0, 0)
            for p, v in ((1, w), (2, r.choice((w, -w, 0.7 * w)))):
                add([p if q in (a, b) else 3 if a < q < b else 0 for q in range(n)], v)
        elif kind == 3:
            c = [r.choice((0, 0, 1, 2, 3)) for _ in range(n)]
            for _ in range(r.randint(2, 4)):
                add([(r.choice((1, 2)) if p in (1, 2) else r.choice((0, 3))) for p in c], r.choice((w, -w, r.uniform(-1, 1))))
        else:
            add([r.choice((0, 0, 0, 1, 2, 3)) for _ in range(n)], w)
    codes.append([0] * n)
    coeffs.append(0.4)
    return np.array(codes, dtype=np.int32), np.array(coeffs)


def rotations(coeffs, time, order, reps):
    """(term, angle / 2) in the order of application."""
    def run(t, o):
        if o == 1:
            return [(i, c * t) for i, c in enumerate(coeffs)]
        if o == 2:
            half = run(t / 2, 1)
            return half + half[::-1]
        p = 1 / (4 - 4 ** (1 / (o - 1)))
        return run(p * t, o - 2) * 2 + run((1 - 4 * p) * t, o - 2) + run(p * t, o - 2) * 2
    return run(time / reps, order) * reps


def rotate(psi, code, phi, conj=False):
    n = len(code)
    if not any(code):
        return psi
    j = np.arange(psi.shape[0])
    x = sum(1 << q for q in range(n) if code[q] in (1, 2))
    yz = sum(1 << q for q in range(n) if code[q] in (2, 3))
    ny = sum(1 for c in code if c == 2)
    par = j & yz
    for sh in (16, 8, 4, 2, 1):
        par = par ^ (par >> sh)
    g = (-1j) ** (ny + 1)
    if conj:
        g = g.conjugate()
    sign = 1.0 - 2.0 * (par & 1)
    shape = (-1,) + (1,) * (psi.ndim - 1)
    return math.cos(phi) * psi + g * math.sin(phi) * sign.reshape(shape) * psi[j ^ x]


@pytest.mark.parametrize("n,order,reps,time,density", [
    (1, 2, 1, 0.3, False), (2, 1, 2, 0.3, False), (3, 2, 1, 0.4, False), (4, 2, 2, 0.4, False), (5, 4, 1, 0.3, False),
    (8, 2, 1, 0.7, False), (11, 1, 2, 0.2, False), (13, 2, 2, 0.3, False), (14, 4, 1, 0.5, False), (17, 1, 1, 3.0, False),
    (19, 2, 1, 0.1, False), (2, 1, 2, 0.3, True), (3, 2, 1, 0.2, True), (6, 2, 2, 0.4, True), (8, 1, 1, 0.4, True)])
def test_rotations_against_complex128(gpulib, n, order, reps, time, density):
    L = gpulib
    for seed in range(3):
        codes, coeffs = hamiltonian(n, 100 * n + seed)
        r = np.random.default_rng(seed)
        N = 1 << (2 * n if density else n)
        psi = r.standard_normal(N) + 1j * r.standard_normal(N)
        psi[r.integers(0, N, N // 4)] = 0.0
        psi /= np.linalg.norm(psi)
        q = L.create(n, density)
        L.set_amps(q, psi)
        h = L.pauli_hamil(codes, coeffs)
        L.lib.applyTrotterCircuit(q, h, time, order, reps)
        got = L.amps(q).copy()
        L.lib.destroyPauliHamil(h)
        L.destroy(q)
        seq = rotations(coeffs, time, order, reps)
        want = psi.reshape(1 << n, -1).T.copy() if density else psi      # rows first
        for t, phi in seq:
            want = rotate(want, codes[t], phi)
        if density:
            want = want.T.copy()                                         # columns first
            for t, phi in seq:
                want = rotate(want, codes[t], phi, conj=True)
            want = want.reshape(-1)
        # each side rounds a rotation's result at most three times, and its
        # coefficients (cosine, sine) and their angle once: 6 x 2^-53 a rotation
        tol = 2 * 6 * 2.0 ** -53 * max(1, len(seq)) * (2 if density else 1) * (1 + np.max(np.abs([p for _, p in seq])))
        assert np.linalg.norm(got - want) <= tol, (n, seed, np.linalg.norm(got - want), tol)
