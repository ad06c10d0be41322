"""calcExpecPauliHamil by tiles (csrc/expec_tile.cu) against the terms one by
one in complex128."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expectation(psi, code):
    n = len(code)
    j = np.arange(psi.shape[0])
    x = sum(1 << q for q in range(n) if code[q] in (1, 2))
    yz = sum(1 << q for q in range(n) if code[q] in (2, 3))
    par = j & yz
    for sh in (16, 8, 4, 2, 1):
        par = par ^ (par >> sh)
    ny = sum(1 for c in code if c == 2)
    return float(np.real(np.vdot(psi, (-1j) ** ny * (1.0 - 2.0 * (par & 1)) * psi[j ^ x])))


def terms(n, seed):
    r = random.Random(seed)
    codes = [[0] * n]
    for _ in range(10):                                     # any string, narrow ones, diagonal ones
        codes.append([r.randrange(4) for _ in range(n)])
        codes.append([r.choice((0, 0, 0, 0, 1, 2, 3)) for _ in range(n)])
        codes.append([r.choice((0, 0, 3)) for _ in range(n)])
    for _ in range(6):                                      # several terms on one X/Y mask
        c = [r.choice((0, 0, 1, 2, 3)) for _ in range(n)]
        for _ in range(r.randint(2, 5)):
            codes.append([r.choice((1, 2)) if v in (1, 2) else r.choice((0, 3)) for v in c])
    for p in range(0, n - 2):                               # equal weights, half the pairs cancel
        for v in (1, 2):
            codes.append([v if q in (p, p + 2) else 3 if q == p + 1 else 0 for q in range(n)])
    co = [r.choice((-0.5, r.uniform(-2, 2))) for _ in codes]
    for k in range(len(codes) - 2 * max(0, n - 2), len(codes)):
        co[k] = -0.5
    return np.array(codes, dtype=np.int32), np.array(co)


def states(N, r):
    z = r.standard_normal(N) + 1j * r.standard_normal(N)
    yield z / np.linalg.norm(z)
    yield z * np.exp2(r.integers(-60, 1, N))                # every magnitude in one tile
    w = np.zeros(N, complex)
    w[r.integers(0, N)] = 0.8 - 0.6j                        # one amplitude, then few next to a large one
    yield w.copy()
    w += 1e-9 * z
    yield w
    yield z * 2.0 ** -400


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 10, 11, 12, 13, 15, 17])
def test_pauli_sums(gpulib, n):
    L = gpulib
    N = 1 << n
    for seed in range(2):
        codes, co = terms(n, 10 * n + seed)
        r = np.random.default_rng(seed)
        for psi in states(N, r):
            q, ws = L.create(n), L.create(n)
            L.set_amps(q, psi)
            h = L.pauli_hamil(codes, co)
            got = L.lib.calcExpecPauliHamil(q, h, ws)
            L.lib.destroyPauliHamil(h)
            L.destroy(q)
            L.destroy(ws)
            want = sum(c * expectation(psi, code) for code, c in zip(codes, co))
            # each side sums products rounded to 2^-53 of |psi_j psi_k| (by tiles
            # 2^-55 of the tile's largest times |psi|): the norm's square, at
            # most log2-deep sums of it, weighted by the coefficients
            scale = float(np.sum(np.abs(co))) * float(np.vdot(psi, psi).real)
            assert abs(got - want) <= 2 * (n + 4) * 2.0 ** -53 * scale, (n, seed, got, want)
