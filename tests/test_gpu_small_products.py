"""Inner products and Pauli expectation values whose products are all far
smaller than the amplitudes that they are made of: every product has to keep
FP64's precision relative to itself, not to the largest amplitude around it
(csrc/fixed_sum.cuh, csrc/reduce.cu, csrc/expec_tile.cu)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = (0.3, 1e-3, 1e-6, 1e-10, 1e-13, math.pi * 1e-16, 1e-20, 1e-40)


def bound(n, products):
    # both sides round each product once and sum at most (n + 8)-deep
    return 2 * (n + 8) * 2.0 ** -53 * math.fsum(products) + 2.0 ** -1060


def near_basis(n, seed, eps):
    """Pairs of states close to two different basis states, neighbours first;
    the rest zero, tiny, or of every magnitude below eps, complex or real."""
    r = np.random.default_rng(seed)
    N = 1 << n
    for a, b in ((0, 1), (1, 0), (N - 2, N - 1), (0, N - 1), tuple(int(v) for v in r.permutation(N)[:2])):
        if a == b:
            continue
        for phase in (1.0, 1j, np.exp(0.7j)):
            for rest in range(3):
                z = r.standard_normal((2, N)) + 1j * r.standard_normal((2, N))
                if rest == 0:
                    z[:] = 0
                elif rest == 1:
                    z *= eps
                else:
                    z = np.real(z) * eps * np.exp2(r.integers(-60, 1, (2, N))) + 0j
                z[0, a], z[0, b] = phase, z[0, b] + 0
                z[1, b], z[1, a] = 1.0, eps
                yield z[0], z[1]


@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 13])
@pytest.mark.parametrize("eps", EPS)
def test_nearly_orthogonal_states(gpulib, n, eps):
    L = gpulib
    bra, ket = L.create(n), L.create(n)
    for u, v in near_basis(n, n, eps):
        L.set_amps(bra, u)
        L.set_amps(ket, v)
        got = L.lib.calcInnerProduct(bra, ket)
        re = np.concatenate([u.real * v.real, u.imag * v.imag])
        im = np.concatenate([u.real * v.imag, -u.imag * v.real])
        assert abs(got.real - math.fsum(re)) <= bound(n, np.abs(re)), (n, eps)
        assert abs(got.imag - math.fsum(im)) <= bound(n, np.abs(im)), (n, eps)
    L.destroy(bra)
    L.destroy(ket)


@pytest.mark.parametrize("eps", EPS)
def test_nearly_orthogonal_density_matrices(gpulib, eps):
    L, n = gpulib, 4
    a, b = L.create(n, True), L.create(n, True)
    for u, v in near_basis(2 * n, 3, eps):
        L.set_amps(a, u)
        L.set_amps(b, v)
        p = np.concatenate([u.real * v.real, u.imag * v.imag])
        assert abs(L.lib.calcDensityInnerProduct(a, b) - math.fsum(p)) <= bound(2 * n, np.abs(p))
    L.destroy(a)
    L.destroy(b)


def magnitude(psi, code):
    """The products of an off-diagonal string's expectation value."""
    n = len(code)
    j = np.arange(psi.shape[0])
    x = sum(1 << q for q in range(n) if code[q] in (1, 2))
    yz = sum(1 << q for q in range(n) if code[q] in (2, 3))
    ny = sum(1 for c in code if c == 2)
    par = j & yz
    for sh in (16, 8, 4, 2, 1):
        par = par ^ (par >> sh)
    sign = 1.0 - 2.0 * (par & 1)
    k = j ^ x
    if ny % 2 == 0:
        p = np.concatenate([sign * psi.real * psi.real[k], sign * psi.imag * psi.imag[k]]) * (1 if ny % 4 == 0 else -1)
    else:
        p = np.concatenate([sign * psi.real * psi.imag[k], -sign * psi.imag * psi.real[k]]) * (1 if ny % 4 == 1 else -1)
    return p


@pytest.mark.parametrize("n", [2, 8, 10, 13, 16])
@pytest.mark.parametrize("eps", EPS)
def test_off_diagonal_strings(gpulib, n, eps):
    L = gpulib
    r = np.random.default_rng(n)
    q, ws = L.create(n), L.create(n)
    for seed in range(3):
        codes = [[1 if k == t else 0 for k in range(n)] for t in (0, 1, n - 1)]
        codes += [[2 if k == t else 0 for k in range(n)] for t in (0, n - 1)]
        for _ in range(4):
            c = [int(v) for v in r.choice((0, 0, 0, 1, 2, 3), n)]
            c[int(r.integers(n))] = int(r.integers(1, 3))
            codes.append(c)
        states = [s for pair in near_basis(n, seed, eps) for s in pair][seed::6]
        for psi in states[:8]:
            # the partner of a large amplitude under some string is small
            L.set_amps(q, psi)
            for code in codes:
                # and with a second string on the same X/Y mask, of another weight
                two = [c if c in (1, 2) else int(v) for c, v in zip(code, r.choice((0, 3), n))]
                co = np.array([0.7, -0.4])
                h = L.pauli_hamil(np.array([code, two], dtype=np.int32), co)
                got = L.lib.calcExpecPauliHamil(q, h, ws)
                L.lib.destroyPauliHamil(h)
                p = np.concatenate([w * magnitude(psi, c) for w, c in zip(co, (code, two))])
                assert abs(got - math.fsum(p)) <= bound(n, np.abs(p)), (n, eps, code, two, got, math.fsum(p))
    L.destroy(q)
    L.destroy(ws)
