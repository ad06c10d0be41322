"""Inner products whose products are all far smaller than the amplitudes that
they are made of: every product has to keep FP64's precision relative to
itself, not to the largest amplitude around it (csrc/fixed_sum.cuh)."""
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
