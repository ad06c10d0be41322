"""calcProbOfAllOutcomes where most high qubits are measured: few or single
items a run, summed by warps (csrc/reduce.cu), on both sides of that line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cases():
    r = np.random.default_rng(3)
    for n in (9, 10, 13, 18):
        for left in (0, 1, 3, 4, 5):                        # unmeasured qubits from 8 up
            high = r.permutation(np.arange(8, n))
            if left >= len(high):
                continue
            for low in ([], [5], [0, 3, 6, 7], list(range(8))):
                yield n, [int(q) for q in r.permutation(np.concatenate([high[left:], low]).astype(int))]
    yield 6, [5, 0]
    yield 19, list(range(19))


@pytest.mark.parametrize("n,qubits", list(cases()))
def test_outcomes(gpulib, n, qubits):
    L, N = gpulib, 1 << n
    j = np.arange(N)
    o = sum(((j >> t) & 1) << b for b, t in enumerate(qubits))
    r = np.random.default_rng(n)
    z = r.standard_normal(N) + 1j * r.standard_normal(N)
    for psi in (z / np.linalg.norm(z), z * np.exp2(r.integers(-80, 4, N))):
        q = L.create(n)
        L.set_amps(q, psi)
        got = np.array(L.calcProbOfAllOutcomes(q, qubits))
        L.destroy(q)
        p = psi.real ** 2 + psi.imag ** 2
        want = np.zeros(1 << len(qubits), np.longdouble)    # (a long sum in double would be the larger error)
        np.add.at(want, o, p.astype(np.longdouble))
        # sums of non-negative terms, at most (n + 8)-deep
        assert np.all(np.abs(got - want) <= 2 * (n + 8) * 2.0 ** -53 * want)
    if n <= 10:
        q = L.create(n, True)
        rho = r.standard_normal(N * N) + 1j * r.standard_normal(N * N)
        L.set_amps(q, rho)
        got = np.array(L.calcProbOfAllOutcomes(q, qubits))
        L.destroy(q)
        d = rho[j * (N + 1)].real
        want, scale = np.zeros(1 << len(qubits), np.longdouble), np.zeros(1 << len(qubits))
        np.add.at(want, o, d.astype(np.longdouble))
        np.add.at(scale, o, np.abs(d))
        assert np.all(np.abs(got - want) <= 2 * (n + 8) * 2.0 ** -53 * scale)
