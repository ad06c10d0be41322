"""applyTrotterCircuit passes that follow one another and each have phase
tables of their own, in the same memory (csrc/pauli_tile.cu), on registers of
many tiles: every pass has to read the tables of its own run."""
import numpy as np
import pytest

from test_gpu_pauli_tile import rotate, rotations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,reps", [(18, 2), (20, 2), (21, 1)])
def test_tables_change_from_pass_to_pass(gpulib, n, reps):
    L = gpulib
    r = np.random.default_rng(n)
    codes, coeffs = [], []
    for run in range(6):
        # a diagonal run on qubits of its own, then a string whose X qubits do
        # not fit the tile of the run before
        pick = r.permutation(n)
        for _ in range(10):
            c = np.zeros(n, int)
            c[pick[r.permutation(10)[:2]]] = 3
            codes.append(c)
            coeffs.append(r.uniform(-2, 2))
        c = np.zeros(n, int)
        c[3 + (np.arange(7) + 7 * run) % (n - 3)] = 1
        codes.append(c)
        coeffs.append(r.uniform(0.2, 1))
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    q = L.create(n)
    L.set_amps(q, psi)
    h = L.pauli_hamil(np.array(codes, dtype=np.int32), np.array(coeffs))
    L.lib.applyTrotterCircuit(q, h, 0.3, 1, reps)
    got = L.amps(q).copy()
    L.lib.destroyPauliHamil(h)
    L.destroy(q)
    seq = rotations(coeffs, 0.3, 1, reps)
    want = psi
    for t, phi in seq:
        want = rotate(want, codes[t], phi)
    # at most 6 roundings a rotation on either side (see test_gpu_pauli_tile.py);
    # a table of another pass turns amplitudes by angles of order 1
    tol = 2 * 6 * 2.0 ** -53 * len(seq) * (1 + max(abs(p) for _, p in seq))
    assert np.linalg.norm(got - want) <= tol
