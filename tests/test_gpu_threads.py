"""Calls from two host threads on registers of their own.  The kernels' launch
configurations depend on the register's size; what one thread's launch needs
must not be taken back by the other's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(n):
    r = np.random.default_rng(n)
    z = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    return z / np.linalg.norm(z)


def gates(L, q, n, rounds):
    for k in range(rounds):
        L.lib.rotateAroundAxis(q, k % n, 0.3, axis())
        L.lib.rotateY(q, (k + 3) % n, 1.1)
        L.lib.rotateZ(q, (k + 5) % n, 0.7)
        L.lib.pauliX(q, (k + 7) % n)


def axis():
    from quantumlab_gb300.quest import Vector
    return Vector(1.0, 2.0, 3.0)


def trotter(L, q, n, rounds):
    codes = np.zeros((n, n), dtype=np.int32)
    for t in range(n):
        codes[t, t], codes[t, (t + 1) % n] = 1 + t % 3, 1 + t % 3
    h = L.pauli_hamil(codes, np.linspace(0.3, 1.0, n))
    ws = L.create(n)
    for _ in range(rounds):
        L.lib.applyTrotterCircuit(q, h, 0.2, 1, 1)
        L.lib.calcExpecPauliHamil(q, h, ws)
    L.destroy(ws)
    L.lib.destroyPauliHamil(h)


# grids of different even shares an SM; tiles of different sizes
@pytest.mark.parametrize("work,sizes,rounds", [(gates, (17, 18), 1500), (gates, (16, 19), 1500), (trotter, (9, 17), 300)])
def test_two_threads(gpulib, work, sizes, rounds):
    L = gpulib
    alone = []
    for n in sizes:
        q = L.create(n)
        L.set_amps(q, state(n))
        work(L, q, n, rounds)
        alone.append(L.amps(q).copy())
        L.destroy(q)
    regs = [L.create(n) for n in sizes]
    for q, n in zip(regs, sizes):
        L.set_amps(q, state(n))
    L.errors.clear()
    ready = threading.Barrier(len(sizes))

    def run(q, n):
        ready.wait()
        work(L, q, n, rounds)

    threads = [threading.Thread(target=run, args=(q, n)) for q, n in zip(regs, sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    errors = list(L.errors)
    L.errors.clear()
    got = [L.amps(q).copy() for q in regs]
    for q in regs:
        L.destroy(q)
    assert not errors, errors[:3]
    for a, b in zip(alone, got):
        assert np.array_equal(a, b)
