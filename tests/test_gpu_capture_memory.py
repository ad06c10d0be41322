"""A captured register gives the device memory of a long flush back."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# the one-launch path (16 qubits) and tensor-core passes (20)
@pytest.mark.parametrize("n,gates", [(16, 6000), (20, 4000)])
def test_long_flush_gives_its_memory_back(gpulib, n, gates):
    L = gpulib
    q = L.create(n)
    assert L.lib.quest_gb300_setCapture(q, 1) == 0
    r = np.random.default_rng(n)

    def circuit(count):
        for _ in range(count):
            a, b = (int(v) for v in r.permutation(n)[:2])
            L.lib.rotateY(q, a, float(r.uniform(-3, 3)))
            L.lib.controlledRotateX(q, a, b, float(r.uniform(-3, 3)))

    circuit(20)
    before = L.lib.calcTotalProb(q)                         # the register's own FP32 copy and a small plan
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    circuit(gates)
    after = L.lib.calcTotalProb(q)
    kept = free - torch.cuda.mem_get_info()[0]
    assert abs(before - 1) < 1e-4 and abs(after - 1) < 1e-2
    assert kept <= 20 << 20, kept
    circuit(20)                                             # and goes on
    assert abs(L.lib.calcTotalProb(q) - 1) < 1e-2
    L.destroy(q)
