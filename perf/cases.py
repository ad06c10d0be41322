"""Performance cases: what a program built on this library has it do, through
the calls that such a program makes (the QuEST C API and its extensions, as
bound by quantumlab_gb300.QuESTLibrary).

Registers live on the GPU.  A pass returns the register's own amplitudes as
tensors over the same device memory.  Results of the FP32 engine are kept as
float32, the precision they carry.
"""
import ctypes as C
import math

import numpy as np
import torch

import quantumlab_gb300 as qg
from quantumlab_gb300 import workloads as W
from quantumlab_gb300.quest import Complex, matrix2

KINDS = ("circuit", "ansatz", "trotter", "noise", "readout", "planned", "captured", "trotter_batch", "swap_tests")


def listed():
    return [
        # The smallest register a program simulates one at a time (one swap test of 16-vectors, a toy
        # circuit): each call is a launch, so call and launch cost is all there is.
        {"name": "circuit_9q", "kind": "circuit", "n": 9, "layers": 4, "dense_start": False},
        # The plain FP64 random circuit at the size the repository quotes it (20 qubits, state in L2).
        {"name": "circuit_20q", "kind": "circuit", "n": 20, "layers": 6, "dense_start": False},
        # The same gates on a state of 1 GiB, mid-circuit (all amplitudes nonzero): every gate streams it.
        {"name": "circuit_26q", "kind": "circuit", "n": 26, "layers": 1, "dense_start": True},
        # A variational circuit of the rotations, controlled rotations and phases that the lab's gate
        # dispatcher issues, odd register size, state as large as L2.
        {"name": "ansatz_23q", "kind": "ansatz", "n": 23, "layers": 1, "dense_start": True},
        # One Trotter step of a Fermi-Hubbard chain in FP64: one call, one Pauli rotation per term.
        {"name": "trotter_22q", "kind": "trotter", "sites": 11, "order": 2, "reps": 1, "time": 0.1},
        # One layer of the noisy density-matrix circuit: gates and three channels on every qubit.
        {"name": "noise_12q", "kind": "noise", "n": 12, "layers": 1, "start_layers": 1},
        # What is read at the end of a Hamiltonian simulation: energy, norm, occupations, joint
        # outcomes, overlap with another state.
        {"name": "readout_24q", "kind": "readout", "sites": 12, "time": 0.35},
        # A compiled fusion plan on a small register (a variational loop): passes of a few microseconds.
        {"name": "planned_16q", "kind": "planned", "n": 16, "layers": 8, "precision": 0},
        # A compiled plan on a large register: tensor-core passes with control qubits, streaming HBM.
        {"name": "planned_26q", "kind": "planned", "n": 26, "layers": 6, "precision": 0},
        # The lab unchanged with op-stream capture on: calls queued, planned, fused and applied.
        {"name": "captured_20q", "kind": "captured", "n": 20, "layers": 8, "precision": 0},
        # A grid of Hubbard instances of 10, 20 and 100 steps run as one batch.
        {"name": "trotter_batch_16q", "kind": "trotter_batch", "sites": 8, "order": 1, "per_dt": 3, "precision": 0},
        # QKMeans distances: every vector against 16 centroids, circuits of 9 to 21 qubits.
        {"name": "swap_tests_16k", "kind": "swap_tests", "count": 1024, "dmin": 4, "dmax": 10},
    ]


def draw(rng):
    kind = rng.choice(KINDS)
    if kind in ("circuit", "ansatz"):
        n = rng.randint(6, 25)
        return {"kind": kind, "n": n, "layers": 1 if n > 22 else rng.randint(1, 4), "dense_start": rng.random() < 0.5}
    if kind == "trotter":
        return {"kind": kind, "sites": rng.randint(4, 11), "order": rng.choice((1, 2)), "reps": rng.choice((1, 2)),
                "time": round(rng.uniform(0.02, 0.3), 3)}
    if kind == "noise":
        return {"kind": kind, "n": rng.randint(4, 11), "layers": rng.choice((1, 2)), "start_layers": rng.randint(0, 3)}
    if kind == "readout":
        return {"kind": kind, "sites": rng.randint(5, 12), "time": round(rng.uniform(0.1, 1.0), 3)}
    if kind == "planned":
        return {"kind": kind, "n": rng.randint(11, 25), "layers": rng.randint(3, 8), "precision": rng.choice((0, 0, 1, 2))}
    if kind == "captured":
        return {"kind": kind, "n": rng.randint(10, 21), "layers": rng.randint(3, 8), "precision": rng.choice((0, 0, 2))}
    if kind == "trotter_batch":
        return {"kind": kind, "sites": rng.randint(6, 8), "order": rng.choice((1, 2)), "per_dt": rng.randint(1, 3),
                "precision": rng.choice((0, 0, 2))}
    d = sorted((rng.randint(2, 10), rng.randint(2, 10)))
    return {"kind": kind, "count": int(round(math.exp(rng.uniform(math.log(8), math.log(1000))))), "dmin": d[0], "dmax": d[1]}


# ------------------------------------------------------------------ handles
class Handle:
    """A library object that is given back when the last tensor or state that uses it goes."""

    def __init__(self, value, free):
        self.value, self.free = value, free

    def __del__(self):
        self.free(self.value)


class DeviceDoubles:
    """An FP64 array of a register's device memory, for torch.as_tensor (which keeps `owner`)."""

    def __init__(self, owner, pointer, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (C.cast(pointer, C.c_void_p).value, False),
                                         "version": 3}


class Register:
    def __init__(self, n, density=False):
        L = qg.load()
        self.q = L.create(n, density=density)
        self.handle = Handle(self.q, L.destroy)
        N = self.q.numAmpsTotal
        self.re = torch.as_tensor(DeviceDoubles(self.handle, self.q.deviceStateVec.real, N), device="cuda")
        self.im = torch.as_tensor(DeviceDoubles(self.handle, self.q.deviceStateVec.imag, N), device="cuda")

    def parts(self):
        return [self.re, self.im]

    def parts32(self):
        return [self.re.float(), self.im.float()]


def hamil(codes, coeffs):
    L = qg.load()
    return Handle(L.pauli_hamil(codes, coeffs), L.lib.destroyPauliHamil)


def random_state(N, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.randn(2, N, generator=g, device="cuda", dtype=torch.float64)
    return z / z.square().sum().sqrt()


# ------------------------------------------------------------------- inputs
def ansatz_ops(n, layers, seed):
    """A variational circuit: single-qubit rotations on every qubit, an entangling ring, controlled
    rotations and phases, one multi-controlled rotation (as in uniformly controlled rotations)."""
    r = W.Xoshiro(seed)
    ang = lambda: math.pi * (2 * r.uniform() - 1)  # noqa: E731
    ops = []
    for layer in range(layers):
        for q in range(n):
            ops += [("h", q), ("ry", q, ang()), ("rz", q, ang())] if layer % 2 == 0 else [("rx", q, ang()), ("ps", q, ang())]
        ops += [("cx", q, (q + 1) % n) for q in range(n)]
        ops += [(("crx", "cry", "crz")[q % 3], q, (q + 2) % n, ang()) for q in range(0, n, 2)]
        ops += [("cp", q, (q + 3) % n, ang()) for q in range(1, n, 2)]
        ops.append(("mscu", n - 1, n - 2, r.randint(n - 2), ang()))
        ops += [("mrz", q, (q + 1) % n, (q + 4) % n, ang()) for q in range(0, n, 4)]
    return ops


def ry_matrix(a):
    return np.array([[math.cos(a / 2), -math.sin(a / 2)], [math.sin(a / 2), math.cos(a / 2)]], dtype=np.complex128)


def circuit_ops(case, seed):
    if case["kind"] == "ansatz":
        return ansatz_ops(case["n"], case["layers"], seed)
    return W.c2_circuit(case["n"], case["layers"], seed)


def calls_of(q, ops):
    """The library calls of a gate list on register q: (function, arguments) pairs."""
    lib = qg.load().lib
    ints = lambda *v: (C.c_int * len(v))(*v)  # noqa: E731
    named = {"cx": lib.controlledNot, "cp": lib.controlledPhaseShift, "h": lib.hadamard, "ps": lib.phaseShift, "rx": lib.rotateX,
             "ry": lib.rotateY, "rz": lib.rotateZ, "crx": lib.controlledRotateX, "cry": lib.controlledRotateY,
             "crz": lib.controlledRotateZ, "deph": lib.mixDephasing, "depol": lib.mixDepolarising, "damp": lib.mixDamping}
    out = []
    for op in ops:
        if op[0] == "cu":
            out.append((lib.compactUnitary, (q, op[1], Complex(op[2], op[3]), Complex(op[4], op[5]))))
        elif op[0] == "mscu":
            out.append((lib.multiStateControlledUnitary, (q, ints(op[1], op[2]), ints(0, 1), 2, op[3], matrix2(ry_matrix(op[4])))))
        elif op[0] == "mrz":
            out.append((lib.multiRotateZ, (q, ints(*op[1:4]), 3, op[4])))
        else:
            out.append((named[op[0]], (q,) + tuple(op[1:])))
    return out


def hubbard(sites, seed):
    r = W.Xoshiro(seed)
    U, t = 1 + 7 * r.uniform(), 0.5 + r.uniform()
    codes, coeffs, _ = W.hubbard_terms(sites, U, t)
    return codes, coeffs


DTS = (0.1, 0.05, 0.01)      # 10, 20 and 100 steps of an evolution over time 1


def batch_instances(case, seed):
    """(codes, coeffs, steps) per instance: a grid over U and the time step."""
    return [hubbard(case["sites"], seed * 1000 + i) + (int(round(1 / DTS[i % 3])),) for i in range(3 * case["per_dt"])]


def swap_inputs(case, seed):
    _, _, vecs, centroids = W.gaussian_mixture_vectors(case["count"], 16, case["dmin"], case["dmax"], seed)
    return W.swap_test_pool(vecs, centroids, case["dmin"], case["dmax"])


READ_QUBITS = tuple(range(0, 10))


def prepare(case, seed):
    L = qg.load()
    lib, kind = L.lib, case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("circuit", "ansatz"):
        s["reg"] = Register(case["n"])
        if case["dense_start"]:
            s["start"] = Register(case["n"])
            z = random_state(1 << case["n"], seed)
            s["start"].re.copy_(z[0])
            s["start"].im.copy_(z[1])
        s["calls"] = calls_of(s["reg"].q, circuit_ops(case, seed))
    elif kind == "trotter":
        s["reg"] = Register(2 * case["sites"])
        s["hamil"] = hamil(*hubbard(case["sites"], seed))
    elif kind == "noise":
        n = case["n"]
        s["reg"], s["start"] = Register(n, density=True), Register(n, density=True)
        pure = Register(n)
        z = random_state(1 << n, seed)
        pure.re.copy_(z[0])
        pure.im.copy_(z[1])
        lib.initPureState(s["start"].q, pure.q)
        for call, args in calls_of(s["start"].q, W.c3_circuit(n, case["start_layers"], seed + 1)):
            call(*args)
        s["calls"] = calls_of(s["reg"].q, W.c3_circuit(n, case["layers"], seed))
        torch.cuda.synchronize()
    elif kind == "readout":
        n = 2 * case["sites"]
        s["reg"], s["other"], s["workspace"] = Register(n), Register(n), Register(n)
        s["hamil"] = hamil(*hubbard(case["sites"], seed))
        for reg, time in ((s["reg"], case["time"]), (s["other"], 0.8 * case["time"])):
            lib.initClassicalState(reg.q, W.neel_index(case["sites"]))
            lib.applyTrotterCircuit(reg.q, s["hamil"].value, time, 1, 1)
    elif kind == "planned":
        n = case["n"]
        s["reg"] = Register(n)
        s["q32"] = Handle(lib.quest_gb300_createQuregF32(n), lib.quest_gb300_destroyQuregF32)
        s["plan"] = Handle(L.plan(n, 6, W.c2_circuit(n, case["layers"], seed)), lib.quest_gb300_planDestroy)
    elif kind == "captured":
        s["reg"] = Register(case["n"])
        lib.quest_gb300_setCapture(s["reg"].q, 1)
        s["calls"] = calls_of(s["reg"].q, W.c2_circuit(case["n"], case["layers"], seed))
    elif kind == "trotter_batch":
        n, inst = 2 * case["sites"], batch_instances(case, seed)
        s["batch"] = Handle(lib.quest_gb300_trotterBatchCreate(n, len(inst)), lib.quest_gb300_trotterBatchDestroy)
        for i, (codes, coeffs, steps) in enumerate(inst):
            h = hamil(codes, coeffs)
            lib.quest_gb300_trotterBatchSetInstance(s["batch"].value, i, h.value, 1.0, case["order"], steps,
                                                    W.neel_index(case["sites"]))
        s["count"], s["reg"] = len(inst), Register(n)
        s["energies"] = np.zeros(len(inst))
    else:
        pool, offsets, dims, ia, ib = swap_inputs(case, seed)
        P = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
        s["batch"] = Handle(lib.quest_gb300_swapTestBatchCreate(P(pool, C.c_double), P(offsets, C.c_longlong), P(dims, C.c_int),
                                                                len(dims), P(ia, C.c_int), P(ib, C.c_int), len(ia)),
                            lib.quest_gb300_swapTestBatchDestroy)
        s["p0"] = np.zeros(len(ia))
    return s


def run(state):
    L = qg.load()
    lib, kind, case = L.lib, state["kind"], state["case"]
    if "precision" in case:
        lib.quest_gb300_setTensorCorePrecision(case["precision"])
    if kind in ("circuit", "ansatz", "noise"):
        reg = state["reg"]
        if "start" in state:
            lib.cloneQureg(reg.q, state["start"].q)
        else:
            lib.initZeroState(reg.q)
        for call, args in state["calls"]:
            call(*args)
        return reg.parts()
    if kind == "trotter":
        reg = state["reg"]
        lib.initClassicalState(reg.q, W.neel_index(case["sites"]))
        lib.applyTrotterCircuit(reg.q, state["hamil"].value, case["time"], case["order"], case["reps"])
        return reg.parts()
    if kind == "readout":
        q, n = state["reg"].q, 2 * case["sites"]
        overlap = lib.calcInnerProduct(state["other"].q, q)
        return {"energy": np.array([lib.calcExpecPauliHamil(q, state["hamil"].value, state["workspace"].q)]),
                "norm": np.array([lib.calcTotalProb(q)]),
                "occupations": np.array([lib.calcProbOfOutcome(q, t, 1) for t in range(n)]),
                "outcomes": L.calcProbOfAllOutcomes(q, READ_QUBITS),
                "overlap": np.array([overlap.real, overlap.imag])}
    if kind == "planned":
        q32, reg = state["q32"].value, state["reg"]
        lib.quest_gb300_initZeroStateF32(q32)
        lib.quest_gb300_applyPlanF32(q32, state["plan"].value)
        lib.quest_gb300_copyToQureg(q32, reg.q)
        return reg.parts32()
    if kind == "captured":
        reg = state["reg"]
        lib.initZeroState(reg.q)
        for call, args in state["calls"]:
            call(*args)
        total = lib.calcTotalProb(reg.q)
        return reg.parts32() + [np.array([total], dtype=np.float32)]
    if kind == "trotter_batch":
        e, reg = state["energies"], state["reg"]
        lib.quest_gb300_trotterBatchRun(state["batch"].value, e.ctypes.data_as(C.POINTER(C.c_double)))
        lib.quest_gb300_trotterBatchCopyState(state["batch"].value, state["count"] - 1, reg.q)
        return [e.astype(np.float32)] + reg.parts32()
    p0 = state["p0"]
    lib.quest_gb300_swapTestBatchRun(state["batch"].value, p0.ctypes.data_as(C.POINTER(C.c_double)))
    return p0.astype(np.float32)


# --------------------------------------------------------------------- work
def gate_work(op, N):
    """(bytes, flops) of one gate call on N FP64 amplitudes: the amplitudes it changes, read and
    written once; 28 flops per complex 2 x 2 product, 12 per real one, 6 per complex product."""
    k = op[0]
    if k == "cu":
        return 32 * N, 14 * N
    if k in ("h", "rx", "ry"):
        return 32 * N, 6 * N
    if k in ("rz", "mrz"):
        return 32 * N, 6 * N
    if k == "ps":
        return 16 * N, 3 * N
    if k == "cx":
        return 16 * N, 0
    if k in ("crx", "cry", "crz"):
        return 16 * N, 3 * N
    if k in ("cp", "mscu"):
        return 8 * N, 1.5 * N
    if k == "deph":
        return 16 * N, N
    return 32 * N, 2 * N                                  # depol, damp


def work(case):
    kind = case["kind"]
    if kind in ("circuit", "ansatz", "noise"):
        N = 1 << (case["n"] * (2 if kind == "noise" else 1))
        ops = W.c3_circuit(case["n"], case["layers"], 1) if kind == "noise" else circuit_ops(case, 1)
        b, f = (32 if kind == "noise" or case["dense_start"] else 16) * N, 0
        for op in ops:
            twice = 2 if kind == "noise" and op[0] in ("cu", "cx") else 1       # rows and columns
            x, y = gate_work(op, N)
            b, f = b + twice * x, f + twice * y
        return {"bytes": b, "flops": f}
    if kind == "trotter":
        N, T = 1 << (2 * case["sites"]), len(hubbard(case["sites"], 1)[1])
        calls = T * case["order"] * case["reps"]
        return {"bytes": 32 * N * calls + 16 * N, "flops": 6 * N * calls}
    if kind == "readout":
        N, codes = 1 << (2 * case["sites"]), hubbard(case["sites"], 1)[0]
        return {"bytes": 32 * N, "flops": N * (4 * len(codes) + 4 + 3 * 2 * case["sites"] + 4 + 8)}
    if kind in ("planned", "captured"):
        N = 1 << case["n"]
        flops = sum(gate_work(op, N)[1] for op in W.c2_circuit(case["n"], case["layers"], 1))
        return {"bytes": 16 * N if kind == "captured" else 8 * N, "flops": flops}
    if kind == "trotter_batch":
        N, T = 1 << (2 * case["sites"]), len(hubbard(case["sites"], 1)[1])
        steps = sum(int(round(1 / dt)) for dt in DTS) * case["per_dt"]
        return {"bytes": 8 * N * 3 * case["per_dt"] + 8 * N, "flops": 6 * N * T * case["order"] * steps}
    dims = range(case["dmin"], case["dmax"] + 1)
    tests = 16 * case["count"]
    return {"bytes": 4 * case["count"] * sum(1 << d for d in dims) / len(dims) + 8 * tests,
            "flops": 6 * tests * sum(1 << (2 * d) for d in dims) / len(dims)}


# -------------------------------------------------------------------- exact
def dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def c128(m):
    return torch.tensor(np.asarray(m, dtype=np.complex128), device=dev())


def index(N):
    return torch.arange(N, device=dev())


def parity(j, mask):
    p = j & mask
    for sh in (32, 16, 8, 4, 2, 1):
        p = p ^ (p >> sh)
    return 1.0 - 2.0 * (p & 1).double()


def apply2(psi, t, u, j, ctrl=0, want=0):
    """u on qubit t of the amplitudes whose bits under ctrl are want."""
    v = psi.view(-1, 2, 1 << t)
    a, b = v[:, 0], v[:, 1]
    new = torch.stack([u[0][0] * a + u[0][1] * b, u[1][0] * a + u[1][1] * b], 1).reshape(-1)
    return new if not ctrl else torch.where((j & ctrl) == want, new, psi)


def compact(a, b):
    return [[a, -b.conjugate()], [b, a.conjugate()]]


def rot(axis, a):
    c, s = math.cos(a / 2), math.sin(a / 2)
    return {"x": [[c, -1j * s], [-1j * s, c]], "y": [[c, -s], [s, c]], "z": [[c - 1j * s, 0], [0, c + 1j * s]]}[axis]


def conj2(u):
    return [[complex(x).conjugate() for x in row] for row in u]


def apply_op(psi, op, j, conj=False, shift=0):
    k = op[0]
    mat = (lambda u: conj2(u)) if conj else (lambda u: u)
    bit = lambda q: 1 << (q + shift)  # noqa: E731
    phase = lambda mask, a: torch.where((j & mask) == mask, psi * complex(math.cos(a), -math.sin(a) if conj else math.sin(a)), psi)  # noqa: E731
    if k == "cu":
        return apply2(psi, op[1] + shift, mat(compact(complex(op[2], op[3]), complex(op[4], op[5]))), j)
    if k == "h":
        f = math.sqrt(0.5)
        return apply2(psi, op[1] + shift, [[f, f], [f, -f]], j)
    if k in ("rx", "ry", "rz"):
        return apply2(psi, op[1] + shift, mat(rot(k[1], op[2])), j)
    if k in ("crx", "cry", "crz"):
        return apply2(psi, op[2] + shift, mat(rot(k[2], op[3])), j, bit(op[1]), bit(op[1]))
    if k == "cx":
        return psi[torch.where((j & bit(op[1])) != 0, j ^ bit(op[2]), j)]
    if k == "ps":
        return phase(bit(op[1]), op[2])
    if k == "cp":
        return phase(bit(op[1]) | bit(op[2]), op[3])
    if k == "mscu":
        return apply2(psi, op[3], rot("y", op[4]), j, bit(op[1]) | bit(op[2]), bit(op[2]))
    if k == "mrz":
        sgn = parity(j, bit(op[1]) | bit(op[2]) | bit(op[3]))
        return psi * torch.complex(torch.full_like(sgn, math.cos(op[4] / 2)), -math.sin(op[4] / 2) * sgn)
    raise ValueError(k)


def apply_channel(rho, op, n):
    t, p = op[1], op[2]
    v = rho.view(1 << (n - t - 1), 2, 1 << (n - 1), 2, 1 << t)        # column bit, row bit of qubit t
    out = v.clone()
    if op[0] == "deph":
        keep = 1 - 2 * p
    elif op[0] == "depol":
        level = 4 * p / 3
        keep = 1 - level
        mean = (v[:, 0, :, 0] + v[:, 1, :, 1]) / 2
        out[:, 0, :, 0] = keep * v[:, 0, :, 0] + level * mean
        out[:, 1, :, 1] = keep * v[:, 1, :, 1] + level * mean
    else:
        keep = math.sqrt(1 - p)
        out[:, 0, :, 0] = v[:, 0, :, 0] + p * v[:, 1, :, 1]
        out[:, 1, :, 1] = (1 - p) * v[:, 1, :, 1]
    out[:, 0, :, 1] = keep * v[:, 0, :, 1]
    out[:, 1, :, 0] = keep * v[:, 1, :, 0]
    return out.reshape(-1)


def pauli_masks(code):
    x = sum(1 << q for q, c in enumerate(code) if c in (1, 2))
    y = sum(1 << q for q, c in enumerate(code) if c == 2)
    z = sum(1 << q for q, c in enumerate(code) if c == 3)
    return x, y, z


def apply_pauli(psi, code, j):
    """P psi for a Pauli string (psi: ... x N)."""
    x, y, z = pauli_masks(code)
    out = psi[..., j ^ x] if x else psi
    return out * (parity(j, y | z) * 1.0) * ((-1j) ** bin(y).count("1"))


def trotter_state(psi, codes, coeffs, time, order, reps, j):
    """coeffs: M x T for psi M x N, or T for psi N."""
    coeffs = np.asarray(coeffs)
    for _ in range(reps):
        seq = list(range(len(codes)))
        for t in (seq if order == 1 else seq + seq[::-1]):
            a = 2 * time / reps / order * coeffs[..., t]
            c, s = np.cos(a / 2), np.sin(a / 2)
            if coeffs.ndim == 2:
                c, s = c128(c)[:, None], c128(s)[:, None]
            psi = c * psi - 1j * s * apply_pauli(psi, codes[t], j)
    return psi


def classical(n, i, rows=()):
    psi = torch.zeros(tuple(rows) + (1 << n,), dtype=torch.complex128, device=dev())
    psi[..., i] = 1
    return psi


def exact(case, seed):
    kind = case["kind"]
    if kind in ("circuit", "ansatz", "planned", "captured"):
        n = case["n"]
        j = index(1 << n)
        psi = torch.complex(*random_state(1 << n, seed)) if case.get("dense_start") else classical(n, 0)
        ops = circuit_ops(case, seed) if kind in ("circuit", "ansatz") else W.c2_circuit(n, case["layers"], seed)
        for op in ops:
            psi = apply_op(psi, op, j)
        out = [psi.real.clone(), psi.imag.clone()]
        return out + [np.array([float(psi.abs().square().sum())])] if kind == "captured" else out
    if kind == "trotter":
        n = 2 * case["sites"]
        codes, coeffs = hubbard(case["sites"], seed)
        psi = trotter_state(classical(n, W.neel_index(case["sites"])), codes, coeffs, case["time"], case["order"],
                            case["reps"], index(1 << n))
        return [psi.real.clone(), psi.imag.clone()]
    if kind == "noise":
        n = case["n"]
        psi = torch.complex(*random_state(1 << n, seed))
        rho = (psi.conj()[:, None] * psi[None, :]).reshape(-1)          # entry (row r, column c) at r + c 2^n
        j = index(1 << (2 * n))
        for op in W.c3_circuit(n, case["start_layers"], seed + 1) + W.c3_circuit(n, case["layers"], seed):
            if op[0] in ("cu", "cx"):
                rho = apply_op(apply_op(rho, op, j), op, j, conj=True, shift=n)
            else:
                rho = apply_channel(rho, op, n)
        return [rho.real.clone(), rho.imag.clone()]
    if kind == "readout":
        n = 2 * case["sites"]
        codes, coeffs = hubbard(case["sites"], seed)
        j = index(1 << n)
        psi, other = (trotter_state(classical(n, W.neel_index(case["sites"])), codes, coeffs, time, 1, 1, j)
                      for time in (case["time"], 0.8 * case["time"]))
        p = psi.abs().square()
        energy = sum(c * float((psi.conj() * apply_pauli(psi, code, j)).real.sum()) for code, c in zip(codes, coeffs))
        o = sum(((j >> q) & 1) << b for b, q in enumerate(READ_QUBITS))
        over = complex((other.conj() * psi).sum())
        return {"energy": np.array([energy]), "norm": np.array([float(p.sum())]),
                "occupations": np.array([float(p[(j >> t) & 1 == 1].sum()) for t in range(n)]),
                "outcomes": torch.zeros(1 << len(READ_QUBITS), dtype=torch.float64, device=dev()).index_add_(0, o, p),
                "overlap": np.array([over.real, over.imag])}
    if kind == "trotter_batch":
        n, inst = 2 * case["sites"], batch_instances(case, seed)
        j = index(1 << n)
        energies, last = np.zeros(len(inst)), None
        for d in range(3):
            members = list(range(d, len(inst), 3))
            codes, co = inst[d][0], np.array([inst[i][1] for i in members])
            psi = trotter_state(classical(n, W.neel_index(case["sites"]), (len(members),)), codes, co, 1.0, case["order"],
                                inst[d][2], j)
            for t, code in enumerate(codes):
                energies[members] += co[:, t] * (psi.conj() * apply_pauli(psi, code, j)).real.sum(-1).cpu().numpy()
            last = psi[-1] if members[-1] == len(inst) - 1 else last
        return [energies, last.real.clone(), last.imag.clone()]
    pool, offsets, dims, ia, ib = swap_inputs(case, seed)
    dots = np.array([np.dot(pool[offsets[a]:offsets[a] + (1 << dims[a])], pool[offsets[b]:offsets[b] + (1 << dims[b])])
                     for a, b in zip(ia, ib)])
    return (1 + dots ** 2) / 2
