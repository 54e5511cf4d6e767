"""What the engine's speed is judged on: calls a user of the package makes,
over the sizes, precisions and circuit kinds of its tests, its benchmark and
its configurations.

listed() names the cases, draw() gives more of the same ranges, prepare()
builds what a caller holds before the call (circuits, states on the device,
plans), run() is one pass through the public API, work() counts what the pass
cannot do without, and exact() restates the result in 64 bits with torch.
"""

import math

import numpy as np
import torch

from qevedo_simulator_b200 import (Batch, Circuit, DeviceState, Plan, _native, estimate, run as run_circuit,
                                   statevector)
from qevedo_simulator_b200.simulator import plan_options

HALF_PI = math.pi / 2


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A few qubits in double precision, the default of statevector(): one
        # call of an interactive session or of a loop over small circuits.
        # Latency, launches and host work.
        {"name": "statevector_7q_c128", "kind": "statevector", "circuit": "mixed", "n": 7, "depth": 8, "bits": 64},
        # The full amplitude vector of the 4x5 grid circuit of depth 20.
        {"name": "statevector_20q_c64", "kind": "statevector", "circuit": "grid", "n": 20, "depth": 20, "bits": 32},
        # Mid-circuit measurement, reset and classical feedback, shot by shot.
        {"name": "dynamic_5q", "kind": "dynamic", "n": 5, "rounds": 5, "shots": 32, "bits": 32},
        # One energy of a small variational problem: an ansatz of 4 layers and
        # the transverse-field Ising Hamiltonian's 2n - 1 Pauli terms.
        {"name": "estimate_13q_c128", "kind": "estimate", "n": 13, "depth": 4, "bits": 64},
        # A program that drives the state gate by gate (a debugger, a
        # front end with its own scheduling): 1-6 qubit unitaries, diagonals
        # and 0-3 controls on any qubits, small and large states.
        {"name": "gates_17q_c128", "kind": "gates", "n": 17, "gates": 40, "bits": 64},
        {"name": "gates_28q_c64", "kind": "gates", "n": 28, "gates": 30, "bits": 32},
        # One-shot apply_ops with default settings in double precision.
        {"name": "oneshot_26q_c128", "kind": "oneshot", "circuit": "grid", "n": 26, "depth": 20, "bits": 64},
        # The 30-qubit depth-20 grid circuit from |0...0> through a plan, the
        # amplitudes left on the device in logical order.
        {"name": "plan_30q_c64", "kind": "plan", "circuit": "grid", "n": 30, "depth": 20, "bits": 32},
        # QFT of a general state through a plan (part of a larger algorithm).
        {"name": "evolve_28q_c64", "kind": "evolve", "circuit": "qft", "n": 28, "depth": 1, "bits": 32},
        # Expectations of a state on the device: every <Z>, and a Pauli sum.
        {"name": "observables_27q_c64", "kind": "observables", "n": 27, "terms": 24, "bits": 32},
        # A million shots of a 28-qubit state.
        {"name": "sample_28q_c64", "kind": "sample", "n": 28, "shots": 1000000, "counted": 0, "bits": 32},
        # One step of a loop over a batch of hardware-efficient ansatz
        # circuits of uneven width: new angles in, every <Z> out.
        {"name": "batch_384", "kind": "batch", "count": 384, "min_width": 10, "max_width": 22, "min_layers": 4,
         "max_layers": 12},
    ]


def draw(rng):
    kind = rng.choice(["statevector", "dynamic", "estimate", "gates", "gates", "oneshot", "plan", "plan", "evolve",
                       "evolve", "observables", "sample", "batch"])
    bits = rng.choice([32, 64])
    if kind == "statevector":
        return {"kind": kind, "circuit": rng.choice(["mixed", "grid", "qft"]), "n": rng.randint(2, 21),
                "depth": rng.randint(2, 24), "bits": bits}
    if kind == "dynamic":
        return {"kind": kind, "n": rng.randint(2, 14), "rounds": rng.randint(2, 6), "shots": rng.randint(4, 32),
                "bits": bits}
    if kind == "estimate":
        return {"kind": kind, "n": rng.randint(4, 22), "depth": rng.randint(2, 8), "bits": bits}
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(9, 28 if bits == 32 else 27), "gates": rng.randint(10, 40),
                "bits": bits}
    if kind == "oneshot":
        return {"kind": kind, "circuit": rng.choice(["mixed", "grid", "qft"]), "n": rng.randint(17, 26),
                "depth": rng.randint(5, 20), "bits": bits}
    if kind == "plan":
        return {"kind": kind, "circuit": rng.choice(["grid", "grid", "qft", "mixed"]), "n": rng.randint(20, 30),
                "depth": rng.randint(8, 20), "bits": 32}
    if kind == "evolve":
        return {"kind": kind, "circuit": rng.choice(["qft", "grid", "mixed"]),
                "n": rng.randint(18, 29 if bits == 32 else 26), "depth": rng.randint(4, 16), "bits": bits}
    if kind == "observables":
        return {"kind": kind, "n": rng.randint(16, 28 if bits == 32 else 27), "terms": rng.randint(8, 30),
                "bits": bits}
    if kind == "sample":
        return {"kind": kind, "n": rng.randint(12, 28 if bits == 32 else 27),
                "shots": int(round(math.exp(rng.uniform(math.log(100), math.log(1000000))))),
                # Outcomes as basis states, or counted by the bits of a few
                # measured qubits (every key then occurs).
                "counted": rng.choice([0, 3]), "bits": bits}
    low = rng.randint(4, 16)
    return {"kind": "batch", "count": int(round(math.exp(rng.uniform(math.log(16), math.log(384))))),
            "min_width": low, "max_width": rng.randint(low, 22), "min_layers": 3, "max_layers": rng.randint(4, 12)}


# ---------------------------------------------------------------- circuits
def program(kind, n, depth, seed):
    """A circuit as (gate name, parameters, qubits) in order."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    if kind == "grid":
        # sqrt(X), sqrt(Y) or sqrt(W) on every qubit, never a qubit's last
        # one again, then CZ on one of four coupler sets of the grid.
        rows = max(r for r in range(1, math.isqrt(n) + 1) if n % r == 0)
        cols = n // rows
        last = [-1] * n
        for layer in range(depth):
            for q in range(n):
                last[q] = int(rng.choice([g for g in range(3) if g != last[q]]))
                out.append([("rx", (HALF_PI,), (q,)), ("ry", (HALF_PI,), (q,)),
                            ("u", (HALF_PI, -math.pi / 4, math.pi / 4), (q,))][last[q]])
            offset = (layer // 2) % 2
            for r in range(rows):
                for c in range(cols):
                    q = r * cols + c
                    if layer % 2 == 0 and c % 2 == offset and c + 1 < cols:
                        out.append(("cz", (), (q, q + 1)))
                    if layer % 2 == 1 and r % 2 == offset and r + 1 < rows:
                        out.append(("cz", (), (q, q + cols)))
    elif kind == "qft":
        # A rotation of every qubit (the state before the transform is then
        # no basis state) and the transform without the final reversal.
        for q in range(n):
            out.append(("ry", (float(rng.random()) * math.tau,), (q,)))
        for t in reversed(range(n)):
            out.append(("h", (), (t,)))
            for c in reversed(range(t)):
                out.append(("cp", (math.pi / float(1 << (t - c)),), (c, t)))
    elif kind == "ansatz":
        for _ in range(depth):
            for q in range(n):
                out.append(("ry", (float(rng.random()) * math.tau,), (q,)))
                out.append(("rz", (float(rng.random()) * math.tau,), (q,)))
            for q in range(n - 1):
                out.append(("cx", (), (q, q + 1)))
    else:
        # `depth` gates per qubit of the standard set.
        names = ["h", "x", "rx", "ry", "rz", "u", "t", "sx", "cx", "cz", "cp", "swap", "ccx", "cswap"]
        for _ in range(depth * n):
            name = names[int(rng.integers(0, 14 if n >= 3 else 12 if n == 2 else 8))]
            width = {"cx": 2, "cz": 2, "cp": 2, "swap": 2, "ccx": 3, "cswap": 3}.get(name, 1)
            count = {"rx": 1, "ry": 1, "rz": 1, "u": 3, "cp": 1}.get(name, 0)
            out.append((name, tuple(float(x) * math.tau for x in rng.random(count)),
                        tuple(int(q) for q in rng.permutation(n)[:width])))
    return out


def circuit_of(prog, n, clbits=0):
    c = Circuit(n, clbits)
    for name, params, qubits in prog:
        if name == "measure":
            c.measure(*qubits)
        elif name == "reset":
            c.reset(*qubits)
        elif name == "feedback":
            c.feedback(params, *qubits)
        else:
            c.gate(name, list(qubits), params)
    return c


def dynamic_program(n, rounds, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    prog = program("mixed", n, 2, seed)
    for k in range(rounds):
        q, t = (int(x) for x in rng.permutation(n)[:2])
        prog += [("measure", (), (q, k)), ("feedback", "X", (t, k)), ("reset", (), (q,)), ("h", (), (q,)),
                 ("cx", (), (q, t)), ("ry", (float(rng.random()) * math.tau,), (t,))]
    return prog


def unitary(rng, k):
    m = rng.standard_normal((1 << k, 1 << k)) + 1j * rng.standard_normal((1 << k, 1 << k))
    q, r = np.linalg.qr(m)
    return np.ascontiguousarray(q * (np.diag(r) / np.abs(np.diag(r))))


def gate_sequence(n, count, seed):
    """(matrix, targets, controls) of gates applied one by one."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i in range(count):
        k = [1, 1, 2, 2, 3, 4, 1, 2, 5, 6][i % 10]
        controls = int(rng.integers(0, 4)) if k <= 2 else 0
        qs = [int(q) for q in rng.permutation(n)[:k + controls]]
        m = np.diag(np.exp(1j * rng.random(1 << k) * math.tau)) if i % 4 == 3 and k <= 4 else unitary(rng, k)
        out.append((m, qs[:k], [(q, bool(rng.integers(0, 2))) for q in qs[k:]]))
    return out


def ansatz_batch(case, seed):
    """(width, gates (layers, width, 2, 2)) of each circuit: RZ(phi) RY(theta)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i in range(case["count"]):
        # Widths and layer counts spread evenly over their ranges; the seed
        # orders them and draws the angles.
        n = case["min_width"] + i % (case["max_width"] - case["min_width"] + 1)
        layers = case["min_layers"] + (7 * i) % (case["max_layers"] - case["min_layers"] + 1)
        theta, phi = rng.random((2, layers, n)) * math.tau
        c, s, e = np.cos(theta / 2), np.sin(theta / 2), np.exp(1j * phi / 2)
        g = np.empty((layers, n, 2, 2), dtype=np.complex128)
        g[..., 0, 0], g[..., 0, 1] = c / e, -s / e
        g[..., 1, 0], g[..., 1, 1] = s * e, c * e
        out.append((n, g))
    return [out[i] for i in rng.permutation(len(out))]


def pauli_terms(n, count, seed):
    """`count` Pauli labels (rightmost letter = qubit 0): neighbours' ZZ, X on
    one qubit, and strings of weight 2 to 6."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for i in range(count):
        s = ["I"] * n
        if i % 3 == 0:
            q = int(rng.integers(0, n - 1))
            s[q] = s[q + 1] = "Z"
        elif i % 3 == 1:
            s[int(rng.integers(0, n))] = "X"
        else:
            for q in rng.permutation(n)[:int(rng.integers(2, 7))]:
                s[int(q)] = "XYZ"[int(rng.integers(0, 3))]
        out.append("".join(s))
    return out


def ising_terms(n):
    """The transverse-field Ising chain's terms as (label, coefficient)."""
    out = []
    for q in range(n):
        if q + 1 < n:
            out.append(("".join("Z" if i in (q, q + 1) else "I" for i in reversed(range(n))), -1.0))
        out.append(("".join("X" if i == q else "I" for i in reversed(range(n))), -0.7))
    return out


def gaussian(n, bits, seed):
    """A normalised vector of independent complex Gaussian amplitudes on the
    device, in the state's precision."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(1 << n, 2, generator=g, device="cuda", dtype=torch.float32 if bits == 32 else torch.float64)
    v *= 1.0 / math.sqrt(2.0 * (1 << n))
    return torch.view_as_complex(v)


# ------------------------------------------------------------------- state
class _Buffer:
    """A DeviceState's amplitudes as a device array (keeps the state)."""

    def __init__(self, st):
        pointer, _ = st.device_buffer()
        self.state = st
        self.__cuda_array_interface__ = {"shape": (1 << st.num_qubits,), "data": (pointer, False), "version": 3,
                                         "typestr": "<c8" if st.precision_bits == 32 else "<c16"}


def device_state(n, bits, amplitudes=None):
    """A state and its amplitude buffer as a torch tensor."""
    st = DeviceState(n, bits)
    view = torch.as_tensor(_Buffer(st), device="cuda")
    if amplitudes is not None:
        view.copy_(amplitudes)
        torch.cuda.synchronize()
    return st, view


def to_logical(st):
    """Brings the state to logical order on the device: the permutation of
    its index bits as at most two passes of disjoint swaps."""
    layout = st.layout()
    if layout == list(range(st.num_qubits)):
        return
    back = {p: q for q, p in enumerate(layout)}  # position -> where its bit belongs
    first, second, seen = [], [], set()
    for start in back:
        if start in seen:
            continue
        cycle, p = [], start
        while p not in seen:
            seen.add(p)
            cycle.append(p)
            p = back[p]
        k = len(cycle)
        for i in range(k):
            j, m = (-i) % k, (1 - i) % k
            if i < j:
                first.append((cycle[i], cycle[j]))
            if i < m:
                second.append((cycle[i], cycle[m]))
    for pairs in (first, second):
        if pairs:
            st.swap_physical(pairs)


def prepare(case, seed):
    kind, s = case["kind"], dict(case)
    if kind == "statevector":
        s["circuit_"] = circuit_of(program(case["circuit"], case["n"], case["depth"], seed), case["n"])
    elif kind == "dynamic":
        s["circuit_"] = circuit_of(dynamic_program(case["n"], case["rounds"], seed), case["n"])
        s["seed"] = seed
    elif kind == "estimate":
        s["circuit_"] = circuit_of(program("ansatz", case["n"], case["depth"], seed), case["n"])
        s["terms_"] = ising_terms(case["n"])
    elif kind == "gates":
        s["gates_"] = gate_sequence(case["n"], case["gates"], seed)
        s["state"], s["view"] = device_state(case["n"], case["bits"], gaussian(case["n"], case["bits"], seed))
    elif kind == "oneshot":
        _native.ensure_cost_model()
        s["ops"] = circuit_of(program(case["circuit"], case["n"], case["depth"], seed), case["n"]).ops()
        s["state"], s["view"] = device_state(case["n"], case["bits"])
        s["options"] = plan_options()
    elif kind in ("plan", "evolve"):
        _native.ensure_cost_model()
        ops = circuit_of(program(case["circuit"], case["n"], case["depth"], seed), case["n"]).ops()
        start = None if kind == "plan" else gaussian(case["n"], case["bits"], seed)
        s["state"], s["view"] = device_state(case["n"], case["bits"], start)
        s["plan"] = Plan(ops, case["n"], case["bits"], plan_options())
    elif kind == "observables":
        s["terms_"] = pauli_terms(case["n"], case["terms"], seed)
        s["state"], s["view"] = device_state(case["n"], case["bits"], gaussian(case["n"], case["bits"], seed))
    elif kind == "sample":
        s["state"], s["view"] = device_state(case["n"], case["bits"], gaussian(case["n"], case["bits"], seed))
        s["uniforms"] = np.random.Generator(np.random.PCG64(seed)).random(case["shots"])
        s["measures"] = [(case["n"] - 1 - 2 * c, c) for c in range(case["counted"])]
    else:
        circuits = ansatz_batch(case, seed)
        s["gates_"] = [g for _, g in circuits]
        s["batch"] = Batch([(n, g, "cx") for n, g in circuits])
    return s


def run(s):
    kind = s["kind"]
    if kind == "statevector":
        return statevector(s["circuit_"], precision="single" if s["bits"] == 32 else "double")
    if kind == "dynamic":
        counts = run_circuit(s["circuit_"], s["shots"], seed=s["seed"],
                             precision="single" if s["bits"] == 32 else "double").counts
        histogram = np.zeros(1 << s["rounds"], dtype=np.int64)
        for key, count in counts.items():
            histogram[int(key, 2)] = count
        return histogram
    if kind == "estimate":
        return estimate(s["circuit_"], s["terms_"], precision="single" if s["bits"] == 32 else "double")
    if kind == "observables":
        return s["state"].expect_z_all(), np.array([s["state"].expect_pauli(t) for t in s["terms_"]])
    if kind == "sample":
        if s["measures"]:
            keys, counts = s["state"].sample_counts(s["uniforms"], s["measures"])
            return keys.view(np.int64), counts.view(np.int64)
        return s["state"].sample_unordered(s["uniforms"]).view(np.int64)
    if kind == "batch":
        s["batch"].set_gates(s["gates_"])
        return s["batch"].run()[0]
    st = s["state"]
    if kind == "gates":
        for matrix, targets, controls in s["gates_"]:
            st.apply(matrix, targets, controls)
    elif kind == "oneshot":
        st.zero()
        st.apply_ops(s["ops"], s["options"])
    elif kind == "plan":
        st.zero()
        st.execute(s["plan"])
    else:
        st.execute(s["plan"])
    to_logical(st)
    return s["view"]


# -------------------------------------------------------------------- work
_FLOPS = {"h": 14, "x": 0, "rx": 14, "ry": 14, "rz": 6, "u": 14, "t": 3, "sx": 14, "cx": 0, "cz": 0.25, "cp": 1.5,
          "swap": 0, "ccx": 0, "cswap": 0}  # per amplitude


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    size = 1 << n
    amps = size * (8 if case.get("bits") == 32 else 16)
    gates = lambda prog: float(sum(_FLOPS[g[0]] for g in prog)) * size  # noqa: E731
    if kind == "statevector":
        return {"bytes": 16 * size, "flops": gates(program(case["circuit"], n, case["depth"], 1))}
    if kind == "dynamic":
        shots = case["shots"]
        return {"bytes": shots * amps, "flops": shots * 14.0 * size * (2 * n + 2 * case["rounds"])}
    if kind == "estimate":
        return {"bytes": 8 * 2 * n, "flops": gates(program("ansatz", n, case["depth"], 1)) + 8.0 * size * (2 * n - 1)}
    if kind == "gates":
        seq = gate_sequence(n, case["gates"], 1)
        share = [0.5 ** len(c) for _, _, c in seq]
        flops = sum(f * (6 if np.count_nonzero(m) <= m.shape[0] else 8 * m.shape[0] - 2)
                    for f, (m, _, _) in zip(share, seq))
        return {"bytes": 2.0 * amps * sum(share), "flops": size * flops}
    if kind in ("oneshot", "plan"):
        return {"bytes": amps, "flops": gates(program(case["circuit"], n, case["depth"], 1))}
    if kind == "evolve":
        return {"bytes": 2 * amps, "flops": gates(program(case["circuit"], n, case["depth"], 1))}
    if kind == "observables":
        return {"bytes": amps * (1 + case["terms"]), "flops": float(size) * (4 + n + 10 * case["terms"])}
    if kind == "sample":
        return {"bytes": amps + 24 * case["shots"], "flops": 4.0 * size}
    parts = [(g.shape[0], w) for w, g in ansatz_batch(case, 1)]
    return {"bytes": sum(64 * l * w + 8 * w for l, w in parts), "flops": sum(14.0 * l * w * 2**w for l, w in parts)}


# ------------------------------------------------------------------- exact
def gate_matrix(name, p):
    """(controls, matrix) in Qiskit's conventions, index bit j = j-th target."""
    r = math.sqrt(0.5)
    if name == "u":
        t, phi, lam = p
        c, s = math.cos(t / 2), math.sin(t / 2)
        return 0, [[c, -np.exp(1j * lam) * s], [np.exp(1j * phi) * s, np.exp(1j * (phi + lam)) * c]]
    if name in ("rx", "ry", "rz"):
        c, s = math.cos(p[0] / 2), math.sin(p[0] / 2)
        return 0, {"rx": [[c, -1j * s], [-1j * s, c]], "ry": [[c, -s], [s, c]],
                   "rz": [[np.exp(-0.5j * p[0]), 0], [0, np.exp(0.5j * p[0])]]}[name]
    x, swap = [[0, 1], [1, 0]], [[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]]
    return {"h": (0, [[r, r], [r, -r]]), "x": (0, x), "t": (0, [[1, 0], [0, np.exp(0.25j * math.pi)]]),
            "sx": (0, [[0.5 + 0.5j, 0.5 - 0.5j], [0.5 - 0.5j, 0.5 + 0.5j]]), "cx": (1, x), "ccx": (2, x),
            "cz": (1, [[1, 0], [0, -1]]), "cp": (1, [[1, 0], [0, np.exp(1j * (p[0] if p else 0))]]),
            "swap": (0, swap), "cswap": (1, swap)}[name]


def apply_exact(v, n, matrix, targets, controls):
    """The gate on the 2^n vector v (complex128), in place."""
    m = np.asarray(matrix, dtype=np.complex128)
    qs = sorted(list(targets) + [q for q, _ in controls], reverse=True)
    shape, top = [], n
    for q in qs:
        shape += [1 << (top - q - 1), 2]
        top = q
    x = v.view(*shape, 1 << top)
    at = {q: 2 * i + 1 for i, q in enumerate(qs)}
    index = [slice(None)] * x.dim()
    for q, value in controls:
        index[at[q]] = int(value)
    parts = []
    for h in range(m.shape[0]):
        for j, q in enumerate(targets):
            index[at[q]] = (h >> j) & 1
        parts.append(x[tuple(index)])
    if np.count_nonzero(m - np.diag(np.diag(m))) == 0:
        for h, part in enumerate(parts):
            if m[h, h] != 1:
                part *= complex(m[h, h])
        return
    old = torch.stack(parts)
    new = (torch.from_numpy(m).to(v.device) @ old.view(len(parts), -1)).view(old.shape)
    del old
    for h, part in enumerate(parts):
        part.copy_(new[h])


def evolve_exact(v, n, prog):
    """A circuit on v in 64 bits; runs of one-qubit gates are multiplied out
    and applied five neighbouring qubits at a time."""
    pending = {}

    def flush():
        for g in range(0, n, 5):
            w = min(5, n - g)
            if not any(q in pending for q in range(g, g + w)):
                continue
            m = np.eye(1)
            for q in range(g, g + w):
                m = np.kron(pending.pop(q, np.eye(2)), m)
            mt = torch.from_numpy(np.ascontiguousarray(m.astype(np.complex128))).to(v.device)
            x = v.view(-1, 1 << w, 1 << g)
            if x.shape[2] == 1:
                y = x.view(-1, 1 << w) @ mt.T
            elif x.shape[0] == 1:
                y = mt @ x[0]
            else:
                y = torch.matmul(mt, x)
            v.copy_(y.reshape(-1))

    for name, params, qubits in prog:
        nc, m = gate_matrix(name, params)
        if len(qubits) == 1:
            q = qubits[0]
            pending[q] = np.asarray(m, dtype=np.complex128) @ pending.get(q, np.eye(2))
            continue
        if any(q in pending for q in qubits):
            flush()
        apply_exact(v, n, m, list(qubits[nc:]), [(q, True) for q in qubits[:nc]])
    flush()
    return v


def zero_exact(n):
    v = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    v[0] = 1
    return v


def pauli_exact(v, n, label):
    """<v|P|v> of a normalised or unnormalised complex128 vector."""
    y = v.clone()
    for q, letter in enumerate(reversed(label)):
        m = {"I": None, "X": [[0, 1], [1, 0]], "Y": [[0, -1j], [1j, 0]], "Z": [[1, 0], [0, -1]]}[letter]
        if m is not None:
            apply_exact(y, n, m, [q], [])
    return float(torch.vdot(v, y).real)


def z_exact(v, n):
    """<Z> of every qubit: total - 2 P(1), unnormalised."""
    p = torch.view_as_real(v).square().sum(-1)
    return [float(p.sum() - 2 * p.view(-1, 2, 1 << q)[:, 1].sum()) for q in range(n)]


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("dynamic", "sample"):
        return None
    if kind in ("statevector", "oneshot", "plan"):
        v = evolve_exact(zero_exact(n), n, program(case["circuit"], n, case["depth"], seed))
        return v.cpu().numpy() if kind == "statevector" else v
    if kind == "estimate":
        v = evolve_exact(zero_exact(n), n, program("ansatz", n, case["depth"], seed))
        return sum(c * pauli_exact(v, n, label) for label, c in ising_terms(n))
    if kind == "batch":
        out = []
        for w, g in ansatz_batch(case, seed):
            v = zero_exact(w)
            i = torch.arange(1 << w, device="cuda")
            # The CX ladder sends bit q to the parity of bits 0..q: index j
            # holds what stood at j ^ (j << 1).
            source = (i ^ (i << 1)) & ((1 << w) - 1)
            for layer in g:
                for q0 in range(0, w, 6):
                    m = np.eye(1)
                    for q in range(q0, min(q0 + 6, w)):
                        m = np.kron(layer[q], m)
                    mt = torch.from_numpy(np.ascontiguousarray(m)).to("cuda")
                    v = torch.matmul(mt, v.view(-1, mt.shape[0], 1 << q0)).reshape(-1)
                v = v[source]
            p = torch.view_as_real(v).square().sum(-1)
            out.append(torch.stack([p.sum() - 2 * p.view(-1, 2, 1 << q)[:, 1].sum() for q in range(w)]))
        return torch.cat(out).cpu().numpy()
    v = gaussian(n, case["bits"], seed).to(torch.complex128)
    if kind == "gates":
        for m, targets, controls in gate_sequence(n, case["gates"], seed):
            apply_exact(v, n, m, targets, controls)
        return v
    if kind == "evolve":
        return evolve_exact(v, n, program(case["circuit"], n, case["depth"], seed))
    return np.array(z_exact(v, n)), np.array([pauli_exact(v, n, t) for t in pauli_terms(n, case["terms"], seed)])
