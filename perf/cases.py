"""What is measured of this framework, and on which inputs.

The cases are the calls that a user's program makes again and again: running a
circuit on a state vector (from a handful of qubits to 30, both precisions,
plain and noisy, with dense blocks and with measurements in the middle),
applying single gates one at a time, sampling the result, and taking batched
gradients.  A case's structure (which gates act where) follows from its own
numbers; the values (angles, unitaries, parameters, states, uniforms) follow
from the seed, as in a program that evaluates one circuit at new parameters.

  listed()            the cases
  draw(rng)           another case of the same ranges
  prepare(case, seed) what a program has before the call: the simulator, the
                      circuit, and its compiled passes
  run(state)          one call
  work(case)          bytes and operations that one call cannot do without
  exact(case, seed)   what run returns, computed in 64 bits by plain torch
"""
from __future__ import annotations

import math

import numpy as np
import torch

PARAMS = {"h": 0, "x": 0, "rx": 1, "ry": 1, "rz": 1, "u3": 3, "cx": 0, "cz": 0, "rzz": 1, "swap": 0}
TWO = {"cx", "cz", "rzz", "swap"}
NAMES = list(PARAMS)
# multiplications and additions per amplitude of the state, by gate
GATE_FLOPS = {"h": 4, "x": 0, "rx": 8, "ry": 6, "rz": 6, "u3": 14, "cx": 0, "cz": 0.5, "rzz": 6, "swap": 0}


# ---- the circuits, as plain lists of (name, qubits) ------------------------------------------
def _pick(rng, qubits, k):
    return [int(q) for q in rng.choice(qubits, size=k, replace=False)]


def _layout(case):
    """[(gate name, qubits)] of a circuit case: `layout` "uniform" draws the
    gates and qubits uniformly; "spread" adds 10 % random two-qubit unitaries
    and takes qubits from the five last ones and the ten first ones; "blocks"
    puts `blocks` dense unitaries on `width` qubits between uniform gates;
    "dynamic" puts `measures` measurements (a third of them resets) between
    them."""
    rng = np.random.default_rng([case["circuit"], case["n"], case["gates"]])
    n, layout = case["n"], case["layout"]
    low, high = list(range(max(0, n - 5), n)), list(range(0, max(1, min(10, n - 5))))
    out = []
    for _ in range(case["gates"]):
        name = NAMES[int(rng.integers(len(NAMES)))]
        if layout == "spread" and rng.random() < 0.1:
            name = "haar2"
        k = 2 if name in TWO or name == "haar2" else 1
        if layout == "spread":
            qs = []
            while len(qs) < k:
                grp = low if rng.random() < 0.5 else high
                q = grp[int(rng.integers(len(grp)))]
                if q not in qs:
                    qs.append(q)
        else:
            qs = _pick(rng, n, k)
        out.append((name, qs))
    if layout == "blocks":
        for i in range(case["blocks"]):
            at = (i + 1) * len(out) // (case["blocks"] + 1)
            out.insert(at, ("haar%d" % case["width"], _pick(rng, n, case["width"])))
    if layout == "dynamic":
        for i in range(case["measures"]):
            at = (i + 1) * len(out) // (case["measures"] + 1)
            out.insert(at, ("reset" if i % 3 == 2 else "measure", _pick(rng, n, 1)))
    return out


def _sweep_layout(case):
    """Every gate class on low, middle and high qubits, one at a time."""
    n = case["n"]
    ones = [n - 1, n - 3, n - 6, n // 2, 0]
    twos = [(n - 2, n - 1), (n - 5, n - 2), (0, n - 1), (n // 2, n - 8), (0, 1)]
    out = [(g, [q]) for g in ("h", "x", "rx", "ry", "rz", "u3") for q in ones]
    return out + [(g, list(t)) for g in ("cx", "cz", "rzz", "swap", "haar2") for t in twos]


def _haar(rng, d):
    z = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
    q, r = np.linalg.qr(z)
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _values(layout, seed):
    """[(name, qubits, angles or matrix)] with values from the seed."""
    rng = np.random.default_rng([11, seed])
    out = []
    for name, qs in layout:
        if name.startswith("haar"):
            v = _haar(rng, 1 << len(qs))
        else:
            v = [float(x) for x in rng.uniform(0.05, 2 * np.pi - 0.05, PARAMS.get(name, 0))]
        out.append((name, qs, v))
    return out


def _circuit(n, gates):
    from quict_b200.core import GATE_BY_NAME, Circuit, Measure, Reset, Unitary
    c = Circuit(n)
    for name, qs, v in gates:
        if name == "measure":
            Measure | c(qs)
        elif name == "reset":
            Reset | c(qs)
        elif name.startswith("haar"):
            Unitary(v) | c(qs)
        else:
            g = GATE_BY_NAME[name]
            (g(*v) if v else g) | c(qs)
    return c


def _matrix(name, v):
    """Gate matrices by their textbook definitions, in 64 bits."""
    if name.startswith("haar"):
        return np.asarray(v)
    i = 1j
    if name == "h":
        return np.array([[1, 1], [1, -1]]) / math.sqrt(2)
    if name == "x":
        return np.array([[0, 1], [1, 0]])
    if name == "cx":
        return np.eye(4)[[0, 1, 3, 2]]
    if name == "cz":
        return np.diag([1, 1, 1, -1])
    if name == "swap":
        return np.eye(4)[[0, 2, 1, 3]]
    c, s = math.cos(v[0] / 2), math.sin(v[0] / 2)
    if name == "rx":
        return np.array([[c, -i * s], [-i * s, c]])
    if name == "ry":
        return np.array([[c, -s], [s, c]])
    if name == "rz":
        return np.diag([c - i * s, c + i * s])
    if name == "rzz":
        return np.diag([c - i * s, c + i * s, c + i * s, c - i * s])
    if name == "u3":
        p, q = np.exp(i * v[1]), np.exp(i * v[2])
        return np.array([[c, -q * s], [p * s, p * q * c]])
    raise ValueError(name)


# ---- plain torch, in 64 bits -----------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _apply(psi, nbits, matrix, axes):
    """`matrix` on the given axes (0 = most significant bit) of a vector of
    2^nbits entries; psi may have a leading batch axis, and then the matrix
    may have one too."""
    batch = psi.shape[0] if psi.dim() == 2 else 1
    k = len(axes)
    order = sorted(axes)
    shape, at, where = [batch], 0, {}
    for a in order:
        shape += [1 << (a - at), 2]
        where[a] = len(shape) - 1
        at = a + 1
    shape.append(1 << (nbits - at))
    front = [0] + [where[a] for a in axes]
    perm = front + [d for d in range(len(shape)) if d not in front]
    t = psi.reshape(shape).permute(perm)
    tail = t.shape
    m = matrix if torch.is_tensor(matrix) else torch.as_tensor(np.asarray(matrix, dtype=np.complex128), device=psi.device)
    t = torch.matmul(m, t.reshape(batch, 1 << k, -1)).reshape(tail)
    back = [0] * len(perm)
    for i, d in enumerate(perm):
        back[d] = i
    return t.permute(back).reshape(psi.shape)


def _exact_circuit(n, gates, uniforms=None):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=_dev())
    psi[0] = 1
    measured, drawn = [], 0
    for name, qs, v in gates:
        if name in ("measure", "reset"):
            t = psi.view(1 << qs[0], 2, -1)
            p0 = float((t[:, 0].real.square() + t[:, 0].imag.square()).sum())
            if name == "measure":
                one = uniforms[drawn % len(uniforms)] > p0
                drawn += 1
                t[:, 0 if one else 1] = 0
                psi *= 1 / math.sqrt(1 - p0 if one else p0)
                measured.append(int(one))
            else:
                t[:, 0] = t[:, 0] / math.sqrt(p0) if math.sqrt(p0) >= 1e-6 else t[:, 1]
                t[:, 1] = 0
        else:
            psi = _apply(psi, n, _matrix(name, v), qs)
    return psi, measured


# ---- circuits on a state vector ----------------------------------------------------------------
class _Uniforms:
    """The uniforms of a run's measurements, the same for every run."""

    def __init__(self, values):
        self.values, self.at = list(values), 0

    def random(self):
        self.at = (self.at + 1) % len(self.values)
        return self.values[self.at - 1]


def _measure_uniforms(case, seed):
    return np.random.default_rng([12, seed]).random(sum(name == "measure" for name, _ in _layout(case)))


def _gates_of(case, seed):
    return _values(_sweep_layout(case) if case["kind"] == "sweep" else _layout(case), seed)


def _prepare_run(case, seed):
    from quict_b200 import _native
    from quict_b200.simulation import StateVectorSimulator
    more = {}
    if case["kind"] == "sweep":
        more["fusion"] = False
    if case["layout"] == "dynamic":
        more["seed"] = _Uniforms(_measure_uniforms(case, seed))
    sim = StateVectorSimulator("GPU", case["precision"], **more)
    circuit = _circuit(case["n"], _gates_of(case, seed))
    sim.run(circuit)
    _native.jit_wait()  # the circuit's passes are compiled from here on
    return {"sim": sim, "circuit": circuit, "dynamic": case["layout"] == "dynamic"}


def _run_run(state):
    out = state["sim"].run(state["circuit"]).tensor
    if state["dynamic"]:
        return {"state": out, "measured": [q.measured for q in state["circuit"].qubits if q.measured is not None]}
    return out


# ---- noisy density matrices ----------------------------------------------------------------------
GAMMA, P1, P2 = 5e-3, 1e-3, 1e-2


def _prepare_dm(case, seed):
    from quict_b200 import _native
    from quict_b200.core import DampingError, DepolarizingError, NoiseModel
    from quict_b200.simulation import DensityMatrixSimulator
    one = [g for g in NAMES if g not in TWO]
    amp = DampingError(amplitude_prob=GAMMA, phase_prob=0)
    model = NoiseModel(basic_gates=NAMES)
    model.add_noise_for_all_qubits(amp.compose(DepolarizingError(P1, 1)), one)
    model.add_noise_for_all_qubits(amp.tensor(amp).compose(DepolarizingError(P2, 2)), sorted(TWO))
    # accumulated: every gate becomes its Kraus set (no random draws)
    sim = DensityMatrixSimulator("GPU", case["precision"], accumulated_mode=True)
    circuit = _circuit(case["n"], _gates_of(case, seed))
    sim.run(circuit, noise_model=model)
    _native.jit_wait()
    return {"sim": sim, "circuit": circuit, "model": model}


def _run_dm(state):
    return state["sim"].run(state["circuit"], noise_model=state["model"]).tensor


def _exact_dm(case, seed):
    n = case["n"]
    paulis = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1, -1])]
    damp = [np.array([[1, 0], [0, math.sqrt(1 - GAMMA)]]), np.array([[0, math.sqrt(GAMMA)], [0, 0]])]
    sup = {}
    for k, p in ((1, P1), (2, P2)):
        ops = paulis if k == 1 else [np.kron(a, b) for a in paulis for b in paulis]
        weights = [1 - p * (len(ops) - 1) / len(ops)] + [p / len(ops)] * (len(ops) - 1)
        dep = sum(w * np.kron(o, o.conj()) for w, o in zip(weights, ops))
        d = damp if k == 1 else [np.kron(a, b) for a in damp for b in damp]
        sup[k] = sum(np.kron(o, o.conj()) for o in d) @ dep
    rho = torch.zeros(1 << (2 * n), dtype=torch.complex128, device=_dev())
    rho[0] = 1
    for name, qs, v in _gates_of(case, seed):
        u = _matrix(name, v)
        rho = _apply(rho, 2 * n, sup[len(qs)] @ np.kron(u, np.conj(u)), qs + [q + n for q in qs])
    return rho.view(1 << n, 1 << n)


# ---- sampling ------------------------------------------------------------------------------------
def _prepare_sample(case, seed):
    from quict_b200.core import Circuit, H
    from quict_b200.simulation import StateVectorSimulator
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    psi = torch.view_as_complex(torch.randn((1 << n, 2), generator=g, device="cuda", dtype=torch.float64))
    psi /= torch.linalg.vector_norm(psi)
    sim = StateVectorSimulator("GPU", case["precision"])
    circuit = Circuit(n)
    H | circuit(0)
    sim.run(circuit, state_vector=psi)
    per = n if case["mode"] == "sequential" else 1
    return {"sim": sim, "uniforms": np.random.default_rng([13, seed]).random(case["shots"] * per), "shots": case["shots"],
            "mode": case["mode"], "counts": case["counts"]}


def _run_sample(state):
    out = state["sim"].sample(state["shots"], uniforms=state["uniforms"], mode=state["mode"], return_counts=state["counts"])
    return np.asarray(out) if state["counts"] else out


# ---- gradients -------------------------------------------------------------------------------------
def _prepare_gradient(case, seed):
    from quict_b200 import _native
    from quict_b200.differentiation import BatchedAdjoint, expectation, hardware_efficient_ansatz, ising_observable
    engine = BatchedAdjoint(hardware_efficient_ansatz(case["n"], case["layers"]), ising_observable(case["n"]), case["precision"])
    params = np.random.default_rng([14, seed]).uniform(0, 2 * np.pi, (case["batch"], 2 * case["n"] * case["layers"]))
    params = torch.tensor(params, dtype=torch.float32 if case["precision"] == "single" else torch.float64, requires_grad=True)
    for _ in range(2):
        expectation(params, engine)
        _native.jit_wait()
    return {"engine": engine, "params": params}


def _run_gradient(state):
    """One training step's share: the energies and their gradients."""
    from quict_b200.differentiation import expectation
    params = state["params"]
    params.grad = None
    energies = expectation(params, state["engine"])
    energies.sum().backward()
    return {"energies": energies.detach(), "gradient": params.grad}


def _exact_gradient(case, seed):
    n, layers = case["n"], case["layers"]
    params = np.random.default_rng([14, seed]).uniform(0, 2 * np.pi, (case["batch"], 2 * n * layers))
    kind = torch.float32 if case["precision"] == "single" else torch.float64
    p = torch.tensor(params, dtype=kind).double().to(_dev())
    x, y = torch.tensor([[0, 1], [1, 0]], dtype=torch.complex128), torch.tensor([[0, -1j], [1j, 0]], dtype=torch.complex128)
    x, y = x.to(p.device), y.to(p.device)
    index = torch.arange(1 << n, device=p.device)
    z = [1.0 - 2.0 * ((index >> (n - 1 - q)) & 1).double() for q in range(n)]
    ring = torch.ones_like(z[0])
    for a in range(n if n > 2 else n - 1):
        b = (a + 1) % n
        ring = ring * (1 - 2 * (((1 - z[a]) / 2) * ((1 - z[b]) / 2)))
    eye = torch.eye(2, dtype=torch.complex128, device=p.device)

    def turn(generator, t):
        return torch.cos(t / 2)[:, None, None] * eye - 1j * torch.sin(t / 2)[:, None, None] * generator

    def phase(t, q):
        return torch.exp(-0.5j * t[:, None] * z[q][None, :])

    rows = []
    for at in range(0, case["batch"], 32):  # a few sets at a time
        t = p[at:at + 32]
        psi = torch.zeros((t.shape[0], 1 << n), dtype=torch.complex128, device=p.device)
        psi[:, 0] = 1
        for layer in range(layers):
            for q in range(n):
                psi = _apply(psi, n, turn(y, t[:, 2 * n * layer + q]), [q])
            for q in range(n):
                psi = psi * phase(t[:, 2 * n * layer + n + q], q)
            psi = psi * ring
        lam = sum(z[q] * z[q + 1] for q in range(n - 1)) * psi
        for q in range(n):
            lam = lam + 0.5 * _apply(psi, n, x, [q])
        energy = (psi.conj() * lam).sum(1).real
        grad = torch.zeros_like(t)
        for layer in reversed(range(layers)):
            psi, lam = psi * ring, lam * ring
            for q in range(n):  # every Rz of a layer sees the same states up to phases
                at_q = 2 * n * layer + n + q
                grad[:, at_q] = (lam.conj() * z[q] * psi).sum(1).imag
                f = phase(-t[:, at_q], q)
                psi, lam = psi * f, lam * f
            for q in range(n):
                at_q = 2 * n * layer + q
                grad[:, at_q] = (lam.conj() * _apply(psi, n, y, [q])).sum(1).imag
                m = turn(y, -t[:, at_q])
                psi, lam = _apply(psi, n, m, [q]), _apply(lam, n, m, [q])
        rows.append((energy, grad))
    return {"energies": torch.cat([e for e, _ in rows]).cpu(), "gradient": torch.cat([g for _, g in rows]).cpu()}


def _qaoa_instances(case, seed):
    """[(qubits, edges, depth, angles)]: graphs and depths from the case, angles from the seed."""
    from quict_b200.differentiation import random_regular_graph
    fixed = np.random.default_rng([15, case["circuit"], case["instances"]])
    values = np.random.default_rng([16, seed])
    out = []
    for _ in range(case["instances"]):
        n = 2 * int(fixed.integers(case["least"] // 2, case["most"] // 2 + 1))
        depth = int(fixed.integers(1, case["depth"] + 1))
        out.append((n, random_regular_graph(n, 3, fixed), depth, values.uniform(0, np.pi, 2 * depth)))
    return out


def _prepare_qaoa(case, seed):
    from quict_b200.differentiation import UnevenQAOABatch
    batch = UnevenQAOABatch(_qaoa_instances(case, seed), case["precision"], mode="persistent")
    batch.capture()
    return {"batch": batch, "dtype": np.float32 if case["precision"] == "single" else np.float64}


def _run_qaoa(state):
    """Energies and gradients of every instance, in the precision that the
    optimiser's angles have."""
    state["batch"].replay()
    got = state["batch"].results()
    return {"energies": np.array([e for e, _ in got], dtype=state["dtype"]),
            "gradients": np.concatenate([g for _, g in got]).astype(state["dtype"])}


def _exact_qaoa(case, seed):
    energies, grads = [], []
    x = torch.tensor([[0, 1], [1, 0]], dtype=torch.complex128, device=_dev())
    eye = torch.eye(2, dtype=torch.complex128, device=_dev())
    for n, edges, depth, angles in _qaoa_instances(case, seed):
        index = torch.arange(1 << n, device=_dev())
        zz = torch.zeros(1 << n, dtype=torch.float64, device=_dev())
        for a, b in edges:
            zz += 1.0 - 2.0 * (((index >> (n - 1 - a)) ^ (index >> (n - 1 - b))) & 1).double()
        cost = (len(edges) - zz) / 2
        psi = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device=_dev())

        def mix(v, beta):
            m = math.cos(beta) * eye - 1j * math.sin(beta) * x
            for q in range(n):
                v = _apply(v, n, m, [q])
            return v

        for k in range(depth):
            psi = mix(psi * torch.exp(0.5j * angles[k] * zz), angles[depth + k])
        lam = cost * psi
        energies.append(float((psi.conj() * lam).sum().real))
        g = np.zeros(2 * depth)
        for k in reversed(range(depth)):
            g[depth + k] = 2 * float(sum((lam.conj() * _apply(psi, n, x, [q])).sum().imag for q in range(n)))
            psi, lam = mix(psi, -angles[depth + k]), mix(lam, -angles[depth + k])
            g[k] = -float((lam.conj() * zz * psi).sum().imag)
            f = torch.exp(-0.5j * angles[k] * zz)
            psi, lam = psi * f, lam * f
        grads.append(g)
    return {"energies": np.array(energies), "gradients": np.concatenate(grads)}


# ---- the cases -------------------------------------------------------------------------------------
def _run_case(name, n, precision, gates, layout, circuit, kind="run", **more):
    return dict({"name": name, "kind": kind, "n": n, "precision": precision, "gates": gates, "layout": layout, "circuit": circuit}, **more)


def listed():
    return [
        # a small circuit, evaluated in the loop of a variational or teaching program: latency counts
        _run_case("run-10q-c128", 10, "double", 60, "uniform", 1),
        # the everyday size: 20 qubits, 200 random gates
        _run_case("run-20q-c128", 20, "double", 200, "uniform", 2),
        # an odd size in single precision, beyond the on-chip caches
        _run_case("run-25q-c64", 25, "single", 300, "uniform", 3),
        # the large runs: 30 qubits, 1000 gates on low and high qubits
        _run_case("run-30q-c128", 30, "double", 1000, "spread", 4),
        _run_case("run-30q-c64", 30, "single", 1000, "spread", 5),
        # gates applied one at a time (a program that steps through a circuit), every class and placement
        _run_case("sweep-28q-c128", 28, "double", 0, "sweep", 0, kind="sweep"),
        # circuits whose oracles or preparations come as dense blocks on several qubits
        _run_case("blocks-20q-c128", 20, "double", 40, "blocks", 6, blocks=4, width=6),
        # measurements and resets in the middle of a circuit
        _run_case("dynamic-25q-c64", 25, "single", 40, "dynamic", 7, measures=6),
        # a noisy 12-qubit device: amplitude damping and depolarising after each gate
        _run_case("noisy-12q-c128", 12, "double", 150, "uniform", 8, kind="dm"),
        # shots from a state, as sample indices on the GPU
        {"name": "sample-26q-c64", "kind": "sample", "n": 26, "precision": "single", "shots": 100000, "mode": "cdf", "counts": False},
        # a training step of a batched variational ansatz: energies and gradients
        {"name": "gradient-16q-c64", "kind": "gradient", "n": 16, "layers": 8, "batch": 256, "precision": "single"},
        # many small optimisation instances of uneven size in one launch
        {"name": "qaoa-32x10..20q-c64", "kind": "qaoa", "instances": 32, "least": 10, "most": 20, "depth": 4, "precision": "single", "circuit": 9},
    ]


def draw(rng):
    precision = rng.choice(["single", "double"])
    circuit = rng.randrange(1 << 20)
    spread = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["run", "run", "run", "sweep", "blocks", "dynamic", "dm", "sample", "gradient", "qaoa"])
    if kind == "run":
        n = rng.randrange(8, 31)
        return _plain(_run_case("", n, precision, spread(20, 1000 if n >= 28 else 400), rng.choice(["uniform", "spread"]), circuit))
    if kind == "sweep":
        return _plain(_run_case("", rng.randrange(18, 29), precision, 0, "sweep", 0, kind="sweep"))
    if kind == "blocks":
        width = rng.randrange(5, 9)
        return _plain(_run_case("", rng.randrange(12, 21), precision, rng.randrange(10, 60), "blocks", circuit, blocks=rng.randrange(1, 5), width=width))
    if kind == "dynamic":
        return _plain(_run_case("", rng.randrange(10, 27), precision, rng.randrange(20, 80), "dynamic", circuit, measures=rng.randrange(2, 9)))
    if kind == "dm":
        return _plain(_run_case("", rng.randrange(5, 13), precision, rng.randrange(30, 151), "uniform", circuit, kind="dm"))
    if kind == "sample":
        n = rng.randrange(8, 28)
        return {"kind": "sample", "n": n, "precision": precision, "shots": spread(100, 200000), "mode": rng.choice(["cdf", "cdf", "sequential"]),
                "counts": n <= 16}
    if kind == "gradient":
        return {"kind": "gradient", "n": rng.randrange(6, 17), "layers": rng.randrange(2, 9), "batch": spread(1, 256), "precision": precision}
    return {"kind": "qaoa", "instances": rng.randrange(4, 33), "least": 10, "most": 2 * rng.randrange(6, 11), "depth": rng.randrange(1, 5),
            "precision": precision, "circuit": circuit}


def _plain(case):
    del case["name"]
    return case


def prepare(case, seed):
    kind = case["kind"]
    make = {"dm": _prepare_dm, "sample": _prepare_sample, "gradient": _prepare_gradient, "qaoa": _prepare_qaoa}.get(kind, _prepare_run)
    state = make(case, seed)
    state["run"] = {"dm": _run_dm, "sample": _run_sample, "gradient": _run_gradient, "qaoa": _run_qaoa}.get(kind, _run_run)
    return state


def run(state):
    return state["run"](state)


def work(case):
    kind = case["kind"]
    size = 16 if case["precision"] == "double" else 8
    if kind == "sample":
        return {"bytes": float(size << case["n"]) + 16.0 * case["shots"], "flops": 4.0 * (1 << case["n"])}
    if kind == "gradient":
        n, units = case["n"], 2 * case["n"] * case["layers"]
        amps = float(case["batch"] << n)
        # forward, the observable, both vectors of the sweep with each generator's inner product
        return {"bytes": 8.0 * case["batch"] * (2 * units + 1), "flops": amps * units * (6 + 2 * 6 + 8)}
    if kind == "qaoa":
        flops = 0.0
        for n, edges, depth, _ in _qaoa_instances(case, 0):
            flops += float(1 << n) * depth * (n * 8 + 6) * 4
        return {"bytes": 16.0 * case["instances"] * (2 * case["depth"] + 1), "flops": flops}
    n = 2 * case["n"] if kind == "dm" else case["n"]
    amps = float(1 << n)
    if kind == "sweep":
        layout = _sweep_layout(case)
        part = {"cx": 0.5, "cz": 0.25, "swap": 0.5}
        return {"bytes": sum(2 * size * amps * part.get(g, 1) for g, _ in layout), "flops": sum(amps * GATE_FLOPS.get(g, 30) for g, _ in layout)}
    flops = 0.0
    for name, qs in _layout(case):
        if name.startswith("haar"):
            flops += amps * (8 * (1 << len(qs)) - 2)
        elif name in ("measure", "reset"):
            flops += amps * 3
        elif kind == "dm":
            flops += amps * (30 if len(qs) == 1 else 126) / 2
        else:
            flops += amps * GATE_FLOPS[name]
    return {"bytes": size * amps, "flops": flops}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None  # whole numbers
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "qaoa":
        return _exact_qaoa(case, seed)
    if kind == "dm":
        return _exact_dm(case, seed)
    if case["n"] > 26 and kind != "sweep":
        return None  # hundreds of gates on gigabytes: too long in plain torch
    gates = _gates_of(case, seed)
    if case["layout"] == "dynamic":
        psi, _ = _exact_circuit(case["n"], gates, _measure_uniforms(case, seed))
        return {"state": psi, "measured": None}
    return _exact_circuit(case["n"], gates)[0]
