"""The work that a program using the engine gives it, as cases that can be timed and compared.

Kinds of case (every one goes through ``B200SvBackend``, the surface that the CLI, ``frontend.run`` and the
C ABI's bindings use):

* ``plan``: a circuit compiled once and executed from |0...0>, as a program that reruns a circuit does
  (``reset_state`` + ``CompiledPlan.execute``); the answer is the state vector and any measurement outcomes.
* ``alias`` / ``cumulative``: drawing shots from a prepared state with explicit variates (the two sampling
  maps of the engine: two or more shots, and single shots or states above 28 qubits).
* ``readout``: a Pauli-sum energy, one Pauli string, and two marginals of a prepared state.
* ``sweep``: a batched QAOA Max-Cut parameter sweep of ragged sizes.
"""
import math
import random

import numpy as np
import torch

from aleph_b200 import circuit as C
from aleph_b200 import workloads
from aleph_b200.backend import B200SvBackend


def listed():
    return [
        # a variational program's inner circuit: a state that fits one SM, where latency is everything
        {"name": "plan_f64_hea_n10", "kind": "plan", "circuit": "hea", "n": 10, "depth": 4, "precision": "f64",
         "measures": 0},
        # the small named benchmark: FP64 brickwall n=20 depth 20 (the state stays in L2)
        {"name": "plan_f64_brickwall_n20", "kind": "plan", "circuit": "brickwall", "n": 20, "depth": 20,
         "precision": "f64", "measures": 0},
        # the named QFT benchmark's circuit at an odd size: few dense gates, many controlled phases, SWAPs
        {"name": "plan_f64_qft_n25", "kind": "plan", "circuit": "qft", "n": 25, "depth": 1, "precision": "f64",
         "measures": 0},
        # dense FP64 layers on a state well above L2: the double-precision main path
        {"name": "plan_f64_brickwall_n27", "kind": "plan", "circuit": "brickwall", "n": 27, "depth": 20,
         "precision": "f64", "measures": 0},
        # Grover search in CX + T gates: permutations and diagonals in plain FP32
        {"name": "plan_f32_grover_n22", "kind": "plan", "circuit": "grover", "n": 22, "depth": 4,
         "precision": "f32", "measures": 0},
        # tensor-core blocks on a state in L2: many short passes
        {"name": "plan_tc32_brickwall_n19", "kind": "plan", "circuit": "brickwall", "n": 19, "depth": 20,
         "precision": "tc32", "measures": 0},
        # the headline circuit (depth-40 brickwall, tensor-core FP32) at 28 qubits
        {"name": "plan_tc32_brickwall_n28", "kind": "plan", "circuit": "brickwall", "n": 28, "depth": 40,
         "precision": "tc32", "measures": 0},
        # mid-circuit measurement: reductions, decisions and collapses between gate passes
        {"name": "plan_f32_measured_n24", "kind": "plan", "circuit": "brickwall", "n": 24, "depth": 4,
         "precision": "f32", "measures": 4},
        # 1024 shots of a scrambled state, the default of every run
        {"name": "alias_f64_n22", "kind": "alias", "n": 22, "shots": 1024, "precision": "f64", "state": "scrambled"},
        # inverse-CDF shots of a large FP32 state
        {"name": "cumulative_f32_n26", "kind": "cumulative", "n": 26, "shots": 4096, "precision": "f32",
         "state": "scrambled"},
        # an energy and marginals of a mid-sized state
        {"name": "readout_f64_n23", "kind": "readout", "n": 23, "terms": 40, "few": 6, "many": 12,
         "precision": "f64", "state": "scrambled"},
        # a QAOA angle sweep: sets that fit shared memory and sets that stream
        {"name": "sweep_f32_384", "kind": "sweep", "sets": 384, "n_lo": 12, "n_hi": 22, "p": 4, "precision": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "plan", "alias", "cumulative", "readout", "sweep"])
    if kind == "plan":
        precision = rng.choice(["f64", "f32", "tc32"])
        circuit = rng.choice(["brickwall", "hea", "qft", "grover", "qaoa"])
        n = rng.randint(3, 26)
        if circuit == "grover":
            n = max(4, n - n % 2)  # n/2 + 1 data qubits and their ancillas
        if circuit == "qaoa":
            n = max(4, n - n % 2)  # 3-regular graphs
        depth = 1 if circuit == "qft" else rng.randint(1, 4) if circuit in ("grover", "qaoa") else rng.randint(2, 20)
        return {"kind": kind, "circuit": circuit, "n": n, "depth": depth, "precision": precision,
                "measures": rng.choice([0, 0, 0, 1, 3])}
    precision = rng.choice(["f64", "f32"])
    state = rng.choice(["scrambled", "product"])
    if kind == "alias":
        return {"kind": kind, "n": rng.randint(4, 22), "shots": _log_int(rng, 2, 20000), "precision": precision,
                "state": state}
    if kind == "cumulative":
        return {"kind": kind, "n": rng.randint(4, 26), "shots": _log_int(rng, 1, 20000), "precision": precision,
                "state": state}
    if kind == "readout":
        n = rng.randint(6, 24)
        return {"kind": kind, "n": n, "terms": _log_int(rng, 1, 100), "few": rng.randint(1, min(10, n)),
                "many": rng.randint(min(n, 11), min(n, 14)), "precision": precision, "state": state}
    lo = rng.randint(4, 14)
    return {"kind": "sweep", "sets": _log_int(rng, 4, 384), "n_lo": lo, "n_hi": rng.randint(lo, 22),
            "p": rng.randint(1, 5), "precision": precision}


# ---- inputs ------------------------------------------------------------------
class _Device:
    """A device allocation as torch sees it (no copy)."""

    def __init__(self, ptr, shape, typestr, keep):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(be, state):
    """The state's amplitudes as a (2^n, 2) tensor of (re, im) on the engine's own memory."""
    ptr, _ = be.state_memory(state)
    typestr = "<f8" if be.precision == "f64" else "<f4"
    return torch.as_tensor(_Device(ptr, (1 << state.num_qubits, 2), typestr, state), device="cuda")


def _graph(n, rng):
    if n % 2 == 0 and n >= 4:
        return workloads.random_3_regular(n, rng)
    edges = set()
    while len(edges) < min((3 * n) // 2, n * (n - 1) // 2):  # as many edges as a 3-regular graph has
        i, j = (int(x) for x in rng.choice(n, 2, replace=False))
        edges.add((min(i, j), max(i, j)))
    return sorted(edges)


def _circuit(case, seed):
    n, depth, rng = case["n"], case["depth"], np.random.default_rng(seed)
    kind = case["circuit"]
    if kind == "brickwall":
        c = workloads.brickwall(n, depth, seed=seed)
    elif kind == "hea":
        c = workloads.build_hea(n, depth, rng.uniform(-math.pi, math.pi, n * (depth + 1)))
    elif kind == "qft":
        c = workloads.qft_product(n, seed=seed)
    elif kind == "grover":
        data = n // 2 + 1
        c = workloads.grover(data, int(rng.integers(0, 1 << data)), depth)
        th = rng.uniform(0.0, math.pi, data)  # a state that depends on every bit of the seed
        for q in range(data):
            c.add(C.Ry(float(th[q])), [q])
    elif kind == "qaoa":
        c = workloads.qaoa_maxcut(n, _graph(n, rng), rng.uniform(0, math.pi, depth), rng.uniform(0, math.pi, depth))
    else:
        raise ValueError(kind)
    for k in range(case["measures"]):  # each measurement after a layer of rotations, so that no outcome is certain
        for q in range(c.num_qubits):
            c.add(C.Ry(float(rng.uniform(0.3, math.pi - 0.3))), [q])
        c.measure(int(rng.integers(0, c.num_qubits)), k)
    return c


def _amplitudes(case, seed):
    """A normalised complex128 state on the GPU. ``scrambled``: complex Gaussian amplitudes, as deep random circuits
    leave them; ``product``: independent qubits at random angles, as shallow ansaetze leave them (a few large
    probabilities and a long tail)."""
    n = case["n"]
    if case["state"] == "scrambled":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        x = torch.randn((1 << n, 2), generator=g, device="cuda", dtype=torch.float64)
        psi = torch.view_as_complex(x)
    else:
        rng = np.random.default_rng(seed)
        psi = torch.ones(1, dtype=torch.complex128, device="cuda")
        for th, ph in zip(rng.uniform(0.2, math.pi - 0.2, n), rng.uniform(0, 2 * math.pi, n)):
            q = torch.tensor([math.cos(th / 2), math.sin(th / 2) * complex(math.cos(ph), math.sin(ph))],
                             dtype=torch.complex128, device="cuda")
            psi = (q[:, None] * psi[None, :]).reshape(-1)
    return psi / torch.linalg.vector_norm(psi)


def _strings(case, seed):
    """A Hamiltonian of random Pauli strings on up to four qubits, Z-only strings as common as mixed ones."""
    n, rng = case["n"], random.Random(seed * 7 + 1)
    terms = []
    for k in range(case["terms"]):
        qs = rng.sample(range(n), rng.randint(1, min(4, n)))
        letters = "Z" if k % 2 == 0 else "XYZ"
        terms.append((rng.uniform(-1, 1), [(q, rng.choice(letters)) for q in qs]))
    return terms


def _queries(case, seed):
    n, rng = case["n"], random.Random(seed * 7 + 2)
    one = [(q, rng.choice("XYZ")) for q in rng.sample(range(n), min(3, n))]
    return one, rng.sample(range(n), case["few"]), rng.sample(range(n), case["many"])


def _sets(case, seed):
    rng = np.random.default_rng(seed)
    graphs = [(int(n), _graph(int(n), rng)) for n in rng.integers(case["n_lo"], case["n_hi"] + 1, case["sets"])]
    shape = (case["sets"], case["p"])
    return graphs, rng.uniform(0, math.pi, shape), rng.uniform(0, math.pi, shape)


def prepare(case, seed):
    seed = int(seed) % (1 << 31)
    be = B200SvBackend(seed=seed, precision=case["precision"])
    s = {"kind": case["kind"], "be": be}
    if case["kind"] == "plan":
        c = _circuit(case, seed)
        s["state"] = be.allocate(c.num_qubits)
        s["plan"] = be.compile(c.num_qubits, c.instructions)
        s["uniforms"] = np.random.default_rng(seed + 1).random(case["measures"]) if case["measures"] else None
        s["amps"] = _view(be, s["state"])
        be.synchronize()
    elif case["kind"] == "sweep":
        s["graphs"], s["gammas"], s["betas"] = _sets(case, seed)
    else:
        s["state"] = be.allocate(case["n"])
        be.synchronize()
        _view(be, s["state"]).copy_(torch.view_as_real(_amplitudes(case, seed)))
        torch.cuda.synchronize()
        rng = np.random.default_rng(seed + 2)
        if case["kind"] == "alias":
            s["variates"] = rng.integers(0, 1 << 64, case["shots"], dtype=np.uint64)
        elif case["kind"] == "cumulative":
            s["variates"] = rng.random(case["shots"])
        else:
            s["terms"] = _strings(case, seed)
            s["one"], s["few"], s["many"] = _queries(case, seed)
    return s


def run(state):
    be, kind = state["be"], state["kind"]
    if kind == "plan":
        be.reset_state(state["state"])
        outcomes = state["plan"].execute(state["state"], state["uniforms"])
        return {"amplitudes": state["amps"], "outcomes": np.array(outcomes, dtype=np.int64)}
    if kind in ("alias", "cumulative"):
        shots = be.sample(state["state"], len(state["variates"]), variates=state["variates"], mode=kind)
        return shots.astype(np.int64)
    if kind == "sweep":
        return be.qaoa_sweep(state["graphs"], state["gammas"], state["betas"])
    energy, values = be.expectation_sum(state["state"], state["terms"], with_terms=True)
    return {"energy": energy, "terms": values, "one": be.expectation_value(state["state"], state["one"]),
            "few": be.probabilities(state["state"], state["few"]),
            "many": be.probabilities(state["state"], state["many"])}


# ---- what a pass cannot do without ----------------------------------------------
_PERMUTATION = ("X", "Cnot", "Swap")
_DIAGONAL = ("Z", "S", "Sdg", "T", "Tdg", "Rz", "Phase", "Cz")


def work(case):
    amp = 16 if case["precision"] == "f64" else 8
    kind = case["kind"]
    if kind == "plan":
        c = _circuit(case, 1)
        size = 1 << c.num_qubits
        flops = 0.0
        for i in c.instructions:
            if isinstance(i, C.Measure):
                flops += 3.0 * size
            elif i.gate.name in _DIAGONAL:
                flops += 6.0 * size / 2 ** (len(i.qubits) + len(i.controls))
            elif i.gate.name not in _PERMUTATION:
                flops += 14.0 * size
        return {"bytes": amp * size, "flops": flops}  # the state is written once; it starts as |0...0>
    if kind == "sweep":
        graphs, _, _ = _sets(case, 1)
        flops = sum(2.0 ** n * (case["p"] * (6.0 + 10.0 * n) + 4.0) for n, _ in graphs)
        return {"bytes": sum(8.0 * (len(e) + 2 * case["p"] + 1) for _, e in graphs), "flops": flops}
    size = 1 << case["n"]
    if kind in ("alias", "cumulative"):
        return {"bytes": amp * size + 16.0 * case["shots"], "flops": 5.0 * size}
    return {"bytes": 4.0 * amp * size + 8.0 * (2 ** case["few"] + 2 ** case["many"]),
            "flops": size * (3.0 * case["terms"] + 12.0)}


def tolerance(case):
    kind, single = case["kind"], case["precision"] != "f64"
    if kind in ("alias", "cumulative"):
        return "exact"
    if kind == "sweep":
        return {"rel": 1e-5, "max": 1e-4} if single else {"rel": 1e-12, "max": 1e-11}
    if kind == "readout":  # FP64 sums of the same amplitudes, in any order
        return {"rel": 1e-11, "max": 1e-9}
    if case["precision"] == "tc32":  # split-BF16 products, some 16 significant bits each: 2e-5 off at depth 20
        return {"rel": 2e-4, "max": 1e-2}
    # FP32: 8.5e-6 off after the 5000 gates of the listed Grover search, 4e-7 after a shallow brickwall; FP64: 3e-15
    return {"rel": 4e-5, "max": 4e-3} if single else {"rel": 1e-13, "max": 1e-11}


# ---- the same answers in 64 bits, in plain torch ----------------------------------
def _matrix(g):
    p = g.params
    c, s = (math.cos(p[0] / 2), math.sin(p[0] / 2)) if p else (0.0, 0.0)
    r = math.sqrt(0.5)
    return {"H": lambda: [[r, r], [r, -r]], "X": lambda: [[0, 1], [1, 0]], "Z": lambda: [[1, 0], [0, -1]],
            "T": lambda: [[1, 0], [0, complex(r, r)]], "Tdg": lambda: [[1, 0], [0, complex(r, -r)]],
            "Phase": lambda: [[1, 0], [0, complex(math.cos(p[0]), math.sin(p[0]))]],
            "Rx": lambda: [[c, -1j * s], [-1j * s, c]], "Ry": lambda: [[c, -s], [s, c]],
            "Rz": lambda: [[complex(c, -s), 0], [0, complex(c, s)]],
            "Unitary1q": lambda: [[complex(x) for x in row] for row in g.matrix]}[g.name]()


def _halves(psi, q, controls=()):
    """The amplitudes with qubit q = 0 and = 1 (controls = 1) as views of psi."""
    n = psi.numel().bit_length() - 1
    t = psi.view([2] * n)
    at = [slice(None)] * n
    for k in controls:
        at[n - 1 - k] = slice(1, 2)
    lo, hi = list(at), list(at)
    lo[n - 1 - q], hi[n - 1 - q] = slice(0, 1), slice(1, 2)
    return t[tuple(lo)], t[tuple(hi)]


def _apply(psi, name, gate, qubits, controls):
    if name == "Cnot":
        name, qubits, controls, m = "X", [qubits[1]], [qubits[0]], [[0, 1], [1, 0]]
    elif name == "Cz":
        name, qubits, controls, m = "Z", [qubits[1]], [qubits[0]], [[1, 0], [0, -1]]
    elif name == "Swap":
        for a, b in ((0, 1), (1, 0), (0, 1)):
            _apply(psi, "Cnot", None, [qubits[a], qubits[b]], [])
        return
    else:
        m = _matrix(gate)
    lo, hi = _halves(psi, qubits[0], controls)
    if m[0][1] == 0 and m[1][0] == 0:
        if m[0][0] != 1:
            lo *= m[0][0]
        if m[1][1] != 1:
            hi *= m[1][1]
        return
    a = lo * m[0][0] + hi * m[0][1]
    hi.copy_(lo * m[1][0] + hi * m[1][1])
    lo.copy_(a)


def _exact_plan(case, seed):
    c = _circuit(case, seed)
    n = c.num_qubits
    if (len(c.instructions) << n) > (3400 << 27):
        return None
    u = iter(np.random.default_rng(seed + 1).random(case["measures"])) if case["measures"] else iter(())
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    outcomes = []
    for i in c.instructions:
        if isinstance(i, C.Measure):
            lo, hi = _halves(psi, i.qubit)
            p1 = float((hi.real ** 2 + hi.imag ** 2).sum())
            p0 = float((lo.real ** 2 + lo.imag ** 2).sum())
            one = p0 < 1e-300 or (p1 >= 1e-300 and next(u) < p1)
            (lo if one else hi).zero_()
            psi /= math.sqrt(p1 if one else p0)
            outcomes.append(int(one))
        else:
            _apply(psi, i.gate.name, i.gate, i.qubits, i.controls)
    return {"amplitudes": torch.view_as_real(psi), "outcomes": np.array(outcomes, dtype=np.int64)}


def _pauli_value(psi, string):
    phi = psi.clone()
    for q, letter in string:
        lo, hi = _halves(phi, q)
        if letter == "Z":
            hi.neg_()
        else:
            a = hi * (1 if letter == "X" else -1j)
            hi.copy_(lo * (1 if letter == "X" else 1j))
            lo.copy_(a)
    return float(torch.vdot(psi, phi).real)


def _marginal(prob, qubits):
    n = prob.numel().bit_length() - 1
    t = prob.view([2] * n)
    keep = [n - 1 - q for q in reversed(qubits)]  # bit 0 of the answer's index is qubits[0]
    rest = [d for d in range(n) if d not in keep]
    return t.permute(keep + rest).reshape(1 << len(qubits), -1).sum(dim=1).cpu().numpy()


def _exact_readout(case, seed):
    psi = _amplitudes(case, seed)
    if case["precision"] != "f64":
        psi = psi.to(torch.complex64).to(torch.complex128)
    terms = _strings(case, seed)
    one, few, many = _queries(case, seed)
    values = [_pauli_value(psi, string) for _, string in terms]
    prob = psi.real ** 2 + psi.imag ** 2
    return {"energy": math.fsum(c * v for (c, _), v in zip(terms, values)), "terms": np.array([c * v for (c, _), v in zip(terms, values)]),
            "one": _pauli_value(psi, one), "few": _marginal(prob, few), "many": _marginal(prob, many)}


def _exact_sweep(case, seed):
    graphs, gammas, betas = _sets(case, seed)
    out = np.zeros(len(graphs))
    for k, (n, edges) in enumerate(graphs):
        z = torch.arange(1 << n, device="cuda")
        cut = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
        for i, j in edges:
            cut += ((z >> i) ^ (z >> j)) & 1
        psi = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")
        for g, b in zip(gammas[k], betas[k]):
            psi *= torch.exp(-1j * g * (len(edges) - 2 * cut))
            c, s = math.cos(b), math.sin(b)
            for q in range(n):
                t = psi.view(-1, 2, 1 << q)
                psi = (c * t - 1j * s * t.flip(1)).reshape(-1)
        out[k] = float(((psi.real ** 2 + psi.imag ** 2) * cut).sum())
    return out


def exact(case, seed):
    seed = int(seed) % (1 << 31)
    if case["kind"] == "plan":
        return _exact_plan(case, seed)
    if case["kind"] == "readout":
        return _exact_readout(case, seed)
    if case["kind"] == "sweep":
        return _exact_sweep(case, seed)
    return None  # bitstrings: whole numbers
