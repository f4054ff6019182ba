"""Edges of the passes and reductions against the oracle or a dense restatement:
wide tiles (smallest states, every class of grouped diagonal, controls on and
off the tile, real and complex matrices with 16 and 32 amplitudes per thread,
gate sequences replaced by the diagonal they multiply out to), shared-memory
passes longer than one staged group, tensor-core passes with more post ops than
a warp has lanes, marginals and Pauli strings on lane, pattern and split qubits,
sweeps over several waves.

Tolerances: FP64 amplitudes 1e-12 and FP32 1e-5 as in the parity tests; FP64
reductions 1e-12 (sums of at most 2^17 terms of a normalised state), FP32 states
are compared on the amplitudes the device holds."""
import numpy as np
import pytest

from aleph_b200 import circuit as C
from aleph_b200 import workloads
from aleph_b200.backend import B200SvBackend, describe_plan
from oracle import oracle
from tests.circuit_gen import random_circuit

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 1e-5, "tc32": 1e-5}


def run_engine(c, precision, **tuning):
    be = B200SvBackend(seed=0, precision=precision)
    for k, v in tuning.items():
        be.set_tuning(k, v)
    st = be.allocate(c.num_qubits)
    be.apply_stream(st, c.instructions)
    return be.statevector(st)


def phase_heavy(n, count, seed):
    """Mostly diagonal gates of every form (sign flips, corner phases on 1 to 3
    qubits, tables, Rz), between dense gates and permutations."""
    rng = np.random.default_rng(seed)
    c = C.Circuit(n)
    for q in range(n):
        c.add(C.Ry(rng.uniform(0, np.pi)), [q])
    for _ in range(count):
        q = [int(x) for x in rng.choice(n, 4, replace=False)]
        t = float(rng.uniform(-np.pi, np.pi))
        kind = rng.integers(0, 10)
        if kind < 2:
            c.add(C.Cz(), q[:2])
        elif kind == 2:
            c.add(C.Ccz(), q[:3])
        elif kind < 5:
            c.add(C.Phase(t), q[:1], controls=q[1:1 + int(rng.integers(0, 3))])
        elif kind == 5:
            c.add(C.Rz(t), q[:1], controls=q[1:1 + int(rng.integers(0, 2))])
        elif kind == 6:
            c.add(C.Unitary2qDiag(np.exp(1j * rng.uniform(0, 6, 4))), q[:2])
        elif kind == 7:
            c.add(C.Cnot(), q[:2])
        elif kind == 8:
            c.add(C.U3(t, 0.3, -0.7), q[:1], controls=q[1:1 + int(rng.integers(0, 3))])
        else:
            c.add(C.H(), q[:1])
    return c


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [12, 13, 17])
@pytest.mark.parametrize("seed", [1, 2])
def test_wide_tiles_match_the_oracle(n, precision, seed):
    c = phase_heavy(n, 160, seed)
    assert len(describe_plan(n, c.instructions, precision, smem_max_n=0)[0]["qubits"]) == 8  # a wide tile
    want, _ = oracle.run(n, c.instructions)
    assert np.abs(run_engine(c, precision, smem_max_n=0) - want).max() <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("tile_r", [4, 5])
@pytest.mark.parametrize("n,phases", [(12, False), (12, True), (13, False), (16, True)])
def test_wide_tiles_real_and_complex_matrices(n, phases, tile_r, precision):
    """One- and two-qubit matrices, real and complex, with and without controls; the
    passes without phases run the smaller kernel."""
    rng = np.random.default_rng(n + tile_r)
    c = C.Circuit(n)
    for _ in range(120):
        q = [int(x) for x in rng.choice(n, 4, replace=False)]
        t = float(rng.uniform(-np.pi, np.pi))
        kind = int(rng.integers(0, 8 if phases else 6))
        if kind == 0:
            c.add(C.Ry(t), q[:1], controls=q[1:1 + int(rng.integers(0, 2))])
        elif kind == 1:
            c.add(C.U3(t, 0.4, 1.1), q[:1], controls=q[1:1 + int(rng.integers(0, 3))])
        elif kind == 2:  # a real pair: fused to one real 4x4
            c.add(C.Ry(t), q[:1]).add(C.H(), q[1:2]).add(C.Cnot(), q[:2]).add(C.Ry(-t), q[1:2])
        elif kind == 3:
            c.add(C.Rx(t), q[:1]).add(C.Cz(), q[:2]).add(C.U3(t, 0.2, 0.1), q[1:2])
        elif kind == 4:
            c.add(C.Cnot(), q[:2])
        elif kind == 5:
            c.add(C.Swap(), q[:2], controls=q[2:3])
        elif kind == 6:
            c.add(C.Phase(t), q[:1], controls=q[1:3])
        else:
            c.add(C.Unitary2qDiag(np.exp(1j * rng.uniform(0, 6, 4))), q[:2])
    passes = describe_plan(n, c.instructions, precision, smem_max_n=0, tile_r=tile_r)
    assert all(len(p["qubits"]) == 8 and p["variant"] == (3 if tile_r == 4 else 0) for p in passes if p["kind"] == 1)
    want, _ = oracle.run(n, c.instructions)
    assert np.abs(run_engine(c, precision, smem_max_n=0, tile_r=tile_r) - want).max() <= TOL[precision]


def test_wide_plans_keep_every_gate():
    for n, c in ((14, random_circuit(14, 300, seed=3)), (25, workloads.qft_product(25, seed=1)),
                 (27, workloads.brickwall(27, 20, seed=2)), (22, workloads.grover(12, 77, 2))):
        wide, warp = describe_plan(n, c.instructions), describe_plan(n, c.instructions, tile_occupancy=2)
        assert sum(p["gates"] for p in wide) == sum(p["gates"] for p in warp) == c.gate_count()
        assert len(wide) <= len(warp)


def diagonal_core_circuit(n, count, seed):
    """Sequences that multiply out to diagonals (Toffolis in CX + T, ZZ rotations,
    CX pairs) and near misses, on overlapping qubits with dense gates between."""
    rng = np.random.default_rng(seed)
    c = C.Circuit(n)
    for q in range(n):
        c.add(C.Ry(rng.uniform(0, np.pi)), [q])
    for _ in range(count):
        a, b, t = (int(x) for x in rng.choice(min(n, 7), 3, replace=False))  # few qubits: blocks meet often
        kind = int(rng.integers(0, 8))
        if kind == 0:
            workloads._toffoli_ct(c, a, b, t)
        elif kind == 1:
            c.add(C.Cnot(), [a, b]).add(C.Rz(rng.uniform(-3, 3)), [b]).add(C.Cnot(), [a, b])
        elif kind == 2:
            c.add(C.Cnot(), [a, b]).add(C.Cnot(), [b, t]).add(C.T(), [t]).add(C.Cnot(), [b, t]).add(C.Cnot(), [a, b])
        elif kind == 3:
            c.add(C.Cnot(), [a, b]).add(C.S(), [b]).add(C.X(), [a]).add(C.Cnot(), [a, b])  # not a diagonal
        elif kind == 4:
            c.add(C.H(), [t]).add(C.Cz(), [a, t]).add(C.Phase(0.3), [b], controls=[t]).add(C.H(), [t])
        elif kind == 5:
            c.add(C.Cnot(), [a, b]).add(C.Cnot(), [a, b])
        elif kind == 6:
            c.add(C.H(), [int(rng.integers(0, n))])
        else:
            c.add(C.Toffoli(), [a, b, t]).add(C.Tdg(), [t]).add(C.Toffoli(), [a, b, t])
    return c


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n,seed", [(13, 1), (13, 2), (14, 3), (18, 4)])
def test_diagonal_cores_match_the_oracle(n, seed, precision):
    c = diagonal_core_circuit(n, 80, seed)
    assert sum(p["gates"] for p in describe_plan(n, c.instructions, precision)) == c.gate_count()
    want, _ = oracle.run(n, c.instructions)
    assert np.abs(run_engine(c, precision) - want).max() <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 12])
def test_shared_memory_passes_longer_than_a_staged_group(n, precision):
    rng = np.random.default_rng(n)
    c = random_circuit(n, 150, seed=n) if n > 3 else C.Circuit(n)
    for k in range(150):
        c.add(C.U3(*rng.uniform(-3, 3, 3)), [int(rng.integers(0, n))])
        if n >= 5 and k % 10 == 0:  # 1024 coefficients each: groups end early
            u, _ = np.linalg.qr(rng.standard_normal((32, 32)) + 1j * rng.standard_normal((32, 32)))
            c.add(C.UnitaryKq(u), [int(x) for x in rng.choice(n, 5, replace=False)])
    want, _ = oracle.run(n, c.instructions)
    for fusion in (1, 0):
        got = run_engine(c, precision, pair_fusion=fusion)
        assert np.abs(got - want).max() <= TOL[precision] * (1 if precision == "f64" else 4)  # 300 FP32 gates


@pytest.mark.parametrize("n", [14, 16])
def test_tensor_core_passes_with_many_post_ops(n):
    rng = np.random.default_rng(n)
    c = C.Circuit(n)
    for q in range(6):
        c.add(C.U3(*rng.uniform(-3, 3, 3)), [q])
    for k in range(33):  # diagonal, across the block's edge: they follow the block
        a, b = int(rng.integers(0, 6)), int(rng.integers(6, n))
        (c.add(C.Cz(), [a, b]) if k % 3 else c.add(C.Phase(0.1 * k), [b], controls=[a]))
        if k % 7 == 0:
            c.add(C.Rz(0.2 * k), [b])
            c.add(C.Unitary2qDiag(np.exp(1j * rng.uniform(0, 6, 4))), [a, b])
    for q in range(n):
        c.add(C.U3(*rng.uniform(-3, 3, 3)), [q])
    want, _ = oracle.run(n, c.instructions)
    assert any(p["post_ops"] > 32 for p in describe_plan(n, c.instructions, "tc32"))
    assert np.abs(run_engine(c, "tc32") - want).max() <= TOL["tc32"]


def random_state(n, precision, seed):
    rng = np.random.default_rng(seed)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    be = B200SvBackend(seed=0, precision=precision)
    st = be.allocate(n)
    be.set_statevector(st, psi / np.linalg.norm(psi))
    return be, st, be.statevector(st)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 3, 5, 6, 9, 13, 17])
def test_marginals_on_lane_pattern_and_split_qubits(n, precision):
    be, st, psi = random_state(n, precision, 7 * n)
    p = np.abs(psi) ** 2
    rng = np.random.default_rng(n)
    sets = [list(range(n)), list(range(n))[::-1], [0], [n - 1], list(range(min(n, 5))), list(range(n // 2, n))]
    sets += [[int(x) for x in rng.choice(n, int(rng.integers(1, n + 1)), replace=False)] for _ in range(4)]
    for qs in sets:
        want = np.zeros(1 << len(qs))
        idx = sum(((np.arange(1 << n) >> q) & 1) << t for t, q in enumerate(qs))
        np.add.at(want, idx, p)
        assert np.abs(be.probabilities(st, qs) - want).max() <= 1e-12


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 4, 6, 11, 15])
def test_pauli_strings_and_sums(n, precision):
    be, st, psi = random_state(n, precision, 11 * n)
    rng = np.random.default_rng(n)
    terms = []
    for k in range(40):
        qs = [int(x) for x in rng.choice(n, int(rng.integers(0, min(n, 4) + 1)), replace=False)]
        terms.append((float(rng.uniform(-1, 1)), [(q, "IXYZ"[int(rng.integers(0, 4))]) for q in qs]))

    def dense(string):
        phi = psi.copy()
        idx = np.arange(1 << n)
        for q, letter in string:
            bit = (idx >> q) & 1
            if letter in "XY":
                phi = phi[idx ^ (1 << q)]
            if letter == "Y":
                phi = phi * np.where(bit == 1, 1j, -1j)
            elif letter == "Z":
                phi = phi * np.where(bit == 1, -1.0, 1.0)
        return float(np.vdot(psi, phi).real)

    want = np.array([c * dense(s) for c, s in terms])
    total, values = be.expectation_sum(st, terms, with_terms=True)
    assert np.abs(values - want).max() <= 1e-12 and abs(total - want.sum()) <= 1e-11
    for (c, s), w in list(zip(terms, want))[:10]:
        assert abs(be.expectation_value(st, s, c) - w) <= 1e-12


@pytest.mark.parametrize("precision,tol", [("f64", 1e-9), ("f32", 2e-5)])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_sweep_passes_with_repeated_edges(p, precision, tol):
    # odd and even layer counts end in different tile kinds; an edge given three times counts three times
    rng = np.random.default_rng(p)
    graphs = []
    for n in (13, 14, 15, 17):
        edges = [(i, (i + 1) % n) for i in range(n)] + [(0, n - 1)] * 3 + [(1, 2), (n - 2, n - 1), (2, n - 2)]
        graphs.append((n, edges))
    gam, bet = rng.uniform(0, np.pi, (4, p)), rng.uniform(0, np.pi, (4, p))
    got = B200SvBackend(seed=0, precision=precision).qaoa_sweep(graphs, gam, bet)
    for k, (n, edges) in enumerate(graphs):
        psi, _ = oracle.run(n, workloads.qaoa_maxcut(n, edges, gam[k], bet[k]).instructions)
        want = sum(0.5 * (1.0 - oracle.expectation(psi, [(i, "Z"), (j, "Z")])) for (i, j) in edges)
        assert abs(got[k] - want) <= tol * max(1.0, abs(want))


@pytest.mark.parametrize("precision,tol", [("f64", 1e-9), ("f32", 2e-5)])
def test_sweep_over_several_waves(precision, tol):
    # 512 MiB of sets share a half of the state buffer: four waves in FP64, two in FP32
    n, edges = 19, [(i, (i + 1) % 19) for i in range(19)] + [(i, i + 9) for i in range(9)]
    rng = np.random.default_rng(3)
    gam, bet = rng.uniform(0, np.pi, (3, 2)), rng.uniform(0, np.pi, (3, 2))
    want = []
    for k in range(3):
        psi, _ = oracle.run(n, workloads.qaoa_maxcut(n, edges, gam[k], bet[k]).instructions)
        want.append(sum(0.5 * (1.0 - oracle.expectation(psi, [(i, "Z"), (j, "Z")])) for (i, j) in edges))
    at = np.arange(250) % 3
    got = B200SvBackend(seed=0, precision=precision).qaoa_sweep([(n, edges)] * 250, gam[at], bet[at])
    assert np.abs(got - np.array(want)[at]).max() <= tol * max(1.0, max(abs(w) for w in want))
