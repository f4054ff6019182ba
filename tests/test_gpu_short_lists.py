"""Gate lists that fit a pass or two: the planner takes warp or wide tiles, whichever
its cost table makes cheaper. Either way the state is the oracle's (FP64 1e-12,
FP32 1e-5), and one gate on a low qubit, which a wide tile could only reach by
two exchanges, goes to a warp tile."""
import numpy as np
import pytest

from aleph_b200 import circuit as C
from aleph_b200.backend import B200SvBackend, describe_plan
from oracle import oracle
from tests.circuit_gen import random_circuit

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 1e-5}


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [13, 16, 22])
@pytest.mark.parametrize("count", [1, 3, 9, 30, 64, 65])
def test_short_lists_match_the_oracle(count, n, precision):
    c = random_circuit(n, count, seed=100 * n + count)
    c.measure(1, 0)  # a second list behind a measurement
    for inst in random_circuit(n, count, seed=count).instructions:
        c.instructions.append(inst)
    for q in range(n):  # a state with weight everywhere
        c.instructions.insert(0, C.GateInstance(C.Ry(0.4 + q), [q]))
    u = [0.7]
    want, _ = oracle.run(n, c.instructions, u)
    be = B200SvBackend(seed=0, precision=precision)
    st = be.allocate(n)
    be.apply_stream(st, c.instructions, measure_uniforms=u)
    assert np.abs(be.statevector(st) - want).max() <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_one_gate_on_a_low_qubit_takes_a_warp_tile(precision):
    for gate, qubits in ((C.H(), [0]), (C.U3(0.3, 0.1, 0.2), [2]), (C.Cnot(), [20, 1])):
        (p,) = describe_plan(24, [C.GateInstance(gate, qubits)], precision)
        assert p["kind"] == "tile" and len(p["qubits"]) == 5
