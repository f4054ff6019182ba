"""A compiled plan on states of either precision: the plan is compiled by one
handle and executed on its own states and on those of a handle of the other
precision, in turn, against the oracle (FP64 states 1e-12, FP32 states 1e-5)."""
import numpy as np
import pytest

from aleph_b200 import circuit as C
from aleph_b200.backend import B200SvBackend
from oracle import oracle
from tests.circuit_gen import random_circuit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32", "tc32"])
@pytest.mark.parametrize("n", [10, 14])
def test_a_plan_runs_on_states_of_either_precision(n, precision):
    c = random_circuit(n, 80, seed=n)
    for q in range(n):  # real and complex matrices: paired, duplicated and plain coefficients
        c.add(C.Ry(0.3 + q), [q]).add(C.U3(0.2 * q, 0.4, 1.1), [(q + 1) % n])
    want, _ = oracle.run(n, c.instructions)
    be = B200SvBackend(seed=0, precision=precision)
    other = B200SvBackend(seed=0, precision="f32" if precision == "f64" else "f64")
    plan = be.compile(n, c.instructions)
    states = [(be, be.allocate(n)), (other, other.allocate(n))]
    for owner, st in states * 2:
        owner.reset_state(st)
        owner.synchronize()
        plan.execute(st)
        be.synchronize()
        tol = 1e-12 if owner.precision == "f64" else 1e-5
        assert np.abs(owner.statevector(st) - want).max() <= tol
