"""What planning costs: a variational program plans again for every new set of
angles, so planning has to stay near the cost of reading the gates, and it has
to grow with the number of gates and not with its square. Ratios of two timings
on this machine, the best of several each, with a wide margin."""
import time

import numpy as np
import pytest

from aleph_b200 import circuit as C
from aleph_b200 import workloads
from aleph_b200.backend import describe_plan
from aleph_b200.circuit import flatten


def best(fn, reps):
    out = float("inf")
    for _ in range(reps):
        t = time.perf_counter()
        fn()
        out = min(out, time.perf_counter() - t)
    return out


@pytest.mark.parametrize("n", [10, 12])
def test_planning_an_ansatz_costs_little_more_than_reading_it(n):
    rng = np.random.default_rng(n)
    f = flatten(workloads.build_hea(n, 4, rng.uniform(-np.pi, np.pi, 5 * n)).instructions)
    as_given = best(lambda: describe_plan(n, f, pair_fusion=False), 60)
    fused = best(lambda: describe_plan(n, f), 60)
    assert fused <= 4.0 * as_given  # 1.6 with fusion on the pair's own 4x4, 9 through 64-amplitude vectors


@pytest.mark.parametrize("n", [10, 16])
def test_planning_grows_with_the_number_of_gates(n):
    # thousands of gates that stay on three qubits form one block
    def circuit(count):
        rng = np.random.default_rng(1)
        c = C.Circuit(n)
        for k in range(count):
            a, b = (int(x) for x in rng.choice(3, 2, replace=False))
            c.add(C.Cnot(), [a, b]).add(C.Rz(0.1 * k), [b]).add(C.Ry(0.3), [a])
        return flatten(c.instructions)

    short, long = circuit(1000), circuit(4000)
    assert best(lambda: describe_plan(n, long), 4) <= 8.0 * best(lambda: describe_plan(n, short), 4)
