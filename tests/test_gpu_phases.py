"""Diagonal gates that the planner joins, cancels or multiplies out, against the
oracle: entries that are no phases, phases next to +1 and -1, and long runs of
small rotations. Every circuit runs on a wide plan (n = 14), a shared-memory one
(n = 10) and, in TC32, on block passes.

Tolerances: FP64 1e-12 and FP32 / TC32 1e-5 on the amplitudes, as in the parity
tests."""
import numpy as np
import pytest

from aleph_b200 import circuit as C
from aleph_b200.backend import B200SvBackend
from oracle import oracle

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 1e-5, "tc32": 1e-5}


def check(n, insts, precision):
    want, _ = oracle.run(n, insts)
    be = B200SvBackend(seed=0, precision=precision)
    if precision == "tc32":
        be.set_tuning("renormalize", 0)  # the blocks are not unitary
    st = be.allocate(n)
    be.apply_stream(st, insts)
    assert np.abs(be.statevector(st) - want).max() <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "f32", "tc32"])
@pytest.mark.parametrize("n", [10, 14])
@pytest.mark.parametrize("pair", [(0.5, 0.5), (2.0, 0.25), (0.0, 0.0), (-1.0, 0.5), (0.5j, 0.5j), (1 + 1e-9, 1.0)])
def test_diagonals_that_are_no_phases_keep_their_modulus(pair, n, precision):
    # a TiledBlock's matrices are taken without a unitarity check
    def diag(c, q):
        return C.GateInstance(C.Unitary1q(np.diag([1.0, c])), [q])

    def cdiag(c, q):
        return C.GateInstance(C.Unitary1q(np.diag([1.0, c])), [q[1]], [q[0]])

    insts = [C.GateInstance(C.H(), [q]) for q in range(3)]
    insts.append(C.TiledBlock([diag(pair[0], 0), diag(pair[1], 0), cdiag(pair[0], [1, 2]), cdiag(pair[1], [1, 2])], 15))
    insts.append(C.GateInstance(C.H(), [0]))
    insts.append(C.TiledBlock([C.GateInstance(C.Cnot(), [0, 1]), diag(pair[0], 1), diag(pair[1], 1),
                               C.GateInstance(C.Cnot(), [0, 1])], 15))
    check(n, insts, precision)


@pytest.mark.parametrize("precision", ["f64", "f32", "tc32"])
@pytest.mark.parametrize("n", [10, 14])
@pytest.mark.parametrize("eps", [1e-8, -1e-10, 3e-12, 0.0])
def test_phases_next_to_a_sign_flip(eps, n, precision):
    # cos(pi - 1e-8) rounds to -1: the angle is in the imaginary part alone
    insts = [C.GateInstance(C.H(), [q]) for q in range(4)]
    insts += [C.GateInstance(C.Rz(np.pi - eps), [0]), C.GateInstance(C.CRz(np.pi - eps), [1, 2])]
    insts += [C.GateInstance(C.Phase(1.0), [3]), C.GateInstance(C.Phase(np.pi - 1.0 - eps), [3])]
    insts += [C.GateInstance(C.H(), [q]) for q in range(4)]
    insts += [C.GateInstance(C.Cnot(), [0, 1]), C.GateInstance(C.Rz(np.pi / 2 - eps), [1]),
              C.GateInstance(C.Cnot(), [0, 1]), C.GateInstance(C.Cnot(), [0, 2]), C.GateInstance(C.Cnot(), [0, 2])]
    insts += [C.GateInstance(C.Phase(np.pi - eps), [2], [0])]
    check(n, insts, precision)


@pytest.mark.parametrize("n", [10, 14])
@pytest.mark.parametrize("angle,count", [(1e-14, 3000), (3e-13, 40), (1e-15, 2000)])
def test_long_runs_of_small_rotations_add_up(angle, count, n):
    # ZZ rotations and phases on the same qubits: each is far below the tolerance, their sum is not
    insts = [C.GateInstance(C.H(), [q]) for q in range(3)]
    for _ in range(count):
        insts += [C.GateInstance(C.Cnot(), [0, 1]), C.GateInstance(C.Rz(angle), [1]), C.GateInstance(C.Cnot(), [0, 1]),
                  C.GateInstance(C.Phase(angle), [2])]
    insts += [C.GateInstance(C.H(), [q]) for q in range(3)]
    check(n, insts, "f64")


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 9, 10, 12, 14])
def test_phase_polynomials_between_gates(n, precision):
    # a thread per amplitude in shared-memory passes, more threads than amplitudes below six qubits
    rng = np.random.default_rng(n)

    def poly():
        masks = [tuple(int(m) for m in rng.integers(1, 1 << n, int(rng.integers(1, 3)))) for _ in range(12)]
        return C.DiagonalPhase(n, [C.PhaseTerm(m, float(rng.uniform(-3, 3))) for m in masks])

    insts = [C.GateInstance(C.H(), [q]) for q in range(n)]
    insts += [poly(), C.GateInstance(C.T(), [0]), poly()]
    insts += [C.GateInstance(C.U3(0.3, 0.4 + q, -1.1), [q]) for q in range(n)] + [poly()]
    check(n, insts, precision)
