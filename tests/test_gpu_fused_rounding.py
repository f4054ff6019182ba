"""The rounding of fused gates does not add up over a circuit in FP64: products of
named gates keep rows of length 1, products of a caller's matrices keep theirs.
n = 6 and 10 are shared-memory passes, n = 14 wide ones."""
import numpy as np
import pytest

from aleph_b200 import circuit as C
from aleph_b200.backend import B200SvBackend

pytestmark = pytest.mark.gpu

LAYERS = 40


def norm2_growth(n, gate):
    """The state's squared norm less 1 after LAYERS of `gate` on every qubit and a
    brick of CNOTs (no two of the gates meet on a qubit without one in between)."""
    insts = []
    for layer in range(LAYERS):
        insts += [C.GateInstance(gate, [q]) for q in range(n)]
        insts += [C.GateInstance(C.Cnot(), [q, (q + 1) % n]) for q in range(layer % 2, n, 2)]
    be = B200SvBackend(seed=0, precision="f64")
    st = be.allocate(n)
    be.apply_stream(st, insts)
    psi = be.statevector(st)
    return float((psi.real.astype(np.longdouble) ** 2).sum() + (psi.imag.astype(np.longdouble) ** 2).sum() - 1)


def row_growth(r):
    return float(2 * np.longdouble(r) ** 2 - 1)


@pytest.mark.parametrize("n", [6, 10, 14])
def test_products_of_named_gates_are_no_worse_than_their_gates(n):
    # gate by gate, each H grows the squared norm by 2 r^2 - 1 = 1.4e-16
    assert abs(norm2_growth(n, C.H())) <= LAYERS * n * row_growth(np.sqrt(0.5))


@pytest.mark.parametrize("n", [6, 10, 14])
def test_a_given_two_qubit_matrix_keeps_its_rows(n):
    # as a Unitary2q and as a UnitaryKq on two qubits, beside named gates
    m = np.eye(4, dtype=complex)[[0, 1, 3, 2]] * (1 + 2.0 ** -51)
    for gate in (C.Unitary2q(m), C.UnitaryKq(m)):
        insts = []
        for layer in range(LAYERS):
            insts += [C.GateInstance(gate, [q, q + 1]) for q in range(0, n, 2)]
            insts += [C.GateInstance(C.S(), [q]) for q in range(0, n, 2)]
        be = B200SvBackend(seed=0, precision="f64")
        st = be.allocate(n)
        be.apply_stream(st, insts)
        gates = LAYERS * n // 2
        want = gates * (float(np.longdouble(1 + 2.0 ** -51) ** 2 - 1))
        assert abs(np.linalg.norm(be.statevector(st)) ** 2 - 1 - want) <= gates * 2.0 ** -52


@pytest.mark.parametrize("n", [6, 10, 14])
def test_products_of_given_matrices_keep_their_rows(n):
    # rows too long by 4 ulp; a product's entries and the arithmetic round by 2^-53 each
    r = np.sqrt(0.5) * (1 + 2.0 ** -50)
    gates = LAYERS * n
    got = norm2_growth(n, C.Unitary1q(np.array([[r, r], [r, -r]], dtype=complex)))
    assert abs(got - gates * row_growth(r)) <= gates * 2.0 ** -52
