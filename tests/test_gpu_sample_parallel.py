"""The parallel sampling builds against the oracle's sequential ones: the whole
alias table (every basis state, at and around its threshold) and the inverse
CDF at and around bin boundaries, for states whose chains stress the parts of
the build: chunks that jump binades, exact ties, zero bins, one-sided stacks.
Bitstrings are whole numbers and the chains are reproduced bit for bit, so the
comparison is exact."""
import numpy as np
import pytest

from aleph_b200.backend import B200SvBackend
from oracle import oracle

pytestmark = pytest.mark.gpu


def make_state(kind: str, n: int, rng) -> np.ndarray:
    size = 1 << n
    if kind == "scrambled":
        psi = rng.standard_normal(size) + 1j * rng.standard_normal(size)
    elif kind == "product":  # a few large probabilities and a long tail: V jumps many binades
        psi = np.ones(1, dtype=np.complex128)
        for th in rng.uniform(0.2, np.pi - 0.2, n):
            psi = np.kron(np.array([np.cos(th / 2), 1j * np.sin(th / 2)]), psi)
    elif kind == "subspace":  # most bins exactly zero
        psi = np.zeros(size, dtype=np.complex128)
        at = rng.choice(size, max(1, size // 16), replace=False)
        psi[at] = rng.standard_normal(at.size) + 1j * rng.standard_normal(at.size)
    elif kind == "ghz":
        psi = np.zeros(size, dtype=np.complex128)
        psi[0] = psi[-1] = 1.0
    elif kind == "uniform":
        psi = np.ones(size, dtype=np.complex128)
    elif kind == "ties":  # |a|^2 = odd^2 * 2^-54: half a unit of every sum in [1/2, 1)
        m = 2 * rng.integers(1 << 10, 1 << 11, size) + 1
        psi = m * 2.0 ** -27 + 0j
        psi[0] = np.sqrt(max(0.0, 1.0 - float((psi[1:].real ** 2).sum())))
        return psi
    return psi / np.linalg.norm(psi)


def device_state(psi, precision):
    be = B200SvBackend(seed=0, precision=precision)
    st = be.allocate(psi.size.bit_length() - 1)
    be.set_statevector(st, psi)
    return be, st, be.statevector(st)  # the state as the device holds it


CASES = [(k, n) for k in ("scrambled", "product", "subspace", "ghz", "uniform") for n in (1, 10, 11, 13, 16)]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind,n", CASES)
def test_alias_table_identical(kind, n, precision):
    be, st, psi = device_state(make_state(kind, n, np.random.default_rng(100 + n)), precision)
    size = psi.size
    prob, alias = oracle.alias_table(psi.real * psi.real + psi.imag * psi.imag)
    edge = np.clip(np.floor(prob * 2.0 ** 32), 0, 2 ** 32 - 1).astype(np.uint64)
    idx = np.arange(size, dtype=np.uint64) << np.uint64(32)
    words = np.concatenate([idx | np.uint64(0xFFFFFFFF), idx | edge, idx | (edge - (edge > 0).astype(np.uint64))])
    got = be.sample(st, words.size, variates=words, mode="alias")
    i, v = (words >> np.uint64(32)).astype(np.int64), (words & np.uint64(0xFFFFFFFF)).astype(np.float64) / 2.0 ** 32
    assert np.array_equal(got, np.where(v < prob[i], i, alias[i].astype(np.int64)).astype(np.uint64))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind,n", [(k, n) for k in ("scrambled", "product", "subspace", "ghz", "uniform", "ties")
                                    for n in (3, 11, 12, 16)])
def test_cumulative_identical_at_bin_boundaries(kind, n, precision):
    be, st, psi = device_state(make_state(kind, n, np.random.default_rng(200 + n)), precision)
    sums = np.add.accumulate(psi.real * psi.real + psi.imag * psi.imag)  # left to right, in order
    rng = np.random.default_rng(n)
    edge = sums[rng.integers(0, psi.size, 60)] / sums[-1]
    u = np.concatenate([edge, np.nextafter(edge, 0), np.nextafter(edge, 2), [0.0, 1 - 2.0 ** -53],
                        rng.random(64)]).clip(0, 1 - 2.0 ** -53)
    want = np.searchsorted(sums, u * sums[-1], side="right")  # the first bin with target < S_i
    want = np.where(want < psi.size, want, np.flatnonzero(psi)[-1]).astype(np.uint64)
    if precision == "f64":
        assert np.array_equal(want, oracle.sample_cumulative(psi, u))
    assert np.array_equal(be.sample(st, u.size, variates=u, mode="cumulative"), want)
