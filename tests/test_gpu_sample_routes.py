"""The routes of sampling against the oracle's sequential builds, exactly: states of
one CTA, states whose chain runs step by step (half of the basis at one
probability: every sum lies on a binade's edge), and tables of many groups."""
import numpy as np
import pytest

from aleph_b200.backend import B200SvBackend
from oracle import oracle

pytestmark = pytest.mark.gpu


def state(kind, n, rng):
    size = 1 << n
    psi = np.zeros(size, dtype=np.complex128)
    if kind == "half":
        psi[rng.permutation(size)[: max(1, size // 2)]] = 1.0
    elif kind == "one":
        psi[int(rng.integers(0, size))] = 1j
    elif kind == "uniform":
        psi += 1.0
    elif kind == "scrambled":
        psi = rng.standard_normal(size) + 1j * rng.standard_normal(size)
    elif kind == "product":
        psi = np.ones(1, dtype=np.complex128)
        for th in rng.uniform(0.2, np.pi - 0.2, n):
            psi = np.kron(np.array([np.cos(th / 2), 1j * np.sin(th / 2)]), psi)
    return psi / np.linalg.norm(psi)


def on_device(kind, n, precision, seed):
    be = B200SvBackend(seed=0, precision=precision)
    st = be.allocate(n)
    be.set_statevector(st, state(kind, n, np.random.default_rng(seed)))
    return be, st, be.statevector(st)  # the state as the device holds it


def check_alias(be, st, psi):
    prob, alias = oracle.alias_table(psi.real * psi.real + psi.imag * psi.imag)
    edge = np.clip(np.floor(prob * 2.0 ** 32), 0, 2 ** 32 - 1).astype(np.uint64)
    idx = np.arange(psi.size, dtype=np.uint64) << np.uint64(32)
    words = np.concatenate([idx | np.uint64(0xFFFFFFFF), idx | edge, idx | (edge - (edge > 0).astype(np.uint64))])
    got = be.sample(st, words.size, variates=words, mode="alias")
    i, v = (words >> np.uint64(32)).astype(np.int64), (words & np.uint64(0xFFFFFFFF)).astype(np.float64) / 2.0 ** 32
    assert np.array_equal(got, np.where(v < prob[i], i, alias[i].astype(np.int64)).astype(np.uint64))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind,n", [("half", 11), ("half", 13), ("half", 17), ("scrambled", 20), ("product", 20)])
def test_alias_tables_of_long_chains(kind, n, precision):
    check_alias(*on_device(kind, n, precision, n))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind", ["scrambled", "product", "half", "one", "uniform"])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 9, 10, 11, 12])
def test_sampling_small_states(n, kind, precision):
    be, st, psi = on_device(kind, n, precision, 31 * n)
    check_alias(be, st, psi)
    sums = np.add.accumulate(psi.real * psi.real + psi.imag * psi.imag)  # left to right, in order
    rng = np.random.default_rng(n)
    edge = sums[rng.integers(0, psi.size, 60)] / sums[-1]
    u = np.concatenate([edge, np.nextafter(edge, 0), np.nextafter(edge, 2), [0.0, 1 - 2.0 ** -53],
                        rng.random(64)]).clip(0, 1 - 2.0 ** -53)
    want = np.searchsorted(sums, u * sums[-1], side="right")
    want = np.where(want < psi.size, want, np.flatnonzero(psi)[-1]).astype(np.uint64)
    assert np.array_equal(be.sample(st, u.size, variates=u, mode="cumulative"), want)


@pytest.mark.parametrize("mode", ["alias", "cumulative"])
@pytest.mark.parametrize("n", [4, 10, 13])
def test_sampling_refuses_a_state_that_is_not_normalised(n, mode):
    from aleph_b200 import abi
    from aleph_b200.backend import BackendError

    for bad in (0.5, np.nan, np.inf):
        be = B200SvBackend(seed=0)
        st = be.allocate(n)
        psi = np.zeros(1 << n, dtype=np.complex128)
        psi[0], psi[-1] = 0.5, bad
        be.set_statevector(st, psi)
        with pytest.raises(BackendError) as e:
            be.sample(st, 8, variates=np.zeros(8, np.uint64 if mode == "alias" else np.float64), mode=mode)
        assert e.value.status == abi.INVALID_STATE


def test_many_shots_of_a_small_state():
    # more shots than one CTA takes: each CTA builds the table for its share
    be, st, psi = on_device("scrambled", 7, "f64", 5)
    words = np.random.default_rng(1).integers(0, 1 << 64, 100_003, dtype=np.uint64)
    assert np.array_equal(be.sample(st, words.size, variates=words, mode="alias"), oracle.sample_alias(psi, words))


@pytest.mark.parametrize("n", [19, 21, 22])
def test_cumulative_draws_up_to_and_above_a_segment_per_chunk(n):
    # n = 21: 1024 blocks and chunks, one kernel scans them and nothing is composed
    be, st, psi = on_device("scrambled", n, "f64", n)
    sums = np.add.accumulate(psi.real * psi.real + psi.imag * psi.imag)
    rng = np.random.default_rng(n)
    edge = sums[rng.integers(0, psi.size, 60)] / sums[-1]
    u = np.concatenate([edge, np.nextafter(edge, 0), np.nextafter(edge, 2), [0.0, 1 - 2.0 ** -53]]).clip(0, 1 - 2.0 ** -53)
    want = np.searchsorted(sums, u * sums[-1], side="right")
    want = np.where(want < psi.size, want, np.flatnonzero(psi)[-1]).astype(np.uint64)
    assert np.array_equal(be.sample(st, u.size, variates=u, mode="cumulative"), want)
