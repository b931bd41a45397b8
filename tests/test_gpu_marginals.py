"""Marginals and the argmax over every shape of mask, against numpy.

The kernels put the lowest five index bits on the lanes, split the rest into
units and chunks, and keep partial sums in fixed scratch: the masks below cover
no, some and all lane bits, no and all high bits, states smaller than a warp,
one and many chunks, and outputs below and above the scratch.
"""
import numpy as np
import pytest

from tests.helpers import random_state

pytestmark = pytest.mark.gpu

ALL = -1
CASES = [(1, 0), (1, 1), (3, 0b101), (5, 0b01010), (6, 0b100000), (6, ALL), (9, 0b101010101), (13, 0),
         (13, 0b11111), (13, 0x1FE0), (14, 0b10000000000001), (16, 0x5555), (16, 0xFFFE), (16, 0x7FFF), (16, ALL),
         (20, 0x3FF), (20, 0xFFC00), (20, 0xAAAAA), (20, 0x7FFFF), (20, ALL)]


def marginal(v, n, mask):
    p = np.abs(v.astype(np.complex128)) ** 2
    rest = tuple(n - 1 - b for b in range(n) if not (mask >> b) & 1)
    return p.reshape((2,) * n).sum(axis=rest).reshape(-1)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,mask", CASES)
def test_marginals(sq, n, mask, prec):
    mask = (1 << n) - 1 if mask == ALL else mask
    v = random_state(n, seed=n, dtype=np.complex128 if prec == "f64" else np.complex64)
    want = marginal(v, n, mask)
    st = sq.State(n, prec).upload(v)
    got = st.marginal_probs(mask)
    # sums of at most 2^20 positive products that add up to 1, in FP64:
    # pairwise over lanes, warps and chunks, at most 2^11 terms in a row
    assert np.abs(got - want).max() < 1e-12
    x, p = st.marginal_argmax(mask)
    assert x == int(np.argmax(want)) and abs(p - want.max()) < 1e-12
    st.free()


@pytest.mark.parametrize("mask", [0b1, 0b11000000, (1 << 12) - 1])
def test_argmax_ties_take_the_lowest(sq, mask):
    """A uniform state: every value has the same probability."""
    n = 12
    st = sq.State(n, "f64").upload(np.full(1 << n, 2.0 ** (-n / 2), dtype=np.complex128))
    x, p = st.marginal_argmax(mask)
    assert x == 0 and p == 2.0 ** -bin(mask).count("1")


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 4, 11, 20])
def test_norm_and_measure_from_one_read(sq, n, prec):
    v = random_state(n, seed=40 + n, dtype=np.complex128 if prec == "f64" else np.complex64)
    st = sq.State(n, prec).upload(v)
    p = np.abs(v.astype(np.complex128)) ** 2
    assert abs(st.norm() - p.sum()) < 1e-12
    for bit in {0, n - 1}:
        one = p[((np.arange(1 << n) >> bit) & 1) == 1].sum()
        assert abs(st.prob_one(bit) - one) < 1e-12
    outcome, q = st.measure_qubit(0, 2.0)  # P(0) is never above 2: the outcome is 1
    one = p[(np.arange(1 << n) >> (n - 1)) & 1 == 1].sum()
    assert outcome == 1 and abs(q - one) < 1e-12
    st.free()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 2, 9, 10, 11, 12, 13, 21])
def test_set_basis(sq, n, prec):
    """Every size from less than a block's run to many, first, last and odd indices."""
    st = sq.State(n, prec)
    for index in sorted({0, 1, (1 << n) - 1, (1 << n) // 3, (1 << n) // 2}):
        st.upload(np.full(1 << n, 2 + 3j))
        got = st.set_basis(index).download()
        assert got[index] == 1 and np.count_nonzero(got) == 1
    st.free()
