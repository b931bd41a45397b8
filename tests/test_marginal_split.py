"""How the read-out of a register is split over blocks (csrc/kernels.cu marginal_chunks): the rule on the CPU, the sums
against numpy on the device, for masks in the low index bits, where one value's sum runs over the whole state."""
import numpy as np
import pytest

from tests import native
from tests.helpers import random_state

RULE = r"""
int main() {
    for (int n = 12; n <= 34; n++)
        for (int lo = 0; lo <= 11; lo++)
            for (int hi = 0; hi <= n - 11 && hi + lo < n; hi++) {
                const uint64_t mask = ((uint64_t(1) << lo) - 1) | (((uint64_t(1) << hi) - 1) << (n - hi));
                const long long runs = 1ll << (n - 11), M = 1ll << __builtin_popcountll(mask);
                long long units = 0, few = 0;
                const int nch = marginal_chunks(n, mask, MARG_SUMS, &units);
                // blocks for every SM wherever there are four runs for each
                if (units < std::min<long long>(256, std::max(1ll, runs / 8))) printf("%d %d %d: %lld units\n", n, lo, hi, units);
                if (nch > 1 && (M * nch > MARG_SUMS || marginal_sums(n, mask) != M * nch)) printf("%d %d %d: sums\n", n, lo, hi);
                const int nf = marginal_chunks(n, mask, REDUCE_SCRATCH_BLOCKS, &few);
                if (nf > 1 && M * nf > REDUCE_SCRATCH_BLOCKS) printf("%d %d %d: few\n", n, lo, hi);
                if ((runs << 11 >> lo >> hi) << (lo + hi) != 1ll << n || units % nch || runs % units) printf("%d %d %d: split\n", n, lo, hi);
            }
    printf("end\n");
}
"""


def test_every_mask_has_blocks(tmp_path):
    assert native.run(tmp_path, RULE) == "end\n"


def marginal(v, n, mask):
    p = np.abs(v.astype(np.complex128)) ** 2
    rest = tuple(n - 1 - b for b in range(n) if not (mask >> b) & 1)
    return p.reshape((2,) * n).sum(axis=rest).reshape(-1)


LOW = [(1 << m) - 1 for m in (1, 4, 5, 6, 8, 10, 11, 12, 13)]
MIXED = [0b10, 0b11111100000, 0x3FF | 1 << 20, 0x7FF | 3 << 19, 0x0F | 0x1F << 16, 0x7FF | 0xFF << 13, 0x700 | 1 << 11]


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("mask", LOW + MIXED)
@pytest.mark.parametrize("n", [14, 21])
def test_low_masks(sq, n, mask, prec):
    mask &= (1 << n) - 1
    v = random_state(n, seed=n, dtype=np.complex128 if prec == "f64" else np.complex64)
    want = marginal(v, n, mask)
    st = sq.State(n, prec).upload(v)
    # sums of at most 2^20 positive products that add up to 1, in FP64, at most 2^11 in a row
    assert np.abs(st.marginal_probs(mask) - want).max() < 1e-12
    x, p = st.marginal_argmax(mask)
    assert x == int(np.argmax(want)) and abs(p - want.max()) < 1e-12
    st.free()


@pytest.mark.gpu
@pytest.mark.parametrize("mask", [0x1F, 0x3FF, 0x7FF, 0x7FF | 3 << 18])
def test_ties_take_the_lowest(sq, mask):
    n = 20
    st = sq.State(n, "f64").upload(np.full(1 << n, 2.0 ** (-n / 2), dtype=np.complex128))
    x, p = st.marginal_argmax(mask)
    assert x == 0 and p == 2.0 ** -bin(mask).count("1")
    st.free()


@pytest.mark.gpu
def test_served_low_masks(sq):
    """The server's slots take the larger scratch at the first request that can use it."""
    n = 18
    masks = [0, 0x3FF, 0b1, 0x7FF, (1 << n) - 1, 0x7FF | 1 << 17, 0x3F]
    rng = np.random.default_rng(3)
    c = sq.Circuit()
    for q in range(n):  # a product state: each qubit's most likely value is known
        a = rng.uniform(0.1, 0.6) + (np.pi / 2 if q % 3 == 0 else 0.0)
        c.append_op(q, 0, 0, [np.cos(a), -np.sin(a), np.sin(a), np.cos(a)])
    st = sq.State(n, "f64").set_basis(0).execute(sq.Plan(c, n, "f64"))
    v = st.download()
    server = sq.Server("f64", max_inflight=2)
    ids = [server.submit(c, n, 0, m) for m in masks]
    done = {r["id"]: r for r in server.drain(len(ids))}
    for i, m in zip(ids, masks):
        want = marginal(v, n, m)
        assert done[i]["status"] == 0
        if m:
            assert done[i]["argmax"] == int(np.argmax(want)) and abs(done[i]["pmax"] - want.max()) < 1e-12
    server.close()
    st.free()
