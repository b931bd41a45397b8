"""Copies of a state between host and device memory (csrc/hostcopy.cpp)."""
import numpy as np
import pytest

from tests import native

ROUTE = r"""
namespace hgm { bool staged(const void *host, size_t bytes); }
int main() {
    const size_t mib = size_t(1) << 20, n = 4 * mib;
    if (hgm_init(0)) return 2;
    char *page = (char *)aligned_alloc(4096, n), *half = (char *)aligned_alloc(4096, n), *man;
    void *pin;
    if (hgm_pinned_alloc(n, &pin) || cudaHostRegister(half, n / 2, cudaHostRegisterDefault) || cudaMallocManaged(&man, n)) return 3;
    printf("%d %d %d\n", staged(page, n), staged(page, mib), staged(page, mib - 1));
    printf("%d %d %d\n", staged(pin, n), staged((char *)pin + 100, n - 100), staged(pin, mib - 1));
    printf("%d %d %d %d\n", staged(half, n), staged(half, n / 2), staged(half + n / 2, n / 2), staged(man, n));
}
"""


@pytest.mark.gpu
def test_page_locked_memory_is_copied_directly(tmp_path):
    assert native.run(tmp_path, ROUTE).split("\n")[:3] == ["1 1 0", "0 0 0", "1 0 1 0"]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [15, 16, 20, 24])
def test_page_locked_round_trip(sq, n):
    import ctypes as C

    from simulador_quantico_b200._lib import check, lib

    rng = np.random.default_rng(n)
    a, b = sq.PinnedArray((1 << n,), np.complex128), sq.PinnedArray((1 << n,), np.complex128)
    a.array[:] = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    st = sq.State(n, "f64")
    check(lib.hgm_state_upload(st.h, C.c_void_p(a.ptr), a.nbytes))
    check(lib.hgm_state_download(st.h, C.c_void_p(b.ptr), b.nbytes))
    assert np.array_equal(a.array, b.array) and np.array_equal(st.download(), a.array)
    st.free()
