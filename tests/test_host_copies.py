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


# pthread_create of the program's own: it fails where `fail_from` says so
THREADS = r"""
#include <dlfcn.h>
#include <pthread.h>
#include <atomic>
#include <cerrno>
#include <functional>
#include <thread>
static std::atomic<int> started{0}, fail_from{1 << 30};
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
    if (started++ >= fail_from) return EAGAIN;
    return ((int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}
namespace hgm { void run_shares(int n, const std::function<void(int)> &share); }
int main(int argc, char **argv) {
    if (atoi(argv[1])) {  // whole copies
        const int n = 18;
        const size_t bytes = size_t(16) << n;
        hgm_state *s;
        double *a = (double *)malloc(bytes), *b = (double *)malloc(bytes);
        for (size_t i = 0; i < bytes / 8; i++) a[i] = (double)i;
        if (hgm_init(0) || hgm_state_create(n, HGM_F64, &s)) return 2;
        for (int k = 0; k < 4; k++) {
            for (size_t i = 0; i < bytes / 8; i++) b[i] = 0;
            started = 0;
            fail_from = k;
            if (hgm_state_upload(s, a, bytes) || hgm_state_download(s, b, bytes)) return 3;
            for (size_t i = 0; i < bytes / 8; i++)
                if (b[i] != a[i]) return 4;
        }
    }
    for (int k = 0; k < 4; k++) {
        std::atomic<int> done[4] = {};
        started = 0;
        fail_from = k;
        run_shares(4, [&](int t) { done[t]++; });
        printf("%d%d%d%d-%d ", (int)done[0], (int)done[1], (int)done[2], (int)done[3], (int)started);
    }
}
"""
SHARES = ["1111-1", "1111-2", "1111-3", "1111-3"]  # each taken once; the threads asked for


def test_every_share_is_taken_without_threads(tmp_path):
    assert native.run(tmp_path, THREADS, 0).split() == SHARES


@pytest.mark.gpu
def test_copies_without_threads(tmp_path):
    assert native.run(tmp_path, THREADS, 1).split() == SHARES


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 20])
def test_two_threads_copy_at_once(sq, n):
    """Whichever way each copy goes, every one is whole."""
    import threading

    states = [sq.State(n, "f64") for _ in range(3)]
    hosts = [np.random.default_rng(k).standard_normal(1 << n) + 1j * k for k in range(3)]
    bad = []

    def work(k):
        for r in range(8):
            states[k].upload(hosts[k] * (r + 1))
            if not np.array_equal(states[k].download(), hosts[k] * (r + 1)):
                bad.append((k, r))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for s in states:
        s.free()


TURNS = r"""
#include <thread>
namespace hgm { std::unique_lock<std::mutex> take_chunks(size_t bytes); }
int main() {
    const size_t mib = size_t(1) << 20;
    auto mine = take_chunks(4 * mib), large = take_chunks(256 * mib);
    auto other = [&] { std::thread([&] { printf("%d", (int)take_chunks(4 * mib).owns_lock()); }).join(); };
    printf("%d%d", (int)mine.owns_lock(), (int)large.owns_lock());
    other();
    mine.unlock();
    other();
}
"""


def test_a_second_copy_does_not_wait_for_the_small_set(tmp_path):
    assert native.run(tmp_path, TURNS) == "1101"
