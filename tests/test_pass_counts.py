"""A plan's passes as they run, where they are reported and weighed: a QFT's qubit reversal is one of them."""
import os
import subprocess
import sys

import pytest

import simulador_quantico_b200 as sq
from simulador_quantico_b200 import workloads as wl
from tests import native

WORK = r"""
int main(int argc, char **argv) {
    const int n = 24;
    hgm_circuit *c = hgm_circuit_new();
    const double x[8] = {0, 0, 1, 0, 1, 0, 0, 0}, s = std::sqrt(0.5), h[8] = {s, 0, s, 0, s, 0, -s, 0};
    for (int t = 0; t < n; t++) hgm_circuit_append_op(c, t, 0, 0, h);
    for (int q = 0; q < n / 2; q++) {
        const int a = q, b = n - 1 - q;
        for (int k = 0; k < 3; k++) hgm_circuit_append_op(c, k == 1 ? a : b, int64_t(1) << (k == 1 ? b : a), int64_t(1) << (k == 1 ? b : a), x);
    }
    hgm_plan *p;
    if (hgm_plan_create(c, n, nullptr, &p)) return 2;
    int64_t passes, run;
    hgm_plan_stats(p, nullptr, &passes, nullptr, nullptr);
    hgm_plan_stream(p, nullptr, nullptr, nullptr, &run);
    printf("%d %d", (int)(run < passes), plan_work((Plan *)p) == (double)run * 16.0 * (1 << n));
}
"""


def test_work_counts_the_passes_that_run(tmp_path):
    assert native.run(tmp_path, WORK) == "1 1"


DEBUG = """
import ctypes as C, numpy as np
import simulador_quantico_b200 as sq
from simulador_quantico_b200 import workloads as wl
L = sq.load_dropin("f64")
for n in (8, 18):
    c = wl.qft(n, 0).build(sq.Circuit())
    host = np.zeros(1 << n, np.complex128)
    host[1] = 1
    L.GpuExecutionWrapper(C.c_void_p(host.ctypes.data), C.c_void_p(c.ref_pts("f64")), n, 4, 8, 1, 64, 2, 1)
"""


@pytest.mark.gpu
def test_debug_line_counts_the_passes_that_run():
    out = subprocess.run([sys.executable, "-c", DEBUG], cwd=native.ROOT, env=dict(os.environ, HYBRID_DEBUG="1"),
                         capture_output=True, text=True, timeout=300, check=True)
    for n in (8, 18):
        stats = sq.Plan(wl.qft(n, 0).build(sq.Circuit()), n, "f64").stats()
        assert stats["passes_run"] <= stats["passes"]
        assert f"qubits={n} " in out.stderr and f"passes={stats['passes_run'] or 1}\n" in out.stderr.split(f"qubits={n} ")[1]
