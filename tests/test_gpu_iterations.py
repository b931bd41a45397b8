"""Many iterations of a plan on a state beyond the chained size: runs of eight
are planned as one (engine.cpp), and the rest runs the plan itself.  The result
is that of the same iterations one call at a time.
"""
import numpy as np
import pytest

from simulador_quantico_b200 import workloads as wl
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


def one_iteration(n, seed):
    g = wl.grover_search(n, seed, 1)
    return wl.CircuitSpec("one", n, 0, g.gates, [g.calls[1]])


@pytest.mark.parametrize("n,prec,iterations", [(22, "f64", 7), (22, "f64", 24), (22, "f64", 29), (23, "f32", 8), (23, "f32", 45)])
def test_iterations_match_single_runs(sq, n, prec, iterations):
    spec = one_iteration(n, 12345)
    v = random_state(n, seed=n, dtype=np.complex128 if prec == "f64" else np.complex64)
    plan = sq.Plan(spec.build(sq.Circuit()), n, prec).upload()
    passes = plan.stats()["passes"]
    a, b = sq.State(n, prec).upload(v), sq.State(n, prec).upload(v)
    l0 = sq.kernel_launches()
    a.execute(plan, iterations)
    launches = sq.kernel_launches() - l0
    # a pass of 64 MiB takes 21 us: 500 us are saved from 24 iterations on
    assert (launches < passes * iterations) == (iterations >= 24)
    for _ in range(iterations):
        b.execute(plan)
    # the same gates; at most 45 iterations of 2 n gates rounded in another order
    assert a.max_abs_diff(b) < (1e-14 if prec == "f64" else 1e-6)
    a.execute(plan, 0)
    assert abs(a.norm() - 1.0) < (1e-12 if prec == "f64" else 1e-4)


def test_iterations_inside_a_capture(sq):
    """A capture forbids the longer plan's allocation: the plan itself is captured."""
    torch = pytest.importorskip("torch")
    n, iterations = 22, 32
    v = random_state(n, seed=3)
    plan = sq.Plan(one_iteration(n, 99).build(sq.Circuit()), n, "f64").upload()
    a, b = sq.State(n, "f64").upload(v), sq.State(n, "f64").upload(v)
    sq.synchronize()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        a.execute(plan, iterations, s.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    b.execute(plan, iterations)
    assert a.max_abs_diff(b) < 1e-14
