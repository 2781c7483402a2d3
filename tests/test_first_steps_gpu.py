"""The first steps of a world: its step graphs are captured as they are needed
where its kernels were built on the device, and beside any capture of the
caller's."""
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300 import GpuMaceLenia, GpuMaceLeniaBatch  # noqa: E402
from cella_nova_gb300.creature import make_creature  # noqa: E402
from cella_nova_gb300.orchestrator import creature_ring_specs  # noqa: E402

pytestmark = pytest.mark.gpu


def empty_world(cr, stream=None):
    sim = GpuMaceLenia((cr.n, cr.n), cr.C, cr.K, cr.c0, cr.c1, cr.mu, cr.sigma, cr.weights,
                       cr.temp, stream=stream)
    sim.upload_state(cr.seed)
    return sim


def built_world(cr, stream=None):
    sim = empty_world(cr, stream)
    specs, w = creature_ring_specs(cr)
    rings = torch.tensor(w, device="cuda")
    torch.cuda.synchronize()
    sim.build_ring_kernels(specs, rings.data_ptr())
    sim.synchronize()
    return sim


def milliseconds(sim, call):
    sim.synchronize()
    t = time.perf_counter()
    call()
    sim.synchronize()
    return 1e3 * (time.perf_counter() - t)


def test_first_step_captures_its_own_graph_only():
    """Ten graphs of 32 steps in all make the set that a layout change captures
    again in a world with uploaded kernels; one step needs one of them."""
    cr = make_creature(1024, 4, seed=1001, radius=(8, 24), seed_box=256)
    with GpuMaceLenia.from_creature(cr) as sim:
        every = min(milliseconds(sim, lambda: sim.set_graph_layout(0)) for _ in range(5))
    first = []
    for _ in range(5):
        with built_world(cr) as sim:
            first.append(milliseconds(sim, lambda: sim.run_steps(1)))
    assert min(first) < every / 2, (first, every)


@pytest.mark.parametrize("n", [128, 512])
def test_graphs_captured_on_demand_step_the_same(n):
    cr = make_creature(n, 3, seed=1002, radius=(n / 24, n / 8), seed_box=n // 2)
    with built_world(cr) as a, built_world(cr) as b:
        for count in (1, 1, 2, 3, 8, 5, 15):
            a.run_steps(count)
            for _ in range(count):
                b.iterate()
            np.testing.assert_array_equal(a.state(), b.state())
        for s in (a, b):   # re-captures what is there, and only that
            s.set_params(cr.mu, cr.sigma, cr.weights, 0.8)
        a.run_steps(4)
        for _ in range(3):
            b.iterate()
        b.iterate_and_render()
        np.testing.assert_array_equal(a.state(), b.state())

def test_first_step_beside_a_capture_on_another_stream():
    cr = make_creature(128, 2, seed=1003, radius=(6, 16), seed_box=64)
    st, x = torch.cuda.Stream(), torch.zeros(4, device="cuda")
    with built_world(cr) as a, built_world(cr) as b:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            x += 1
            a.run_steps(3)
        b.run_steps(3)
        np.testing.assert_array_equal(a.state(), b.state())
        g.replay()
        torch.cuda.synchronize()
        assert x.tolist() == [1.0] * 4   # capturing runs nothing
        np.testing.assert_array_equal(a.state(), b.state())   # the graph holds no step


def test_last_kernel_set_under_capture():
    """cg_set_kernel_device only enqueues work, also with the last kernel."""
    cr = make_creature(128, 2, seed=1004, radius=(6, 16), seed_box=64)
    spec = torch.view_as_real(torch.tensor(np.asarray(cr.kspec, np.complex64),
                                           device="cuda")).contiguous()
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with empty_world(cr, st.cuda_stream) as a, empty_world(cr) as b:
        a.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            for k in range(cr.K):
                a.set_kernel_device(spec[k].data_ptr(), k)
        with torch.cuda.stream(st):
            g.replay()
        for k in range(cr.K):
            b.set_kernel_device(spec[k].data_ptr(), k)
        a.run_steps(5)
        b.run_steps(5)
        np.testing.assert_array_equal(a.state(), b.state())


def test_first_batch_step_beside_a_capture():
    """A batch that lacks a kernel captures its graphs with its first step."""
    cr = make_creature(64, 2, seed=1005, radius=(4, 10), seed_box=32)

    class Partial(GpuMaceLeniaBatch):
        def set_kernel(self, world, k, spec):
            if k > 0:
                super().set_kernel(world, k, spec)

    st, x = torch.cuda.Stream(), torch.zeros(4, device="cuda")
    with Partial([cr, cr]) as a, Partial([cr, cr]) as b:
        a.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            x += 1
            a.run_steps(5)
        b.run_steps(5)
        np.testing.assert_array_equal(a.state(1), b.state(1))
