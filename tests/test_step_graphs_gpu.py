"""The step graphs: every split of a step count into graphs of 8, 4, 2 and 1
steps (batch: 4 and 1), and a world whose graphs do not exist yet."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300 import GpuMaceLenia, GpuMaceLeniaBatch  # noqa: E402
from cella_nova_gb300.creature import make_creature  # noqa: E402
from cella_nova_gb300.orchestrator import creature_ring_specs  # noqa: E402

pytestmark = pytest.mark.gpu


def creature(n, C, seed):
    return make_creature(n, C, seed=seed, radius=(max(2.0, n / 16), n / 6), seed_box=n // 2)


@pytest.mark.parametrize("n", [64, 512])   # one stream, and a stream per channel
@pytest.mark.parametrize("counts", [(1, 2, 3), (5, 7), (6, 1, 14), (0, 15)])
def test_step_counts_equal_single_steps(n, counts):
    cr = creature(n, 3, 900 + n)
    with GpuMaceLenia.from_creature(cr) as a, GpuMaceLenia.from_creature(cr) as b:
        for c in counts:
            a.run_steps(c)
            for _ in range(c):
                b.iterate()
            np.testing.assert_array_equal(a.state(), b.state())


@pytest.mark.parametrize("mode", [0, 1])
def test_batch_step_counts_equal_single_worlds(mode):
    # ten worlds of one side: more than mode 1's lane groups
    crs = [creature(64, 1 + i % 3, 910 + i) for i in range(10)] + [creature(512, 2, 930)]
    with GpuMaceLeniaBatch(crs) as b:
        for side in (64, 512):
            b.set_mode(side, mode)
        for c in (5, 8, 3):
            b.run_steps(c)
        for i, cr in enumerate(crs):
            with GpuMaceLenia.from_creature(cr) as s:
                s.run_steps(16)
                np.testing.assert_array_equal(b.state(i), s.state(), err_msg=f"world {i}")


def device_built(cr, stream):
    sim = GpuMaceLenia((cr.n, cr.n), cr.C, cr.K, cr.c0, cr.c1, cr.mu, cr.sigma, cr.weights,
                       cr.temp, stream=stream)
    specs, w = creature_ring_specs(cr)
    rings = torch.tensor(w, device="cuda")
    torch.cuda.synchronize()
    sim.build_ring_kernels(specs, rings.data_ptr())
    sim.upload_state(cr.seed)
    sim.synchronize()
    return sim


def test_first_steps_under_capture():
    """Steps of a world whose own graphs were never captured, enqueued into
    the caller's capture: replayed, they are the steps."""
    cr = creature(128, 2, 950)
    st = torch.cuda.Stream()
    with device_built(cr, st.cuda_stream) as a, device_built(cr, None) as b:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            a.run_steps(2)
        for _ in range(2):
            g.replay()
        torch.cuda.synchronize()
        b.run_steps(4)
        np.testing.assert_array_equal(a.state(), b.state())
        a.run_steps(3)     # and its own graphs after that
        b.run_steps(3)
        np.testing.assert_array_equal(a.state(), b.state())
