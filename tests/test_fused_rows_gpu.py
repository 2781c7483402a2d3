"""Chains of steps, whose diffusion takes the next step's forward row pass
with it, against the same steps one by one, whose kernels are separate; and
both graph layouts where the fused kernel runs on the channels' streams."""
import numpy as np
import pytest

from cella_nova_gb300 import GpuMaceLenia
from cella_nova_gb300.creature import make_creature

pytestmark = pytest.mark.gpu


def creature(n, C, seed):
    return make_creature(n, C, seed=seed, radius=(max(2.0, n / 16), max(3.0, n / 6)),
                         seed_box=n // 2)


@pytest.mark.parametrize("n", [16, 32, 128, 256])
@pytest.mark.parametrize("C", [1, 3])
def test_chains_equal_single_steps(n, C):
    cr = creature(n, C, 980 + n)
    with GpuMaceLenia.from_creature(cr) as a, GpuMaceLenia.from_creature(cr) as b:
        for count in (2, 15, 8):
            a.run_steps(count)
            for _ in range(count):
                b.iterate()
            np.testing.assert_array_equal(a.state(), b.state())


@pytest.mark.parametrize("r2c", [0, 1, 2, 3, 4])   # from 3 on nothing is fused
def test_layouts_agree_512(r2c):
    cr = creature(512, 3, 985)
    with GpuMaceLenia.from_creature(cr) as a, GpuMaceLenia.from_creature(cr) as b:
        for s in (a, b):
            s.set_variants([r2c, 0, 0, 0])
        b.set_graph_layout(1)
        for count in (11, 4):
            a.run_steps(count)
            b.run_steps(count)
            np.testing.assert_array_equal(a.state(), b.state())
        a.iterate_and_render()
        b.iterate_and_render()
        np.testing.assert_array_equal(a.download_render_packed(), b.download_render_packed())
