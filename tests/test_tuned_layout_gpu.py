"""The tuner leaves the graph layout alone where both layouts are one graph."""
import pytest

from cella_nova_gb300 import GpuMaceLenia
from cella_nova_gb300.creature import make_creature

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 128, 256])
def test_small_sides_keep_their_layout(n):
    cr = make_creature(n, 2, seed=1010, radius=(max(2.0, n / 16), max(3.0, n / 6)),
                       seed_box=n // 2)
    with GpuMaceLenia.from_creature(cr) as sim:
        for layout in (0, 1):
            sim.set_graph_layout(layout)
            for _ in range(8):   # timing one graph twice would pick either
                sim.autotune(reps=2)
                assert sim.graph_layout() == layout
