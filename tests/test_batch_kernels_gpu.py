"""Kernels replaced in a batch whose size classes step their worlds as graph
branches (mode 1): each world's column pass follows that world's own spectra,
real or complex, whatever the other worlds hold."""
import numpy as np
import pytest

from cella_nova_gb300 import GpuMaceLenia, GpuMaceLeniaBatch
from cella_nova_gb300.creature import make_creature

pytestmark = pytest.mark.gpu


def skewed(spec, dy, dx):
    """The spectrum of the kernel moved by (dy, dx): not point-symmetric."""
    f = np.fft.fftfreq(spec.shape[0])
    return (spec * np.exp(-2j * np.pi * (dy * f[:, None] + dx * f[None, :]))).astype(np.complex64)


@pytest.mark.parametrize("n", [64, 512, 1024])
def test_replaced_kernels_of_one_world(n):
    crs = [make_creature(n, 2, seed=960 + i, radius=(max(2.0, n / 24), n / 10), seed_box=n // 2)
           for i in range(2)]
    crs[1].kspec[0] = skewed(crs[1].kspec[0], 3, 5)   # one world is complex throughout
    with GpuMaceLeniaBatch(crs) as b, GpuMaceLenia.from_creature(crs[0]) as a:
        b.set_mode(n, 1)
        # real, then complex, then real again
        for spec in (None, skewed(crs[0].kspec[1], 2, 1), crs[0].kspec[1]):
            if spec is not None:
                b.set_kernel(0, 1, spec)
                a.set_kernel(spec, 1)
            b.run_steps(5)
            a.run_steps(5)
            np.testing.assert_array_equal(b.state(0), a.state())
        with GpuMaceLenia.from_creature(crs[1]) as s:
            s.run_steps(15)
            np.testing.assert_array_equal(b.state(1), s.state())
