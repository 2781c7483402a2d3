"""The quotients of the diffusion adjoint at the ends of the FP32 range."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300.autograd import LeniaWorld  # noqa: E402
from cella_nova_gb300.creature import make_creature, ring_kernel  # noqa: E402

pytestmark = pytest.mark.gpu


def box_in_order(y):
    """The 3x3 toroidal sum, row by row from the top left, in FP32."""
    s = np.zeros_like(y)
    for di in (1, 0, -1):
        for dj in (1, 0, -1):
            s = s + np.roll(y, (di, dj), (0, 1))
    return s


@pytest.mark.parametrize("scale", [2.0 ** -140, 2.0 ** -126, 2.0 ** -112, 2.0 ** -101, 1.0,
                                   2.0 ** 100, 2.0 ** 125, 2.0 ** 127])
@pytest.mark.parametrize("infinite", [False, True])
def test_quotients_are_divisions(scale, infinite):
    """No kernel feeds or reads channel 1, so A is 1 and Z is 9 there, and its
    state gradient is the 3x3 sum of the incoming one divided by 9."""
    n = 64
    cr = make_creature(n, 2, seed=970, c0=[0], c1=[0], seed_box=n // 2, radius=(4, 10))
    h = np.stack([ring_kernel(n, R, b) for R, b in zip(cr.ring_radius, cr.ring_weights)])
    rng = np.random.default_rng(971)
    ybar = rng.standard_normal((2, n, n)).astype(np.float32)
    y = (np.clip(ybar[1], -1.9, 1.9) * np.float64(scale)).astype(np.float32)
    if infinite:
        y[10, 20], y[40, 0] = np.inf, -np.inf
    ybar[1] = y
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        want = box_in_order(y) / np.float32(9)
    dev = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    x, yb = dev(cr.seed), dev(ybar)
    w = LeniaWorld(n, 2, cr.c0, cr.c1, cr.temp)
    w.load(cr.mu, cr.sigma, cr.weights, dev(h))
    xbar = torch.empty_like(x)
    pg = torch.zeros(3, dtype=torch.float64, device="cuda")
    assert w.lib.cg_step_backward(w.h, P(x), P(yb), P(xbar), P(pg), None) == 0
    torch.cuda.synchronize()
    w.close()
    got = xbar.cpu().numpy()
    assert np.isfinite(got[0]).all()
    np.testing.assert_array_equal(got[1], want)
