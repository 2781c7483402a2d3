"""The growth adjoint's FP32 partial sums do not depend on whether a world's
variants were set."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300.autograd import LeniaWorld  # noqa: E402
from cella_nova_gb300.creature import make_creature, ring_kernel  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 128, 256])
def test_variants_in_use_set_again_change_no_gradient(n):
    """Setting the variants that a world has leaves its parameter gradients as
    they were, up to the order in which at most 32 CTAs' FP64 sums are added
    (31 roundings of 2^-53 of the sum of their sizes, which random signs keep
    below 100 of the largest gradient: 4e-13); another grouping of the FP32
    sums before that would show as 1e-8."""
    cr = make_creature(n, 2, seed=995, c0=[0, 1, 0], c1=[1, 0, 0], seed_box=n // 2,
                       radius=(max(2.0, n / 16), n / 6))
    h = np.stack([ring_kernel(n, R, b) for R, b in zip(cr.ring_radius, cr.ring_weights)])
    x = torch.tensor(cr.seed, dtype=torch.float32, device="cuda")
    ybar = torch.tensor(np.random.default_rng(n).standard_normal(cr.seed.shape),
                        dtype=torch.float32, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    pgs = []
    for again in (False, True):
        w = LeniaWorld(n, cr.C, cr.c0, cr.c1, cr.temp)
        if again:
            v = (ctypes.c_int * 4)()
            assert w.lib.cg_get_variants(w.h, v) == 0
            w.set_variants(list(v))
        w.load(cr.mu, cr.sigma, cr.weights, torch.tensor(h, dtype=torch.float32, device="cuda"))
        xbar = torch.empty_like(x)
        pg = torch.zeros((3, cr.K), dtype=torch.float64, device="cuda")
        assert w.lib.cg_step_backward(w.h, P(x), P(ybar), P(xbar), P(pg), None) == 0
        torch.cuda.synchronize()
        w.close()
        pgs.append(pg.cpu())
    size = pgs[0].abs().amax(dim=1, keepdim=True)
    assert float(((pgs[1] - pgs[0]).abs() / size).max()) <= 1e-12
