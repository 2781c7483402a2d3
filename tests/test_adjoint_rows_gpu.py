"""The adjoint's row kernels at the sides where their rows land by tensor
copies: the two routes of the rule that chooses (more CTAs than places) and
every CTA shape give the same bits."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300.autograd import LeniaWorld  # noqa: E402
from cella_nova_gb300.creature import make_creature, ring_kernel  # noqa: E402

pytestmark = pytest.mark.gpu


# CTAs per plane, against 608 places: 256 with variant 0 and 64 with variant 2
# of the inverse row pass at 1024, 1024 and 256 at 2048.  So with variant 0
# (variant 2) the planes land from 3 (10) planes on at 1024 and always (from 3
# on) at 2048: the first case never lands, the second its growth rows in one
# shape only, the last two everything or nothing by shape
@pytest.mark.parametrize("n,c0,c1", [
    (1024, [0], [0]),
    (1024, [0, 1, 0, 1], [1, 0, 0, 1]),
    (2048, [0], [0]),
    (2048, [0, 1], [1, 0]),
])
def test_routes_and_shapes_give_the_same_bits(n, c0, c1):
    C = max(c0 + c1) + 1
    cr = make_creature(n, C, seed=1700 + n, c0=c0, c1=c1, seed_box=n // 4, radius=(8, 24))
    h = torch.tensor(np.stack([ring_kernel(n, R, b)
                               for R, b in zip(cr.ring_radius, cr.ring_weights)]),
                     dtype=torch.float32, device="cuda")
    rng = np.random.default_rng(n)
    x = torch.tensor(cr.seed, dtype=torch.float32, device="cuda")
    ybar = torch.tensor(rng.standard_normal(cr.seed.shape), dtype=torch.float32, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    ref = None
    for variants in ([2, 0, 2, 1], [1, 0, 1, 1], [0, 0, 0, 1]):
        w = LeniaWorld(n, C, cr.c0, cr.c1, cr.temp)
        w.set_variants(variants)
        w.load(cr.mu, cr.sigma, cr.weights, h)
        xbar = torch.empty_like(x)
        pg = torch.zeros(3 * cr.K, dtype=torch.float64, device="cuda")
        kg = torch.zeros((cr.K, n // 2, n, 2), dtype=torch.float32, device="cuda")
        hbar = torch.empty_like(h)
        assert w.lib.cg_step_backward(w.h, P(x), P(ybar), P(xbar), P(pg), P(kg)) == 0
        assert w.lib.cg_kernel_grad_spatial(w.h, P(kg), P(hbar)) == 0
        torch.cuda.synchronize()
        w.close()
        assert torch.isfinite(xbar).all() and float(xbar.abs().max()) > 0
        if ref is None:
            ref = (xbar, hbar)
        else:
            assert torch.equal(xbar, ref[0]), variants
            assert torch.equal(hbar, ref[1]), variants
