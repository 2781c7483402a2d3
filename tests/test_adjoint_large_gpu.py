"""One step's VJP at the large sides against FP64 autograd, on both routes of
the adjoint's row kernels (rows gathered, and landed by tensor copies)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300.autograd import LeniaWorld  # noqa: E402
from cella_nova_gb300.creature import make_creature, ring_kernel  # noqa: E402
from oracle import autograd_ref as AR  # noqa: E402

pytestmark = pytest.mark.gpu


# CTAs of the growth adjoint: 256 per kernel at 1024 with variant 0 (64 with
# variant 2), 1024 (256) at 2048; rows land from 609 CTAs on
@pytest.mark.parametrize("n,c0,c1", [(1024, [0], [0]), (1024, [0, 1, 0, 1], [1, 0, 0, 1]),
                                     (2048, [0], [0])])
def test_vjp_matches_fp64(n, c0, c1):
    C = max(c0 + c1) + 1
    cr = make_creature(n, C, seed=990 + n, c0=c0, c1=c1, seed_box=n // 4, radius=(8, 24))
    h = np.stack([ring_kernel(n, R, b) for R, b in zip(cr.ring_radius, cr.ring_weights)])
    h = h.astype(np.float32)
    rng = np.random.default_rng(n)
    x = torch.tensor(cr.seed, dtype=torch.float32)
    ybar = torch.tensor(rng.standard_normal(cr.seed.shape), dtype=torch.float32)
    f64 = lambda a: torch.tensor(np.asarray(a, np.float64), requires_grad=True)
    xt, mu, sg, ww, ht = f64(x), f64(cr.mu), f64(cr.sigma), f64(cr.weights), f64(h)
    out = AR.step(xt, torch.fft.fft2(ht), cr.c0, cr.c1, mu, sg, ww, cr.temp)
    ref = torch.autograd.grad(torch.sum(out * ybar.double()), [xt, mu, sg, ww, ht])
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    for variants in (None, [0, 0, 0, 0], [2, 0, 2, 1]):
        w = LeniaWorld(n, C, cr.c0, cr.c1, cr.temp)
        if variants:
            w.set_variants(variants)
        w.load(cr.mu, cr.sigma, cr.weights, torch.tensor(h, device="cuda"))
        xd, yd = x.cuda(), ybar.cuda()
        xbar = torch.empty_like(xd)
        pg = torch.zeros(3 * cr.K, dtype=torch.float64, device="cuda")
        kg = torch.zeros((cr.K, n // 2, n, 2), dtype=torch.float32, device="cuda")
        hbar = torch.empty((cr.K, n, n), dtype=torch.float32, device="cuda")
        assert w.lib.cg_step_backward(w.h, P(xd), P(yd), P(xbar), P(pg), P(kg)) == 0
        assert w.lib.cg_kernel_grad_spatial(w.h, P(kg), P(hbar)) == 0
        torch.cuda.synchronize()
        w.close()
        for got, r in zip([xbar, *pg.reshape(3, -1), hbar], ref):
            # the adjoint's bar (test_adjoint_gpu.py)
            assert float((got.cpu().double() - r).abs().max() / r.abs().max()) < 1e-4, variants
