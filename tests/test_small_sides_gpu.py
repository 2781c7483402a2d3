"""Small grid sides: the many-CTA shapes, the column pass whose CTAs share a
tile's kernels, and the growth adjoint's row chains, at the edges of each."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300 import GpuMaceLenia  # noqa: E402
from cella_nova_gb300.autograd import LeniaWorld  # noqa: E402
from cella_nova_gb300.creature import make_creature, ring_kernel  # noqa: E402
from oracle import autograd_ref as AR  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def creature(n, C, c0, c1, seed):
    return make_creature(n, C, seed=seed, c0=c0, c1=c1, seed_box=n // 2,
                         radius=(max(2.0, n / 16), max(4.0, n / 6)))


# kernels per input channel that a grid's CTAs share unevenly (7, 5 and 1),
# not at all (2 channels, 1 kernel), and the most there can be (64)
MAPS = {"uneven": (3, [0] * 7 + [1] * 5 + [2], [0, 1, 2] * 4 + [1]),
        "one": (2, [1], [0]),
        "most": (1, [0] * 64, [0] * 64)}


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512])
@pytest.mark.parametrize("name", list(MAPS))
def test_step_matches_fp64(n, name):
    C, c0, c1 = MAPS[name]
    cr = creature(n, C, c0, c1, 700 + n)
    with GpuMaceLenia.from_creature(cr) as sim:
        for _ in range(2):
            x = sim.state()
            sim.iterate()
            ref, _, _ = O.step_np(x.astype(np.float64), cr.kspec.astype(np.complex128), cr.c0,
                                  cr.c1, cr.mu.astype(np.float64), cr.sigma.astype(np.float64),
                                  cr.weights.astype(np.float64), cr.temp)
            assert np.abs(sim.state() - ref).max() <= 1e-5   # the step's bar (test_step_gpu.py)


@pytest.mark.parametrize("n", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("chosen", [None, [0, 0, 0, 0], [2, 2, 2, 1]])
def test_growth_adjoint_rows(n, chosen):
    """One step's VJP with the rows chained as in an untuned world and as
    after a choice of variants, with kernels that all feed one channel."""
    cr = creature(n, 2, [0, 1, 0], [1, 1, 1], 800 + n)
    h = np.stack([ring_kernel(n, R, b) for R, b in zip(cr.ring_radius, cr.ring_weights)])
    rng = np.random.default_rng(n)
    x = torch.tensor(cr.seed, dtype=torch.float32, device="cuda")
    ybar = torch.tensor(rng.standard_normal(cr.seed.shape), dtype=torch.float32, device="cuda")
    w = LeniaWorld(n, cr.C, cr.c0, cr.c1, cr.temp)
    if chosen:
        w.set_variants(chosen)
    w.load(cr.mu, cr.sigma, cr.weights, torch.tensor(h, dtype=torch.float32, device="cuda"))
    xbar = torch.empty_like(x)
    pg = torch.zeros(3 * cr.K, dtype=torch.float64, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    assert w.lib.cg_step_backward(w.h, P(x), P(ybar), P(xbar), P(pg), None) == 0
    torch.cuda.synchronize()
    f64 = lambda a: torch.tensor(np.asarray(a, np.float64), requires_grad=True)
    xt, mu, sg, ww = f64(x.cpu()), f64(cr.mu), f64(cr.sigma), f64(cr.weights)
    ks = torch.fft.fft2(torch.tensor(h, dtype=torch.complex128))
    out = AR.step(xt, ks, cr.c0, cr.c1, mu, sg, ww, cr.temp)
    ref = torch.autograd.grad(torch.sum(out * ybar.cpu().double()), [xt, mu, sg, ww])
    w.close()
    for got, r in zip([xbar, *pg.reshape(3, -1)], ref):   # the adjoint's bar (test_adjoint_gpu.py)
        assert float((got.cpu().double() - r).abs().max() / r.abs().max()) < 1e-4
