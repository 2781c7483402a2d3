"""DiffusionLeniaGPU's parameters: the padded ring weights, and gradients that
are tensors of their own."""
import pytest

torch = pytest.importorskip("torch")

from cella_nova_gb300 import autograd  # noqa: E402
from cella_nova_gb300._abi import MAX_RINGS  # noqa: E402
from cella_nova_gb300.creature import make_creature  # noqa: E402


class HostWorld:
    """Stands in for the world, which rings() only asks for its device."""

    def __init__(self, *args):
        self.device = torch.device("cpu")


def padded(weights):
    return torch.stack([torch.nn.functional.pad(b, (0, MAX_RINGS - b.numel())) for b in weights])


@pytest.fixture
def model(monkeypatch):
    monkeypatch.setattr(autograd, "LeniaWorld", HostWorld)
    return autograd.DiffusionLeniaGPU(make_creature(32, 2, seed=5, radius=(2, 5), seed_box=16),
                                      device="cpu", autotune=False)


def test_rings_first_seen_in_inference_mode(model):
    with torch.inference_mode():
        assert torch.equal(model.rings(), padded(model.ring_weights))
    coef = torch.arange(float(len(model.ring_weights) * MAX_RINGS)).view(-1, MAX_RINGS)
    (model.rings() * coef).sum().backward()
    for k, b in enumerate(model.ring_weights):
        assert torch.equal(b.grad, coef[k, :b.numel()].to(b.dtype))


def test_rings_of_other_counts(model):
    before = model.rings()
    for count in (1, 3, MAX_RINGS, MAX_RINGS + 1):   # what is beyond the last ring is not read
        weights = torch.arange(1.0, count + 1, dtype=torch.float64)
        model.ring_weights[1] = torch.nn.Parameter(weights)
        with torch.inference_mode():
            assert torch.equal(model.rings(), padded(model.ring_weights))
        model.rings().sum().backward()
        assert torch.equal(model.ring_weights[1].grad, (weights <= MAX_RINGS).double())
    assert before.shape == (len(model.ring_weights), MAX_RINGS)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_gradients_share_no_storage(dtype):
    m = autograd.DiffusionLeniaGPU(make_creature(64, 2, seed=6, radius=(4, 10), seed_box=32),
                                   autotune=False)
    leaves = [p.detach().to(dtype).requires_grad_() for p in (m.mu, m.sigma, m.weights)]
    xT = autograd.unroll_rings(m.world, m.specs, m.seed, *leaves, m.rings(), 2, 2)
    (xT ** 2).sum().backward()
    for p in leaves:
        g = p.grad
        assert g.dtype == dtype and torch.isfinite(g).all()
        assert g.untyped_storage().nbytes() == g.numel() * g.element_size()
        assert g.storage_offset() == 0


@pytest.mark.gpu
def test_rings_first_seen_under_capture():
    m = autograd.DiffusionLeniaGPU(make_creature(64, 2, seed=7, radius=(4, 10), seed_box=32),
                                   autotune=False)
    padded(m.ring_weights)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = m.rings()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, padded(m.ring_weights))
