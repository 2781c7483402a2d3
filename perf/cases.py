"""Workloads that measure the framework through its public entry points.

Five kinds of work, each what a program that uses the package does with it:

* ``run``     a world (:class:`GpuMaceLenia`) stepped on the device, the state
              left there for the next consumer on the GPU;
* ``host``    the same world fed from host arrays and read back into them;
* ``batch``   many worlds of uneven size stepped together
              (:class:`GpuMaceLeniaBatch`), their states read back;
* ``grad``    the differentiable unroll (:class:`DiffusionLeniaGPU`): forward,
              loss, backward;
* ``search``  one Adam iteration of several candidates
              (:class:`GradientSearch`).

A case is a dict of plain values.  ``prepare`` builds what the program holds
before the call, ``run`` is one pass, ``exact`` the same result in 64 bits by
plain torch.  Worlds keep stepping from pass to pass, as a simulation does.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from cella_nova_gb300 import GpuMaceLenia, GpuMaceLeniaBatch
from cella_nova_gb300.autograd import DiffusionLeniaGPU
from cella_nova_gb300.creature import Creature, all_pairs
from cella_nova_gb300.search import AdamConfig, GradientSearch

L2_BYTES = 129e6
# no case costs more than this many kernel updates (grid points x kernels x
# steps, gradients counted by GRAD_COST)
GRAD_COST = 4.5
MAX_COST = 1024 * 1024 * 9 * 16 * GRAD_COST
LR = AdamConfig(lr_seed=1e-3, lr_params=1e-3, lr_rings=1e-2)


def _case(name, kind, n, C, K, steps, **more):
    c = {"name": name, "kind": kind, "n": n, "C": C, "K": K, "steps": steps,
         "symmetric": True, "tuned": False, "temp": 1.0}
    c.update(more)
    return c


def listed():
    return [
        # one tick of a small creature on screen: nothing but launch latency
        _case("tick64", "run", 64, 3, 9, 1),
        # a parameter sweep's small world, ten steps between looks
        _case("run256", "run", 256, 3, 9, 10),
        # a creature with its own channel wiring and skewed kernels (complex
        # spectra), an odd number of steps, used as it comes (no tuner)
        _case("run512_irregular", "run", 512, 4, 11, 5, symmetric=False, temp=1.2),
        # the reference's ordinary grid, tuned once and run
        _case("run1024", "run", 1024, 3, 9, 8, tuned=True),
        # the large single-channel Lenia world, used as it comes
        _case("run2048_c1", "run", 2048, 1, 1, 4),
        # the headline: the largest grid, three channels, all pairs
        _case("run2048", "run", 2048, 3, 9, 8, tuned=True),
        # the reference's host loop: seeds in, some steps, state out
        _case("host512", "host", 512, 3, 9, 10),
        # a population of creatures of uneven size screened together
        _case("batch_mixed", "batch", 1024, 3, 9, 8, tuned=True, worlds=10, n_min=64, pick=5),
        # gradients of a small creature, as a notebook takes them
        _case("grad128", "grad", 128, 2, 4, 16, tuned=True, every=8),
        # gradients at the reference's ordinary grid
        _case("grad1024", "grad", 1024, 3, 9, 16, tuned=True, every=8),
        # a population optimised together, one Adam iteration
        _case("search256", "search", 256, 3, 9, 16, tuned=True, every=8, worlds=6),
    ]


def _cost(c):
    f = GRAD_COST if c["kind"] in ("grad", "search") else 1.0
    if c["kind"] == "batch":
        return sum(n * n * K for n, _, K, _ in _batch_shapes(c)) * c["steps"]
    return c["n"] ** 2 * max(c["K"], c["C"]) * c["steps"] * f * c.get("worlds", 1)


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "host", "batch", "grad", "search"])
    lo, hi = {"run": (4, 11), "host": (6, 10), "batch": (7, 10), "grad": (6, 10),
              "search": (6, 9)}[kind]
    while True:
        n = 1 << rng.randint(lo, hi)
        C = rng.choice([1, 2, 3, 3, 4, 5])
        K = C * C if C <= 4 and rng.random() < 0.5 else rng.randint(max(1, C - 1), 3 * C)
        c = _case("", kind, n, C, K, rng.choice([1, 2, 3, 5, 8]),
                  symmetric=rng.random() < 0.7, tuned=rng.random() < 0.5,
                  temp=round(rng.uniform(0.5, 1.2), 2))
        del c["name"]
        if kind == "batch":
            c.update(worlds=rng.randint(2, 12), n_min=64, pick=rng.randint(0, 999))
        if kind in ("grad", "search"):   # ring kernels, built on the GPU
            c.update(symmetric=True, steps=rng.choice([5, 8, 12, 16]), every=rng.choice([4, 8]))
        if kind == "search":
            c.update(worlds=rng.randint(2, 8))
        if _cost(c) <= MAX_COST:
            return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _maps(C, K, rng):
    """Channel read and channel fed by each kernel: all pairs where K = C^2,
    otherwise drawn (channels may be unused or used several times)."""
    if K == C * C:
        return all_pairs(C)
    return (rng.integers(0, C, K).astype(np.uint32), rng.integers(0, C, K).astype(np.uint32))


def _shells(n, R, B, dtype=torch.float64):
    """(B, n, n): the Lenia ring kernel's shells exp(4 - 1/(t(1-t)))."""
    d = (torch.arange(n, device="cuda", dtype=dtype) + n // 2) % n - n // 2
    r = torch.sqrt(d[:, None] ** 2 + d[None, :] ** 2) / R
    idx = torch.floor(r * B)
    t = r * B - idx
    inside = (t > 0) & (t < 1) & (r < 1)
    t = torch.where(inside, t, torch.full_like(t, 0.5))
    core = torch.where(inside, torch.exp(4 - 1 / (t * (1 - t))), torch.zeros_like(t))
    return torch.stack([torch.where(idx == l, core, torch.zeros_like(core)) for l in range(B)])


def _creature(n, C, K, temp, seed, symmetric=True, spectra=True):
    """A creature of random Lenia rings; ``symmetric=False`` skews every
    kernel by a linear ramp, so that its spectrum is complex."""
    rng = np.random.default_rng(seed)
    c0, c1 = _maps(C, K, rng)
    lo = max(2.0, 12.0 * n / 1024)
    hi = min(max(30.0 * n / 1024, lo + 2.0), n / 2 - 1)
    R = rng.uniform(lo, hi, K).astype(np.float32).astype(np.float64)
    rings, kspec = [], np.empty((K, n, n) if spectra else (K, 0, 0), np.complex64)
    for k in range(K):
        b = rng.uniform(0.25, 1.0, 1 + k % 3)
        rings.append(b.astype(np.float32).astype(np.float64).tolist())
        if spectra:
            h = torch.tensordot(torch.tensor(rings[k], dtype=torch.float64, device="cuda"),
                                _shells(n, float(R[k]), len(rings[k])), dims=1)
            if not symmetric:
                d = (torch.arange(n, device="cuda", dtype=torch.float64) + n // 2) % n - n // 2
                h = h * (1 + 0.5 * d[None, :] / float(R[k]))
            kspec[k] = torch.fft.fft2(h / h.sum()).to(torch.complex64).cpu().numpy()
    mu = rng.uniform(0.05, 0.3, K).astype(np.float32)
    # growth bumps no narrower than 0.03: narrower ones make a few-channel
    # world chaotic within ten steps, and no two roundings then agree
    sigma = rng.uniform(0.03, 0.08, K).astype(np.float32)
    w = rng.uniform(0.1, 1.0, K)
    for c in range(C):
        if (c1 == c).any():
            w[c1 == c] /= w[c1 == c].sum()
    box = min(256, n // 2)
    o = (n - box) // 2
    x = np.zeros((C, n, n))
    x[:, o:o + box, o:o + box] = rng.random((C, box, box), dtype=np.float32)
    return Creature(n=n, C=C, K=K, seed=x, kspec=kspec, c0=c0, c1=c1, mu=mu, sigma=sigma,
                    weights=w.astype(np.float32), temp=float(np.float32(temp)), ring_radius=R,
                    ring_weights=rings)


def _batch_shapes(c):
    """(n, C, K, temp) of a batch's worlds: powers of two from n_min to n
    alike, the first of them n."""
    rng = np.random.default_rng(c["pick"])
    lo, hi = int(math.log2(c["n_min"])), int(math.log2(c["n"]))
    out = []
    for i in range(c["worlds"]):
        n = c["n"] if i == 0 else 1 << int(rng.integers(lo, hi + 1))
        C = int(rng.integers(1, c["C"] + 1))
        K = C * C if rng.random() < 0.5 else int(rng.integers(C, 2 * C + 2))
        out.append((n, C, K, round(float(rng.uniform(0.5, 1.2)), 2)))
    return out


def _creatures(c, seed):
    if c["kind"] == "batch":
        return [_creature(n, C, K, t, [seed, i], c["symmetric"])
                for i, (n, C, K, t) in enumerate(_batch_shapes(c))]
    spectra = c["kind"] in ("run", "host")
    return [_creature(c["n"], c["C"], c["K"], c["temp"], [seed, i], c["symmetric"], spectra)
            for i in range(c.get("worlds", 1))]


def _target(x):
    """The seed moved by (+8, +16) pixels: what the unroll should reach."""
    return np.roll(x, (8, 16), axis=(-2, -1))


class _DeviceState:
    """The world's current state as an array on the GPU (keeps the world)."""

    def __init__(self, sim):
        self.sim = sim
        self.__cuda_array_interface__ = {
            "shape": (sim.num_channels, sim.n, sim.n), "typestr": "<f4", "version": 2,
            "data": (sim.channel_ptr(), False)}


def prepare(case, seed):
    kind, crs = case["kind"], _creatures(case, seed)
    if kind in ("run", "host"):
        # on torch's default stream (1: the legacy stream), as a program that
        # hands the state on to torch has it
        sim = GpuMaceLenia.from_creature(crs[0], stream=1)
        if case["tuned"]:
            sim.autotune()
        return {"case": case, "sim": sim, "seed": crs[0].seed}
    if kind == "batch":
        b = GpuMaceLeniaBatch(crs, stream=1)
        if case["tuned"]:
            b.autotune()
        return {"case": case, "batch": b}
    if kind == "grad":
        model = DiffusionLeniaGPU(crs[0], autotune=case["tuned"])
        target = torch.tensor(_target(crs[0].seed), dtype=torch.float32, device="cuda")
        return {"case": case, "model": model, "target": target}
    search = GradientSearch(crs, [_target(cr.seed) for cr in crs], T=case["steps"],
                            every=case["every"], adam=LR, autotune=case["tuned"])
    return {"case": case, "search": search}


def run(state):
    case = state["case"]
    if case["kind"] == "run":
        sim = state["sim"]
        sim.run_steps(case["steps"])
        return torch.as_tensor(_DeviceState(sim), device="cuda")
    if case["kind"] == "host":
        sim = state["sim"]
        for c in range(case["C"]):
            sim.upload_channel(state["seed"][c], c)
        sim.run_steps(case["steps"])
        return sim.download_all_channels()
    if case["kind"] == "batch":
        b = state["batch"]
        b.run_steps(case["steps"])
        return [b.state(w) for w in range(case["worlds"])]
    if case["kind"] == "grad":
        model = state["model"]
        model.zero_grad(set_to_none=True)
        xT = model(case["steps"], case["every"])
        loss = torch.mean((xT - state["target"]) ** 2)
        loss.backward()
        return {"xT": xT.detach(), "loss": loss.detach(), "seed": model.seed.grad,
                "mu": model.mu.grad, "sigma": model.sigma.grad, "weights": model.weights.grad,
                "rings": torch.cat([b.grad for b in model.ring_weights])}
    search = state["search"]
    search.run(1)
    return [{"seed": c.seed, "params": c.params, "rings": c.rings, "xT": c.xT, "g_seed": c.g0,
             "g_params": c.pgrad, "g_rings": c.ring_grad, "loss": c.loss} for c in search.cands]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _step_work(n, C, K, symmetric, steps):
    """Bytes: the state in and out and the kernels' half spectra (real when
    every kernel is point-symmetric), once, or once per step where they
    exceed the L2 cache.  Flops: real 2-D transforms of every channel and
    kernel, the products, the growth and the 3 x 3 redistribution."""
    px = n * n
    moved = 8.0 * C * px + K * px / 2 * (4 if symmetric else 8)
    fft = 2.5 * px * 2 * math.log2(n)
    flops = (C + K) * fft + K * px * (3 + 8) + 25.0 * C * px
    return moved * (steps if moved > L2_BYTES else 1), flops * steps


def work(case):
    if case["kind"] == "batch":
        parts = [_step_work(n, C, K, case["symmetric"], case["steps"])
                 for n, C, K, _ in _batch_shapes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    n, C, K = case["n"], case["C"], case["K"]
    moved, flops = _step_work(n, C, K, case["symmetric"], case["steps"])
    if case["kind"] in ("grad", "search"):
        # seed in, target in, state and seed gradient out; backward: twice the
        # forward's transforms
        moved, flops = 16.0 * C * n * n, 3 * flops
        if case["kind"] == "search":   # Adam: moments in and out, seed out
            moved += 20.0 * C * n * n
    return {"bytes": moved * case.get("worlds", 1), "flops": flops * case.get("worlds", 1)}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------

def _box(a):
    a = a + torch.roll(a, 1, -1) + torch.roll(a, -1, -1)
    return a + torch.roll(a, 1, -2) + torch.roll(a, -1, -2)


def _step64(x, spec, c0, c1, mu, sigma, w, temp):
    """spec: the kernels' spectra on the half plane of rfft2."""
    n = x.shape[-1]
    X = torch.fft.rfft2(x)
    acc = [torch.zeros_like(x[0]) for _ in range(x.shape[0])]
    for k in range(len(c0)):
        u = torch.fft.irfft2(X[int(c0[k])] * spec[k], s=(n, n))
        g = 2 * torch.exp(-((u - mu[k]) ** 2) / (2 * sigma[k] ** 2)) - 1
        acc[int(c1[k])] = acc[int(c1[k])] + w[k] * g
    A = torch.exp(temp * torch.stack(acc))
    return A * _box(x / _box(A))


def _d(a):
    return torch.tensor(np.asarray(a, np.float64), device="cuda")


def _half_spectra(kspec):
    """The uploaded spectra's Hermitian part (all that a real state's real
    convolution uses), on the half plane."""
    out = []
    for s in kspec:
        s = torch.tensor(s, device="cuda").to(torch.complex128)
        m = torch.roll(torch.flip(s, (0, 1)), (1, 1), (0, 1)).conj()
        out.append(((s + m) / 2)[:, :s.shape[0] // 2 + 1].contiguous())
    return out


def _run64(cr, steps):
    x, spec = _d(cr.seed), _half_spectra(cr.kspec)
    with torch.no_grad():
        for _ in range(steps):
            x = _step64(x, spec, cr.c0, cr.c1, _d(cr.mu), _d(cr.sigma), _d(cr.weights), cr.temp)
    return x


def _grad64(cr, steps):
    """x_T, the loss and its gradients with ring kernels built from their
    ring weights."""
    leaf = {"seed": _d(cr.seed), "mu": _d(cr.mu), "sigma": _d(cr.sigma), "weights": _d(cr.weights)}
    bs = [_d(b).requires_grad_() for b in cr.ring_weights]
    for t in leaf.values():
        t.requires_grad_()
    spec = []
    for b, R in zip(bs, cr.ring_radius):
        h = torch.tensordot(b, _shells(cr.n, float(R), len(b)), dims=1)
        spec.append(torch.fft.rfft2(h / h.sum()))
    x = leaf["seed"]
    for _ in range(steps):
        x = checkpoint(_step64, x, spec, cr.c0, cr.c1, leaf["mu"], leaf["sigma"],
                       leaf["weights"], cr.temp, use_reentrant=False)
    loss = torch.mean((x - _d(_target(cr.seed))) ** 2)
    loss.backward()
    out = {k: t.grad for k, t in leaf.items()}
    out.update(xT=x.detach(), loss=loss.detach(), rings=[b.grad for b in bs])
    return out


def exact(case, seed):
    crs = _creatures(case, seed)
    if case["kind"] == "run":
        return _run64(crs[0], case["steps"])
    if case["kind"] == "host":
        return _run64(crs[0], case["steps"]).reshape(-1)
    if case["kind"] == "batch":
        return [_run64(cr, case["steps"]) for cr in crs]
    if case["kind"] == "grad":
        g = _grad64(crs[0], case["steps"])
        g["rings"] = torch.cat(g["rings"])
        return g
    out = []
    for cr in crs:
        g = _grad64(cr, case["steps"])
        rings, grings = torch.zeros((2, cr.K, 8), dtype=torch.float64, device="cuda")
        for k, b in enumerate(cr.ring_weights):
            rings[k, :len(b)] = _d(b)
            grings[k, :len(b)] = g["rings"][k]
        params = torch.cat([_d(cr.mu), _d(cr.sigma), _d(cr.weights)])
        gp = torch.cat([g["mu"], g["sigma"], g["weights"]])

        def adam(p, q, lr):   # the first step: both moments are the gradient's own
            return p - lr * q / (q.abs() + LR.eps)

        out.append({"seed": adam(_d(cr.seed), g["seed"], LR.lr_seed),
                    "params": adam(params, gp, LR.lr_params),
                    "rings": adam(rings, grings, LR.lr_rings), "xT": g["xT"],
                    "g_seed": g["seed"], "g_params": gp, "g_rings": grings,
                    "loss": g["loss"].reshape(1)})
    return out
