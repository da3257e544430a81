"""Workloads of the 1D hybrid time-stepper for performance measurements.

``listed()`` is a fixed set of cases, ``draw(rng)`` gives further ones of the same
kinds and ranges.  ``prepare`` builds what a user's program holds before the call
(states, solvers, networks), ``run`` is one pass through the package's public entry
points, ``work`` what that pass cannot do without, and ``exact`` the same outputs
from plain torch in 64 bits.

Kinds:

* ``burgers_step``       one no-grad solver.step with a correction, as an evaluation
                         loop with its own corrector issues it;
* ``ks_step_grad``       one solver.step with a correction and its backward, as a
                         training loop with its own corrector issues it;
* ``burgers_rollout``    a fused solver rollout (data generation, baselines without
                         a network); with ``grad`` its backward too (fitting initial
                         states or a fixed correction through the solver);
* ``ks_rollout``         the same for Kuramoto-Sivashinsky, within a horizon where
                         the chaotic dynamics still determine the digits;
* ``burgers_ragged``     thousands of rows of different n, nu, dt, dx in one launch;
* ``burgers_cnn``        simulate_rollout with the periodic CNN corrector, evaluation;
                         with ``grad`` the training step's rollout, loss and backward;
* ``fno``                the FNO corrector alone on a batch of states: evaluation, or
                         forward, loss and backward (pre-training on stored pairs);
* ``ks_fno_train``       simulate_rollout of the KS solver with the FNO corrector,
                         loss and backward (the unrolled training step).
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from inc_b200.batched import RaggedBurgers
from inc_b200.correctors import FNO1D, PeriodicCNN1D
from inc_b200.rollout import burgers_rollout, ks_rollout, simulate_rollout
from inc_b200.solvers import BurgersSolverTorch, KSSolverTorch

DEV = "cuda:0"
TWO_PI = 2 * math.pi


# ---------------------------------------------------------------------------- cases
def listed():
    return [
        # one step of an evaluation loop at the small Burgers configuration: launch latency
        dict(name="burgers_step_32x128", kind="burgers_step", B=32, n=128, scheme="ssprk3"),
        # one differentiated KS step, an odd batch of short rows: latency of a training loop
        dict(name="ks_step_grad_37x64", kind="ks_step_grad", B=37, n=64, L=22.0, dt=0.2),
        # the small Burgers configuration, 200 fused steps: one dependency chain per row
        dict(name="burgers_rollout_32x128", kind="burgers_rollout", B=32, n=128, steps=200, grad=False),
        # a differentiable Burgers unroll, checkpoints every 8 steps
        dict(name="burgers_rollout_grad_256x256", kind="burgers_rollout", B=256, n=256, steps=32, grad=True),
        # the KS configuration (1024 rows of 256 cells) over the horizon that stays comparable
        dict(name="ks_rollout_1024x256", kind="ks_rollout", B=1024, n=256, steps=40, L=64.0, dt=0.25, grad=False),
        # a differentiable KS unroll of the training shape, checkpoints every 8 steps
        dict(name="ks_rollout_grad_512x512", kind="ks_rollout", B=512, n=512, steps=64, L=100.0, dt=0.2, grad=True),
        # the ragged batch: 4096 rows of 64..512 cells, 500 steps
        dict(name="burgers_ragged_4096", kind="burgers_ragged", B=4096, steps=500),
        # evaluation of the Burgers CNN corrector, 32-step unroll
        dict(name="burgers_cnn_256x256", kind="burgers_cnn", B=256, n=256, steps=32, grad=False),
        # its training step (rollout, loss, backward)
        dict(name="burgers_cnn_train_256x256", kind="burgers_cnn", B=256, n=256, steps=32, grad=True),
        # the FNO corrector evaluated on the KS training batch
        dict(name="fno_512x512", kind="fno", B=512, n=512, width=64, modes=16, grad=False),
        # pre-training the FNO on stored pairs: an odd batch of shorter rows, forward and backward
        dict(name="fno_train_201x256", kind="fno", B=201, n=256, width=64, modes=16, grad=True),
        # the unrolled KS + FNO training step of the training shape, 8 steps
        dict(name="ks_fno_train_256x512", kind="ks_fno_train", B=256, n=512, steps=8, width=64, modes=16, L=100.0,
             dt=0.2),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    top = max(work(c)["flops"] for c in listed())
    while True:  # a case within the largest listed one's work
        case = _draw(rng)
        if work(case)["flops"] <= top:
            return case


def _draw(rng):
    kind = rng.choice(["burgers_step", "ks_step_grad", "burgers_rollout", "ks_rollout", "burgers_ragged",
                       "burgers_cnn", "burgers_cnn", "fno", "fno", "ks_fno_train"])
    if kind == "burgers_step":
        return dict(kind=kind, B=_log_int(rng, 1, 4096), n=rng.choice([32, 64, 128, 256, 512]),
                    scheme=rng.choice(["euler", "ssprk3"]))
    if kind == "ks_step_grad":
        n = rng.choice([32, 64, 128, 256, 512])
        return dict(kind=kind, B=_log_int(rng, 1, 1024), n=n, L=rng.uniform(0.2, 0.4) * n, dt=rng.choice([0.1, 0.2]))
    if kind == "burgers_rollout":
        return dict(kind=kind, B=_log_int(rng, 1, 2048), n=rng.choice([64, 128, 256, 512]),
                    steps=_log_int(rng, 4, 200), grad=rng.random() < 0.5)
    if kind == "ks_rollout":
        n = rng.choice([64, 128, 256, 512])
        return dict(kind=kind, B=_log_int(rng, 1, 1024), n=n, steps=_log_int(rng, 4, 40), L=rng.uniform(0.2, 0.25) * n,
                    dt=rng.choice([0.1, 0.2]), grad=rng.random() < 0.5)
    if kind == "burgers_ragged":
        return dict(kind=kind, B=_log_int(rng, 100, 4096), steps=_log_int(rng, 20, 400))
    if kind == "burgers_cnn":
        return dict(kind=kind, B=_log_int(rng, 1, 512), n=rng.choice([64, 128, 256, 512]), steps=_log_int(rng, 4, 32),
                    grad=rng.random() < 0.5)
    if kind == "fno":
        return dict(kind=kind, B=_log_int(rng, 1, 512), n=rng.choice([64, 128, 256, 512]),
                    width=rng.choice([32, 64, 64]), modes=rng.choice([8, 12, 16]), grad=rng.random() < 0.5)
    n = rng.choice([128, 256, 512])
    return dict(kind=kind, B=_log_int(rng, 1, 256), n=n, steps=_log_int(rng, 2, 8), width=rng.choice([32, 64, 64]),
                modes=rng.choice([8, 12, 16]), L=rng.uniform(0.2, 0.25) * n, dt=0.2)


# ---------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _sines(g, B, n, K=5):
    """sum_k A_k sin(k x + phi_k), A ~ U[-0.5, 0.5], on a period of 2 pi."""
    x = torch.arange(n, device=DEV, dtype=torch.float64) * (TWO_PI / n)
    k = torch.arange(1, K + 1, device=DEV, dtype=torch.float64)
    a, ph = _rand(g, B, K) - 0.5, TWO_PI * _rand(g, B, K)
    return (a[..., None] * torch.sin(k[:, None] * x + ph[..., None])).sum(1)


def _cosines(g, B, n, K=8):
    """sum_k a_k cos(2 pi k x / L + phi_k), a_k ~ N(0, 1) / k."""
    x = torch.arange(n, device=DEV, dtype=torch.float64) / n
    k = torch.arange(1, K + 1, device=DEV, dtype=torch.float64)
    a = torch.randn(B, K, generator=g, device=DEV, dtype=torch.float64) / k
    ph = TWO_PI * _rand(g, B, K)
    return (a[..., None] * torch.cos(TWO_PI * k[:, None] * x + ph[..., None])).sum(1)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _draw_params(net, g):
    """The network's parameters redrawn from the generator: U(+-1/sqrt(fan in)), and the
    reference's U[0, 1) / (in * out) for the Fourier layers' complex weights."""
    with torch.no_grad():
        for p in net.parameters():
            if p.is_complex():
                scale = 1.0 / (p.shape[0] * p.shape[1])
                p.copy_(torch.complex(scale * _rand(g, *p.shape), scale * _rand(g, *p.shape)))
            else:
                fan = p[0].numel() if p.dim() > 1 else 32
                p.copy_((2 * _rand(g, *p.shape) - 1) / math.sqrt(max(fan, 1)))
    return net


def _ragged_sizes(B):
    """Row lengths of the ragged batch: U{64, 128, 256, 512}, one draw per batch size."""
    g = torch.Generator().manual_seed(B)
    return torch.tensor([64, 128, 256, 512])[torch.randint(4, (B,), generator=g)]


def _burgers_dt(n):
    """A quarter of dx over the typical speed 1.5."""
    return 0.25 * TWO_PI / n / 1.5


def _burgers_solver(case):
    n = case["n"]
    return BurgersSolverTorch(SimpleNamespace(
        resolution=n, dt=_burgers_dt(n), x=None, adaptive_CFL=None, L=TWO_PI, nu=0.01, device=torch.device(DEV),
        convection_term="WENO", equation_type="viscosity", batch_size=case["B"],
        time_scheme=case.get("scheme", "ssprk3")))


def _ks_solver(case):
    ds = torch.full((case["B"],), case["L"], device=DEV)
    return KSSolverTorch(SimpleNamespace(resolution=case["n"], dt=case["dt"], device=torch.device(DEV),
                                         domain_size=ds, alpha=torch.zeros(case["B"], device=DEV),
                                         time_scheme="ETRK2")), ds


def _inputs(case, seed):
    """The case's arrays, FP32 on the GPU; ``exact`` starts from the same ones."""
    g = _gen(seed)
    kind, B = case["kind"], case["B"]
    f = lambda t: t.float().contiguous()  # noqa: E731
    if kind == "burgers_ragged":
        ns = _ragged_sizes(B)
        nu = torch.exp(math.log(1e-3) + math.log(50.0) * _rand(g, B)).cpu()
        dx = TWO_PI / ns.double()
        rows, peak = [None] * B, torch.zeros(B, dtype=torch.float64)
        for n in (64, 128, 256, 512):
            idx = (ns == n).nonzero().reshape(-1)
            u = _sines(g, len(idx), n).cpu() if len(idx) else torch.zeros(0, n)
            for i, r in zip(idx.tolist(), u):
                rows[i], peak[i] = r.float().numpy(), float(r.abs().max())
        dt = 0.4 * torch.minimum(dx / peak.clamp_min(1e-12), dx * dx / nu)
        return dict(ns=ns, rows=rows, nu=nu.numpy(), dt=dt.numpy(), dx=dx.numpy())
    n = case["n"]
    if kind in ("burgers_step", "burgers_rollout", "burgers_cnn"):
        u = f(_sines(g, B, n))
    elif kind == "fno":
        u = f(_cosines(g, B, n))
    else:
        u = f(0.5 * _cosines(g, B, n))
    out = dict(u=u)
    if kind in ("burgers_step", "ks_step_grad", "ks_rollout"):
        out["s"] = f(0.01 * _normal(g, B, n))
    if kind in ("burgers_cnn", "fno", "ks_fno_train"):
        torch.manual_seed(seed)
        if kind == "burgers_cnn":
            net = PeriodicCNN1D()
        else:
            net = FNO1D(L=case.get("L", 64.0), modes=case["modes"], width=case["width"])
        out["net"] = _draw_params(net.to(DEV), g)
    if kind == "ks_step_grad" or case.get("grad") or kind == "ks_fno_train":
        # the target of the mean-square loss: frames for rollouts, a state otherwise
        shape = (B, case["steps"], n) if "steps" in case else (B, n)
        out["target"] = f(0.1 * _normal(g, *shape))
    return out


def prepare(case, seed):
    st = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind == "burgers_ragged":
        st["batch"] = RaggedBurgers(st["rows"], st["nu"], st["dt"], st["dx"], device=DEV)
    elif kind in ("burgers_step", "burgers_rollout", "burgers_cnn"):
        st["solver"] = _burgers_solver(case)
    elif kind != "fno":
        st["solver"], st["ds"] = _ks_solver(case)
    if "target" in st:
        st["u"].requires_grad_(True)
        if "s" in st:
            st["s"].requires_grad_(True)
    return st


# ---------------------------------------------------------------------------- a pass
def _mse(a, b):
    return ((a - b) ** 2).mean()


def _grads(st, names=("u", "s")):
    out = {k: st[k].grad for k in names if k in st}
    if "net" in st:
        out["params"] = [p.grad for p in st["net"].parameters()]
    return out


def _zero(st):
    for k in ("u", "s"):
        if k in st:
            st[k].grad = None
    if "net" in st:
        st["net"].zero_grad(set_to_none=True)


def run(st):
    case = st["case"]
    kind, grad = case["kind"], "target" in st
    if kind == "burgers_ragged":
        return st["batch"].rollout(case["steps"])
    if grad:
        _zero(st)
    with torch.set_grad_enabled(grad):
        if kind == "burgers_step":
            st["solver"].correction_s = st["s"]
            out = st["solver"].step(st["u"])
        elif kind == "ks_step_grad":
            st["solver"].correction_s = st["s"]
            out = st["solver"].step(st["u"], st["ds"])
        elif kind == "burgers_rollout":
            out = burgers_rollout(st["solver"], st["u"], case["steps"])
        elif kind == "ks_rollout":
            out = ks_rollout(st["solver"], st["u"], case["steps"], st["ds"], s=st["s"])
        elif kind == "burgers_cnn":
            out, corr = simulate_rollout(st["net"], st["solver"], st["u"], case["steps"], "INC")
            if not grad:
                return dict(frames=out, corrections=corr)
        elif kind == "fno":
            out = st["net"](st["u"])
        else:
            out, corr = simulate_rollout(st["net"], st["solver"], st["u"], case["steps"], "INC", L=st["ds"])
        if not grad:
            return out
        loss = _mse(out, st["target"])
    loss.backward()
    return dict(out=out.detach(), **_grads(st))


# ---------------------------------------------------------------------------- what it needs
def _fno_work(case):
    """Multiply-adds of the lift, the four layers (pointwise product; the Fourier branch as
    a transform to and from the kept modes and their mixing) and the projection."""
    n, w, m = case["n"], case["width"], case["modes"]
    fft = 2 * 2.5 * math.log2(n)
    layer = 2 * w * w + 2 * fft / 2 * w + 8 * w * w * m / n
    return 4 * w + 4 * layer + 2 * w * 128 + 2 * 128


def work(case):
    kind, B = case["kind"], case["B"]
    if kind == "burgers_ragged":
        cells = float(_ragged_sizes(B).sum())
        return dict(bytes=8 * cells, flops=503 * cells * case["steps"])
    n, steps = case["n"], case.get("steps", 1)
    cells = float(B * n)
    if kind == "burgers_step":
        return dict(bytes=12 * cells, flops=(503 if case["scheme"] == "ssprk3" else 165) * cells)
    if kind == "burgers_rollout":
        if case["grad"]:  # frames out, target in, their gradient, the state in and its gradient out
            return dict(bytes=cells * (8 + 8 * steps), flops=3 * 503 * cells * steps)
        return dict(bytes=cells * (4 + 4 * steps), flops=503 * cells * steps)
    ks = 2 * (10 * math.log2(n) + 12)
    if kind == "ks_step_grad":
        return dict(bytes=cells * 24, flops=3 * ks * cells)
    if kind == "ks_rollout":
        if case["grad"]:
            return dict(bytes=cells * (16 + 8 * steps), flops=3 * ks * cells * steps)
        return dict(bytes=cells * (8 + 4 * steps), flops=ks * cells * steps)
    if kind == "burgers_cnn":
        net = 21120 + 503
        if case["grad"]:
            return dict(bytes=cells * (8 + 8 * steps), flops=3 * net * cells * steps)
        return dict(bytes=cells * (4 + 8 * steps), flops=net * cells * steps)
    w = case["width"]
    params = 8.0 * 4 * w * w * case["modes"] + 4.0 * (4 * w * w + 128 * w)
    if kind == "fno":
        if case["grad"]:
            return dict(bytes=16 * cells + 2 * params, flops=3 * _fno_work(case) * cells)
        return dict(bytes=8 * cells + params, flops=_fno_work(case) * cells)
    return dict(bytes=cells * (8 + 8 * steps) + 2 * params, flops=3 * (_fno_work(case) + ks) * cells * steps)


# ---------------------------------------------------------------------------- 64 bits
def _weno(f, right):
    """WENO5-JS values of f at the right interface of every cell (the right-biased form is
    the mirrored stencil around cell i + 1)."""
    r = lambda k: torch.roll(f, -k, -1)  # noqa: E731
    a, b, c, d, e = (r(3), r(2), r(1), r(0), r(-1)) if right else (r(-2), r(-1), r(0), r(1), r(2))
    if right:  # stencils in the reference's order: (i-1, i, i+1), (i, i+1, i+2), (i+1, i+2, i+3)
        a, b, c, d, e = e, d, c, b, a
        q = (11 * c - 7 * b + 2 * a) / 6, (2 * d + 5 * c - b) / 6, (-e + 5 * d + 2 * c) / 6
        s = (3 * c - 4 * b + a, d - b, 3 * e - 4 * d + c)
    else:
        q = (2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6
        s = (a - 4 * b + 3 * c, b - d, 3 * c - 4 * d + e)
    curv = (a - 2 * b + c, b - 2 * c + d, c - 2 * d + e)
    w = [g / (1e-6 + 13 / 12 * k * k + 0.25 * t * t) ** 2 for g, k, t in zip((0.1, 0.6, 0.3), curv, s)]
    return (w[0] * q[0] + w[1] * q[1] + w[2] * q[2]) / (w[0] + w[1] + w[2])


def _burgers_rhs(u, dx, nu, s=None):
    alpha = u.abs().max(dim=1, keepdim=True).values
    flux = 0.5 * u * u
    h = _weno(0.5 * (flux + alpha * u), False) + _weno(0.5 * (flux - alpha * u), True)
    r = -(h - torch.roll(h, 1, -1)) / dx + nu * (torch.roll(u, 1, -1) - 2 * u + torch.roll(u, -1, -1)) / (dx * dx)
    return r if s is None else r + s


def _burgers_step(u, dx, dt, nu, s=None, scheme="ssprk3"):
    u1 = u + dt * _burgers_rhs(u, dx, nu, s)
    if scheme == "euler":
        return u1
    u2 = 0.75 * u + 0.25 * (u1 + dt * _burgers_rhs(u1, dx, nu, s))
    return u / 3 + 2 / 3 * (u2 + dt * _burgers_rhs(u2, dx, nu, s))


def _ks_coefficients(case):
    k = TWO_PI * torch.fft.rfftfreq(case["n"], 1.0 / case["n"], device=DEV, dtype=torch.float64)
    k = k / torch.tensor(case["L"], dtype=torch.float32).double().item()
    lop, dt = k * k - k ** 4, case["dt"]
    e, small = torch.exp(lop * dt), lop.abs() < 1e-6
    safe = torch.where(small, torch.ones_like(lop), lop)
    p1 = torch.where(small, torch.full_like(lop, dt), (e - 1) / safe)
    p2 = torch.where(small, torch.full_like(lop, dt / 2), (e - 1 - lop * dt) / (safe * safe * dt))
    ik = torch.complex(torch.zeros_like(k), k)
    ik[-1] = 0  # the Nyquist derivative is imaginary in physical space
    return e, p1, p2, -0.5 * ik


def _ks_step(u, co, s=None):
    e, p1, p2, d = co
    n = u.shape[-1]
    sh = 0 if s is None else torch.fft.rfft(s)
    for _ in range(2):
        n1 = d * torch.fft.rfft(u * u)
        a = e * torch.fft.rfft(u) + p1 * (n1 + sh)
        ui = torch.fft.irfft(a, n=n)
        u = torch.fft.irfft(a + p2 * (d * torch.fft.rfft(ui * ui) - n1), n=n)
    return u


def _cnn(p, u):
    x = u.unsqueeze(1)
    for i in range(4):
        x = F.conv1d(F.pad(x, (2, 2), mode="circular"), p[2 * i], p[2 * i + 1])
        x = F.gelu(x) if i < 3 else x
    return x.squeeze(1)


def _fno(p, u, L):
    """p: the parameters by name, in 64 bits; L a number or [B] domain sizes."""
    n = u.shape[-1]
    if isinstance(L, torch.Tensor):
        grid = L.reshape(-1, 1) * torch.linspace(0, 1, n, dtype=u.dtype, device=u.device)
    else:
        grid = torch.linspace(0, L, n, dtype=u.dtype, device=u.device).expand(u.shape)
    h = torch.einsum("wc,bcn->bwn", p["fc0.weight"], torch.stack([u, grid], 1)) + p["fc0.bias"][:, None]
    for i in range(4):
        w = p[f"conv{i}.weights1"]
        m = w.shape[-1]
        modes = torch.einsum("bim,iom->bom", torch.fft.rfft(h)[..., :m], w)
        spec = torch.fft.irfft(F.pad(modes, (0, n // 2 + 1 - m)), n=n)
        h = spec + torch.einsum("oi,bin->bon", p[f"w{i}.weight"][:, :, 0], h) + p[f"w{i}.bias"][:, None]
        h = F.gelu(h) if i < 3 else h
    h = F.gelu(torch.einsum("oi,bin->bon", p["fc1.weight"], h) + p["fc1.bias"][:, None])
    return (torch.einsum("oi,bin->bon", p["fc2.weight"], h) + p["fc2.bias"][:, None]).squeeze(1)


def _params64(net):
    return {k: v.detach().to(torch.complex128 if v.is_complex() else torch.float64).requires_grad_(True)
            for k, v in net.named_parameters()}


def _unroll(step, u, steps, grad):
    frames = []
    for _ in range(steps):
        u = checkpoint(step, u, use_reentrant=False) if grad else step(u)
        frames.append(u)
    return torch.stack(frames, 1)


def exact(case, seed):
    ins = _inputs(case, seed)
    kind = case["kind"]
    if kind == "burgers_ragged":
        out = [None] * case["B"]
        for n in (64, 128, 256, 512):
            idx = [i for i, v in enumerate(ins["ns"].tolist()) if v == n]
            if not idx:
                continue
            col = lambda a: torch.tensor(a[idx], device=DEV, dtype=torch.float64).reshape(-1, 1)  # noqa: E731
            u = torch.stack([torch.from_numpy(ins["rows"][i]) for i in idx]).to(DEV).double()
            nu, dt, dx = col(ins["nu"]), col(ins["dt"]), col(ins["dx"])
            for _ in range(case["steps"]):
                u = _burgers_step(u, dx, dt, nu)
            for i, row in zip(idx, u):
                out[i] = row
        return torch.cat(out)
    grad = "target" in ins
    leaf = {k: ins[k].double().requires_grad_(grad) for k in ("u", "s") if k in ins}
    u, s, n = leaf["u"], leaf.get("s"), case["n"]
    p = _params64(ins["net"]) if "net" in ins else {}
    if kind.startswith("burgers"):
        dx, dt, nu = TWO_PI / n, _burgers_dt(n), 0.01
    elif kind != "fno":
        co = _ks_coefficients(case)
    with torch.set_grad_enabled(grad):
        if kind == "burgers_step":
            out = _burgers_step(u, dx, dt, nu, s, case["scheme"])
        elif kind == "burgers_rollout":
            out = _unroll(lambda v: _burgers_step(v, dx, dt, nu), u, case["steps"], grad)
        elif kind == "ks_step_grad":
            out = _ks_step(u, co, s)
        elif kind == "ks_rollout":
            out = _unroll(lambda v: _ks_step(v, co, s), u, case["steps"], grad)
        elif kind == "fno":
            out = _fno(p, u, 64.0)
        elif kind == "ks_fno_train":
            ds = torch.full((case["B"],), case["L"], device=DEV).double()
            out = _unroll(lambda v: _ks_step(v, co, _fno(p, v, ds)), u, case["steps"], grad)
        else:
            q = list(p.values())
            if not grad:
                frames, corr = [], []
                for _ in range(case["steps"]):
                    corr.append(_cnn(q, u))
                    u = _burgers_step(u, dx, dt, nu, corr[-1])
                    frames.append(u)
                return dict(frames=torch.stack(frames, 1), corrections=torch.stack(corr, 1))
            out = _unroll(lambda v: _burgers_step(v, dx, dt, nu, _cnn(q, v)), u, case["steps"], grad)
        if not grad:
            return out.detach()
        loss = _mse(out, ins["target"].double())
    loss.backward()
    res = dict(out=out.detach(), **{k: v.grad for k, v in leaf.items()})
    if p:
        res["params"] = [v.grad for v in p.values()]
    return res
