"""The whole FNO corrector on the GPU (inc_fno_forward / inc_fno_backward): outputs and every
gradient against its FP64 copy on torch's FFTs, at the edges of its ranges (one row, odd
batches, rows of half a tile to four tiles, the widths and mode counts it takes), rows of
very different magnitude, and the calls that keep the general path."""
import pytest
import torch

from inc_b200.correctors import FNO1D, fp64_copy

pytestmark = pytest.mark.gpu
TOL, GTOL = 1e-5, 1e-4  # max abs error over max abs FP64 value, as for the layers' own tests


def _rel(a, ref):
    a, ref = (torch.view_as_real(t) if t.is_complex() else t for t in (a.detach().cpu(), ref.detach().cpu()))
    return (a.double() - ref).abs().max().item() / max(ref.abs().max().item(), 1e-30)


def _net(width, modes, L=16):
    torch.manual_seed(width + modes)
    return FNO1D(L=L, modes=modes, width=width)


def _fused(y):
    return "FNOFn" in type(y.grad_fn).__name__


@pytest.mark.parametrize("B,n,width,modes", [
    (1, 64, 32, 1), (1, 512, 64, 16), (3, 64, 64, 16), (5, 128, 32, 5), (7, 256, 64, 12), (2, 512, 32, 16),
    (65, 128, 64, 16), (149, 64, 64, 7), (150, 256, 32, 16), (301, 128, 64, 3)])
def test_fno_matches_fp64(cuda, B, n, width, modes):
    net = _net(width, modes)
    g = torch.Generator().manual_seed(B + n)
    u = torch.randn(B, n, generator=g, dtype=torch.float64)
    L = 20.0 + torch.rand(B, generator=g, dtype=torch.float64)
    gy = torch.randn(B, n, generator=g, dtype=torch.float64)
    ref = fp64_copy(net)
    ur = u.clone().requires_grad_(True)
    yr = ref(ur, L.float().double())
    yr.backward(gy)
    net = net.to(cuda)
    uc = u.float().to(cuda).requires_grad_(True)
    y = net(uc, L.float().to(cuda))
    assert _fused(y)
    y.backward(gy.float().to(cuda))
    with torch.no_grad():
        assert _rel(net(uc, L.float().to(cuda)), yr) < TOL  # evaluation
    assert _rel(y, yr) < TOL
    assert _rel(uc.grad, ur.grad) < GTOL
    for (name, p), (_, pr) in zip(net.named_parameters(), ref.named_parameters()):
        assert _rel(p.grad, pr.grad) < GTOL, name


def test_fno_rows_of_different_magnitude_and_non_finite(cuda):
    """Each trajectory's tiles have their own scales: small and large states beside each other
    and beside a non-finite one, each as accurate as alone."""
    net = _net(64, 16)
    u = torch.randn(6, 128, generator=torch.Generator().manual_seed(0), dtype=torch.float64)
    u *= torch.tensor([0.0, 1e-6, 1.0, 1.0, 30.0, 1e3], dtype=torch.float64)[:, None]
    ref = fp64_copy(net)
    with torch.no_grad():
        yr = ref(u)
        u[2, 40] = float("nan")
        y = net.to(cuda)(u.float().to(cuda)).cpu()
    assert torch.isnan(y[2]).any()
    for r in (0, 1, 3, 4, 5):
        assert _rel(y[r], yr[r]) < TOL, r


def test_fno_general_path_is_kept_and_agrees(cuda):
    """Hooked layers, a domain size that needs a gradient, and shapes outside the fused kernels
    run layer by layer, with the same results."""
    net = _net(64, 16).to(cuda)
    u = torch.randn(4, 128, generator=torch.Generator().manual_seed(1)).to(cuda).requires_grad_(True)
    y = net(u)
    assert _fused(y)
    seen = []
    h = net.conv1.register_forward_hook(lambda m, i, o: seen.append(o.shape))
    yh = net(u)
    h.remove()
    assert not _fused(yh) and seen == [(4, 64, 128)]
    assert _rel(yh, y.double()) < TOL
    L = torch.full((4,), 16.0, device=cuda, requires_grad=True)
    yl = net(u, L)
    yl.sum().backward()
    assert not _fused(yl) and L.grad is not None and _rel(yl, y.double()) < TOL
    for width, modes, n in ((16, 8, 128), (64, 20, 128), (64, 16, 32)):
        out = _net(width, modes).to(cuda)(torch.randn(2, n, device=cuda))
        assert out.shape == (2, n) and not _fused(out)


def test_fno_partial_gradients_and_permuted_input(cuda):
    """Only what asks for a gradient gets one; a permuted (non-contiguous) state is taken."""
    net = _net(32, 8).to(cuda)
    u = torch.randn(128, 3, generator=torch.Generator().manual_seed(2)).to(cuda).t()
    assert not u.is_contiguous()
    net(u).square().mean().backward()
    full = [p.grad.clone() for p in net.parameters()]
    net.zero_grad()
    for p in net.parameters():
        p.requires_grad_(False)
    net.w2.weight.requires_grad_(True)
    uc = u.contiguous().requires_grad_(True)
    net(uc).square().mean().backward()
    assert uc.grad is not None
    for (name, p), g in zip(net.named_parameters(), full):
        assert (p.grad is None) if name != "w2.weight" else torch.equal(p.grad, g), name


@pytest.mark.parametrize("offset", [1, 3])
def test_fno_parameters_at_odd_offsets(cuda, offset):
    """Parameters that are views into one buffer, 4-byte aligned only: the same bits."""
    torch.manual_seed(offset)
    net = FNO1D(L=16.0, modes=8, width=32).to(cuda)
    u = torch.randn(5, 64, device=cuda)

    def grads():
        net.zero_grad()
        y = net(u)
        y.square().sum().backward()
        return [y.detach()] + [p.grad.clone() for p in net.parameters()]

    want = grads()
    with torch.no_grad():
        for p in net.parameters():
            if not p.is_complex():
                buf = torch.empty(p.numel() + offset, device=cuda)
                buf[offset:].copy_(p.reshape(-1))
                p.data = buf[offset:].view(p.shape)
    assert net._fused(u, 16.0) and net.fc2.weight.data_ptr() % 16 != 0
    for a, b in zip(grads(), want):
        assert torch.equal(a, b)


def test_fno_pending_conjugation_is_not_read_raw(cuda):
    net = FNO1D(L=16.0, modes=8, width=32).to(cuda)
    net.conv1.weights1 = torch.nn.Parameter(net.conv1.weights1.detach().conj())
    assert net.conv1.weights1.is_conj() and not net._fused(torch.randn(2, 64, device=cuda), 16.0)


@pytest.mark.parametrize("wanted", ["u", "fc2.bias", "fc1.bias", "conv3.weights1", "w3.bias", "conv1.weights1",
                                    "w1.weight", "conv0.weights1", "w0.weight", "fc0.bias"])
def test_fno_backward_leaves_out_what_is_frozen(cuda, monkeypatch, wanted):
    """With one gradient asked for, the backward is given that one alone (NULL for the others,
    whose kernels it leaves out) and its bits are those of the full backward."""
    from inc_b200 import _native as nat
    net = _net(32, 8).to(cuda)
    u = torch.randn(5, 128, generator=torch.Generator().manual_seed(3)).to(cuda).requires_grad_(True)
    net(u).square().sum().backward()
    full = dict({n: p.grad.clone() for n, p in net.named_parameters()}, u=u.grad.clone())
    net.zero_grad()
    u = u.detach().requires_grad_(wanted == "u")
    for n, p in net.named_parameters():
        p.requires_grad_(n == wanted)
    given = []

    class Lib:
        def __getattr__(self, name):
            return getattr(lib, name)

        def inc_fno_backward(self, *args):
            g = args[6]._obj
            for field, _ in g._fields_:
                v = getattr(g, field)
                given.extend([v] if v is None or isinstance(v, int) else list(v))
            return lib.inc_fno_backward(*args)

    lib = nat.lib()
    monkeypatch.setattr(nat, "lib", lambda: Lib())
    net(u).square().sum().backward()
    assert sum(v is not None for v in given) == 1 and len(given) == 19
    got = u.grad if wanted == "u" else dict(net.named_parameters())[wanted].grad
    assert torch.equal(got, full[wanted])


def _ks(B, n, cuda):
    from types import SimpleNamespace

    from inc_b200.solvers import KSSolverTorch
    L = torch.linspace(0.2, 0.3, B).mul(n).to(cuda)
    return KSSolverTorch(SimpleNamespace(resolution=n, dt=0.1, device=cuda, domain_size=L,
                                         alpha=torch.zeros(B, device=cuda), time_scheme="ETRK2")), L


@pytest.mark.parametrize("checkpoint_every", [None, 2])
def test_fno_in_the_ks_loop(cuda, monkeypatch, checkpoint_every):
    """simulate_rollout's unrolled training step through FNOFn (each row its own domain size, every
    parameter used at every step) against the same loop layer by layer."""
    from inc_b200 import correctors
    from inc_b200.rollout import simulate_rollout
    B, n, steps = 5, 128, 4
    g = torch.Generator().manual_seed(4)
    u0, target = torch.randn(B, n, generator=g).to(cuda), torch.randn(B, steps, n, generator=g).to(cuda)
    calls = []
    apply = correctors.FNOFn.apply
    monkeypatch.setattr(correctors.FNOFn, "apply", lambda *a: (calls.append(1), apply(*a))[1])
    got = []
    for native in (True, False):
        net = _net(32, 8).to(cuda)
        if not native:
            net.conv2.register_forward_hook(lambda *a: None)
        solver, L = _ks(B, n, cuda)
        u = u0.clone().requires_grad_(True)
        del calls[:]
        frames, corrections = simulate_rollout(net, solver, u, steps, "INC", L=L, checkpoint_every=checkpoint_every)
        (((frames - target) ** 2).mean() + corrections.square().mean()).backward()
        assert len(calls) == (0 if not native else steps if checkpoint_every is None else 2 * steps)
        got.append([frames, corrections, u.grad] + [p.grad for p in net.parameters()])
    for a, b in zip(*got):
        assert _rel(a, b.detach().to(torch.complex128 if b.is_complex() else torch.float64)) < 1e-5


def test_fno_training_step_in_a_graph(cuda):
    """Forward and backward captured in one CUDA graph and replayed for new states: the eager bits."""
    net = _net(64, 16).to(cuda)
    g = torch.Generator().manual_seed(5)
    states = [torch.randn(7, 256, generator=g).to(cuda) for _ in range(2)]
    static = states[0].clone()
    params = list(net.parameters())

    def step(u):
        y = net(u)
        assert _fused(y)
        return [y.detach()] + list(torch.autograd.grad(y.square().mean(), params))

    side = torch.cuda.Stream(cuda)
    side.wait_stream(torch.cuda.current_stream(cuda))
    with torch.cuda.stream(side):
        step(static)
    torch.cuda.current_stream(cuda).wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(static)
    for u in (states[1], states[0]):
        static.copy_(u)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(out, step(u)):
            assert torch.equal(a, b)


def test_fno_evaluation_in_a_graphed_rollout(cuda):
    from inc_b200.graphs import GraphedRollout
    from inc_b200.rollout import simulate_rollout
    B, n, steps = 6, 64, 5
    net = _net(32, 8).to(cuda)
    g = torch.Generator().manual_seed(6)
    a, b = (torch.randn(B, n, generator=g).to(cuda) for _ in range(2))
    solver, L = _ks(B, n, cuda)
    assert net._fused(a, L)
    replay = GraphedRollout(net, solver, a, steps, domain_size=L)
    for u in (b, a):
        frames, corrections = replay(u)
        with torch.no_grad():
            want = simulate_rollout(net, _ks(B, n, cuda)[0], u, steps, "INC", L=L)
        assert torch.equal(frames, want[0]) and torch.equal(corrections, want[1])


def test_fno_second_derivative_is_refused(cuda):
    """A penalty on dL/du needs what the native backward does not record: an error, not a term that
    silently contributes nothing."""
    net = _net(32, 8).to(cuda)
    u = torch.randn(2, 64, device=cuda, requires_grad=True)
    (gu,) = torch.autograd.grad(net(u).square().sum(), u, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        (net(u).square().sum() + gu.square().sum()).backward()
