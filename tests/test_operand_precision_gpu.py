"""The tensor-core products keep FP32's accuracy whatever the sizes of the operands beside
each other: channels whose activations are a power of two smaller and whose next layer's weights
are as much larger, cells far from one large cell, and short rows.  Errors are against
FP64 and are bounded by those of FP32 arithmetic on the same inputs (torch's layers, the
layer-by-layer FNO, the replaying CNN backward).  Factors: 4 for one tensor or channel against
another evaluation's, whose rounding scatters; 1.25 where errors are averaged over seeds."""
import copy

import pytest
import torch

from inc_b200 import fused
from inc_b200.correctors import FNO1D, PeriodicCNN1D, fp64_copy
from tests.test_fused_gpu import _params, _sim_params, _u0, fp32_convs  # noqa: F401

pytestmark = pytest.mark.gpu


def _err(a, ref):
    """Relative L2 error."""
    a, ref = (torch.view_as_real(t) if t.is_complex() else t for t in (a.detach().cpu(), ref.detach().cpu()))
    return ((a.double() - ref.double()).norm() / ref.double().norm().clamp_min(1e-300)).item()


def _fno_errors(net, ref, u, gy, cuda, native):
    """Errors of y, dL/du and every parameter's gradient; those of the layers next to the
    rescaled channels are the worst over these channels."""
    net = copy.deepcopy(net).to(cuda)
    if not native:
        net.conv1.register_forward_hook(lambda *a: None)  # a hooked layer: layer by layer
    uc = u.float().to(cuda).requires_grad_(True)
    y = net(uc)
    assert ("FNOFn" in type(y.grad_fn).__name__) == native
    y.backward(gy.float().to(cuda))
    ur = u.clone().requires_grad_(True)
    yr = ref(ur)
    grads = torch.autograd.grad(yr, [ur] + list(ref.parameters()), gy)
    out = dict(y=_err(y, yr), u=_err(uc.grad, grads[0]))
    axis = {"fc1.weight": 1, "conv3.weights1": 1, "w3.weight": 0}
    for (name, p), g in zip(net.named_parameters(), grads[1:]):
        if name in axis:
            out[name] = max(_err(a, b) for a, b in zip(p.grad.unbind(axis[name]), g.unbind(axis[name])))
        else:
            out[name] = _err(p.grad, g)
    return out


@pytest.mark.parametrize("width,e", [(64, 6), (64, 20), (32, 10)])
def test_fno_channels_of_different_size(cuda, width, e):
    """Every second channel between the last layer and fc1 2^-e times as large, its weights in
    fc1 2^e times: no GELU stands between them, so the function is the same and an FP32
    evaluation rounds the same."""
    torch.manual_seed(width)
    net = FNO1D(L=20.0, modes=12, width=width)
    g = torch.Generator().manual_seed(e)
    u, gy = (torch.randn(7, 256, generator=g, dtype=torch.float64) for _ in range(2))
    fp32 = _fno_errors(net, fp64_copy(net), u, gy, cuda, native=False)
    scale = 2.0 ** (-e * (torch.arange(width) % 2).float())
    with torch.no_grad():
        net.conv3.weights1 *= scale[None, :, None]
        net.w3.weight *= scale[:, None, None]
        net.w3.bias *= scale
        net.fc1.weight /= scale
    for name, err in _fno_errors(net, fp64_copy(net), u, gy, cuda, native=True).items():
        assert err <= 4 * fp32[name], name


def _corrections(net, u, N, cuda, steps=1, dt=None):
    """The corrections of every step, [B, steps, N]."""
    from inc_b200.solvers import BurgersSolverTorch
    params = _sim_params(_params(N, B=u.shape[0]), u.shape[0], "euler", cuda)
    params.dt = params.dt if dt is None else dt
    return fused.burgers_cnn_rollout(net, BurgersSolverTorch(params), u, steps)[1]


@pytest.mark.parametrize("e", [6, 20])
def test_cnn_hidden_channels_of_different_size(cuda, e):
    N = 128
    torch.manual_seed(e)
    net = PeriodicCNN1D()
    scale = 2.0 ** (-e * (torch.arange(32) % 2).float())
    with torch.no_grad():
        net.convs[1].weight *= scale[:, None, None]
        net.convs[1].bias *= scale
        net.convs[2].weight /= scale[:, None]
    u = torch.tensor(_u0(4, N, seed=e), dtype=torch.float32)
    with torch.no_grad():
        ref = copy.deepcopy(net).double()(u.double())
        fp32 = _err(net(u), ref)
        assert _err(_corrections(net.to(cuda), u.to(cuda), N, cuda)[:, 0], ref) <= 4 * fp32


@pytest.mark.parametrize("N,size", [(64, 1e3), (256, 1e6), (512, 1e9)])
def test_cnn_cells_far_from_a_large_one(cuda, N, size):
    torch.manual_seed(N)
    net = PeriodicCNN1D()
    u = torch.tensor(_u0(3, N, seed=N), dtype=torch.float32)
    u[:, 20] = size
    with torch.no_grad():
        ref = copy.deepcopy(net).double()(u.double())
        fp32 = net(u)
        got = _corrections(net.to(cuda), u.to(cuda), N, cuda)[:, 0]
    far = torch.arange(N)[40:]  # beyond the receptive field of cell 20
    assert _err(got[:, far], ref[:, far]) <= 4 * _err(fp32[:, far], ref[:, far])


def _hidden_gradients(net, u, w, cuda, monkeypatch, record):
    """(native, FP64) gradients of the hidden weights of sum(w * corrections), steps that leave the
    state as it is (dt = 1e-30): each is the network's at u."""
    ref = copy.deepcopy(net).double()
    (ref(u.double())[:, None] * w.double()).sum().backward()
    net = copy.deepcopy(net).to(cuda)
    with monkeypatch.context() as m:
        if not record:
            m.setattr(fused, "ACTS_BYTES_MAX", 0)
        c = _corrections(net, u.to(cuda), u.shape[1], cuda, w.shape[1], 1e-30)
        (c * w.to(cuda)).sum().backward()
    return [(net.convs[i].weight.grad, ref.convs[i].weight.grad) for i in (1, 2)]


def test_cnn_hidden_weight_gradients_of_one_short_row(cuda, monkeypatch):
    """Their operands are rounded no more coarsely than the replaying backward's."""
    N, steps = 64, 4
    total = {}
    for seed in range(8):
        torch.manual_seed(seed)
        net = PeriodicCNN1D()
        u = torch.tensor(_u0(1, N, seed=seed), dtype=torch.float32)
        w = torch.randn(1, steps, N, generator=torch.Generator().manual_seed(seed))
        for record in (True, False):
            for i, (a, r) in enumerate(_hidden_gradients(net, u, w, cuda, monkeypatch, record)):
                total[record, i] = total.get((record, i), 0.0) + _err(a, r) ** 2
    for i in range(2):
        assert total[True, i] <= 1.25 ** 2 * total[False, i], i


@pytest.mark.parametrize("B,N,steps,e", [(5, 256, 4, 6), (3, 512, 5, 20), (9, 64, 4, 12)])
def test_cnn_hidden_weight_gradients_by_channel(cuda, monkeypatch, B, N, steps, e):
    """Each channel's gradient on its own, every second channel's activations 2^-e times as large
    (and its adjoint 2^e): a small channel's sums are as accurate as a large one's.  The mean
    square over the 32 channels scatters less than one tensor's error: factor 2."""
    torch.manual_seed(N)
    net = PeriodicCNN1D()
    scale = 2.0 ** (-e * (torch.arange(32) % 2).float())
    with torch.no_grad():
        net.convs[1].weight *= scale[:, None, None]
        net.convs[1].bias *= scale
        net.convs[2].weight /= scale[:, None]
    u = torch.tensor(_u0(B, N, seed=N), dtype=torch.float32)
    w = torch.randn(B, steps, N, generator=torch.Generator().manual_seed(N))
    rms = {}
    for record in (True, False):
        grads = _hidden_gradients(net, u, w, cuda, monkeypatch, record)
        rms[record] = [sum(_err(a.select(axis, c), r.select(axis, c)) ** 2 for c in range(32)) ** 0.5
                       for axis, (a, r) in enumerate(grads)]  # conv 1's output channels, conv 2's input channels
    for i in range(2):
        assert rms[True][i] <= 2 * rms[False][i], i


def test_cnn_hidden_gradients_with_weight_rows_of_different_size(cuda, monkeypatch):
    """The same scaling under a loss of one sign (truncation adds up over cells), each channel
    on its own, averaged over seeds."""
    N, e = 256, 12
    scale = 2.0 ** (-e * (torch.arange(32) % 2).float())
    total = {True: [0.0, 0.0], False: [0.0, 0.0]}
    for seed in range(6):
        torch.manual_seed(seed)
        net = PeriodicCNN1D()
        with torch.no_grad():
            net.convs[1].weight *= scale[:, None, None]
            net.convs[1].bias *= scale
            net.convs[2].weight /= scale[:, None]
        u = torch.tensor(_u0(4, N, seed=seed), dtype=torch.float32)
        for record in (True, False):
            for axis, (a, r) in enumerate(_hidden_gradients(net, u, torch.ones(4, 4, N), cuda, monkeypatch, record)):
                total[record][axis] += sum(_err(a.select(axis, c), r.select(axis, c)) ** 2 for c in range(32))
    for i in range(2):
        assert total[True][i] <= 1.25 ** 2 * total[False][i], i


def _one_channel(bias):
    """A network of channel 0 alone, centre taps of 1 (every sum is one value), `bias` before
    the second and third GELU."""
    net = PeriodicCNN1D()
    with torch.no_grad():
        for p in net.parameters():
            p.zero_()
        for i, conv in enumerate(net.convs):
            conv.weight[0, 0, 2] = 1.0
            if i in (1, 2):
                conv.bias[0] = bias
    return net


def test_gelu_derivative_has_no_systematic_error(cuda):
    """GELU's errors depend on its argument alone, so a mean error does not average out over
    cells.  With 10 before the later GELUs (derivative 1) dL/du is GELU' at u exactly; its mean
    error over bins of 1/4 (65,536 cells: 1e-10 of rounding) is at most 4e-9 where |u| < 1/2
    and 1e-8, FP32 erff's own, elsewhere."""
    B, N = 128, 512
    net = _one_channel(10.0).to(cuda)
    g = torch.Generator().manual_seed(0)
    for k in range(-6, 6):
        u = ((k + torch.rand(B, N, generator=g)) / 4).to(cuda).requires_grad_(True)
        _corrections(net, u, N, cuda, 1, 1e-30).sum().backward()
        z = u.detach().double()
        exact = 0.5 * torch.erfc(-z / 2 ** 0.5) + z * torch.exp(-0.5 * z * z) / (2 * torch.pi) ** 0.5
        error = (u.grad.double() - exact)
        assert error.abs().max() < 2e-7
        assert abs(error.mean().item()) < (4e-9 if -2 <= k < 2 else 1e-8), k


def test_cnn_overflow_before_a_gelu(cuda):
    """GELU is infinite at +infinity, as 0.5 z (1 + erf(z / sqrt 2)) is: the third layer's input
    overflows in cell 20, which the last layer passes on, and to its neighbours with weight 0."""
    N = 128
    net = _one_channel(0.0).to(cuda)
    u = torch.zeros(2, N, device=cuda)
    u[:, 20] = 1e38
    want = torch.zeros(2, N)
    want[:, 18:23] = float("nan")
    want[:, 20] = float("inf")
    with torch.no_grad():
        net.convs[2].weight[0, 0, 2] = 10.0
        got = _corrections(net, u, N, cuda, 1, 1e-30)[:, 0].cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    keep = ~torch.isnan(want)
    assert torch.equal(got[keep], want[keep])


@pytest.mark.parametrize("N", [64, 256, 512])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_cnn_non_finite_cell_leaves_the_others(cuda, N, bad):
    """A non-finite cell of the state, and of the adjoint, leaves cells beyond its reach as they are."""
    torch.manual_seed(N)
    net = PeriodicCNN1D()
    g = torch.Generator().manual_seed(N)
    u = torch.tensor(_u0(3, N, seed=N), dtype=torch.float32)
    w = torch.randn(3, 1, N, generator=g)
    far = torch.arange(N)[40:]
    uc = u.to(cuda).requires_grad_(True)
    net = net.to(cuda)
    (_corrections(net, uc, N, cuda, 1, 1e-30) * w.to(cuda)).sum().backward()
    want, uc.grad = uc.grad[:, far].clone(), None
    w[:, :, 20] = bad
    (_corrections(net, uc, N, cuda, 1, 1e-30) * w.to(cuda)).sum().backward()
    assert not torch.isfinite(uc.grad[:, 20]).any()
    assert _err(uc.grad[:, far], want) < 1e-6
    with torch.no_grad():
        clean = _corrections(net, u.to(cuda), N, cuda, 1, 1e-30)[:, 0, far]
        u[:, 20] = bad
        got = _corrections(net, u.to(cuda), N, cuda, 1, 1e-30)[:, 0]
    assert not torch.isfinite(got[:, 20]).any() and _err(got[:, far], clean) < 1e-6


@pytest.mark.parametrize("B,n", [(600, 512), (1200, 256), (592, 512)])
def test_fno_gradients_of_large_batches(cuda, B, n):
    """Past 16 SM counts of tiles the weight gradients take whole rows at a time (592 rows of 512 on 148
    SMs are the last that do not): sums of up to 512 full-scale terms in the accumulators."""
    torch.manual_seed(B)
    net = FNO1D(L=20.0, modes=16, width=32)
    g = torch.Generator().manual_seed(n)
    u, gy = (torch.randn(B, n, generator=g, dtype=torch.float64).to(cuda) for _ in range(2))
    ref = fp64_copy(net).to(cuda)
    fp32 = _fno_errors(net, ref, u, gy, cuda, native=False)
    for name, err in _fno_errors(net, ref, u, gy, cuda, native=True).items():
        assert err <= 4 * fp32[name], name
