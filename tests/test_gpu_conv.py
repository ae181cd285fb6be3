"""Convolution-as-GEMM (overlapping-row TMA view) against F.conv1d."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from nmtgminor_b200 import ops
from nmtgminor_b200.ops import conv as C
from nmtgminor_b200.parallel.flat import FlatParameterStore


@pytest.mark.parametrize("Ci,Co,k,s,act", [(512, 512, 3, 2, "gelu"), (512, 512, 2, 2, "none"), (80, 256, 3, 1, "gelu"),
                                           (256, 256, 3, 2, "relu")])
def test_conv1d_gemm_forward_backward(Ci, Co, k, s, act):
    torch.manual_seed(0)
    B, T = 3, 101
    conv = torch.nn.Conv1d(Ci, Co, k, stride=s).cuda()
    ref = torch.nn.Conv1d(Ci, Co, k, stride=s).cuda()
    ref.load_state_dict(conv.state_dict())
    store = FlatParameterStore(conv, "cuda")
    x = torch.randn(B, T, Ci, device="cuda").bfloat16().requires_grad_()
    y = C.conv1d(x, conv.weight, conv.bias, s, act)
    xr = x.detach().float().requires_grad_()
    with torch.no_grad():
        ref.weight.copy_(conv.weight.work.float())
        ref.bias.copy_(conv.bias.work.float())
    yr = C.conv1d_reference(xr, ref.weight, ref.bias, s, act)
    assert y.shape == yr.shape
    scale = yr.abs().max().item()
    assert (y.float() - yr).abs().max().item() / scale < 2e-2
    g = torch.randn_like(yr)
    (y.float() * g).sum().backward()
    (yr * g).sum().backward()
    torch.cuda.synchronize()
    assert ops.check_status() == 0
    rel = lambda a, b: ((a - b).abs().max() / (b.abs().max() + 1e-6)).item()
    assert rel(x.grad.float(), xr.grad) < 3e-2
    assert rel(conv.weight.main_grad, ref.weight.grad) < 3e-2
    assert rel(conv.bias.main_grad, ref.bias.grad) < 3e-2
    print("overlapping-row descriptors accepted:", C._OVERLAP_OK[0])


def test_feature_extractor_gemm_path_matches_library_path():
    from nmtgminor_b200.models.speech_encoders import ConvFeatureExtractor
    torch.manual_seed(0)
    specs = [(64, 10, 5), (64, 3, 2), (64, 3, 2), (64, 2, 2)]
    for mode in ("layer_norm", "default"):
        fe = ConvFeatureExtractor(specs, mode=mode, conv_bias=True).cuda()
        wav = torch.randn(2, 4000, device="cuda")
        want = fe(wav)                     # library path (no working copies yet)
        FlatParameterStore(fe, "cuda")
        got = fe(wav)
        assert got.shape == want.shape
        assert (got.float() - want).abs().max().item() / want.abs().max().item() < 5e-2


@pytest.mark.parametrize("channels,taps,stride,B,samples,bias", [(256, 1, 1, 1, 1, True), (512, 10, 5, 1, 10, False), (512, 10, 5, 3, 2347, True),
                                                                 (256, 16, 64, 2, 1105, False), (512, 3, 2, 5, 64, True)])
def test_front_end_kernels(channels, taps, stride, B, samples, bias):
    """Convolution + LayerNorm + GELU and LayerNorm + GELU against 64 bits: results differ by their rounding to the
    8 significant bits of bf16 (at most 2^-8 of the value) and by the 32-bit
    sums, whose error in a unit-variance row stays below 2^-23 * (taps + channels) over the deviation of the row."""
    g = torch.Generator().manual_seed(taps * channels + samples)
    rand = lambda *s: torch.randn(*s, generator=g).cuda()
    wav, w, b = rand(B, samples), rand(channels, 1, taps), rand(channels) if bias else None
    norm = torch.nn.LayerNorm(channels).cuda()
    with torch.no_grad():
        norm.weight.copy_(1 + 0.2 * rand(channels))
        norm.bias.copy_(0.3 * rand(channels))
    T = (samples - taps) // stride + 1
    rows = T + 3

    def want(y):
        return F.gelu(F.layer_norm(y, (channels,), norm.weight.double(), norm.bias.double(), norm.eps))

    def check(got, ref):
        error = (got.double() - ref).abs()
        assert (error <= ref.abs() * 2 ** -8 + 2 ** -23 * (taps + channels) * 8).all(), error.max()
    out = torch.full((B * rows, channels), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.ext().conv_norm_gelu(wav, w, b, norm.weight, norm.bias, norm.eps, out, rows, T, stride)
    check(out.view(B, rows, channels)[:, :T], want(F.conv1d(wav.double().unsqueeze(1), w.double(), None if b is None else b.double(), stride=stride)
                                                   .transpose(1, 2)))
    assert (out.view(B, rows, channels)[:, T:] == 7).all()
    x, then = rand(B * rows, channels).bfloat16(), torch.full_like(out[:B * (T + 1)], 7.0)
    ops.ext().norm_gelu(x, B, rows, norm.weight, norm.bias, norm.eps, then, T + 1, T)
    check(then.view(B, T + 1, channels)[:, :T], want(x.view(B, rows, channels)[:, :T].double()))
    assert (then.view(B, T + 1, channels)[:, T:] == 7).all()


@pytest.mark.parametrize("samples", [400, 719, 4001])
@pytest.mark.parametrize("conv_bias", [False, True])
def test_frozen_front_end_matches_the_general_path(samples, conv_bias):
    """The same layers with and without gradients; strides 5, 2, 2, 3 leave tails of every length behind an utterance."""
    from nmtgminor_b200.models.speech_encoders import ConvFeatureExtractor
    torch.manual_seed(samples)
    fe = ConvFeatureExtractor([(256, 10, 5), (256, 3, 2), (256, 2, 2), (256, 4, 3)], conv_bias=conv_bias).cuda()
    FlatParameterStore(fe, "cuda")
    wav = torch.randn(3, samples + 8, device="cuda")[:, 3:3 + samples]
    want = fe(wav)
    with torch.no_grad():
        assert C.frozen_front_end(wav, fe.convs, fe.norms) is not None
        got = fe(wav)
    assert got.shape == want.shape and got.dtype == want.dtype
    assert (got - want).abs().max().item() / want.abs().max().item() < 5e-2
    fe.norms[0].register_forward_hook(lambda *a: None)           # a hook that has to be called
    with torch.no_grad():
        assert C.frozen_front_end(wav, fe.convs, fe.norms) is None


@pytest.mark.parametrize("shape", [(1, 1, 4), (3, 5, 8), (48, 3, 128), (1024, 64, 128), (2, 7, 1024)])
def test_weight_norm_kernels(shape):
    """Weight and gradients against 64 bits; the columns' sums are of rows = shape[0] * shape[1] products in 32 bits, whose error stays below
    2^-24 * rows times the sum of their sizes."""
    torch.manual_seed(shape[0])
    conv = torch.nn.utils.parametrizations.weight_norm(torch.nn.Conv1d(shape[1], shape[0], shape[2]).cuda(), dim=2)
    gain, v = conv.parametrizations.weight.original0, conv.parametrizations.weight.original1
    with torch.no_grad():
        gain.mul_(1 + 0.3 * torch.randn_like(gain))
    w = C.weight_normed(conv)
    dw = torch.randn_like(w)
    dv, dg = torch.autograd.grad(w, (v, gain), dw, retain_graph=True)
    vd, gd = v.detach().double().requires_grad_(), gain.detach().double().requires_grad_()
    n = vd.square().sum((0, 1), keepdim=True).sqrt()
    want = vd * (gd / n)
    wv, wg = torch.autograd.grad(want, (vd, gd), dw.double())
    part = 2 ** -24 * (shape[0] * shape[1] + 8)
    size = (dw.double() * vd).abs().sum((0, 1), keepdim=True) / n       # what the terms of dg add up to without their signs
    assert ((w - want).abs() <= part * want.abs()).all()
    assert ((dg - wg).abs() <= 2 * part * size).all()
    assert ((dv - wv).abs() <= 2 * part * (gd / n).abs() * (dw.abs() + vd.abs() * size / n)).all()
    # a second derivative: the gradient as differentiable operations
    dv2, dg2 = torch.autograd.grad(w, (v, gain), dw, create_graph=True)
    assert dv2.requires_grad and torch.allclose(dv2, dv, rtol=1e-4, atol=1e-5) and torch.allclose(dg2, dg, rtol=1e-4, atol=1e-4)
    conv.register_forward_hook(lambda *a: None)
    assert C.weight_normed(conv) is None


def test_modes_see_the_operations_that_kernels_replace():
    """Under a dispatch or function mode (a counter, a trace) the normalisation of the weights and the front end are tensor operations."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    from nmtgminor_b200.models.speech_encoders import ConvFeatureExtractor, ConvPositionalEmbedding

    class Dispatched(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Called(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    seen, pos = [], ConvPositionalEmbedding(128, 16, 2).cuda()
    x = torch.randn(2, 40, 128, device="cuda")
    want = torch.autograd.grad(pos(x).square().sum(), list(pos.parameters()))
    with Dispatched():
        loss = pos(x).square().sum()
        assert any("norm" in name for name in seen)
        del seen[:]
        got = torch.autograd.grad(loss, list(pos.parameters()))
        assert any("norm" in name for name in seen)
    for a, b in zip(got, want):
        # the library's convolution rounds its operands to 11 bits (2^-11 each), and weights a last bit apart round differently
        assert (a - b).norm() <= 2 ** -10 * b.norm()
    fe = ConvFeatureExtractor([(256, 10, 5), (256, 3, 2)]).cuda()
    FlatParameterStore(fe, "cuda")
    wav = torch.randn(2, 4000, device="cuda")
    with torch.no_grad():
        for mode in (Dispatched(), Called()):
            with mode:
                assert C.weight_normed(pos.conv) is None and C.frozen_front_end(wav, fe.convs, fe.norms) is None
        with torch.device("cuda"):            # a default device is no such mode
            assert C.weight_normed(pos.conv) is not None and C.frozen_front_end(wav, fe.convs, fe.norms) is not None
    # a graph that is recorded under the mode's eyes later: the forward pass ran outside
    loss = pos(x).square().sum()
    del seen[:]
    with Dispatched():
        torch.autograd.grad(loss, list(pos.parameters()))
    assert any("sum" in name for name in seen)


@pytest.mark.parametrize("masked", [False, True])
def test_a_speech_encoder_waits_for_the_device_once(masked):
    """Lengths reach the host before the front end runs; masks that are drawn from them go the other way without a wait."""
    import warnings

    from nmtgminor_b200.models.speech_encoders import Wav2Vec2Encoder
    p = 0.5 if masked else 0.0
    enc = Wav2Vec2Encoder(dim=128, layers=2, heads=2, ffn=256, conv_layers=[(256, 10, 5), (256, 3, 2)], pos_kernel=16, pos_groups=2, mask_prob=p,
                          mask_length=3, mask_channel_prob=p, mask_channel_length=8).cuda().train()
    FlatParameterStore(enc, "cuda")
    source = torch.randn(3000, 3, 2, device="cuda")
    source[:, :, 0] = torch.arange(3000, device="cuda")[:, None] < torch.tensor([3000, 1234, 700], device="cuda")
    x, seqs = enc(source)
    assert x.shape[0] == int(seqs.cu[-1]) == sum(((n - 10) // 5 + 1 - 3) // 2 + 1 for n in (3000, 1234, 700)) and torch.isfinite(x).all()
    with warnings.catch_warnings(record=True) as seen:
        warnings.simplefilter("always")
        torch.cuda.set_sync_debug_mode("warn")
        try:
            enc(source)
        finally:
            torch.cuda.set_sync_debug_mode("default")
    waits = ["%s:%d" % (w.filename, w.lineno) for w in seen if "called a synchronizing" in str(w.message)]
    assert len(waits) == 1, waits
