"""1-D convolution over channels-last sequences as a tensor-core GEMM without an im2col buffer.

For ``x`` [B, T, Ci] (channels last, time padded to a multiple of the stride) the im2col row of output frame
``(b, t)`` is the contiguous run ``x[b, t*s : t*s + k, :]``: ``k * Ci`` elements starting ``s * Ci`` elements after
the previous row.  That is an ordinary 2-D tensor whose rows overlap, which a TMA descriptor (row stride ``s * Ci``,
row length ``k * Ci``) reads directly, so the convolution is ONE ``gemm(A_view, W[Co, k*Ci])`` with the bias and the
activation in the epilogue.  If the driver refuses descriptors with overlapping rows the same result is produced
from ``k`` GEMMs over non-overlapping single-tap views.  The weight gradient is the transposed product over the same
view; the input gradient is ``k`` GEMMs that scatter each tap back into its strided slot.

Used for the wav2vec2 feature extractor layers after the first (512 channels, k 3 / 2, stride 2) and the Whisper
stem (80 -> 1280 k3, 1280 -> 1280 k3 s2), replacing cuDNN calls of the reference (onmt/models/speech_recognizer/
fairseq_wav2vec2/wav2vec2.py ``ConvFeatureExtractionModel``; onmt/models/whisper/whisper_encoder.py conv1 / conv2).
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from . import ACT_IDS, _act_backward, empty_rows, ext, fused_param, gemm

_OVERLAP_OK = [None]      # None = untested, True / False once the driver answered


def conv1d_reference(x, weight, bias=None, stride: int = 1, act: str = "none"):
    """x [B, T, Ci], weight [Co, Ci, k] -> [B, T_out, Co] (plain PyTorch)."""
    y = F.conv1d(x.transpose(1, 2).float(), weight.float(), None if bias is None else bias.float(), stride=stride).transpose(1, 2)
    if act == "gelu":
        y = F.gelu(y)
    elif act == "relu":
        y = F.relu(y)
    elif act in ("silu", "swish"):
        y = F.silu(y)
    return y.to(x.dtype)


def _padded_input(x, k: int, s: int):
    """Copy x into a zero-tailed buffer whose time axis is a multiple of the stride; returns (flat [rows, Ci], Tp)."""
    B, T, Ci = x.shape
    Tp = (T + s - 1) // s * s
    buf = torch.zeros((B * Tp + k, Ci), dtype=torch.bfloat16, device=x.device)
    buf[:B * Tp].view(B, Tp, Ci)[:, :T].copy_(x)
    return buf, Tp


def _overlap_view(buf, M: int, k: int, s: int, Ci: int):
    return buf.as_strided((M, k * Ci), (s * Ci, 1))


def _tap_view(buf, M: int, tap: int, s: int, Ci: int):
    return buf.as_strided((M, Ci), (s * Ci, 1), storage_offset=tap * Ci)


class _Conv1dFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w_work, b_work, gw, gb, stride, act, need_dx):
        B, T, Ci = x.shape
        Co, _, k = w_work.shape
        s = stride
        buf, Tp = _padded_input(x, k, s)
        M = B * Tp // s
        wg = w_work.permute(0, 2, 1).reshape(Co, k * Ci).contiguous()          # [Co, k*Ci], tap-major like the rows of A
        out = empty_rows(M, Co, x.device)
        pre = empty_rows(M, Co, x.device) if act != 0 else None
        done = False
        if _OVERLAP_OK[0] is not False:
            try:
                gemm(_overlap_view(buf, M, k, s, Ci), wg, out, bias=b_work, preact=pre, act=act)
                _OVERLAP_OK[0] = done = True
            except RuntimeError as exc:
                if "cuTensorMapEncodeTiled" not in str(exc):
                    raise
                _OVERLAP_OK[0] = False
        if not done:
            acc = out if act == 0 else pre
            for tap in range(k):
                gemm(_tap_view(buf, M, tap, s, Ci), wg[:, tap * Ci:(tap + 1) * Ci], acc, bias=b_work if tap == 0 else None,
                     residual=acc if tap > 0 else None)
            if act != 0:
                a = pre.float()
                out.copy_((F.relu(a) if act == 1 else F.gelu(a) if act == 2 else F.silu(a)).to(out.dtype))
        T_out = (T - k) // s + 1
        ctx.save_for_backward(buf, wg, pre if pre is not None else out)
        ctx.cfg = (B, T, Tp, Ci, Co, k, s, act, T_out, need_dx, M)
        ctx.gw, ctx.gb = gw, gb
        return out.view(B, Tp // s, Co)[:, :T_out]

    @staticmethod
    def backward(ctx, dy):
        buf, wg, pre = ctx.saved_tensors
        B, T, Tp, Ci, Co, k, s, act, T_out, need_dx, M = ctx.cfg
        # frames past T_out (they straddle two utterances or the zero tail) received no gradient
        dz = torch.zeros((M, Co), dtype=torch.bfloat16, device=dy.device)
        dz.view(B, Tp // s, Co)[:, :T_out].copy_(dy)
        if act != 0:
            dz = _act_backward(dz, pre, act)
            dz.view(B, Tp // s, Co)[:, T_out:].zero_()
        if ctx.gw is not None:
            dwg = torch.zeros((Co, k * Ci), dtype=torch.float32, device=dy.device)
            if _OVERLAP_OK[0]:
                gemm(dz, _overlap_view(buf, M, k, s, Ci), dwg, a_mn_major=True, b_mn_major=True, accumulate=True, allow_split_k=True)
            else:
                for tap in range(k):
                    gemm(dz, _tap_view(buf, M, tap, s, Ci), dwg[:, tap * Ci:(tap + 1) * Ci], a_mn_major=True, b_mn_major=True,
                         accumulate=True, allow_split_k=True)
            ctx.gw.add_(dwg.view(Co, k, Ci).permute(0, 2, 1))
        if ctx.gb is not None:
            ext().colsum(dz, ctx.gb)
        dx = None
        if need_dx:
            dbuf = torch.zeros_like(buf)
            for tap in range(k):
                # tap `tap` of every frame lands in its own strided slot; later taps add to what earlier taps wrote
                slot = _tap_view(dbuf, M, tap, s, Ci)
                gemm(dz, wg[:, tap * Ci:(tap + 1) * Ci], slot, b_mn_major=True, residual=slot if tap >= s else None)
            dx = dbuf[:B * Tp].view(B, Tp, Ci)[:, :T]
        return dx, None, None, None, None, None, None, None


def conv1d(x, weight, bias=None, stride: int = 1, act: str = "none", padding: int = 0):
    """Channels-last 1-D convolution: ``x`` [B, T, Ci], ``weight`` [Co, Ci, k] (the ``nn.Conv1d`` layout).

    Takes the GEMM path for parameters with bf16 working copies when ``stride * Ci`` and ``Ci`` are multiples of 8;
    anything else (the single-channel first wav2vec2 layer, grouped convolutions) runs ``F.conv1d``."""
    act_id = ACT_IDS[act]
    if padding:
        x = F.pad(x, (0, 0, padding, padding))
    Ci = x.shape[-1]
    if not (fused_param(weight) and x.is_cuda and Ci % 8 == 0 and (stride * Ci) % 8 == 0 and weight.shape[1] == Ci):
        return conv1d_reference(x, weight, bias, stride, act)
    gw = weight.main_grad if weight.requires_grad else None
    gb = bias.main_grad if (bias is not None and bias.requires_grad) else None
    xin = x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16)
    if not torch.is_grad_enabled():
        gw = gb = None
    return _Conv1dFn.apply(xin, weight.work, bias.work if bias is not None else None, gw, gb, int(stride), act_id,
                           bool(x.requires_grad and torch.is_grad_enabled()))


def _watched() -> bool:
    """Whether a mode or a hook of all modules has to see the tensor operations that a kernel would replace.  (The mode of a default
    device only looks at calls that make tensors.)"""
    return (torch._C._len_torch_dispatch_stack() > 0
            or any(type(m) is not torch.utils._device.DeviceContext for m in torch.overrides._get_current_function_mode_stack())
            or torch.is_autocast_enabled() or torch.jit.is_tracing() or torch._C._are_functorch_transforms_active()
            or torch.autograd.forward_ad._current_level >= 0 or torch.nn.modules.module._has_any_global_hook())


def _hooked(*modules) -> bool:
    return any(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks for m in modules)


def _front_end_layer(i, conv, norm, channels: int, device) -> bool:
    """Whether layer ``i`` is of the kind that the kernels of csrc/frontend.cu take."""
    if not (type(conv) is torch.nn.Conv1d and type(norm) is torch.nn.LayerNorm and tuple(norm.normalized_shape) == (channels,)
            and norm.weight is not None and norm.bias is not None and not _hooked(norm)):
        return False
    w = conv.weight
    if not all(p.dtype == torch.float32 and p.device == device for p in (norm.weight, norm.bias, w)):
        return False
    if conv.out_channels != channels or conv.groups != 1 or conv.dilation != (1,) or conv.padding != (0,):
        return False
    if i == 0:
        return conv.in_channels == 1 and conv.kernel_size[0] <= 16 and conv.stride[0] <= 64
    return conv.in_channels == channels and fused_param(w) and (conv.bias is None or fused_param(conv.bias))


def frozen_front_end(wav, convs, norms):
    """Strided convolutions over ``wav`` [B, samples], LayerNorm over the channels and GELU behind each, without gradients: ``[B, T, C]``
    (bf16).  The first convolution, every norm and every GELU run in the kernels of csrc/frontend.cu, which leave their frames where the
    next convolution's overlapping rows are read.  None for layers that these do not take (256 or 512 channels as one or two 16-byte
    vectors a lane) and under the tracers and modes that have to see tensor operations."""
    C = convs[0].out_channels
    if (torch.is_grad_enabled() or _watched() or type(wav) is not torch.Tensor or not wav.is_cuda or wav.dim() != 2 or wav.shape[0] == 0
            or C not in (256, 512) or _OVERLAP_OK[0] is False):
        return None
    T = wav.shape[1]
    for i, (conv, norm) in enumerate(zip(convs, norms)):
        if not _front_end_layer(i, conv, norm, C, wav.device) or T < conv.kernel_size[0]:
            return None
        T = (T - conv.kernel_size[0]) // conv.stride[0] + 1
    B, T = wav.shape
    for i, (conv, norm) in enumerate(zip(convs, norms)):
        k, s = conv.kernel_size[0], conv.stride[0]
        T = (T - k) // s + 1
        # rows for the next convolution: whole strides of every utterance, and the overhang of the last one's frames.  Those past T are
        # never read by a frame that is kept
        nk, ns = (convs[i + 1].kernel_size[0], convs[i + 1].stride[0]) if i + 1 < len(convs) else (0, 1)
        rows = -(-T // ns) * ns
        out = torch.empty((B * rows + nk, C), dtype=torch.bfloat16, device=wav.device)
        affine = (norm.weight.detach().contiguous(), norm.bias.detach().contiguous(), norm.eps)
        if i == 0:
            bias = conv.bias.detach().float() if conv.bias is not None else None
            ext().conv_norm_gelu(wav.detach().float().contiguous(), conv.weight.detach().contiguous(), bias, *affine, out, rows, T, s)
        else:
            y = empty_rows(B * had // s, C, wav.device)
            taps = conv.weight.work.permute(0, 2, 1).reshape(C, k * C).contiguous()
            try:
                gemm(_overlap_view(buf, y.shape[0], k, s, C), taps, y, bias=conv.bias.work if conv.bias is not None else None)
                _OVERLAP_OK[0] = True
            except RuntimeError as exc:
                if "cuTensorMapEncodeTiled" not in str(exc):
                    raise
                _OVERLAP_OK[0] = False
                return None
            ext().norm_gelu(y, B, had // s, *affine, out, rows, T)
        buf, had = out, rows
    return buf[:B * had].view(B, had, C)


class _WeightNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, v, gain):
        w, norm = ext().weight_norm_fwd(v, gain)
        ctx.save_for_backward(v, gain, norm)
        return w

    @staticmethod
    def backward(ctx, dw):
        v, gain, norm = ctx.saved_tensors
        if torch.is_grad_enabled() or _watched():          # a graph of the gradient is wanted, or its operations: the same as those
            dims = tuple(range(v.dim() - 1))
            n = v.square().sum(dims, keepdim=True).sqrt()
            dot = (dw * v).sum(dims, keepdim=True)
            return (gain / n) * (dw - v * (dot / n.square())), (dot / n).view_as(gain)
        dw = dw.contiguous()
        if dw.data_ptr() % 16:
            dw = dw.clone()
        return ext().weight_norm_bwd(dw, v, gain, norm)


def weight_normed(conv):
    """Weight of a convolution under ``parametrizations.weight_norm(conv, dim=last)`` from the kernels of csrc/weight_norm.cu; None where
    something else parametrises it, or a form, mode or tracer needs the tensor operations."""
    from torch.nn.utils import parametrizations, parametrize
    chain = getattr(conv, "parametrizations", None)
    if chain is None or set(chain.keys()) != {"weight"} or len(chain.weight) != 1 or parametrize._cache_enabled:
        return None
    norm, gain, v = chain.weight[0], chain.weight.original0, chain.weight.original1
    if type(norm) is not parametrizations._WeightNorm or norm.dim not in (v.dim() - 1, -1):
        return None
    lanes = v.shape[-1] // 4
    if (_watched() or _hooked(conv, norm, chain.weight)
            or not all(type(p) in (torch.Tensor, torch.nn.Parameter) and p.is_cuda and p.dtype == torch.float32 and p.is_contiguous()
                       and p.data_ptr() % 16 == 0 for p in (v, gain))
            or v.device != gain.device or gain.numel() != v.shape[-1] or v.numel() == 0 or v.shape[-1] % 4 or lanes > 256 or lanes & (lanes - 1)):
        return None
    return _WeightNormFn.apply(v, gain)
