"""Patch embedding of the vision encoders: a convolution whose stride is its kernel size is a linear layer on patches.

``patch_embed(conv, pixels)`` is ``conv(pixels).flatten(2).transpose(1, 2)``: ``[B, C, H, W]`` pixels to ``[B, patches, hidden]`` tokens.  On
the native path one kernel (``csrc/patchify.cu``) lays the patches out as rows, padded to whole 16 bytes, and the tcgen05 GEMM does
the rest; everything that is not the plain form (hooks on the module, a forward of its own, gradients for the pixels, other strides,
tensor subclasses, autocast, tracing, transforms, modes and timers that want to see the convolution) is left to the module.  (cuDNN runs these shapes on a general kernel: 384 x 384 pixels, patches of 14, 1152 channels 138 us, here 12.)
"""

from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.autograd import forward_ad
from torch.utils._device import DeviceContext

from . import _native as nat
from .gemm import gemm
from .linear import colsum

nat.declare("csb_patchify", [nat.vp] * 2 + [nat.i64] * 3 + [nat.i32] * 8 + [nat.vp])


class _PatchEmbedFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias):
        B, C, H, W = x.shape
        N, _, ph, pw = weight.shape
        gh, gw, K = H // ph, W // pw, C * ph * pw
        Kp = (K + 7) // 8 * 8
        x = x if x.stride(3) == 1 else x.contiguous()
        patches = torch.empty((B * gh * gw, Kp), dtype=x.dtype, device=x.device)
        _patchify(x, patches, B, C, gh, gw, ph, pw)
        w2 = weight.reshape(N, K)
        if Kp != K or w2.data_ptr() % 16:
            wp = torch.empty((N, Kp), dtype=x.dtype, device=x.device)
            _patchify(w2, wp, N, 1, 1, 1, 1, K)  # rows of K as rows of Kp
            w2 = wp
        y = gemm(patches, w2, bias=bias)
        ctx.save_for_backward(*([patches] if ctx.needs_input_grad[1] else []))
        ctx.w_shape, ctx.has_bias = weight.shape, bias is not None
        return y.view(B, gh * gw, N)

    @staticmethod
    def backward(ctx, dy):
        N = ctx.w_shape[0]
        dy2 = nat.dense(dy.reshape(-1, N))
        dw = db = None
        again = torch.is_grad_enabled() and dy.requires_grad  # the gradients are linear in dy and may be differentiated once more
        if ctx.needs_input_grad[1]:
            (patches,) = ctx.saved_tensors
            K = ctx.w_shape[1] * ctx.w_shape[2] * ctx.w_shape[3]
            dw = dy2.t() @ patches if again else gemm(dy2, patches, a_mn_major=True, b_mn_major=True)
            dw = dw[:, :K].reshape(ctx.w_shape)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy2.sum(0) if again else colsum(dy2)
        return None, dw, db


def _patchify(x, out, B, C, gh, gw, ph, pw):
    s = x.stride()
    sb, sc, sh = (s[0], s[1], s[2]) if x.dim() == 4 else (s[0], 0, 0)
    nat.check(nat.lib().csb_patchify(x.data_ptr(), out.data_ptr(), sb, sc, sh, B, C, gh, gw, ph, pw, out.shape[1],
                                     int(x.data_ptr() % 4 == 0 and sb % 2 == 0 and sc % 2 == 0 and sh % 2 == 0 and pw % 2 == 0), nat.stream()),
              "csb_patchify")


_FORWARD, _CONV_FORWARD, _CONV2D = nn.Conv2d.forward, nn.Conv2d._conv_forward, F.conv2d


def _observed() -> bool:
    """Whether something between the caller and the kernels is to see the operators: a transform, a mode, a tracer, a replaced conv2d."""
    return (forward_ad._current_level >= 0 or torch._C._functorch.peek_interpreter_stack() is not None or torch._C._len_torch_dispatch_stack() > 0
            or (torch._C._len_torch_function_stack() > 0
                and not all(isinstance(m, DeviceContext) for m in torch.overrides._get_current_function_mode_stack()))
            or torch.compiler.is_compiling() or torch.jit.is_tracing()
            or F.conv2d is not _CONV2D or nn.Conv2d.forward is not _FORWARD or nn.Conv2d._conv_forward is not _CONV_FORWARD)


def _plain(conv: nn.Module, x: torch.Tensor) -> bool:
    if type(conv) is not nn.Conv2d or "forward" in vars(conv) or "_conv_forward" in vars(conv):
        return False
    w, b = conv.weight, conv.bias
    return (all(type(t) in (torch.Tensor, nn.Parameter) for t in ((x, w) if b is None else (x, w, b)))
            and x.is_cuda and w.device == x.device and x.dtype == w.dtype == torch.bfloat16 and not nat.LIBRARY_MODE
            and x.dim() == 4 and x.shape[1] == w.shape[1] and conv.stride == conv.kernel_size and conv.padding == (0, 0)
            and conv.dilation == (1, 1) and conv.groups == 1 and x.shape[2] >= w.shape[2] and x.shape[3] >= w.shape[3] and x.shape[0] > 0
            and w.shape[0] % 8 == 0 and (b is None or b.dtype == torch.bfloat16)
            and not (torch.is_grad_enabled() and x.requires_grad) and not torch.is_autocast_enabled()
            and not (conv._forward_hooks or conv._forward_pre_hooks or conv._backward_hooks or conv._backward_pre_hooks)
            and not nn.modules.module._has_any_global_hook() and not _observed())


def patch_embed(conv: nn.Conv2d, pixels: torch.Tensor) -> torch.Tensor:
    if _plain(conv, pixels):
        return _PatchEmbedFn.apply(pixels, conv.weight, conv.bias)
    return conv(pixels).flatten(2).transpose(1, 2)
