"""Patch embedding as patches x weight against the convolution in 64 bits, and what is left to the module."""

import pytest
import torch
import torch.nn as nn

from cornstarch_b200.ops import _native as nat
from cornstarch_b200.ops.patch import patch_embed

BF16 = torch.bfloat16


def _conv(C, N, p, bias, device="cuda"):
    torch.manual_seed(C + N + p)
    return nn.Conv2d(C, N, p, p, bias=bias).to(device=device, dtype=BF16)


def _pixels(B, C, H, W, form):
    g = torch.Generator(device="cuda").manual_seed(H + W)
    big = torch.randn(B, C, H + 2, W + 3, generator=g, device="cuda").to(BF16)
    return {"plain": big[..., :H, :W].contiguous(), "odd offset": big[:, :, 1 : H + 1, 1 : W + 1], "even offset": big[:, :, 2 : H + 2, 2 : W + 2],
            "channels last": big[..., :H, :W].contiguous(memory_format=torch.channels_last)}[form]


# patches of 588 (padded to 592), 25 (to 32, odd rows), 768 elements; pixels left over at the right and bottom; one patch
@pytest.mark.gpu
@pytest.mark.parametrize("B,C,H,W,p,N", [(1, 3, 384, 384, 14, 72), (2, 3, 45, 31, 14, 72), (3, 1, 20, 24, 5, 8), (2, 3, 32, 48, 16, 264), (1, 3, 14, 14, 14, 8)])
@pytest.mark.parametrize("form", ["plain", "odd offset", "even offset", "channels last"])
@pytest.mark.parametrize("bias", [False, True])
def test_patch_embed(B, C, H, W, p, N, form, bias):
    conv, x = _conv(C, N, p, bias), _pixels(B, C, H, W, form)
    before = nat.launch_count
    y = patch_embed(conv, x)
    assert nat.launch_count > before
    dy = torch.randn(y.shape, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(BF16)
    y.backward(dy)
    ref = _conv(C, N, p, bias).double()
    yr = ref(x.double()).flatten(2).transpose(1, 2)
    yr.backward(dy.double())
    assert y.shape == yr.shape
    pairs = [(y, yr), (conv.weight.grad, ref.weight.grad)] + ([(conv.bias.grad, ref.bias.grad)] if bias else [])
    for a, r in pairs:  # one rounding to bf16
        assert a.shape == r.shape and (a.double() - r).norm() <= 2.0**-8 * r.norm()


@pytest.mark.gpu
def test_what_is_left_to_the_module():
    conv, x = _conv(3, 16, 14, True), _pixels(1, 3, 28, 28, "plain")
    want = conv(x).flatten(2).transpose(1, 2)

    def launches(c, t):
        before = nat.launch_count
        y = patch_embed(c, t)
        assert (y.double() - want.double()).norm() <= 2.0**-7 * want.double().norm()  # two roundings to bf16
        return nat.launch_count - before

    assert launches(conv, x) > 0
    xg = x.clone().requires_grad_()
    assert launches(conv, xg) == 0
    patch_embed(conv, xg).sum().backward()
    assert xg.grad is not None
    seen = []
    handle = conv.register_forward_hook(lambda *a: seen.append(1))
    assert launches(conv, x) == 0 and seen
    handle.remove()
    overlapping = nn.Conv2d(3, 16, 14, 7).to("cuda", BF16)
    assert torch.equal(patch_embed(overlapping, x), overlapping(x).flatten(2).transpose(1, 2))


def test_cpu_path():
    conv, x = _conv(3, 16, 14, True, "cpu"), torch.randn(2, 3, 30, 28).to(BF16)
    assert torch.equal(patch_embed(conv, x), conv(x).flatten(2).transpose(1, 2))
