"""Patch embedding as patches x weight against the convolution in 64 bits, and what is left to the module."""

import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

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


class _Sub(torch.Tensor):
    pass


def _own_forward(conv, x):
    conv.forward = lambda t: nn.Conv2d.forward(conv, t) * 2
    return patch_embed(conv, x), 2 * _module(conv, x)


def _own_class_forward(conv, x):
    with pytest.MonkeyPatch.context() as m:
        m.setattr(nn.Conv2d, "forward", lambda self, t: self._conv_forward(t, self.weight, self.bias) * 2)
        return patch_embed(conv, x), 2 * _module(conv, x)


def _subclass_weight(conv, x):
    conv.weight = nn.Parameter(conv.weight.detach().as_subclass(_Sub))
    y = patch_embed(conv, x)
    assert isinstance(y, _Sub)
    return y.as_subclass(torch.Tensor), _module(conv, x).as_subclass(torch.Tensor)


def _forward_mode(conv, x):
    from torch.autograd import forward_ad

    t = torch.ones_like(conv.weight)
    weight = conv.weight.detach()
    del conv.weight  # a dual tensor in its place
    with torch.no_grad(), forward_ad.dual_level():
        conv.weight = forward_ad.make_dual(weight, t)
        y = forward_ad.unpack_dual(patch_embed(conv, x))
        assert y.tangent is not None
        return y.tangent, F.conv2d(x, t, None, conv.stride).flatten(2).transpose(1, 2)


def _vmap(conv, x):
    xs = torch.stack([x, x + 1])
    return torch.vmap(lambda t: patch_embed(conv, t))(xs), torch.stack([_module(conv, t) for t in xs])


def _timer(conv, x):
    from cornstarch_b200.testing.timer import TimerContextManager

    with TimerContextManager("torch.nn.functional.conv2d") as t:
        y = patch_embed(conv, x)
    assert len(t.get_elapsed_times()["torch.nn.functional.conv2d"]) == 1
    return y, _module(conv, x)


def _dispatch_mode(conv, x):
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with Mode():
        y = patch_embed(conv, x)
    assert torch.ops.aten.convolution.default in seen
    return y, _module(conv, x)


def _module(conv, x):
    with torch.no_grad():
        return F.conv2d(x, conv.weight, conv.bias, conv.stride).flatten(2).transpose(1, 2)


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("case", [_own_forward, _own_class_forward, _subclass_weight, _forward_mode, _vmap, _timer, _dispatch_mode])
def test_a_module_that_something_else_changes_or_watches(case, device):
    conv, x = _conv(3, 16, 14, True, device), torch.randn(2, 3, 28, 42, generator=torch.Generator().manual_seed(0)).to(device, BF16)
    got, want = case(conv, x)
    assert torch.equal(got.detach(), want.detach())


@pytest.mark.gpu
def test_gradients_of_the_gradients():
    conv, x = _conv(3, 16, 14, True), _pixels(2, 3, 28, 42, "plain")
    v, u = torch.randn_like(conv.weight), torch.randn_like(conv.bias)
    out = []
    for embed in (lambda: patch_embed(conv, x), lambda: conv(x).flatten(2).transpose(1, 2)):
        y = embed().float()
        dw, db = torch.autograd.grad((y**3).sum(), [conv.weight, conv.bias], create_graph=True)
        out.append([dw, db, *torch.autograd.grad([dw, db], [conv.weight, conv.bias], [v, u])])
    for a, b in zip(*out):  # bf16 activations, cubed: two or three roundings on either side
        assert (a.double() - b.double()).norm() <= 2.0**-5 * b.double().norm()


@pytest.mark.gpu
def test_a_gradient_off_the_16_byte_grid():
    conv, x = _conv(3, 16, 14, True), _pixels(2, 3, 28, 42, "plain")
    dy = torch.randn(12 * 16 + 1, device="cuda").to(BF16)[1:].view(2, 6, 16)
    grads = []
    for d in (dy, dy.clone()):
        grads.append(torch.autograd.grad(patch_embed(conv, x), [conv.weight, conv.bias], d))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.gpu
@pytest.mark.parametrize("frozen", [False, True])
def test_patches_are_kept_for_the_weight_only(frozen):
    conv, x = _conv(3, 16, 14, True), _pixels(2, 3, 28, 42, "plain")
    conv.weight.requires_grad_(not frozen)
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t.shape) or t, lambda t: t):
        y = patch_embed(conv, x)
    assert kept == ([] if frozen else [(12, 592)])
    y.sum().backward()
    assert torch.equal(conv.bias.grad, torch.full_like(conv.bias, 12)) and (conv.weight.grad is None) == frozen


def test_cpu_path():
    conv, x = _conv(3, 16, 14, True, "cpu"), torch.randn(2, 3, 30, 28).to(BF16)
    assert torch.equal(patch_embed(conv, x), conv(x).flatten(2).transpose(1, 2))
