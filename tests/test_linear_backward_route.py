"""Which linear backward passes go through the one native call, and that every other form gets its gradients on the general
path.  Runs on the CPU: ``gemm`` is its fp32 statement there, and the native library is one that records the calls."""

import pytest
import torch

from cornstarch_b200.ops import _native as nat
from cornstarch_b200.ops import linear as L

BF16 = torch.bfloat16


class _Recorder:
    def __init__(self):
        self.calls = 0

    def csb_colsum_parts(self, rows):
        return rows

    def csb_linear_bwd(self, *args):
        self.calls += 1
        return 0


@pytest.fixture
def lib(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(nat, "lib", lambda: rec)
    monkeypatch.setattr(nat, "status_word", lambda device=None: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(nat, "stream", lambda: 0)
    return rec


def _randn(*shape):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))).to(BF16)


def _layer(x, w, b, dy, main_w=None, main_b=None):
    """Gradients of x, w and b as a program sees them: in ``main_grad`` where there is one."""
    x, w = x.detach().requires_grad_(), w.detach().requires_grad_()
    b = b.detach().requires_grad_() if b is not None else None
    for t, m in ((w, main_w), (b, main_b)):
        if t is not None and m is not None:
            t.main_grad = m
    L._LinearFn.apply(x, 1, None, None, w, b).backward(dy)
    return [x.grad, *(t.main_grad if hasattr(t, "main_grad") else t.grad for t in (w, b) if t is not None)]


def _check(got, x, w, b, dy, base=0.0):
    want = [dy.double() @ w.double(), dy.double().t() @ x.double() + base] + ([dy.double().sum(0) + base] if b is not None else [])
    for a, r in zip(got, want):
        # one rounding to bf16 (2^-9 of the value), two where the result is added to a buffer
        assert (a.double() - r).norm() <= 2.0**-8 * r.norm()


def test_plain_layers_take_the_native_call(lib):
    _layer(_randn(9, 40), _randn(24, 40), _randn(24), _randn(9, 24))
    _layer(_randn(9, 40), _randn(24, 40), None, _randn(9, 24), torch.zeros(24, 40))
    assert lib.calls == 2


@pytest.mark.parametrize("w_dtype,b_dtype", [(torch.float16, None), (torch.float64, None), (torch.float16, torch.float16),
                                             (BF16, torch.float16), (torch.float32, torch.float64)])
def test_buffers_of_other_types_are_not_the_kernels(lib, w_dtype, b_dtype):
    """The kernels write bf16 and fp32.  A buffer of another type goes the general way (where the GEMM refuses it on the GPU) and
    is never taken for bf16."""
    x, w, dy, b = _randn(9, 40), _randn(24, 40), _randn(9, 24), _randn(24) if b_dtype is not None else None
    got = _layer(x, w, b, dy, torch.ones(24, 40, dtype=w_dtype), None if b is None else torch.ones(24, dtype=b_dtype))
    assert lib.calls == 0
    _check(got, x, w, b, dy, base=1.0)


def _misaligned(t):
    """``t`` as a contiguous view four elements into a flat buffer: 8 bytes off the 16-byte grid."""
    flat = torch.zeros(t.numel() + 8, dtype=t.dtype)
    flat[4 : 4 + t.numel()] = t.flatten()
    return flat[4 : 4 + t.numel()].view(t.shape)


def _row_of_wider(t):
    """The one row ``t`` from columns 4.. of a wider row: contiguous, and off the grid."""
    wide = torch.zeros(3, t.shape[1] + 12, dtype=t.dtype)
    wide[0, 4 : 4 + t.shape[1]] = t[0]
    return wide[:1, 4 : 4 + t.shape[1]]


@pytest.mark.parametrize("which", ["x", "dy", "both"])
@pytest.mark.parametrize("form,T", [(_misaligned, 9), (_misaligned, 1), (_row_of_wider, 1)])
@pytest.mark.parametrize("main", [False, True])
def test_operands_off_the_grid_take_the_general_path(lib, which, form, T, main):
    """The TMA loads of the native call need 16-byte aligned rows; the general path repacks such an operand."""
    x, w, dy = _randn(T, 40), _randn(24, 40), _randn(T, 24)
    xs, dys = (form(x) if which != "dy" else x), (form(dy) if which != "x" else dy)
    for t, u in ((xs, x), (dys, dy)):
        assert t.is_contiguous() and torch.equal(t, u)

    class GivesDy(torch.autograd.Function):  # the gradient that reaches the layer is this tensor, not a copy
        @staticmethod
        def forward(ctx, y):
            return y.float().sum()

        @staticmethod
        def backward(ctx, g):
            return dys

    xr, wr = xs.detach().requires_grad_(), w.detach().requires_grad_()
    if main:
        wr.main_grad = torch.zeros(24, 40)
    GivesDy.apply(L._LinearFn.apply(xr, 1, None, None, wr, None)).backward()
    assert lib.calls == 0
    _check([xr.grad, wr.main_grad if main else wr.grad], x, w, None, dy)


def test_gradients_of_several_projections_change_one_by_one(lib):
    """They may lie in one buffer, but a change of one in place is no change of the others: an autograd graph that holds one of
    them stays valid."""
    w, b = _randn(48, 40), _randn(48)
    ws = [t.detach().requires_grad_() for t in torch.split(w, [24, 8, 16])]
    bs = [t.detach().requires_grad_() for t in torch.split(b, [24, 8, 16])]
    x = _randn(9, 40).requires_grad_()
    L._LinearFn.apply(x, 3, None, None, *ws, *bs).backward(_randn(9, 48))
    assert lib.calls == 1
    for ts in (ws, bs):
        with torch.no_grad():
            ts[0].grad.fill_(2.0)
            ts[2].grad.fill_(3.0)
        z = torch.ones_like(ts[0], requires_grad=True)
        loss = (z * ts[0].grad).sum()
        torch.optim.SGD(ts[1:], lr=0.1).zero_grad(set_to_none=False)
        ts[2].grad.mul_(0.5)
        loss.backward()
        assert (z.grad == 2).all() and (ts[0].grad == 2).all() and not ts[1].grad.any() and not ts[2].grad.any()
