"""The native route's backward where the pass is not the ordinary one that the forward was: a batch of gradients, a mode around the
backward alone, saved-tensor hooks that change what is not part of the saved data; and arguments the operators refuse."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


def _qkv(n=64):
    return [torch.randn(1, 2, n, 64, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda").half().requires_grad_() for i in range(3)]


def test_a_batch_of_gradients():
    from aotriton_b200 import autograd
    ins = _qkv()
    do = torch.randn(3, 1, 2, 64, 64, device="cuda").half()
    out = autograd.scaled_dot_product_attention(*ins, dropout_p=0.2)
    want = [torch.autograd.grad(out, ins, g, retain_graph=True) for g in do]
    for a, w in zip(torch.autograd.grad(out, ins, do, is_grads_batched=True, retain_graph=True), zip(*want)):
        assert torch.equal(a, torch.stack(w))
    with pytest.raises(RuntimeError):      # the Function has no rule for it
        torch.autograd.grad(autograd.attention(*ins), ins, do, is_grads_batched=True)
    for a, w in zip(torch.autograd.grad(out, ins, do[0]), want[0]):
        assert torch.equal(a, w)


class _Names(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("kind", ["sdpa", "sdpa_dropout", "attention", "attention_dropout", "packed"])
def test_a_mode_around_the_backward_alone(kind):
    from aotriton_b200 import autograd
    ins = _qkv(100)
    p = 0.2 if "dropout" in kind else 0.0
    cu = torch.tensor([0, 30, 100], dtype=torch.int32, device="cuda")
    call = {"sdpa": lambda: autograd.scaled_dot_product_attention(*ins, dropout_p=p, is_causal=True), "packed": lambda: autograd.varlen_attention(
        *ins, cu, cu, 70, 70, causal=True, dropout_p=0.1), "attention": lambda: autograd.attention(*ins, causal=(20, 3), dropout_p=p)}[kind.split("_")[0]]
    want = torch.autograd.grad(call().sum(), ins)
    out = call().sum()
    mode = _Names()
    mode.seen = []
    with mode:
        got = torch.autograd.grad(out, ins)
    if "sdpa" in kind:
        assert "aotriton_b200.attn_bwd.default" in mode.seen
    else:      # the Function's gradients and scratch
        assert sum("aten.empty_like" in s for s in mode.seen) >= 4
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_saved_tensor_hooks_do_not_see_the_seed():
    from aotriton_b200 import autograd
    ins = _qkv(200)
    want = torch.autograd.grad(autograd.attention(*ins, dropout_p=0.3).sum(), ins)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.dtype), t)[1], lambda t: t if t.is_floating_point() else t + 1):
        out = autograd.attention(*ins, dropout_p=0.3)
    assert seen == [torch.float16] * 4 + [torch.float32]
    for a, b in zip(torch.autograd.grad(out.sum(), ins), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("bad", [dict(philox_seed=1 << 63), dict(philox_offset1=1 << 63), dict(philox_seed="5"), dict(philox_offset1=0.5)])
@pytest.mark.parametrize("p", [0.0, 0.2])
def test_numbers_the_operator_refuses(bad, p):
    from aotriton_b200 import autograd
    with pytest.raises((RuntimeError, TypeError, OverflowError)):
        autograd.scaled_dot_product_attention(*_qkv(), dropout_p=p, **bad)
