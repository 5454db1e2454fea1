"""Arguments of the native route that the operators refuse, and saved-tensor hooks that change what is not part of the saved data."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(n=64):
    return [torch.randn(1, 2, n, 64, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda").half().requires_grad_() for i in range(3)]


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
