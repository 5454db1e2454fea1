"""Arguments of the native route that the operators refuse."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(n=64):
    return [torch.randn(1, 2, n, 64, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda").half().requires_grad_() for i in range(3)]


@pytest.mark.parametrize("bad", [dict(philox_seed=1 << 63), dict(philox_offset1=1 << 63), dict(philox_seed="5"), dict(philox_offset1=0.5)])
@pytest.mark.parametrize("p", [0.0, 0.2])
def test_numbers_the_operator_refuses(bad, p):
    from aotriton_b200 import autograd
    with pytest.raises((RuntimeError, TypeError, OverflowError)):
        autograd.scaled_dot_product_attention(*_qkv(), dropout_p=p, **bad)
