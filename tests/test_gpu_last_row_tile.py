"""Rows of the last tile beyond a sequence's end take the last row's mask bounds, so they run through the kernels with whatever
lies behind the sequence.  Nothing of that may reach a stored row: results are bit for bit those of a run whose
neighbouring sequence holds ordinary values.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("poison", [3.0e4, float("inf"), float("nan")])
@pytest.mark.parametrize("D", [64, 128, 192])
@pytest.mark.parametrize("n,causal", [(1, True), (57, True), (185, True), (129, False), (300, (40, 0)), (383, False)])
def test_neighbour_stays_out(n, causal, D, poison):
    from aotriton_b200 import autograd, cabi
    lens, Hq, Hk = [n, 200], 4, 2
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda h: torch.randn(1, sum(lens), h, D, generator=g, device="cuda", dtype=torch.bfloat16).transpose(1, 2)
    q, k, v, do = mk(Hq), mk(Hk), mk(Hk), mk(Hq)
    cu = torch.tensor([0, n, sum(lens)], dtype=torch.int32, device="cuda")

    def run(ts, p):
        q, k, v, do = ts
        q, k, v = (t.clone().requires_grad_() for t in (q, k, v))
        out = autograd.varlen_attention(q, k, v, cu, cu, max(lens), max(lens), causal=causal, dropout_p=p)
        return [t[:, :, :n].clone() for t in (out.detach(),) + torch.autograd.grad(out, (q, k, v), do)]

    poisoned = [t.clone() for t in (q, k, v, do)]
    for t in poisoned:
        t[:, :, n:] = poison
    for p in (0.0, 0.1):
        for name, a, b in zip(("out", "dq", "dk", "dv"), run((q, k, v, do), p), run(poisoned, p)):
            assert torch.isfinite(a).all() and torch.equal(a, b), f"{name}, dropout {p}"
    assert cabi.lib().ab200_kernel_status(0) == 0
