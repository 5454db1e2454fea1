"""dK/dV and dQ of the general kernels in one launch, against the same kernels in separate stage calls (equal
bit for bit), and the calls that must not take it: dQ in the place of an input."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hk,Sq,Sk,D,bias", [
    (1, 1, 1, 1, 1, 8, False), (2, 4, 2, 33, 95, 64, True), (1, 2, 2, 200, 31, 64, False), (1, 6, 2, 97, 64, 100, True),
    (1, 2, 1, 40, 50, 160, False),      # head dims above 128: two launches
])
@pytest.mark.parametrize("in_place", [False, True])
def test_equal_to_separate_stages(B, Hq, Hk, Sq, Sk, D, bias, in_place):
    from aotriton_b200 import cabi
    g = torch.Generator(device="cuda").manual_seed(Sq + D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, do, k, v = mk(B, Hq, Sq, D), mk(B, Hq, Sq, D), mk(B, Hk, Sk, D), mk(B, Hk, Sk, D)
    b = mk(B, Hq, Sq, Sk) if bias else None
    kw = dict(sm_scale=D ** -0.5, bias=b)
    out, lse = torch.empty_like(q), torch.empty(B * Hq, Sq, device="cuda")
    assert cabi.attn_fwd(q, k, v, out, lse, **kw) == 0

    def backward(dq, do, *stages):
        dk, dv, db = torch.full_like(k, float("nan")), torch.full_like(v, float("nan")), torch.full_like(b, float("nan")) if bias else None
        delta = torch.empty_like(lse)
        n0 = cabi.lib().ab200_launch_count()
        for stage in stages:
            assert cabi.attn_bwd(q, k, v, out, do, dq, dk, dv, lse, delta, dbias=db, stage=stage, **kw) == 0
        assert cabi.lib().ab200_last_bwd_family() == 1
        one = stages == ("all",) and D <= 128 and dq.data_ptr() != do.data_ptr()
        assert cabi.lib().ab200_launch_count() - n0 == (2 if one else 3)
        return [dq, dk, dv] + ([db] if bias else [])

    want = backward(torch.full_like(q, float("nan")), do, "preprocess", "dkdv", "dq")
    mine = do.clone()
    got = backward(mine if in_place else torch.full_like(q, float("nan")), mine, "all")
    for x, y in zip(got, want):
        assert not torch.isnan(y).any() and torch.equal(x, y)
