"""dropout_p = 1, which is accepted: nothing is kept, dV is zero and so is every score's gradient but for delta's part (zero here), on both
kernel families."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,D,family", [(torch.float16, 64, 2), (torch.bfloat16, 128, 2), (torch.float16, 256, 2), (torch.float16, 60, 1), (torch.float32, 64, 1)])
@pytest.mark.parametrize("bias", [False, True])
def test_nothing_is_kept(dt, D, family, bias):
    from aotriton_b200 import cabi
    g = torch.Generator(device="cuda").manual_seed(D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    q, k, v, do = (mk(1, 2, 100, D) for _ in range(4))
    b = mk(1, 2, 100, 104)[..., :100] if bias else None
    lse = (q.float() @ k.float().transpose(-1, -2) * 0.1 + (b.float() if bias else 0)).logsumexp(-1)[0]
    nan = lambda t: torch.full_like(t, float("nan"))
    dq, dk, dv, db = nan(q), nan(k), nan(v), nan(b) if bias else None
    # (out = 0, so that delta is: the forward's own output is 0 * infinity)
    assert cabi.attn_bwd(q, k, v, torch.zeros_like(q), do, dq, dk, dv, lse, torch.empty_like(lse), bias=b, dbias=db, sm_scale=0.1, dropout_p=1.0,
                         philox_seed=torch.tensor([3], dtype=torch.uint64, device="cuda")) == 0
    assert cabi.lib().ab200_last_bwd_family() == family
    for t in (dq, dk, dv) + ((db,) if bias else ()):
        assert (t == 0).all()
