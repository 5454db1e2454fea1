"""Where the backward rounds with dropout, on values that are known exactly: one query that sees n keys with equal scores (Q = 0 or
K = 0), so that P = 1 / n, and products with a single term.

  dV = cast(keep ? P / (1 - p) : 0) dO: scaled in fp32 and rounded to 16 bits once.  The values of n and p are such that rounding P
       before it is scaled gives another number, while an error of 1e-5 in P does not.
  dS = P (keep ? dP / (1 - p) : 0  -  delta): with delta = fp32(dP / (1 - p)) a kept score's is exactly zero, if the scaled dP is
       rounded to fp32 before delta is subtracted.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

SEED, OFFSET = 0x5EED, 11


def _setting(dt, d, n, p):
    import numpy as np
    from oracle import philox
    dev = dict(device="cuda", dtype=dt)
    keep = torch.from_numpy(np.array(philox.keep_mask(SEED, OFFSET, 0, 0, 1, 1, n, 1, n, p)[0])).cuda()
    assert 0 < int(keep.sum()) < n
    kw = dict(sm_scale=1.0, dropout_p=p, philox_seed=torch.tensor([SEED], dtype=torch.uint64, device="cuda"), philox_offset2=OFFSET)
    lse = torch.full((1, 1), float(n), device="cuda").log()
    return dev, keep, kw, lse, torch.zeros(1, 1, 1, d, **dev), torch.zeros(1, 1, n, d, **dev)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,p", [(22, 0.2), (24, 0.6)])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_probabilities_are_scaled_before_they_are_rounded(d, bias, n, p, dt):
    from aotriton_b200 import cabi
    dev, keep, kw, lse, q, k = _setting(dt, d, n, p)
    b = torch.zeros(1, 1, 1, n, **dev) if bias else None
    scale = 1 / (1 - torch.tensor(p))
    want, twice = (torch.tensor(1.0 / n) * scale).to(dt), (torch.tensor(1.0 / n).to(dt).float() * scale).to(dt)
    assert want != twice
    do = torch.ones_like(q)
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(k)
    assert cabi.attn_bwd(q, k, torch.zeros_like(k), torch.zeros_like(q), do, dq, dk, dv, lse, torch.zeros_like(lse), stage="dkdv", bias=b, **kw) == 0
    assert cabi.lib().ab200_last_bwd_family() == 2
    assert torch.equal(dv, torch.where(keep, want.cuda(), 0).to(dt).view(1, 1, n, 1).expand_as(dv))


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("stage", ["dkdv", "dq"])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_scaled_dp_is_rounded_before_delta_is_subtracted(d, bias, stage, dt):
    from aotriton_b200 import cabi
    n, p, x = 22, 0.3, 1000.0
    dev, keep, kw, lse, q, k = _setting(dt, d, n, p)
    b = torch.zeros(1, 1, 1, n, **dev) if bias else None
    v, do = torch.zeros_like(k), torch.zeros_like(q)
    v[..., 0], do[..., 0] = x, 1.0
    scale = 1 / (1 - torch.tensor(p))
    delta = (x * scale).cuda().view(1, 1)
    assert float(x * scale) != x * float(scale)      # (a product that is not rounded leaves 5e-5 behind)
    if stage == "dq":
        k[0, 0, range(n), range(n)] = 1.0      # dQ[j] = dS[j]
    else:
        q[..., 0] = 1.0                        # dK[j][0] = dS[j]
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(k)
    assert cabi.attn_bwd(q, k, v, torch.zeros_like(q), do, dq, dk, dv, lse, delta, stage=stage, bias=b, **kw) == 0
    assert cabi.lib().ab200_last_bwd_family() == 2
    ds = dq[0, 0, 0, :n] if stage == "dq" else dk[0, 0, :, 0]
    assert torch.equal(ds[keep], torch.zeros_like(ds[keep]))
    torch.testing.assert_close(ds[~keep].float(), (-delta[0] / n).expand(int((~keep).sum())), atol=0, rtol=2 ** -8)
