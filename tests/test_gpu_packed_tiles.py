"""Forward of token-packed batches, whose grid counts the row tiles of all sequences: empty and one-token
sequences, lengths around a tile, more sequences than a warp looks at in one step, more than the search takes.

Each sequence must come out as the dense call on it alone does (the same kernel on the same blocks in the same
order): bit for bit.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,causal", [(64, False), (128, True), (256, True)])
@pytest.mark.parametrize("lens", [
    [300], [0, 17], [256, 0, 0, 257, 1, 255, 512],
    [int(x) for x in np.random.RandomState(1).randint(0, 600, 32)],
    [int(x) for x in np.random.RandomState(2).randint(0, 300, 45)],
    [int(x) for x in np.random.RandomState(3).randint(17, 60, 130)],
])
def test_equal_to_dense_calls(lens, D, causal):
    from aotriton_b200 import cabi
    dt, Hq, Hk, total = torch.bfloat16, 4, 2, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(total)
    q, k, v = (torch.randn(1, total, h, D, generator=g, device="cuda").to(dt).transpose(1, 2) for h in (Hq, Hk, Hk))
    starts = [0] + [int(x) for x in np.cumsum(lens)]
    cu = torch.tensor(starts, dtype=torch.int32, device="cuda")
    kw = dict(sm_scale=D ** -0.5)
    if causal:
        kw.update(causal_type=3, window_left=cabi.WINDOW_BOTTOM_RIGHT, window_right=cabi.WINDOW_BOTTOM_RIGHT)
    out, lse = torch.full_like(q, float("nan")), torch.full((Hq, total), float("nan"), device="cuda")
    assert cabi.attn_fwd(q, k, v, out, lse, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(lens), max_seqlen_k=max(lens),
                         **kw) == 0
    assert not torch.isnan(out.float()).any() and not torch.isnan(lse).any()
    for a, b in zip(starts, starts[1:]):
        if b - a <= 16:          # (short sequences alone take the split-key kernel, which sums in another order)
            continue
        one, lse1 = torch.empty(1, Hq, b - a, D, dtype=dt, device="cuda"), torch.empty(Hq, b - a, device="cuda")
        assert cabi.attn_fwd(q[:, :, a:b], k[:, :, a:b], v[:, :, a:b], one, lse1, **kw) == 0
        assert torch.equal(out[:, :, a:b], one) and torch.equal(lse[:, a:b], lse1)
    torch.cuda.synchronize()
    assert cabi.lib().ab200_kernel_status(0) == 0
