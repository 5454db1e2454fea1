"""General kernels: rows that see nothing near a non-finite token are not touched by it.

A masked pair weighs zero, and zero times a non-finite value is not zero, so the kernels only contract over tokens
that some nearby row sees.  "Nearby" is 16 aligned rows against 16 aligned tokens: where no pair of such a tile is
unmasked, results equal those of the run without the non-finite token, bit for bit.
"""
import pytest
import torch

from oracle import attention as A

pytestmark = pytest.mark.gpu
TL, BR = A.TOP_LEFT, A.BOTTOM_RIGHT


def _tiles(mask):
    """True where some pair of the 16 x 16 tile around (m, n) is unmasked."""
    sq, sk = mask.shape
    m = torch.zeros(sq + -sq % 16, sk + -sk % 16, dtype=torch.bool)
    m[:sq, :sk] = mask
    t = m.view(m.shape[0] // 16, 16, -1, 16).any(3).any(1)
    return t.repeat_interleave(16, 0).repeat_interleave(16, 1)[:sq, :sk]


@pytest.mark.parametrize("poison", [float("nan"), float("inf")])
@pytest.mark.parametrize("D", [64, 100, 160])
@pytest.mark.parametrize("Sq,Sk,causal", [(90, 90, (3, TL, TL)), (70, 130, (3, BR, BR)), (150, 150, (3, 20, 5))])
def test_masked_tokens_stay_out(Sq, Sk, causal, D, poison):
    from aotriton_b200 import cabi
    g = torch.Generator(device="cuda").manual_seed(Sq)
    mk = lambda h, s: torch.randn(1, h, s, D, generator=g, device="cuda")
    q, do, k, v = mk(2, Sq), mk(2, Sq), mk(1, Sk), mk(1, Sk)
    kw = dict(sm_scale=D ** -0.5, causal_type=causal[0], window_left=causal[1], window_right=causal[2])
    near = _tiles(A.window_mask(Sq, Sk, *causal))

    def run(q, k, v, do):
        out, lse = torch.empty_like(q), torch.empty(2, Sq, device="cuda")
        delta = torch.empty_like(lse)
        dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
        assert cabi.attn_fwd(q, k, v, out, lse, **kw) == 0 and cabi.lib().ab200_last_fwd_family() == 1
        assert cabi.attn_bwd(q, k, v, out, do, dq, dk, dv, lse, delta, **kw) == 0 and cabi.lib().ab200_last_bwd_family() == 1
        return [t.cpu() for t in (out, dq, dk, dv)]

    clean = run(q, k, v, do)
    for n in (0, 21, Sk // 2, Sk - 1):
        kp, vp = k.clone(), v.clone()
        kp[:, :, n] = vp[:, :, n] = poison
        got = run(q, kp, vp, do)
        rows = ~near[:, n]
        for a, b in zip(got[:2], clean[:2]):
            assert torch.equal(a[:, :, rows], b[:, :, rows]), f"key {n}"
    for m in (0, 21, Sq // 2, Sq - 1):
        qp, dop = q.clone(), do.clone()
        qp[:, :, m] = dop[:, :, m] = poison
        got = run(qp, k, v, dop)
        keys = ~near[m]
        for a, b in zip(got[2:], clean[2:]):
            assert torch.equal(a[:, :, keys], b[:, :, keys]), f"query {m}"
