"""Dropout keep bits that pass from the dK/dV kernel to the dQ kernel through dBias, where it is written: the rule on the CPU, and
on the GPU the gradients of one call against those of separate stage calls, where every kernel draws its own bits -- the same
arithmetic, so equal bit for bit, dBias included.
"""
import ctypes as C

import pytest
import torch

TL, BR = -2147483647, -2147483646


def _tiles(sq=300, sk=1100, d=72, bias=None, dbias=None, p=0.1, alias=None):
    from aotriton_b200 import cabi
    mk = lambda h, n: torch.empty(2, h, n, d, dtype=torch.float16)
    q, k, v, out, do, dq, dk, dv = mk(4, sq), mk(2, sk), mk(2, sk), mk(4, sq), mk(4, sq), mk(4, sq), mk(2, sk), mk(2, sk)
    lse = torch.empty(8, sq)
    dbias = torch.empty(2, 4, sq, sk, dtype=torch.float16) if dbias is None else dbias
    bias = torch.empty_like(dbias) if bias is None else bias
    if alias == "bias":
        bias = dbias
    a = cabi.make_bwd_args(q, k, v, out, do, dq, dk, dv, lse, torch.empty_like(lse), bias=bias, dbias=dbias, sm_scale=1.0, dropout_p=p)
    return cabi.lib().ab200_debug_keep_tiles(C.byref(a))


def test_rule():
    mk = lambda *s: torch.empty(*s, dtype=torch.float16)
    in_dq = 32                                              # head dim 72: 1024 keys
    assert _tiles(sk=1104) == 34                            # whole tiles only
    assert _tiles(sk=1088) == 34 and _tiles(sk=2048) == 64 and _tiles(sk=24) == 0
    assert _tiles(sk=1104, d=56) == 34                      # (no room in dQ at this head dim)
    assert _tiles(sk=1104, p=0.0) == 0
    assert _tiles(sk=1100) == in_dq                         # rows off a 16-byte boundary
    assert _tiles(sk=1104, dbias=mk(2, 4, 300, 1112)[..., :1104]) == 34
    assert _tiles(sk=1104, dbias=mk(2, 1, 300, 1104).expand(2, 4, 300, 1104), bias=mk(2, 4, 300, 1104)) == in_dq
    assert _tiles(sk=1104, alias="bias") == in_dq           # dBias in the bias' place: it is still read


CASES = [
    # B, Hq, Hk, Sq, Sk, D, causal
    (1, 2, 2, 32, 32, 64, (0, 0, 0)),
    (1, 2, 1, 31, 400, 64, (0, 0, 0)),              # no whole row group
    (1, 4, 2, 391, 1104, 72, (0, 0, 0)),            # partial tile at the end, keys beyond dQ's room
    (2, 2, 2, 129, 2200, 128, (3, BR, BR)),
    (1, 4, 1, 640, 640, 128, (3, 130, 65)),         # tiles masked on both sides
    (1, 2, 2, 200, 96, 56, (3, TL, TL)),
    (1, 2, 1, 257, 328, 256, (0, 0, 0)),            # wide: dK from dBias behind the dQ kernel
    (1, 2, 2, 320, 504, 192, (3, TL, TL)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", CASES)
def test_equal_to_separate_stages(case, dt):
    from aotriton_b200 import cabi
    B, Hq, Hk, Sq, Sk, D, (ct, wl, wr) = case
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk + D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    q, do, k, v, bias = mk(B, Hq, Sq, D), mk(B, Hq, Sq, D), mk(B, Hk, Sk, D), mk(B, Hk, Sk, D), mk(B, Hq, Sq, Sk)
    kw = dict(sm_scale=D ** -0.5, causal_type=ct, window_left=wl, window_right=wr, dropout_p=0.3,
              philox_seed=torch.tensor([0x5ca1ab1e12345], dtype=torch.uint64, device="cuda"),
              philox_offset1=torch.tensor([0xfffffff0], dtype=torch.uint64, device="cuda"), philox_offset2=7)
    out, lse = torch.empty_like(q), torch.empty(B * Hq, Sq, device="cuda")
    assert cabi.attn_fwd(q, k, v, out, lse, bias=bias, **kw) == 0

    def backward(*stages):
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v, bias)]
        delta = torch.empty_like(lse)
        for stage in stages:
            assert cabi.attn_bwd(q, k, v, out, do, *grads[:3], lse, delta, bias=bias, dbias=grads[3], stage=stage, **kw) == 0
        return grads

    got, want = backward("all"), backward("preprocess", "dkdv", "dq")
    assert cabi.lib().ab200_kernel_status(0) == 0
    for name, a, b in zip(("dq", "dk", "dv", "dbias"), got, want):
        assert not torch.isnan(b.float()).any()
        if D > 128 and name == "dk":      # (from dBias in the one call, by a kernel of its own in stages)
            torch.testing.assert_close(a, b, atol=2e-2, rtol=2e-2)
        else:
            assert torch.equal(a, b), f"{name}: {float((a.float() - b.float()).abs().max())}"
