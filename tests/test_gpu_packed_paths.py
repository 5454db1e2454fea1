"""Two everyday uses of packed sequences through the Python entry point, each sequence against the oracle: a training
step without dropout, and decoding (one query per sequence against its cached keys).

Tolerances: those of test_gpu_parity.py (atol = rtol = 2e-2 bf16, 1e-2 fp16).
"""
import numpy as np
import pytest
import torch

from oracle import attention as A
from _util import ATOL, close

pytestmark = pytest.mark.gpu


def _packed(lens, h, d, dt, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(1, sum(lens), h, d, generator=g).to(dt).transpose(1, 2)


def _cu(lens):
    return [0] + [int(x) for x in np.cumsum(lens)]


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,causal", [(128, True), (128, False), (64, True), (192, True)])
def test_training_step(D, causal, dt):
    from aotriton_b200 import autograd
    lens, Hq, Hk = [1, 64, 129, 0, 300, 515, 128], 4, 2
    q, do, k, v = (_packed(lens, h, D, dt, i) for i, h in enumerate((Hq, Hq, Hk, Hk)))
    qd, kd, vd = (t.cuda().requires_grad_() for t in (q, k, v))
    cu = _cu(lens)
    cud = torch.tensor(cu, dtype=torch.int32, device="cuda")
    out = autograd.varlen_attention(qd, kd, vd, cud, cud, max(lens), max(lens), causal=causal)
    got = [out.detach()] + list(torch.autograd.grad(out, (qd, kd, vd), do.cuda()))
    for a, b in zip(cu, cu[1:]):
        if a == b:
            continue
        s = slice(a, b)
        mask = A.window_mask(b - a, b - a, 3, A.TOP_LEFT, A.TOP_LEFT) if causal else None
        ref = A.attention(q[:, :, s], k[:, :, s], v[:, :, s], sm_scale=D ** -0.5, mask=mask, dout=do[:, :, s])
        for name, t in zip(("out", "dq", "dk", "dv"), got):
            ok, err = close(t[:, :, s].float().cpu(), getattr(ref, name), ATOL[dt])
            assert ok, f"{name} of tokens {a}..{b}: max err {err}"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Hq,Hk,D,count", [(32, 8, 128, 9), (8, 8, 64, 40), (16, 2, 128, 3)])
def test_decoding_step(Hq, Hk, D, count, dt):
    from aotriton_b200 import autograd, cabi, flash
    rng = np.random.default_rng(count)
    lens = [int(x) for x in rng.integers(1, 3000, count)]
    lens[0], lens[-1] = 1, 2999
    q, k, v = _packed([1] * count, Hq, D, dt, 1), _packed(lens, Hk, D, dt, 2), _packed(lens, Hk, D, dt, 3)
    cu = _cu(lens)
    t32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    with torch.no_grad():
        out = autograd.varlen_attention(q.cuda(), k.cuda(), v.cuda(), t32(list(range(count + 1))), t32(cu), 1, max(lens),
                                        causal=flash.CausalType.BOTTOM_RIGHT)
    assert cabi.lib().ab200_last_fwd_family() == 2
    for z, (a, b) in enumerate(zip(cu, cu[1:])):
        ref = A.attention(q[:, :, z:z + 1], k[:, :, a:b], v[:, :, a:b], sm_scale=D ** -0.5)
        ok, err = close(out[:, :, z:z + 1].float().cpu(), ref.out, ATOL[dt])
        assert ok, f"sequence {z} of {b - a} keys: max err {err}"
    assert cabi.lib().ab200_kernel_status(0) == 0
