"""The register-tiled kernels (fp32; 16-bit rows the tensor cores do not take) at the edges of their tiles: 32 rows, blocks of 64
columns (32 above head dim 64), the forward's blocks dealt to two groups of warps.

Against the same formulas in 64 bits.  fp32: sums of up to 300 products of N(0, 1) values, each rounded to 2^-24, and exponentials
good to 2^-22; 1e-4 (atol = rtol) is the suite's bound for fp32 (test_gpu_parity.py).  fp16 likewise 1e-2.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
ATOL = {torch.float32: 1e-4, torch.float16: 1e-2}


def _reference(q, k, v, do, mask):
    q, k, v, do = (t.double() for t in (q, k, v, do))
    g = q.shape[1] // k.shape[1]
    k, v = (t.repeat_interleave(g, 1) for t in (k, v))
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    s = q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5
    if mask is not None:
        s = s.masked_fill(~mask, float("-inf"))
    out = s.softmax(-1).nan_to_num(0.0) @ v
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), do)
    fold = lambda t: t.unflatten(1, (-1, g)).sum(2)
    return out.detach(), dq, fold(dk), fold(dv)


@pytest.mark.parametrize("dt,D", [(torch.float32, 64), (torch.float32, 128), (torch.float32, 80), (torch.float32, 33),
                                  (torch.float16, 60), (torch.float16, 100)])
@pytest.mark.parametrize("sq,sk", [(1, 1), (31, 33), (32, 64), (33, 65), (64, 128), (65, 129), (97, 31), (130, 193), (300, 257)])
@pytest.mark.parametrize("causal", [False, True])
def test_edges(sq, sk, causal, dt, D):
    from aotriton_b200 import autograd, cabi
    if causal and sq > sk:
        pytest.skip("rows without a key: covered elsewhere")
    g = torch.Generator(device="cuda").manual_seed(sq * 1000 + sk)
    mk = lambda h, n: torch.randn(2, h, n, D, generator=g, device="cuda").to(dt)
    q, k, v, do = mk(4, sq), mk(2, sk), mk(2, sk), mk(4, sq)
    mask = torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril() if causal else None
    ref = _reference(q, k, v, do, mask)
    ins = [t.clone().requires_grad_() for t in (q, k, v)]
    out = autograd.attention(*ins, causal=causal)
    got = (out.detach(),) + torch.autograd.grad(out, ins, do)
    assert cabi.lib().ab200_last_fwd_family() == 1
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, ref):
        torch.testing.assert_close(a.double(), b, atol=ATOL[dt], rtol=ATOL[dt], msg=lambda m: f"{name}: {m}")


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads", [1, 24])
def test_split_row_tiles(heads, D):
    """Few row tiles: two CTAs share the blocks of one (1 x 1024 rows); many (24 heads): one CTA each.  Grouped heads, so that the
    blocks run over several of them."""
    from aotriton_b200 import autograd
    g = torch.Generator(device="cuda").manual_seed(heads)
    mk = lambda h: torch.randn(1, h, 1024, D, generator=g, device="cuda")
    q, k, v, do = mk(2 * heads), mk(heads), mk(heads), mk(2 * heads)
    ref = _reference(q, k, v, do, torch.ones(1024, 1024, dtype=torch.bool, device="cuda").tril())
    ins = [t.clone().requires_grad_() for t in (q, k, v)]
    out = autograd.attention(*ins, causal=True)
    for name, a, b in zip(("out", "dq", "dk", "dv"), (out.detach(),) + torch.autograd.grad(out, ins, do), ref):
        torch.testing.assert_close(a.double(), b, atol=1e-4, rtol=1e-4, msg=lambda m: f"{name}: {m}")


@pytest.mark.parametrize("D", [32, 64, 100, 128])
@pytest.mark.parametrize("rows", [1, 5, 127, 500, 2000])
def test_fp32_delta(rows, D):
    """delta = rowsum(O * dO): the 16-byte path and, from rows that are not aligned to it, the scalar one."""
    from aotriton_b200 import autograd
    g = torch.Generator(device="cuda").manual_seed(rows)
    mk = lambda: torch.randn(1, 2, rows, D + 1, generator=g, device="cuda")
    base = [mk() for _ in range(4)]
    def run(ts):
        ins = [t.requires_grad_() for t in ts[:3]]
        out = autograd.attention(*ins, causal=True)
        return torch.autograd.grad(out, ins, ts[3])
    aligned = run([t[..., :D].contiguous() for t in base])
    loose = run([t[..., :D].detach() for t in base])
    for a, b in zip(aligned, loose):
        torch.testing.assert_close(a, b, atol=1e-4, rtol=1e-4)
