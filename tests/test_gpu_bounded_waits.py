"""Bounded waits that run out in the kernels test_gpu_robustness.py does not reach: the split-key forward, where one
CTA of a cluster gives up and its peers meet it at the cluster barriers; the forward with one tile per CTA and dropout,
whose drawing warps then wait for the softmax warps; dK formed from dBias.

One copy is left out with a wait limit of about a million cycles.  The kernel must return, the status word must name
it, further work must be refused until the reset, and the next call must give what an undisturbed one gives.
"""
import pytest
import torch

from _util import randn_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what,drop,lo,hi", [("split keys", 1, 0x5000, 0x6000), ("keep bits", 1, 0x100, 0x1000),
                                             ("dk from dbias", 4, 0x4000, 0x5000)])
def test_runs_out_cleanly(what, drop, lo, hi):
    from aotriton_b200 import cabi
    L = cabi.lib()
    dt = torch.float16
    Hq, Sq, Sk, D = {"split keys": (2, 1, 2048, 128), "keep bits": (1, 640, 640, 256), "dk from dbias": (1, 128, 128, 256)}[what]
    q, k, v, do = (t.cuda() for t in randn_inputs((1, Hq, Sq, D), (1, 1, Sk, D), (1, 1, Sk, D), dt, seed=1))
    out, lse, delta = torch.empty_like(q), torch.empty(Hq, Sq, device="cuda"), torch.empty(Hq, Sq, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    prob = dict(sm_scale=D ** -0.5)
    if what == "keep bits":
        prob.update(dropout_p=0.2, philox_seed=torch.tensor([3], dtype=torch.uint64, device="cuda"),
                    philox_offset1=torch.tensor([1], dtype=torch.uint64, device="cuda"))
    bias = torch.randn(1, Hq, Sq, Sk, device="cuda").to(dt) if what == "dk from dbias" else None
    db = torch.empty_like(bias) if bias is not None else None
    backward = bias is not None

    def call():
        if backward:
            return cabi.attn_bwd(q, k, v, out, do, *grads, lse, delta, bias=bias, dbias=db, **prob)
        return cabi.attn_fwd(q, k, v, out, lse, bias=bias, **prob)

    stream = torch.cuda.current_stream().cuda_stream
    assert L.ab200_kernel_status(1) == 0
    assert cabi.attn_fwd(q, k, v, out, lse, bias=bias, **prob) == 0
    results = grads + [db] if backward else [out, lse]
    assert call() == 0
    torch.cuda.synchronize()
    want = [t.clone() for t in results]
    L.ab200_debug_bounded_wait_test(drop, 1000)
    try:
        assert call() == 0
        assert call() == 0      # queued behind the first: starts after the failure and leaves at once
    finally:
        L.ab200_debug_bounded_wait_test(0, 0)
    assert L.ab200_stream_check(stream) == 719
    code = L.ab200_kernel_status(0)
    assert lo <= code < hi, hex(code)
    assert call() == 719
    assert L.ab200_kernel_status(1) == code
    assert L.ab200_stream_check(stream) == 0
    for t in results:
        t.fill_(float("nan"))
    assert call() == 0
    torch.cuda.synchronize()
    for a, b in zip(results, want):
        assert torch.equal(a, b)
