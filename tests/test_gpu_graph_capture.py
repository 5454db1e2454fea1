"""The operators under CUDA graph capture: every launch goes into the graph, nothing on the way asks the runtime
for something a capturing stream refuses, and a replay gives what the plain call gives, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TL = -2147483647


@pytest.mark.parametrize("dt,B,Hq,Hk,Sq,Sk,D,p", [
    (torch.bfloat16, 2, 4, 2, 200, 200, 128, 0.0),       # tile kernels
    (torch.float16, 1, 2, 2, 256, 256, 64, 0.2),
    (torch.float16, 1, 2, 1, 130, 200, 256, 0.0),        # wide heads
    (torch.bfloat16, 2, 8, 2, 1, 700, 128, 0.0),         # split keys
    (torch.float32, 1, 2, 2, 100, 90, 64, 0.1),          # general kernels
])
def test_replay_equals_call(dt, B, Hq, Hk, Sq, Sk, D, p):
    from aotriton_b200 import cabi
    g = torch.Generator(device="cuda").manual_seed(Sq + D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dt)
    q, do, k, v = mk(B, Hq, Sq, D), mk(B, Hq, Sq, D), mk(B, Hk, Sk, D), mk(B, Hk, Sk, D)
    kw = dict(sm_scale=D ** -0.5)
    if Sq > 1:
        kw.update(causal_type=3, window_left=TL, window_right=TL)
    if p:
        kw.update(dropout_p=p, philox_seed=torch.tensor([7], dtype=torch.uint64, device="cuda"),
                  philox_offset1=torch.tensor([3], dtype=torch.uint64, device="cuda"))
    out, lse, delta = torch.empty_like(q), torch.empty(B * Hq, Sq, device="cuda"), torch.empty(B * Hq, Sq, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    results = [out, lse] + grads

    def step():
        return (cabi.attn_fwd(q, k, v, out, lse, **kw), cabi.attn_bwd(q, k, v, out, do, *grads, lse, delta, **kw))

    assert step() == (0, 0)
    torch.cuda.synchronize()
    want = [t.clone() for t in results]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    n0 = cabi.lib().ab200_launch_count()
    with torch.cuda.graph(graph, stream=stream):
        codes = step()
    assert codes == (0, 0) and cabi.lib().ab200_launch_count() > n0
    for _ in range(2):
        for t in results:
            t.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(results, want):
            assert torch.equal(a, b)
    assert cabi.lib().ab200_kernel_status(0) == 0


def test_autograd_step_replays():
    """The Python entry points: outputs, log-sum-exp and gradients come from the graph's memory pool."""
    from aotriton_b200 import autograd
    mk = lambda h: torch.randn(2, h, 150, 64, device="cuda", dtype=torch.float16).requires_grad_()
    q, k, v = mk(4), mk(2), mk(2)
    do = torch.randn(2, 4, 150, 64, device="cuda", dtype=torch.float16)

    def step():
        out = autograd.attention(q, k, v, causal=True, dropout_p=0.1, philox_seed=11)
        return (out,) + torch.autograd.grad(out, (q, k, v), do)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            want = step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a.detach(), b.detach())
