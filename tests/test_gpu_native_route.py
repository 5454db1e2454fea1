"""The entry points' native route against the Function and the operators it stands for: the same bits over the forms a call
takes, and the other way taken wherever a mode, a transform or a tensor is not ordinary."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


def _rand(*s, dt=torch.float16, seed=0):
    return torch.randn(*s, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dt)


@pytest.fixture
def python_way(monkeypatch):
    from aotriton_b200 import autograd
    return lambda: monkeypatch.setattr(autograd, "_attend", lambda *a: None)


def _step(call, ins, do):
    ins = [t.detach().requires_grad_() for t in ins]
    out = call(*ins)
    outs = out if isinstance(out, tuple) else (out,)
    return [o.detach() for o in outs] + list(torch.autograd.grad(outs[0], ins, do))


def _layouts(b, h, n, d, dt, seed):
    yield _rand(b, h, n, d, dt=dt, seed=seed)
    yield _rand(b, n, h, d, dt=dt, seed=seed).transpose(1, 2)
    yield _rand(b, h, n, 2 * d, dt=dt, seed=seed)[..., :d]


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("kind", ["attention", "causal", "window", "bias", "expanded_bias", "dropout", "lse", "sdpa", "sdpa_bias_dropout"])
def test_same_bits_as_the_python_way(kind, layout, dt, python_way):
    from aotriton_b200 import autograd
    q, k, v, do = (list(_layouts(2, h, n, 64, dt, i))[layout] for i, (h, n) in enumerate(((4, 150), (2, 200), (2, 200), (4, 150))))
    ins = [q, k, v]
    if "bias" in kind:
        ins.append(_rand(2, 4, 150, 200, dt=dt, seed=9) if kind != "expanded_bias" else _rand(2, 1, 150, 200, dt=dt, seed=9).expand(2, 4, 150, 200))
    call = {
        "attention": lambda *a: autograd.attention(*a),
        "causal": lambda *a: autograd.attention(*a, causal=True, sm_scale=0.2),
        "window": lambda *a: autograd.attention(*a, causal=(40, 7)),
        "bias": lambda *a: autograd.attention(*a),
        "expanded_bias": lambda *a: autograd.attention(*a),
        "dropout": lambda *a: autograd.attention(*a, dropout_p=0.3, philox_seed=(1 << 63) + 5, philox_offset1=(1 << 64) - 7),
        "lse": lambda *a: autograd.attention(*a, return_lse=True),
        "sdpa": lambda *a: autograd.scaled_dot_product_attention(*a, is_causal=True, enable_gqa=True),
        "sdpa_bias_dropout": lambda *a: autograd.scaled_dot_product_attention(*a, dropout_p=0.1, enable_gqa=True, scale=0.3),
    }[kind]
    seen = []
    native = autograd._native.attend
    class Spy:
        attend = staticmethod(lambda *a: (seen.append(r := native(*a)), r)[1])
        last_bwd_family, note_bwd_family = autograd._native.last_bwd_family, autograd._native.note_bwd_family
    try:
        keep, autograd._native = autograd._native, Spy
        got = _step(call, ins, do)
        with torch.no_grad():
            plain = call(*ins)
    finally:
        autograd._native = keep
    assert len(seen) == 2 and all(s is not None for s in seen)
    python_way()
    want = _step(call, ins, do)
    for a, b in zip(got, want):
        assert a.stride() == b.stride() and torch.equal(a, b)
    plain = plain if isinstance(plain, tuple) else (plain,)
    for a, b in zip(plain, want):
        assert not a.requires_grad and torch.equal(a, b)


@pytest.mark.parametrize("p", [0.0, 0.2])
def test_packed_same_bits(p, python_way):
    from aotriton_b200 import autograd
    lens = [1, 77, 130, 300]
    cu = torch.tensor([0, 1, 78, 208, 508], dtype=torch.int32, device="cuda")
    q, k, v, do = (_rand(1, 508, h, 64, seed=i).transpose(1, 2) for i, h in enumerate((4, 2, 2, 4)))
    call = lambda *a: autograd.varlen_attention(*a, cu, cu, max(lens), max(lens), causal=True, dropout_p=p, return_lse=True)
    got = _step(call, (q, k, v), do)
    assert autograd.last_bwd_family == 2
    python_way()
    for a, b in zip(got, _step(call, (q, k, v), do)):
        assert a.stride() == b.stride() and torch.equal(a, b)


def _qkv(grad=True):
    return [_rand(1, 2, 64, 64, seed=i).requires_grad_(grad) for i in range(3)]


def test_saved_tensor_hooks_and_versions():
    from aotriton_b200 import autograd
    q, k, v = _qkv()
    want = torch.autograd.grad(autograd.attention(q, k, v).sum(), (q, k, v))
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
        out = autograd.attention(q, k, v)
    assert len(packed) == 5      # q, k, v, out, log-sum-exp
    for a, b in zip(torch.autograd.grad(out.sum(), (q, k, v)), want):
        assert torch.equal(a, b)
    x = q.detach().clone().requires_grad_()
    y = x * 1
    out = autograd.attention(y, k, v)
    with torch.no_grad():
        y.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


def test_second_derivatives_stay_refused():
    from aotriton_b200 import autograd
    q, k, v = _qkv()
    out = autograd.scaled_dot_product_attention(q, k, v)
    g, = torch.autograd.grad(out.float().square().sum(), q, create_graph=True)
    with pytest.raises(RuntimeError):
        g.sum().backward()


def test_modes_see_the_operators():
    from aotriton_b200 import autograd

    class Names(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    mode = Names()
    mode.seen = []
    q, k, v = _qkv()
    with mode:
        autograd.scaled_dot_product_attention(q, k, v).sum().backward()
    assert "aotriton_b200.attn_fwd.default" in mode.seen and "aotriton_b200.attn_bwd.default" in mode.seen
    from torch._subclasses.fake_tensor import FakeTensorMode
    plain = [t.detach() for t in (q, k, v)]
    with FakeTensorMode() as fake:
        f = [fake.from_tensor(t) for t in plain]
        assert autograd.scaled_dot_product_attention(*f).shape == q.shape


def test_transforms_stay_refused():
    from aotriton_b200 import autograd
    q, k, v = _qkv(False)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda q: autograd.attention(q, k, v).sum())(q)
    import torch.autograd.forward_ad as fwd
    with fwd.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError)):
            autograd.attention(fwd.make_dual(q, torch.ones_like(q)), k, v)


def test_other_tensors_go_the_python_way():
    from aotriton_b200 import autograd
    q, k, v = _qkv(False)

    class Sub(torch.Tensor):
        pass

    args = lambda **kw: {**dict(q=q, k=k, v=v, b=None, cu_q=None, cu_k=None, max_q=0, max_k=0, sm_scale=1.0, dropout_p=0.0, causal=False,
                                return_lse=False, seed=1, offset1=2, op=False), **kw}
    assert autograd._attend(**args()) is not None
    for bad in (dict(q=q.as_subclass(Sub)), dict(q=q.cpu()), dict(k=k.float()), dict(q=q[0]), dict(q=q.transpose(2, 3)), dict(q=q[:, :, :0]),
                dict(dropout_p=0.5, seed=-1), dict(dropout_p=0.5, offset1=1 << 64), dict(sm_scale=torch.tensor(1.0)), dict(return_lse=1)):
        assert autograd._attend(**args(**bad)) is None, bad
    with pytest.raises(RuntimeError, match="attn_fwd failed"):
        autograd.attention(q, k, v, dropout_p=-0.5)


def test_gradients_follow_the_stream():
    from aotriton_b200 import autograd
    q, k, v = _qkv()
    want = torch.autograd.grad(autograd.attention(q, k, v).sum(), (q, k, v))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        got = torch.autograd.grad(autograd.attention(q, k, v).sum(), (q, k, v))
    torch.cuda.current_stream().wait_stream(side)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
