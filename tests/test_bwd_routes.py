"""CPU: which route a backward takes, and on a pretended device how many launches that is."""
import ctypes as C

import pytest
import torch

from aotriton_b200 import cabi
from test_host_fake_device import _bwd_args, fake      # noqa: F401 (a fixture)


def _launches(L, a):
    n0 = L.ab200_launch_count()
    assert L.ab200_attn_bwd(C.byref(a), None) == 0 and L.ab200_last_bwd_family() == 1
    return L.ab200_launch_count() - n0


@pytest.mark.parametrize("dtype,D,B,H,S,want", [
    (cabi.DTYPE_FP32, 64, 1, 1, 1, 2), (cabi.DTYPE_FP32, 128, 4, 16, 2048, 2),      # preprocess, dK/dV and dQ
    (cabi.DTYPE_FP16, 60, 4, 16, 2048, 2), (cabi.DTYPE_FP16, 124, 4, 8, 1024, 2),
    (cabi.DTYPE_FP16, 100, 4, 16, 1023, 3), (cabi.DTYPE_BF16, 124, 4, 16, 992, 2),   # 4096 working CTAs; 3968
    (cabi.DTYPE_FP32, 160, 1, 2, 64, 3),                                             # head dims above 128
])
def test_general_backward_in_one_launch_or_two(fake, dtype, D, B, H, S, want):      # noqa: F811
    a = _bwd_args(dtype=dtype, D=D, B=B, Hq=H, Hk=H, S=S)
    elt = 4 if dtype == cabi.DTYPE_FP32 else 2
    for i, v in enumerate((a.q, a.out, a.dout, a.dq, a.k, a.v, a.dk, a.dv)):      # (apart, whatever their size)
        v.ptr = (i + 1) << 34
        assert v.size[0] * v.stride[0] * elt < 1 << 34
    a.lse, a.delta = 10 << 34, 11 << 34
    assert _launches(fake, a) == want
    a.dq.ptr = a.dout.ptr      # dQ over dO: dK/dV must have read it
    assert _launches(fake, a) == 3


def test_dk_from_dbias_rule():
    """dK comes from dBias only where dBias keeps every value the dQ kernel writes, in rows a tile map can describe, and
    where dQ, written before dK is formed, leaves the inputs alone."""
    mk = lambda *s, dt=torch.float16: torch.empty(*s, dtype=dt)

    def ask(dqk=256, sq=130, sk=136, dt=torch.float16, family=0, dbias="", dq=None, **kw):
        q, do, k, v = mk(2, 4, sq, dqk, dt=dt), mk(2, 4, sq, dqk, dt=dt), mk(2, 2, sk, dqk, dt=dt), mk(2, 2, sk, dqk, dt=dt)
        bias = mk(2, 4, sq, sk, dt=dt)
        db = {"": lambda: mk(2, 4, sq, sk, dt=dt), "bshd": lambda: mk(2, sq, 4, sk, dt=dt).transpose(1, 2),
              "padded": lambda: mk(2, 4, sq, sk + 8, dt=dt)[..., :sk], "over bias": lambda: bias,
              "one batch": lambda: mk(1, 4, sq, sk, dt=dt).expand(2, 4, sq, sk), "none": lambda: None,
              "off": lambda: mk(2, 4, sq, sk + 8, dt=dt)[..., 1:sk + 1], "short": lambda: mk(2, 4, sq - 1, sk, dt=dt)}[dbias]()
        grads = [q if dq == "q" else mk(2, 4, sq, dqk, dt=dt), mk(2, 2, sk, dqk, dt=dt), mk(2, 2, sk, dqk, dt=dt)]
        lse = torch.empty(8, sq)
        a = cabi.make_bwd_args(q, k, v, mk(2, 4, sq, dqk, dt=dt), do, *grads, lse, torch.empty_like(lse), bias=bias, dbias=db,
                               sm_scale=1.0, **kw)
        old = cabi.lib().ab200_set_kernel_family(family)
        try:
            return cabi.lib().ab200_debug_dk_from_dbias(C.byref(a))
        finally:
            cabi.lib().ab200_set_kernel_family(old)

    assert ask() == 1 and ask(dqk=136) == 1 and ask(dt=torch.bfloat16) == 1 and ask(family=2) == 1
    assert ask(dbias="bshd") == 1 and ask(dbias="padded") == 1
    assert ask(dbias="none") == 0 and ask(dqk=128) == 0
    assert ask(sk=131) == 0 and ask(dbias="off") == 0                    # rows off a 16-byte boundary
    assert ask(dbias="one batch") == 0 and ask(dbias="short") == 0       # values lost
    assert ask(dbias="over bias") == 0 and ask(dq="q") == 0              # over something still read
    assert ask(dt=torch.float32) == 0 and ask(dqk=260) == 0 and ask(family=1) == 0      # general kernels
    cu = torch.tensor([0, 130, 260], dtype=torch.int32)
    assert ask(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=130, max_seqlen_k=136, varlen_type=cabi.VARLEN_PADDED) == 0
