"""CPU, on a pretended device: how many launches a backward takes on each of its routes."""
import ctypes as C

import pytest

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
