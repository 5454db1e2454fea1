"""CPU, on a pretended device of 148 SMs: which forwards the split-key kernel takes and how it cuts them."""
import ctypes as C

import pytest
import torch

from aotriton_b200 import cabi
from test_host_fake_device import fake      # noqa: F401 (a fixture)


def _plan(L, B, Hq, Hk, Sq, Sk, D, dt=torch.bfloat16, family=0, bias=False, **kw):
    mk = lambda *s: torch.empty(*s, dtype=dt)
    q, k = mk(B, Hq, Sq, D), mk(B, Hk, Sk, D)
    a = cabi.make_fwd_args(q, k, k, torch.empty_like(q), None, bias=mk(B, Hq, Sq, Sk) if bias else None, sm_scale=1.0, **kw)
    old = L.ab200_set_kernel_family(family)
    try:
        n = L.ab200_debug_split_keys(C.byref(a), None)
    finally:
        L.ab200_set_kernel_family(old)
    return (n & 0xff, n >> 8 & 0xff, n >> 16) if n > 0 else n


def test_which_calls(fake):      # noqa: F811
    assert _plan(fake, 1, 4, 4, 16, 300, 128) != 0
    assert _plan(fake, 1, 4, 4, 17, 300, 128) == 0                                  # too many queries
    assert _plan(fake, 1, 4, 4, 1, 300, 136) == 0 and _plan(fake, 1, 4, 4, 1, 300, 60) == 0
    assert _plan(fake, 1, 4, 4, 1, 300, 128, bias=True) == 0 and _plan(fake, 1, 4, 4, 1, 300, 128, dropout_p=0.1) == 0
    assert _plan(fake, 1, 4, 4, 1, 300, 128, dt=torch.float32) == 0 and _plan(fake, 1, 4, 4, 1, 300, 128, family=1) == 0
    assert _plan(fake, 1, 4, 4, 1, 300, 60, family=2) == -801


@pytest.mark.parametrize("shape,want", [
    ((1, 1, 1, 1, 1, 128), (1, 4, 6)), ((1, 1, 1, 1, 192, 128), (1, 4, 6)),      # a piece has at least two tiles of 64 keys
    ((1, 1, 1, 1, 193, 128), (2, 4, 6)), ((1, 1, 1, 1, 449, 64), (4, 4, 12)), ((1, 1, 1, 1, 961, 64), (8, 8, 12)),
    ((18, 8, 1, 1, 2000, 128), (8, 8, 6)), ((19, 8, 1, 1, 2000, 128), (8, 4, 3)),      # 144 and 152 CTAs: one an SM, two
    ((37, 8, 1, 1, 2000, 128), (8, 4, 3)), ((38, 8, 1, 1, 2000, 128), (4, 4, 3)),      # 296 places
    ((74, 8, 1, 1, 2000, 128), (4, 4, 3)), ((75, 8, 1, 1, 2000, 128), (2, 4, 3)), ((149, 8, 1, 1, 2000, 128), (1, 4, 3)),
    ((18, 32, 1, 1, 2000, 128), (8, 4, 6)), ((19, 32, 1, 1, 2000, 128), (4, 4, 6)),      # 32-row tiles of 128: one CTA an SM
])
def test_cut(fake, shape, want):      # noqa: F811
    assert _plan(fake, *shape) == want
