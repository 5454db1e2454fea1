"""Tensors read natively into the parameter structs, against the views built one by one in Python: the ordinary
forms agree field by field, everything else is left to the Python way (and refused or taken as it was there)."""
import pytest
import torch

from aotriton_b200 import flash

_p = flash._p


def _fields(view):
    return view.data_ptr, list(view.sizes), list(view.strides), view.dtype


TENSORS = [torch.empty(2, 3, 4, 8, dtype=torch.float16), torch.empty(2, 4, 3, 8, dtype=torch.bfloat16).transpose(1, 2),
           torch.empty(2, 3, 4, 16)[..., :8], torch.empty(1, 1, 1, 1), torch.empty(2, 0, 4, 8),
           torch.empty(1, 3, 4, 8).expand(2, 3, 4, 8)]


@pytest.mark.parametrize("i", range(len(TENSORS)))
def test_ordinary_tensors(i):
    t, lse, scalar, null = TENSORS[i], torch.empty(6, 4), torch.zeros(1, dtype=torch.uint64), torch.empty(0, dtype=torch.int32)
    f = flash._fwd_params()
    assert _p.set_fwd_views(f, flash._DTYPES, t, t, t, None, lse, t, scalar, null, scalar, null, None, null)
    for got in (f.Q, f.K, f.V, f.Out):
        assert _fields(got) == _fields(flash.mk_aotensor(t))
    for got in (f.B, f.encoded_softmax):
        assert _fields(got) == _fields(flash.mk_aotensor(None, if_empty_then_like=t))
    assert _fields(f.L) == _fields(flash.mk_aotensor(lse))
    for got, want in ((f.philox_seed_ptr, scalar), (f.philox_offset1, null), (f.philox_seed_output, scalar),
                      (f.persistent_atomic_counter, null)):
        assert (got.data_ptr, got.dtype) == (flash.mk_aotensor(want).data_ptr, flash.mk_aotensor(want).dtype)
    b = flash._bwd_params()
    assert _p.set_bwd_views(b, flash._DTYPES, t, t, t, t, t, t, t, t, t, None, lse, scalar, null)
    for got in (b.Q, b.K, b.V, b.B, b.Out, b.DO, b.DK, b.DV, b.DQ):
        assert _fields(got) == _fields(flash.mk_aotensor(t))
    assert _fields(b.DB) == _fields(flash.mk_aotensor(None, if_empty_then_like=t))


@pytest.mark.parametrize("bad", [None, torch.empty(2, 3, 4), torch.empty(2, 3, 4, 8).transpose(2, 3),
                                 torch.empty(2, 3, 4, 8, dtype=torch.complex64)])
def test_other_forms_are_left_alone(bad):
    t, lse, null = TENSORS[0], torch.empty(6, 4), torch.empty(0, dtype=torch.uint64)
    assert not _p.set_fwd_views(flash._fwd_params(), flash._DTYPES, bad, t, t, None, lse, t, null, null, null, null, None, null)
    assert not _p.set_bwd_views(flash._bwd_params(), flash._DTYPES, t, t, t, None, t, bad, t, t, t, None, lse, null, null)
    with pytest.raises(Exception):
        flash.attn_fwd(bad, t, t, None, 1.0, lse, t, 0.0, null, null, 0, null, null, None, False, null)


def test_scalars_on_the_device():
    from aotriton_b200 import autograd
    for v in (0, 1, (1 << 63) - 1, 1 << 63, (1 << 64) - 1):
        assert autograd._device_u64("cpu", v).item() == v and autograd._device_u64("cpu", v).dtype == torch.uint64
    for v in (-1, 1 << 64):
        with pytest.raises(OverflowError):
            autograd._device_u64("cpu", v)
    seed, off = autograd._philox_tensors("cpu", 0.5, 7, (1 << 64) - 1)
    assert (seed.item(), off.item()) == (7, autograd.DEFAULT_PHILOX_OFFSET_2 - 1)
    assert autograd._philox_tensors("cpu", 0.0, 7, 3)[0].numel() == 0
