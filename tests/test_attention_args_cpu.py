"""Operand checks of the attention entry points that need no GPU: which views are copied, which addresses are refused."""
import ctypes
import os

import pytest
import torch

from msamp.ops import native, nn as K


def _view(offset, strides, shape=(2, 5, 3, 64)):
    need = offset + 1 + sum((n - 1) * s for n, s in zip(shape, strides))
    return torch.randn(need, dtype=torch.float32).bfloat16().as_strided(shape, strides, offset)


def test_readable_rows_are_passed_on():
    for strides in ((960, 192, 64, 1), (960, 64, 320, 1), (5 * 256, 256, 72, 1), (960, 192, 0, 1)):
        t = _view(0, strides)
        assert K._rows16(t) is t
        assert K._rows16(_view(8, strides)).data_ptr() % 16 == 0


@pytest.mark.parametrize('offset, strides', [
    (4, (960, 192, 64, 1)),       # contiguous, starts 8 bytes into its buffer
    (1, (960, 192, 64, 1)),
    (4, (1000, 200, 64, 1)),      # what the backward of a concatenation along the last axis hands over
    (0, (960, 196, 64, 1)),       # rows of 392 bytes
    (0, (1, 10, 50, 200)),
    (0, (0, 0, 0, 0)),            # gradient of a sum
])
def test_other_rows_are_copied(offset, strides):
    t = _view(offset, strides)
    c = K._rows16(t)
    assert c.data_ptr() != t.data_ptr() and c.data_ptr() % 16 == 0 and c.is_contiguous() and torch.equal(c, t)


def test_size_one_axis_with_an_odd_stride_is_copied():
    t = _view(0, (3, 192, 64, 1), (1, 5, 3, 64))    # contiguous by definition, but the stride of the batch is 6 bytes
    assert t.is_contiguous() and K._rows16(t).stride(0) % 8 == 0


@pytest.mark.skipif(not os.path.exists(native.LIB_PATH), reason='kernel library not built')
@pytest.mark.parametrize('family', ['', 'tc_'])
@pytest.mark.parametrize('which, n', [('fwd', 4), ('bwd', 8)])
def test_misaligned_addresses_are_refused(family, which, n):
    """No launch and no driver call: the addresses below belong to nothing."""
    entry = getattr(native.lib(), f'msamp_attention_{family}{which}')
    strides = (ctypes.c_int64 * 24)(*([960, 192, 64] * 8))
    f32 = 1 << 20
    for bad in range(n):
        a = [((1 << 20) + (8 if i == bad else 0)) for i in range(n)]
        ptrs = a[:4] + [f32] if which == 'fwd' else a[:4] + [f32] + a[4:] + [f32]
        rc = entry(*ptrs, strides, 2, 3, 5, 64, 0.125, 1, None)
        assert rc != 0 and b'16-byte aligned' in native.lib().msamp_last_error(), (bad, rc)
