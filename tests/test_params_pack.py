"""The packed parameter block holds what the ctypes structure would, also for values that a field cannot hold."""
import ctypes

import pytest

from flash_attn_b200 import _lib

FIELDS = [n for n, _ in _lib.FwdParams._fields_]


def values(**over):
    v = {n: i + 1 for i, n in enumerate(FIELDS)}
    v.update(softmax_scale=0.125, p_dropout=0.1, window_left=-1, window_right=-1, q_pos0=-5, k_pos0=1 << 40, seed=(1 << 64) - 1)
    v.update(over)
    return [v[n] for n in FIELDS]


@pytest.mark.parametrize("over", [{}, dict(lse=0, workspace=0, workspace_bytes=0, status=0, stream=0),
                                  dict(softmax_scale=1e300), dict(seed=-1), dict(batch=1 << 32)])
def test_packed_block_is_the_structure(over):
    v = values(**over)
    packed = _lib.pack_params(*v)
    assert len(packed) == ctypes.sizeof(_lib.FwdParams)
    got, want = _lib.FwdParams.from_buffer_copy(packed), _lib.FwdParams(*v)
    for n in FIELDS:
        assert getattr(got, n) == getattr(want, n), n
