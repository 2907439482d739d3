"""What b2_recur_prep refuses, it refuses on every path: rows of more channels than fit shared memory (host checks, no GPU)."""
import ctypes

import pytest

from b200attn import _lib


@pytest.mark.parametrize("dk", [128, 124])           # heads that the vector form takes, and not
def test_rows_of_too_many_channels(dk):
    lib = _lib.load()
    buf = ctypes.create_string_buffer(64)
    p = ctypes.addressof(buf) + 15 & ~15             # aligned and never read: the call is refused on the host
    H = 51200 // (3 * dk) + 1                        # q, k and v rows of H heads: more than 51200 fp32 numbers
    rc = lib.b2_recur_prep(p, 3 * H * dk, _lib.ACT_BF16, 4, H, H, dk, dk, 1, None, 0, 0, 0.0, 1.0, 1.0, None, 0, 0, 0, -1,
                           _lib.DECAY_HEAD_CONST, 0, None, 0, None, p, 1.0, p, p, p, 1, None, p, None, p, None)
    assert rc == _lib.B2_EUNSUPPORTED and b"do not fit shared memory" in lib.b2_last_error()
