"""What a prompt pass decides before it launches anything, from its sizes alone.  No GPU needed."""
import ctypes as C

import pytest

from ksearch_b200 import _lib

E2B, E4B, TINY, MHA = (8, 1, 256), (8, 2, 256), (4, 1, 128), (8, 8, 128)   # query heads, KV heads, head size


def _pass(shape, max_seq, window, n, base):
    span = C.c_uint(0)
    return _lib.load().ks_debug_prompt_pass(*shape, max_seq, window, n, base, C.byref(span)) != 0, span.value


@pytest.mark.parametrize("max_seq", [1, 64, 100, 4096, 5000, 131072])
def test_the_image_launch_covers_what_the_pass_sees_and_little_more(max_seq):
    slot = -(-max_seq // 64)
    for n in (1, 9, 64, 65, 300, 2048):
        for base in (0, 1, 63, 64, 511, 512, 2048, 4095, 100000):
            if base + n > max_seq:
                continue
            need, span = -(-(base + n) // 64), _pass(E4B, max_seq, 0, n, base)[1]
            assert need <= span <= slot and span < 2 * need
