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
            assert need <= span <= slot and span < max(2 * need, 33)


@pytest.mark.parametrize("n_kv,hd,max_seq,n_slots", [(1, 256, 4096, 1), (2, 256, 4096, 8), (2, 256, 131072, 1), (32, 256, 1024, 8), (1, 128, 64, 64)])
def test_decoded_tiles_leave_the_memory_that_others_need(n_kv, hd, max_seq, n_slots):
    """As many tiles as the slots hold, up to 256 MB but one slot's at least, and none where that would cut into the spare memory."""
    lib, most, spare = _lib.load(), 1 << 62, 3 << 30
    one, slot = n_kv * (64 * hd * 8 + 4), -(-max_seq // 64)
    tiles = lib.ks_debug_image_tiles(n_kv, hd, max_seq, n_slots, most, spare)
    assert slot <= tiles <= n_slots * slot
    assert tiles == n_slots * slot or tiles == max(slot, (256 << 20) // one)
    need = tiles * one
    assert lib.ks_debug_image_tiles(n_kv, hd, max_seq, n_slots, spare + need, spare) == tiles
    for free in (spare + need - 1, spare, spare - 1, need, 0):
        assert lib.ks_debug_image_tiles(n_kv, hd, max_seq, n_slots, free, spare) == 0


# microseconds per layer: rows share their context / every row by itself (E2B- and E4B-shaped layers, one slot)
@pytest.mark.parametrize("shape,window,n,base,shared,rows", [
    (E2B, 0, 256, 0, 120.8, 114.3), (E2B, 0, 384, 0, 133.4, 140.4), (E2B, 0, 128, 256, 95.3, 87.6), (E2B, 0, 256, 256, 123.1, 127.6),
    (E2B, 0, 96, 512, 91.9, 86.4), (E2B, 0, 160, 512, 112.8, 118.3), (E2B, 0, 64, 1024, 108.9, 82.3), (E2B, 0, 128, 1024, 105.5, 108.8),
    (E2B, 0, 48, 2048, 95.3, 93.8), (E2B, 0, 64, 2048, 109.5, 97.4), (E2B, 0, 80, 2048, 98.2, 124.6), (E2B, 0, 32, 4096, 107.9, 89.2), (E2B, 0, 48, 4096, 98.0, 123.5),
    (E2B, 128, 192, 1024, 109.7, 98.5), (E2B, 128, 640, 1024, 186.0, 198.6), (E2B, 1024, 64, 4096, 107.2, 80.3),
    (E4B, 0, 256, 0, 176.6, 171.2), (E4B, 0, 448, 0, 252.5, 268.9), (E4B, 0, 128, 256, 133.1, 124.3), (E4B, 0, 256, 256, 178.5, 186.8),
    (E4B, 0, 64, 1024, 133.4, 100.8), (E4B, 0, 160, 1024, 159.3, 187.3), (E4B, 0, 48, 2048, 142.3, 114.6), (E4B, 0, 64, 2048, 148.5, 119.6),
    (E4B, 0, 80, 2048, 142.9, 169.0), (E4B, 0, 32, 4096, 135.9, 105.4), (E4B, 0, 48, 6000, 153.9, 169.2),
    (E4B, 128, 256, 4096, 203.7, 190.2), (E4B, 512, 128, 4096, 158.7, 141.4), (E4B, 1024, 96, 4096, 159.2, 146.6), (E4B, 1024, 64, 1024, 133.2, 98.8),
    (TINY, 0, 192, 512, 55.6, 51.3), (TINY, 0, 448, 512, 68.9, 75.1), (TINY, 0, 128, 1024, 80.0, 56.2), (TINY, 0, 320, 1024, 61.3, 75.6),
    (MHA, 0, 128, 0, 56.7, 53.1), (MHA, 0, 192, 0, 59.1, 68.8), (MHA, 0, 32, 256, 47.2, 38.5), (MHA, 0, 24, 2048, 54.5, 69.7),
])
def test_prompt_rows_take_the_faster_form_of_attention(shape, window, n, base, shared, rows):
    """Away from the line (within 3 % either form will do) the rule picks the form that was measured faster."""
    took = shared if _pass(shape, 8192, window, n, base)[0] else rows
    assert took <= 1.03 * min(shared, rows)
