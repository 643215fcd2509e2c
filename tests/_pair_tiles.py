"""Shapes that reach each tile width of the CTA-pair GEMM, found with the library's own rule."""
import functools

PLAIN, FUSED, FLOAT8 = 0, 1, 2
WIDTHS = {PLAIN: set(range(32, 241, 16)), FUSED: set(range(32, 193, 32)), FLOAT8: set(range(32, 225, 32))}


@functools.lru_cache(None)
def shapes(form, sms=148):
    """{width: (ms, n)} with the least ms * n of a search; n is ragged (7 past a multiple of 16) wherever that costs nothing."""
    from sparse import _ext
    rule = _ext.lib().sp24_pair_tile_columns
    found = {}
    for ms in range(256, 4097, 256):
        for n in [1] + list(range(7, 18000, 16)):
            w = rule(ms, n, form, sms)
            if w not in found or ms * n < found[w][0] * found[w][1]:
                found[w] = (ms, n)
    return found
