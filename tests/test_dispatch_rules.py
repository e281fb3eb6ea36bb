"""Rules that choose between kernels with the same results, asked on the CPU: no output shows which one ran."""
import ctypes as C

import apus_b200


def rule(mangled, restype, *argtypes):
    f = getattr(apus_b200.lib(), mangled)
    f.restype, f.argtypes = restype, argtypes
    return f


def test_item_rows_follow_the_routings_to_be_expected():
    """64-row work items are for experts with more than 32 rows.  A padded exchange brings world * tokens * topk slots, of
    which one in `world` is filled (moe.py, forward_padded): decode steps stay with items of 32."""
    rows = rule("_ZN4apus12tc_item_rowsExiib", C.c_int, C.c_longlong, C.c_int, C.c_int, C.c_bool)
    E, topk = 256, 6
    for world in (2, 4, 8):
        nl = E // world
        for tokens in (1, 18, 32, 64, 128):                        # per rank
            slots = world * tokens * topk
            want = 64 if tokens * world * topk / E > 29 else 32   # rows per expert
            assert rows(slots, nl, E, True) == want, (world, tokens)
    assert rows(8 * 32 * topk, 32, E, True) == 32 and rows(8 * 32 * topk, 32, E, False) == 64
    for tokens, want in ((512, 32), (1200, 32), (1400, 64), (2048, 64)):
        assert rows(tokens * topk, E, E, False) == want
    assert rows(0, 0, E, True) == 32


def test_taller_tiles_of_the_f32_linears_only_where_they_save_waves():
    pays = rule("_ZN4apus10seq64_paysExx", C.c_bool, C.c_longlong, C.c_longlong)
    up = lambda a, b: -(-a // b)   # noqa: E731
    for tokens, rows, want in ((32, 4736, False), (32, 4768, True), (32, 9472, True), (32, 9504, False), (320, 1024, False), (512, 1024, True),
                               (2048, 1024, True)):
        assert pays(up(rows, 32) * up(tokens, 32), up(rows, 64) * up(tokens, 32)) == want, (tokens, rows)
