"""The height of the phase-field tiles of a level never computes many more rows than the best height would (CPU)."""
import ctypes as C

from hpcrack_b200 import lib as L


def test_no_wasted_rows(full=16, least=4):
    tile_rows = L.load()._ZN3hpc9tile_rowsEiii  # hpc::tile_rows(int ny, int full, int least)
    tile_rows.argtypes, tile_rows.restype = [C.c_int] * 3, C.c_int
    heights = [h for h in (4, 8, 16) if least <= h <= full]
    computed = lambda ny, h: -(-ny // (h - 1)) * h  # noqa: E731: a tile of h rows finishes h - 1
    for ny in range(2, 400):
        h = tile_rows(ny, full, least)
        assert h in heights
        assert 3 * computed(ny, h) <= 4 * min(computed(ny, q) for q in heights), ny
