"""Host-side bounds of the kernels' launches, against a restatement of how rows reach threads and
chunks (no GPU). The bounds are internal functions of the library, called by their C++ names."""
import ctypes

import pytest

from tpchq01_gpu_b200 import _lib

LAYOUTS = {"pair": 0, "pair_filter": 1, "separate": 2, "separate_filter": 3, "uncompressed": 4}


def internal(name, restype, argtypes):
    f = getattr(ctypes.CDLL(_lib.LIB_PATH), name)
    f.restype, f.argtypes = restype, argtypes
    return f


@pytest.mark.parametrize("placement", range(5))
@pytest.mark.parametrize("layout", sorted(LAYOUTS))
def test_a_scan_launch_gives_a_thread_at_most_32768_rows(layout, placement):
    """Tiles go round the CTAs, a tile's rows evenly over the consumer threads; the rows after the
    last whole tile go a row a thread, CTAs with a tile less first."""
    most = internal("_ZN2q124scan_max_rows_per_launchEiij", ctypes.c_uint64, [ctypes.c_int, ctypes.c_int, ctypes.c_uint32])
    tile_rows = internal("_ZN2q114scan_tile_rowsEii", ctypes.c_uint32, [ctypes.c_int, ctypes.c_int])
    R = tile_rows(LAYOUTS[layout], placement)
    per_thread = 4 if layout == "uncompressed" else 12
    threads = R // per_thread
    for grid in [1, 2, 3, 7, 147, 148]:
        bound = most(LAYOUTS[layout], placement, grid)
        assert 0 < bound <= 1 << 31 and bound % 128 == 0
        for rows in [bound, bound - 1, bound - R + 1, bound - R * grid + R - 1]:
            tiles, tail = divmod(rows, R)
            extra = tiles % grid
            for cta in {0, extra, max(extra - 1, 0), grid - 1}:
                turn = (cta - extra) % grid
                own_tiles = tiles // grid + (1 if cta < extra else 0)
                own_tail = len(range(turn * threads, tail, grid * threads))
                assert own_tiles * per_thread + own_tail <= 32768, (grid, rows, cta)
