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


class ChunkPool:
    """One CTA's reservations in the group-key partition's pass 1 (64 partitions, rounds of 3072
    records, chunks of 256, reserved 128 at a time): a partition's new chunks of a round lie
    together, and those of a round that no longer fit the grab go to a new one."""

    def __init__(self):
        self.room = [0] * 64
        self.left = self.reserved = 0

    def round(self, records):
        assert sum(records.values()) <= 3072
        need = fit = 0
        for p in sorted(records):
            rest = max(0, records[p] - self.room[p])
            want = -(-rest // 256)
            self.room[p] += 256 * want - records[p]
            need += want
            if need <= self.left:
                fit = need
        if need > self.left:
            more = max(need - fit, 128)
            self.reserved += more
            self.left = more - (need - fit)
        else:
            self.left -= need


def wasteful_order(rounds):
    """Rounds whose passing rows come in an order that leaves 11 chunks of every grab unused: nine
    partitions open a chunk for one record, then are filled three at a time, so that each grab has
    been used to 117 chunks when one partition wants 12. The last round opens every partition."""
    def rest(n):
        return {0: 3072 - n}
    cycle = [{**rest(9), **{p: 1 for p in range(1, 10)}}] + [rest(0)] * 8
    for first in (1, 4, 7):
        cycle += [rest(0)] * 9 + [{**rest(765), **{p: 255 for p in range(first, first + 3)}}]
    for i in range(rounds - 1):
        yield cycle[i % len(cycle)]
    yield {**rest(63), **{p: 1 for p in range(1, 64)}}


@pytest.mark.parametrize("ctas", [1, 2, 4, 8])
def test_partition_chunks_stay_within_their_bound(ctas):
    """The directory entries cleared for a segment cover every chunk its CTAs reserve, also where a
    full segment's rows come in the order that wastes the most."""
    bound = internal("_ZN2q124groupkey_part_max_chunksEmj", ctypes.c_uint64, [ctypes.c_uint64, ctypes.c_uint32])
    rounds = 6 * (1 << 24) // 3072 // ctas
    pool = ChunkPool()
    for r in wasteful_order(rounds):
        pool.round(r)
    assert pool.reserved > 1.093 * rounds * 12   # the order does what it is made for
    assert ctas * pool.reserved <= bound(ctas * rounds * 3072, ctas)


def test_partition_chunks_of_small_and_uniform_segments():
    bound = internal("_ZN2q124groupkey_part_max_chunksEmj", ctypes.c_uint64, [ctypes.c_uint64, ctypes.c_uint32])
    for rounds in [1, 2, 3, 50]:
        for spread in [1, 3, 64]:
            pool = ChunkPool()
            for _ in range(rounds):
                pool.round({p: 3072 // spread for p in range(spread)})
            assert pool.reserved <= bound(rounds * 3072, 1), (rounds, spread)
