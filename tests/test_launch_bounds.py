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


class BatchInstance(ctypes.Structure):
    _fields_ = [("col", ctypes.c_void_p * 6), ("rows", ctypes.c_uint64), ("cutoff", ctypes.c_int32),
                ("num_groups", ctypes.c_uint32), ("mode", ctypes.c_uint32), ("pad", ctypes.c_uint32),
                ("acc", ctypes.c_void_p), ("out", ctypes.c_void_p)]


class BatchItem(ctypes.Structure):
    _fields_ = [("instance", ctypes.c_uint32), ("first_tile", ctypes.c_uint32), ("num_tiles", ctypes.c_uint32),
                ("pad", ctypes.c_uint32)]


def batch_items(rows, num_groups, ctas):
    """The work items (instance, first tile, tiles) of a batch of equal group counts, in the order they are claimed."""
    plan = internal("_ZN2q110batch_planEPKNS_16BatchInstanceDevEjjjRSt6vectorINS_9BatchItemESaIS4_EERNS_11BatchParamsE", None,
                    [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p])
    inst = (BatchInstance * len(rows))()
    for i, n in enumerate(rows):
        inst[i].rows, inst[i].num_groups, inst[i].mode = n, num_groups, 1
    vector = (ctypes.c_void_p * 3)()          # an empty std::vector: first, last, end of storage
    params = ctypes.create_string_buffer(4096)
    plan(inst, len(rows), 0, ctas, vector, params)
    n = ((vector[1] or 0) - (vector[0] or 0)) // ctypes.sizeof(BatchItem)
    items = ctypes.cast(vector[0], ctypes.POINTER(BatchItem))
    return [(items[i].instance, items[i].first_tile, items[i].num_tiles) for i in range(n)]


@pytest.mark.parametrize("num_groups", [4, 64, 1024, 2500])
@pytest.mark.parametrize("rows,most", [([1_000_003], 1.7), ([2_000_003], 1.5), ([4_000_003], 1.3), ([5_000_001], 1.3), ([8_000_003], 1.2),
                                       ([20_000_001], 1.2), ([100_000_003], 1.1), ([100_003] * 8, 1.7),
                                       ([2_500_001] * 2, 1.4), ([500_001] * 8, 1.4), ([1_000_001] * 16, 1.4)])
def test_batch_pieces_even_out_the_ctas(num_groups, rows, most):
    """Every tile is in one item, and CTAs that claim the items in turn end within `most` times an equal share (a piece
    in two CTAs and none in the others' second turn made it twice the share)."""
    ctas = 148
    tiles = [-(-n // 2048) for n in rows]
    items = batch_items(rows, num_groups, ctas)
    for i, n in enumerate(tiles):
        own = sorted((first, size) for inst, first, size in items if inst == i)
        assert [first for first, _ in own] == [sum(size for _, size in own[:k]) for k in range(len(own))]
        assert sum(size for _, size in own) == n
        assert all(0 < size <= (1023 if num_groups <= 4 else 4096) for _, size in own)
    busy = [0] * ctas
    for _, _, size in items:
        k = busy.index(min(busy))
        busy[k] += size
    assert max(busy) <= most * sum(tiles) / ctas
