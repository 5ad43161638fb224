"""The high-cardinality paths of the group-key shared placement against the oracle. Above 256
groups the library chooses on the device, from a sample of the rows, among: one pass with a
shared slot per key < 4096 (3-stage ring above 2048 groups; larger keys into global
accumulators), every passing row straight into global accumulators (few passing rows over spread
keys), and, above 4096 groups, a two-pass radix partition (rows partitioned by key into 8-byte
records, then one shared-memory slot table per 4096-key partition). Q1_GROUPKEY_PATH forces each
path so that all are checked: group counts on both sides of the
partition width, uniform and Zipf keys, cutoffs from nothing to everything passing, ragged and
tiny row counts, few-CTA launches (partition changes and table flushes inside a CTA) and a
launch that crosses the 2^27-row segment boundary (against the global placement and the row
count). Tolerance 0."""
import ctypes

import numpy as np
import pytest
import torch

import gen_np
import tpchq01_gpu_b200 as q
from oracle import py_oracle as O
from tpchq01_gpu_b200 import _lib
from test_gpu_groupkey import check, device_cols, keys_for, run_gpu, widen, zipf_cdf

pytestmark = pytest.mark.gpu

ROWS = 400_037
SEED = 555


PATHS = ["partitioned", "single", "global", "auto"]


@pytest.fixture(scope="module")
def table(cuda):
    comp = gen_np.compress(gen_np.generate(SEED, 0, ROWS))
    c, keep = device_cols(comp)
    return comp, c, keep


@pytest.fixture(params=PATHS)
def path(request, monkeypatch):
    if request.param == "auto":
        monkeypatch.delenv("Q1_GROUPKEY_PATH", raising=False)
    else:
        monkeypatch.setenv("Q1_GROUPKEY_PATH", request.param)
    return request.param


@pytest.mark.parametrize("num_groups", [257, 1024, 1025, 2049, 3000, 4096])
@pytest.mark.parametrize("dist", ["uniform", "zipf"])
@pytest.mark.parametrize("path", ["single", "global", "auto"], indirect=True)
def test_wide_tables_match_oracle(table, path, num_groups, dist):
    """257..4096 groups: the path is chosen on the device; the single pass keeps (group, discount)
    cells up to 1024 groups and one slot per group above."""
    comp, c, _ = table
    keys, _ = keys_for(num_groups, dist)
    for cutoff in [727000, 727600, 729999, 730089]:
        check(comp, keys, num_groups, cutoff, run_gpu(c, keys, num_groups, "shared_mem_per_thread", cutoff))


@pytest.mark.parametrize("num_groups", [4097, 8191, 12288, 65536])
@pytest.mark.parametrize("dist", ["uniform", "zipf"])
def test_two_paths_match_oracle(table, path, num_groups, dist):
    comp, c, _ = table
    keys, _ = keys_for(num_groups, dist)
    for cutoff in [727000, 727600, 729999, 730089]:
        check(comp, keys, num_groups, cutoff, run_gpu(c, keys, num_groups, "shared_mem_per_thread", cutoff))


@pytest.mark.parametrize("rows", [1, 31, 2047, 2048, 2049, 4097, 65_537])
def test_small_and_ragged(table, path, rows):
    comp, _, _ = table
    part = {k: (v[:rows].copy() if isinstance(v, np.ndarray) and len(v) == ROWS else v) for k, v in comp.items()}
    c, keep = device_cols(part)
    keys = gen_np.group_keys_uniform(SEED + rows, 0, rows, 65536)
    check(part, keys, 65536, 730089, run_gpu(c, keys, 65536, "shared_mem_per_thread", 730089))


@pytest.mark.parametrize("blocks", [1, 3])
@pytest.mark.parametrize("dist", ["uniform", "zipf"])
def test_few_ctas(table, path, blocks, dist):
    """Few CTAs: each walks many partitions in pass 2 (a table flush at every change) and stages
    every partition's records in pass 1."""
    comp, c, _ = table
    keys, _ = keys_for(65536, dist)
    check(comp, keys, 65536, 729999, run_gpu(c, keys, 65536, "shared_mem_per_thread", 729999, blocks=blocks))


def test_domain_edges(table, path):
    """Rows outside the slot tables' fast domain reduce straight into the accumulators."""
    comp, _, _ = table
    wide = widen(comp, 4242, frac=0.05)
    c, keep = device_cols(wide)
    for dist in ["uniform", "zipf"]:
        keys, _ = keys_for(40000, dist)
        for cutoff in [729999, 730089]:
            check(wide, keys, 40000, cutoff, run_gpu(c, keys, 40000, "shared_mem_per_thread", cutoff))


def test_key_out_of_range_is_reported(table, path):
    comp, c, _ = table
    keys, _ = keys_for(5000, "uniform")
    keys = keys.copy()
    keys[12345] = 5000
    with pytest.raises(q.Q1Error) as e:
        run_gpu(c, keys, 5000, "shared_mem_per_thread", 730089)
    assert e.value.status == 6


@pytest.mark.parametrize("path", ["partitioned", "auto"], indirect=True)
def test_crosses_segment_boundary(cuda, path):
    """2^27 + 4099 rows: two segments of the partitioned path. Same table as the global placement,
    and the counts add up to the rows that pass."""
    rows = (1 << 27) + 4099
    L = q.lib()
    stream = torch.cuda.current_stream()
    sh = ctypes.c_void_p(stream.cuda_stream)
    cols = {k: torch.empty(rows * w + 64, dtype=torch.uint8, device="cuda")
            for k, w in [("shipdate", 2), ("discount", 1), ("extendedprice", 4), ("tax", 1), ("quantity", 1)]}
    flags = torch.empty(4 * ((rows + 15) // 16) + 64, dtype=torch.uint8, device="cuda")
    out = _lib.CompressedHostOut()
    for k, t in cols.items():
        setattr(out, k, t.data_ptr())
    out.flags = flags.data_ptr()
    _lib.check(L.q1_generate_compressed_device(SEED + 9, 0, rows, 0, ctypes.byref(out), sh))
    c = _lib.CompressedColumns()
    for k, t in cols.items():
        setattr(c, k, t.data_ptr())
    G = 65536
    cdf = torch.from_numpy(zipf_cdf(G).view(np.int32).copy()).cuda()
    keys = torch.empty(rows + 16, dtype=torch.int32, device="cuda")
    scratch = torch.empty(int(L.q1_groupkey_scratch_bytes(G)) // 8 + 2, dtype=torch.int64, device="cuda")
    cutoff = 729999
    ship = cols["shipdate"][: 2 * rows].view(torch.int16).to(torch.int32)
    passing = int((ship <= cutoff - 727563).sum())
    del ship
    for cdf_arg in [None, cdf]:
        _lib.check(L.q1_generate_group_keys_device(SEED + 9, 0, rows, G,
                                                   None if cdf_arg is None else ctypes.c_void_p(cdf_arg.data_ptr()),
                                                   ctypes.c_void_p(keys.data_ptr()), sh))
        res = []
        for placement in ["shared_mem_per_thread", "global"]:
            o = torch.zeros(G * 12, dtype=torch.int64, device="cuda")
            _lib.check(L.q1_launch_groupkey(q.placement_id(placement), ctypes.byref(c), ctypes.c_void_p(keys.data_ptr()),
                                            G, rows, cutoff, None, ctypes.c_void_p(scratch.data_ptr()),
                                            ctypes.c_void_p(o.data_ptr()), sh))
            _lib.check(L.q1_sync_check(sh))
            res.append(o.cpu().numpy().view(np.uint64).reshape(G, 6, 2))
        assert np.array_equal(res[0], res[1])
        assert int(res[0][:, 0, 0].sum()) == passing and not res[0][:, 0, 1].any()


@pytest.mark.parametrize("num_groups", [64, 1000, 4096, 65536])
@pytest.mark.parametrize("blocks", [0, 1, 3])
def test_one_key_many_rows(table, monkeypatch, num_groups, blocks):
    """Most rows of one key, one discount and the largest quantity: one partition takes every record of a
    tile (several chunks a round), and one cell's count and quantity pass 65,536 and 2^16 many times
    over (the carries of a packed word). The other keys' rows fall on partial chunks of 1 to 257
    records."""
    comp, _, _ = table
    comp = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in comp.items()}
    n = len(comp["shipdate"])
    hot = num_groups - 1
    keys = np.full(n, hot, dtype=np.uint32)
    at = 1000
    for j, run in enumerate([1, 31, 32, 33, 255, 256, 257, 1500]):
        keys[at:at + run] = j * 7 % num_groups
        at += 20_011
    rest = keys == hot
    comp["quantity"][rest] = 255
    comp["discount"][rest] = 5
    c, keep = device_cols(comp)
    for forced in ["single", "partitioned"] if num_groups > 4096 else ["single"]:
        monkeypatch.setenv("Q1_GROUPKEY_PATH", forced)
        check(comp, keys, num_groups, 730089, run_gpu(c, keys, num_groups, "shared_mem_per_thread", 730089, blocks))


@pytest.mark.parametrize("num_groups,rows", [(3000, 1 << 25), (3500, (1 << 25) - 1), (3500, 1 << 25), (4096, (1 << 25) + 1),
                                             (4097, (3 << 19) - 1), (4097, 3 << 19), (65536, (3 << 19) + 1)])
@pytest.mark.parametrize("dist", ["uniform", "zipf"])
def test_path_choice_lines(table, monkeypatch, num_groups, rows, dist):
    """Rows around the lines from which the path is chosen on the device: the table over and over, for cutoffs that
    let no row, few rows and all rows pass."""
    monkeypatch.delenv("Q1_GROUPKEY_PATH", raising=False)
    comp, _, _ = table
    keys, _ = keys_for(num_groups, dist)
    whole, rest = divmod(rows, ROWS)

    def repeat(t, n):
        return torch.cat([t.view(-1, n // ROWS).repeat(whole, 1).view(-1), t[: rest * (n // ROWS)]])

    names = ["shipdate", "quantity", "discount", "tax", "extendedprice"]
    dev = {k: torch.from_numpy(np.ascontiguousarray(comp[k]).view(np.uint8).copy()).cuda() for k in names}
    dev = {k: repeat(t, t.numel()) for k, t in dev.items()}
    dkeys = torch.from_numpy(keys.astype(np.uint32).view(np.uint8).copy()).cuda()
    dkeys = repeat(dkeys, dkeys.numel())
    c = _lib.CompressedColumns()
    for k in names:
        setattr(c, k, dev[k].data_ptr())
    scratch = torch.zeros(int(q.lib().q1_groupkey_scratch_bytes(num_groups)) // 8 + 2, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for cutoff in [727000, 727600, 730089]:
        out = torch.zeros(num_groups * 12, dtype=torch.int64, device="cuda")
        _lib.check(q.lib().q1_launch_groupkey(3, ctypes.byref(c), dkeys.data_ptr(), num_groups, rows, cutoff, None,
                                              scratch.data_ptr(), out.data_ptr(), stream))
        _lib.check(q.lib().q1_sync_check(stream))
        got = q.decode_aggregates(out.cpu().numpy().view(np.uint64), num_groups)
        part = {k: (v[:rest] if isinstance(v, np.ndarray) and len(v) == ROWS else v) for k, v in comp.items()}
        want = whole * q.decode_aggregates(O.q1_groupkey(comp, keys, num_groups, cutoff)[0], num_groups)
        want = want + q.decode_aggregates(O.q1_groupkey(part, keys[:rest], num_groups, cutoff)[0], num_groups)
        assert np.array_equal(got, want), cutoff


@pytest.mark.parametrize("num_groups", [5000, 65536])
@pytest.mark.parametrize("blocks", [0, 1, 3])
def test_path_choice_with_few_ctas_and_domain_edges(table, monkeypatch, num_groups, blocks):
    """The choice on the device, on a table large enough for it, in few CTAs and with rows outside the tables'
    fast domain; a key out of range is reported whatever path is taken."""
    monkeypatch.delenv("Q1_GROUPKEY_PATH", raising=False)
    comp, _, _ = table
    comp = {k: np.tile(comp[k], 5) for k in ["shipdate", "quantity", "discount", "tax", "extendedprice"]}
    assert len(comp["shipdate"]) > 3 << 19
    wide = widen(comp, 77, frac=0.02)
    c, keep = device_cols(wide)
    for dist in ["uniform", "zipf"]:
        keys = np.tile(keys_for(num_groups, dist)[0], 5)
        for cutoff in [727600, 729999]:
            check(wide, keys, num_groups, cutoff, run_gpu(c, keys, num_groups, "shared_mem_per_thread", cutoff, blocks))
        keys[123_456] = num_groups
        for cutoff in [727600, 740000]:
            if cutoff == 740000 or wide["shipdate"][123_456] <= cutoff - 727563:
                with pytest.raises(q.Q1Error) as e:
                    run_gpu(c, keys, num_groups, "shared_mem_per_thread", cutoff, blocks)
                assert e.value.status == 6


@pytest.mark.parametrize("rows", [20_011, 300_007, 1_000_003])
def test_frequent_large_keys_take_no_longer(cuda, monkeypatch, rows):
    """65,536 groups: tables whose rows are nearly all of one key, or of eight, that the single pass has no slot
    for, against spread keys (4 times allowed; 1.0 M rows of one key took 78 times as long in the single pass)."""
    monkeypatch.delenv("Q1_GROUPKEY_PATH", raising=False)
    groups = 65536
    comp = gen_np.compress(gen_np.generate(SEED + 40, 0, rows))
    c, keep = device_cols(comp)
    out = torch.zeros(groups * 12, dtype=torch.int64, device="cuda")
    scratch = torch.zeros(int(q.lib().q1_groupkey_scratch_bytes(groups)) // 8 + 2, dtype=torch.int64, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def best(keys):
        d = torch.from_numpy(keys.astype(np.uint32).view(np.int32).copy()).cuda()
        times = []
        for _ in range(8):
            out.zero_()
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda._sleep(200_000)   # the launches are queued before the first begins
            ev[0].record()
            _lib.check(q.lib().q1_launch_groupkey(3, ctypes.byref(c), ctypes.c_void_p(d.data_ptr()), groups, rows, 740000,
                                                  None, ctypes.c_void_p(scratch.data_ptr()),
                                                  ctypes.c_void_p(out.data_ptr()), stream))
            ev[1].record()
            _lib.check(q.lib().q1_sync_check(stream))
            times.append(ev[0].elapsed_time(ev[1]))
        check(comp, keys, groups, 740000, out.cpu().numpy().view(np.uint64))
        return min(times)

    spread = gen_np.group_keys_uniform(SEED + 41, 0, rows, groups)
    one = np.where(np.arange(rows) % 10, 50_000, spread).astype(np.uint32)
    eight = (spread & 7) * 8000 + 5000
    t = [best(k) for k in [spread, one, eight.astype(np.uint32)]]
    assert t[1] < 4 * t[0] and t[2] < 4 * t[0], t
