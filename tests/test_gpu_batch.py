"""Batched aggregation (q1_batch_*): many instances in one persistent kernel over a device tile
queue, replayed as a CUDA graph, placements chosen by the autotuner. Every instance's result
must equal the oracle and the plain per-instance launch (q1_launch_groupkey) bit for bit."""
import ctypes
import os

import numpy as np
import pytest
import torch

import gen_np
import tpchq01_gpu_b200 as q
from oracle import py_oracle as O
from tpchq01_gpu_b200 import _lib

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 100, 2047, 2048, 2049, 4096 + 3, 10_000, 65_537, 300_011, 1_000_003]
GROUPS = [1, 4, 8, 64, 1024, 3000]


def make_instances(seed=77, n=30):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        rows = SIZES[i % len(SIZES)]
        g = GROUPS[(i * 7) % len(GROUPS)]
        cutoff = int(rng.integers(729906, 730090)) if i % 5 else [727000, 740000, 728826, 729999, 729906][(i // 5) % 5]
        cols = gen_np.generate(seed * 1000 + i, 0, rows)
        comp = gen_np.compress(cols)
        if i % 7 == 3 and rows:
            # rows at the edges of the compressed domain: the shared tables' exact slow path
            r2 = np.random.default_rng(i)
            idx = r2.choice(rows, max(1, rows // 20), replace=False)
            comp["discount"][idx] = r2.integers(0, 101, len(idx))
            comp["tax"][idx] = r2.integers(0, 256, len(idx))
            comp["extendedprice"][idx] = r2.integers(0, 2**32, len(idx), dtype=np.uint64).astype(np.uint32)
            comp["quantity"][idx] = r2.integers(0, 256, len(idx))
        keys = gen_np.group_keys_uniform(seed * 1000 + i, 0, rows, g)
        out.append((comp, keys, g, cutoff))
    return out


def to_device(instances):
    keep, descs, outs = [], [], []
    for comp, keys, g, cutoff in instances:
        rows = len(keys)
        d = {k: torch.from_numpy(np.ascontiguousarray(comp[k]).view(np.uint8).copy()).cuda()
             for k in ["shipdate", "discount", "extendedprice", "tax", "quantity"]}
        d["keys"] = torch.from_numpy(np.ascontiguousarray(keys).view(np.uint8).copy()).cuda()
        out = torch.zeros(g * 12 + 2, dtype=torch.int64, device="cuda")
        bi = _lib.BatchInstance()
        for k in ["shipdate", "discount", "extendedprice", "tax", "quantity"]:
            setattr(bi.cols, k, d[k].data_ptr())
        bi.keys = d["keys"].data_ptr()
        bi.rows = rows
        bi.cutoff_day = cutoff
        bi.num_groups = g
        bi.aggregates = out.data_ptr()
        keep.append(d)
        descs.append(bi)
        outs.append(out)
    arr = (_lib.BatchInstance * len(descs))(*descs)
    return arr, outs, keep


def oracle_tables(instances):
    res = []
    for comp, keys, g, cutoff in instances:
        buf, flag = O.q1_groupkey(comp, keys, g, cutoff)
        assert flag == 0
        res.append(buf)
    return res


def read(out, g):
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint64)[: g * 12]


def run_batch(arr, n, opts, stream, runs=2):
    b = ctypes.c_void_p()
    _lib.check(q.lib().q1_batch_create(arr, n, ctypes.byref(opts), ctypes.c_void_p(stream), ctypes.byref(b)))
    try:
        for _ in range(runs):
            _lib.check(q.lib().q1_batch_run(b, ctypes.c_void_p(stream)))
        _lib.check(q.lib().q1_sync_check(ctypes.c_void_p(stream)))
        desc = _lib.BatchDesc()
        _lib.check(q.lib().q1_batch_describe(b, ctypes.byref(desc)))
        modes = []
        for i in range(n):
            m = ctypes.c_int32(-1)
            _lib.check(q.lib().q1_batch_instance_mode(b, i, ctypes.byref(m)))
            modes.append(m.value)
        return desc, modes
    finally:
        q.lib().q1_batch_destroy(b)


@pytest.fixture(scope="module")
def data(cuda):
    inst = make_instances()
    return inst, oracle_tables(inst)


@pytest.mark.parametrize("use_graph", [1, 0])
@pytest.mark.parametrize("chunk", [0, 1, 7])
def test_batch_equals_oracle(data, use_graph, chunk):
    inst, want = data
    arr, outs, keep = to_device(inst)
    opts = _lib.BatchOpts(use_graph, 0, chunk, 0, None)
    stream = torch.cuda.current_stream().cuda_stream
    desc, modes = run_batch(arr, len(inst), opts, stream)   # two runs: outputs are overwritten, not doubled
    assert desc.instances == len(inst) and desc.uses_graph == use_graph
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        assert np.array_equal(read(outs[i], g), want[i]), f"instance {i} (rows={len(keys)}, groups={g})"


def test_batch_accumulate_mode(data):
    inst, want = data
    arr, outs, keep = to_device(inst)
    opts = _lib.BatchOpts(1, 1, 0, 0, None)
    stream = torch.cuda.current_stream().cuda_stream
    run_batch(arr, len(inst), opts, stream, runs=2)
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        got = q.decode_aggregates(read(outs[i], g), g)
        assert np.array_equal(got, 2 * q.decode_aggregates(want[i], g))


def test_autotuner_modes_cache_and_parity(data, tmp_path):
    inst, want = data
    arr, outs, keep = to_device(inst)
    cache = str(tmp_path / "tune.txt")
    stream = torch.cuda.current_stream().cuda_stream
    desc, modes = run_batch(arr, len(inst), _lib.BatchOpts(1, 0, 0, 2, cache.encode()), stream)
    assert os.path.exists(cache) and desc.tuned_classes > 0
    text = open(cache).read()
    assert "mode " in text and "chunk " in text
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        assert modes[i] in (0, 1, 2)
        if g > 4:
            assert modes[i] != 0
        assert np.array_equal(read(outs[i], g), want[i])
    # second batch reuses the cache: no class is measured again
    arr2, outs2, keep2 = to_device(inst)
    desc2, modes2 = run_batch(arr2, len(inst), _lib.BatchOpts(1, 0, 0, 1, cache.encode()), stream)
    assert desc2.tuned_classes == 0 and modes2 == modes
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        assert np.array_equal(read(outs2[i], g), want[i])


def test_batch_equals_plain_launches(data):
    """One launch per instance (q1_launch_groupkey) gives the same tables as the batch."""
    inst, want = data
    arr, outs, keep = to_device(inst)
    stream = torch.cuda.current_stream().cuda_stream
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        rows = len(keys)
        out = torch.zeros(g * 12 + 2, dtype=torch.int64, device="cuda")
        scratch = torch.zeros(int(q.lib().q1_groupkey_scratch_bytes(g)) // 8 + 2, dtype=torch.int64, device="cuda")
        placement = 1 if g <= 8 else 3
        _lib.check(q.lib().q1_launch_groupkey(placement, ctypes.byref(arr[i].cols), ctypes.c_void_p(arr[i].keys), g,
                                              rows, cutoff, None, ctypes.c_void_p(scratch.data_ptr()),
                                              ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(stream)))
        _lib.check(q.lib().q1_sync_check(ctypes.c_void_p(stream)))
        assert np.array_equal(read(out, g), want[i])


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shared", [False, True])
def test_batch_tables_are_stored_or_summed(cuda, shared, offset):
    """Each run overwrites what the tables held (empty groups too); instances that share a table sum in it. Tables
    start at any 8-byte boundary."""
    inst = [i for i in make_instances(seed=91, n=24) if i[2] in (4, 64, 1024)]
    arr, outs, keep = to_device(inst)
    table = {}
    for i, w in enumerate(oracle_tables(inst)):
        g = inst[i][2]
        t = g if shared else i   # a table per group count, or per instance
        table.setdefault(t, [outs[i].fill_(-7), 0])
        table[t][1] = table[t][1] + q.decode_aggregates(w, g)
        arr[i].aggregates = table[t][0].data_ptr() + 8 * offset
    stream = torch.cuda.current_stream().cuda_stream
    run_batch(arr, len(inst), _lib.BatchOpts(1, 0, 0, 0, None), stream)
    for t, (out, total) in table.items():
        g = t if shared else inst[t][2]
        got = q.decode_aggregates(out.cpu().numpy().view(np.uint64)[offset : offset + g * 12], g)
        assert np.array_equal(got, total), (t, g)


@pytest.mark.parametrize("chunk", [0, 1])
def test_batch_many_small_instances(cuda, chunk):
    """Rows at the edges of a ring tile and of a team's turn, more instances per CTA than it keeps run descriptors
    for, and every engine (the cells, the slots and, from a cache file, the global one) in the same CTAs."""
    rows = [1, 1023, 1024, 1025, 2048, 2049, 3072, 3073, 5 * 1024 + 7]
    groups = [1, 4, 64, 65, 1024, 1025, 3000]
    inst = []
    for i in range(63):
        n, g = rows[i % len(rows)], groups[i % len(groups)]
        comp = gen_np.compress(gen_np.generate(4000 + i, 0, n))
        inst.append((comp, gen_np.group_keys_uniform(4000 + i, 0, n, g), g, 729999))
    want = oracle_tables(inst)
    arr, outs, keep = to_device(inst)
    copies = 45   # 2835 instances
    big = (_lib.BatchInstance * (len(inst) * copies))(*[arr[i % len(inst)] for i in range(len(inst) * copies)])
    tables = []
    for i in range(len(big)):
        tables.append(torch.full((inst[i % len(inst)][2] * 12,), 5, dtype=torch.int64, device="cuda"))
        big[i].aggregates = tables[i].data_ptr()
    stream = torch.cuda.current_stream().cuda_stream
    run_batch(big, len(big), _lib.BatchOpts(1, 0, chunk, 0, None), stream)
    torch.cuda.synchronize()
    for i in range(len(big)):
        got = tables[i].cpu().numpy().view(np.uint64)
        assert np.array_equal(got, want[i % len(inst)]), (i, inst[i % len(inst)][2], len(inst[i % len(inst)][1]))


def test_batch_modes_from_a_cache_file(cuda, tmp_path):
    """Placements read from a cache file: global for some classes; 0, an earlier file's register placement, is the
    shared table."""
    inst = []
    for i, (n, g) in enumerate([(5000, 4), (5000, 64), (70001, 65), (70001, 3000), (5000, 1), (70001, 1024)]):
        comp = gen_np.compress(gen_np.generate(4100 + i, 0, n))
        inst.append((comp, gen_np.group_keys_uniform(4100 + i, 0, n, g), g, 740000))
    want = oracle_tables(inst)
    arr, outs, keep = to_device(inst)
    mode = [0, 2, 2, 1, 2, 0]
    cache = tmp_path / "tune.txt"
    lines = [f"mode {int(np.log2(len(k)))} {g} 10 {m}" for (c, k, g, d), m in zip(inst, mode)]
    cache.write_text("# cache\n" + "\n".join(lines) + "\n")
    stream = torch.cuda.current_stream().cuda_stream
    desc, modes = run_batch(arr, len(inst), _lib.BatchOpts(1, 0, 0, 1, str(cache).encode()), stream)
    assert modes == [m or 1 for m in mode] and desc.tuned_classes == 0
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        assert np.array_equal(read(outs[i], g), want[i]), (i, g)


def few_group_columns(kind, rows, seed):
    """Columns of instances of up to four groups: ordinary, all rows alike, over the whole compressed
    domain, or all at its upper edge."""
    comp = gen_np.compress(gen_np.generate(seed, 0, rows))
    r = np.random.default_rng(seed)
    if kind == "alike":
        for k, v in [("quantity", 50), ("discount", 5), ("tax", 5), ("extendedprice", 10_494_950), ("shipdate", 7)]:
            comp[k][:] = v
    elif kind == "domain":
        comp["discount"][:] = r.integers(0, 101, rows)
        comp["tax"][:] = r.integers(0, 256, rows)
        comp["extendedprice"][:] = r.integers(0, 2**32, rows, dtype=np.uint64).astype(np.uint32)
        comp["quantity"][:] = r.integers(0, 256, rows)
        comp["shipdate"][:] = r.integers(0, 32768, rows)
    elif kind == "edge":
        for k, v in [("quantity", 255), ("discount", 0), ("tax", 255), ("extendedprice", 0xFFFFFFFF), ("shipdate", 32767)]:
            comp[k][:] = v
    return comp


@pytest.mark.parametrize("chunk", [0, 1])
@pytest.mark.parametrize("kind", ["ordinary", "alike", "domain", "edge"])
def test_batch_of_few_groups(cuda, kind, chunk):
    """One to five groups, rows at the edges of a ring tile and of a team's turn, one key for nearly all rows or
    keys spread evenly, beside instances of the other engines."""
    inst = []
    for i, rows in enumerate([1, 255, 256, 1023, 1024, 1025, 2 * 1024 + 7, 3 * 1024, 50_001, 300_011]):
        for g in [1, 2, 3, 4, 5, 64, 1000]:
            keys = gen_np.group_keys_uniform(600 + i, 0, rows, g)
            if (i + g) % 2:
                keys[rows // 10:] = g - 1
            inst.append((few_group_columns(kind, rows, 5000 + 10 * i + g), keys, g, [729999, 760330][i % 2]))
    want = oracle_tables(inst)
    arr, outs, keep = to_device(inst)
    stream = torch.cuda.current_stream().cuda_stream
    run_batch(arr, len(inst), _lib.BatchOpts(1, 0, chunk, 0, None), stream)
    for i, (comp, keys, g, cutoff) in enumerate(inst):
        assert np.array_equal(read(outs[i], g), want[i]), (len(keys), g)


def test_few_group_key_out_of_range_is_reported(cuda):
    inst = make_instances(seed=12, n=30)
    inst = [x for x in inst if x[2] == 4 and len(x[1]) > 1000][:1]
    comp, keys, g, _ = inst[0]
    keys = keys.copy()
    keys[len(keys) // 2] = 4
    arr, outs, keep = to_device([(comp, keys, g, 740000)])
    stream = torch.cuda.current_stream().cuda_stream
    with pytest.raises(q.Q1Error) as e:
        run_batch(arr, 1, _lib.BatchOpts(1, 0, 0, 0, None), stream)
    assert e.value.status == 6


@pytest.fixture(scope="module")
def alike_rows(cuda):
    """18 million rows for every SM, all alike: each CTA gets more than 2^24 of them."""
    n = 18_000_003 * torch.cuda.get_device_properties(0).multi_processor_count
    cols = {k: torch.full((n,), v, dtype=d, device="cuda") for k, v, d in [
        ("shipdate", 7, torch.int16), ("quantity", 255, torch.uint8), ("discount", 0, torch.uint8),
        ("tax", 0, torch.uint8), ("extendedprice", 0, torch.int32)]}
    cols["keys"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    return n, cols


@pytest.mark.parametrize("num_groups,price,discount,tax", [
    (1, (1 << 24) - 1, 10, 8), (4, (1 << 24) - 1, 10, 8), (64, (1 << 24) - 1, 10, 8), (1024, (1 << 24) - 1, 10, 8),
    (2500, (1 << 24) - 1, 10, 8), (1, (1 << 32) - 1, 0, 255), (4, (1 << 32) - 1, 0, 255)])
def test_batch_flushes_within_an_instance(alike_rows, num_groups, price, discount, tax):
    """More than 2^24 rows of one instance in every CTA, all of one cell with the largest quantity: without a
    flush after at most 2^23 of them, the cell's 32-bit quantity would wrap. Of up to four groups also with
    values outside the cells' domain: without a flush after 2^21 of them, the slots' words would."""
    n, cols = alike_rows
    key = num_groups - 1
    cols["keys"].fill_(key)
    cols["discount"].fill_(discount)
    cols["tax"].fill_(tax)
    cols["extendedprice"].fill_(price if price < 1 << 31 else price - (1 << 32))
    out = torch.zeros(num_groups * 12, dtype=torch.int64, device="cuda")
    bi = (_lib.BatchInstance * 1)()
    for k in ["shipdate", "discount", "extendedprice", "tax", "quantity"]:
        setattr(bi[0].cols, k, cols[k].data_ptr())
    bi[0].keys, bi[0].rows, bi[0].cutoff_day, bi[0].num_groups = cols["keys"].data_ptr(), n, 729999, num_groups
    bi[0].aggregates = out.data_ptr()
    stream = torch.cuda.current_stream().cuda_stream
    run_batch(bi, 1, _lib.BatchOpts(1, 0, 0, 0, None), stream, runs=1)
    got = q.decode_aggregates(read(out, num_groups), num_groups)
    dp = (100 - discount) * price
    want = np.zeros((num_groups, 6), dtype=object)
    want[key] = [n, n * 25500, n * price, n * discount, n * dp, n * dp * (100 + tax)]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("num_groups", [1, 2, 4])
def test_few_groups_take_no_longer_for_rows_alike(cuda, num_groups):
    """The time of an instance of up to four groups does not hang on its values: rows of one key, discount and tax,
    and rows of any discount and tax, against ordinary ones (1.5 times allowed; cells that all rows add to took
    2.7 times)."""
    rows = 20_000_001
    g = torch.Generator(device="cuda")
    g.manual_seed(3)

    def column(lo, hi, dtype):
        return torch.randint(lo, hi, (rows,), generator=g, device="cuda", dtype=dtype)

    cols = {"shipdate": column(0, 2500, torch.int16), "quantity": column(1, 51, torch.uint8),
            "discount": column(0, 11, torch.uint8), "tax": column(0, 9, torch.uint8),
            "extendedprice": column(90_000, 10_494_950, torch.int32), "keys": column(0, num_groups, torch.int32)}
    out = torch.zeros(num_groups * 12, dtype=torch.int64, device="cuda")
    bi = (_lib.BatchInstance * 1)()
    for k in ["shipdate", "discount", "extendedprice", "tax", "quantity"]:
        setattr(bi[0].cols, k, cols[k].data_ptr())
    bi[0].keys, bi[0].rows, bi[0].cutoff_day, bi[0].num_groups = cols["keys"].data_ptr(), rows, 729999, num_groups
    bi[0].aggregates = out.data_ptr()
    stream = torch.cuda.current_stream()
    b = ctypes.c_void_p()
    opts = _lib.BatchOpts(1, 0, 0, 0, None)
    _lib.check(q.lib().q1_batch_create(bi, 1, ctypes.byref(opts), ctypes.c_void_p(stream.cuda_stream), ctypes.byref(b)))

    def best():
        times = []
        for _ in range(12):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for _ in range(5):
                _lib.check(q.lib().q1_batch_run(b, ctypes.c_void_p(stream.cuda_stream)))
            ev[1].record()
            torch.cuda.synchronize()
            times.append(ev[0].elapsed_time(ev[1]))
        return min(times)
    try:
        ordinary = best()
        cols["tax"].copy_(column(0, 256, torch.int32))
        cols["discount"].copy_(column(0, 101, torch.int32))
        any_value = best()
        cols["tax"].fill_(5)
        cols["discount"].fill_(5)
        cols["keys"].fill_(0)
        alike = best()
        _lib.check(q.lib().q1_sync_check(ctypes.c_void_p(stream.cuda_stream)))
    finally:
        torch.cuda.synchronize()
        q.lib().q1_batch_destroy(b)
    assert any_value < 1.5 * ordinary and alike < 1.5 * ordinary, (ordinary, any_value, alike)


@pytest.mark.parametrize("num_groups", [65, 97, 500, 1023, 1024])
def test_batch_cells_of_spaced_keys(cuda, num_groups):
    """Keys of every step-th group: the (group, discount) cells' groups' words lie in an order of their own."""
    rows = 100_003
    inst = []
    for step in [1, 32, 128]:
        comp = gen_np.compress(gen_np.generate(700 + step, 0, rows))
        inst.append((comp, gen_np.group_keys_uniform(700 + step, 0, rows, num_groups) // step * step, num_groups, 740000))
    want = oracle_tables(inst)
    arr, outs, keep = to_device(inst)
    run_batch(arr, len(inst), _lib.BatchOpts(1, 0, 0, 0, None), torch.cuda.current_stream().cuda_stream)
    for i in range(len(inst)):
        assert np.array_equal(read(outs[i], num_groups), want[i])


def test_cells_of_spaced_keys_take_no_longer(cuda):
    """1024 groups, the keys multiples of 128, against spread keys (1.5 times allowed; with the groups' words in the
    order of the groups, and so in one bank, 2.1 times)."""
    rows, groups = 60_000_001, 1024
    g = torch.Generator(device="cuda")
    g.manual_seed(4)

    def column(lo, hi, dtype):
        return torch.randint(lo, hi, (rows,), generator=g, device="cuda", dtype=dtype)

    cols = {"shipdate": column(0, 2500, torch.int16), "quantity": column(1, 51, torch.uint8),
            "discount": column(0, 11, torch.uint8), "tax": column(0, 9, torch.uint8),
            "extendedprice": column(90_000, 10_494_950, torch.int32), "keys": column(0, groups, torch.int32)}
    out = torch.zeros(groups * 12, dtype=torch.int64, device="cuda")
    bi = (_lib.BatchInstance * 1)()
    for k in ["shipdate", "discount", "extendedprice", "tax", "quantity"]:
        setattr(bi[0].cols, k, cols[k].data_ptr())
    bi[0].keys, bi[0].rows, bi[0].cutoff_day, bi[0].num_groups = cols["keys"].data_ptr(), rows, 729999, groups
    bi[0].aggregates = out.data_ptr()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    b = ctypes.c_void_p()
    opts = _lib.BatchOpts(1, 0, 0, 0, None)
    _lib.check(q.lib().q1_batch_create(bi, 1, ctypes.byref(opts), stream, ctypes.byref(b)))

    def best():
        times = []
        for _ in range(8):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for _ in range(3):
                _lib.check(q.lib().q1_batch_run(b, stream))
            ev[1].record()
            torch.cuda.synchronize()
            times.append(ev[0].elapsed_time(ev[1]))
        return min(times)
    try:
        spread = best()
        cols["keys"].copy_(cols["keys"] % 8 * 128)
        spaced = best()
        _lib.check(q.lib().q1_sync_check(stream))
    finally:
        torch.cuda.synchronize()
        q.lib().q1_batch_destroy(b)
    assert spaced < 1.5 * spread, (spread, spaced)


@pytest.mark.parametrize("chunk", [1, 7, 1000, 100_000])
def test_describe_reports_the_chunk_asked_for(cuda, chunk):
    """Also one larger than any instance, or than a work item may be; without one, the largest piece."""
    inst = [x for x in make_instances(seed=5, n=30) if len(x[1])]
    arr, outs, keep = to_device(inst)
    stream = torch.cuda.current_stream().cuda_stream
    desc, _ = run_batch(arr, len(inst), _lib.BatchOpts(1, 0, chunk, 0, None), stream, runs=1)
    assert desc.chunk_tiles == chunk
    desc, _ = run_batch(arr, len(inst), _lib.BatchOpts(1, 0, 0, 0, None), stream, runs=1)
    assert 1 <= desc.chunk_tiles <= max(-(-len(k) // 2048) for _, k, _, _ in inst)
