"""Performance cases: the work a user of this framework has it do, through its public entry points.

Six kinds of work, each over the range of sizes and options it is used with:

  query     Q1Context.run on a loaded table: the reference's whole query, from the zeroed aggregates
            to the result on the host, over a table in HBM or streamed from pinned host memory
  scan      launch_compressed / launch_uncompressed on caller-owned device columns, any table
            placement, flag packing and filter pushdown (with the bitmap made in the same pass)
  groupkey  q1_launch_groupkey: group by a uint32 key, uniform or Zipf, 2 to 65,536 groups
  batch     q1_batch_run: many independent group-key tables in one execution of a prepared batch
  tbl       q1_tbl_parse_device: dbgen lineitem text to reference-typed columns
  serve     q1_server_submit / q1_server_wait: a burst of mixed requests to a running server

Tables are made on the GPU from the seed with TPC-H lineitem's distributions (dates, flags derived
from them, quantity 1-50, price = quantity x unit price, discount 0-10 %, tax 0-8 %).
"""
import ctypes
import math

import numpy as np
import torch

import tpchq01_gpu_b200 as q
from tpchq01_gpu_b200 import _lib

FRAME = 727563                         # day number of 1992-01-01
CURRENT_DAY = 728826 - FRAME           # 1995-06-17: decides the return flag and the line status
LAST_ORDER = 729968 - FRAME            # 1998-08-02
CUTOFF = 729999                        # l_shipdate <= 1998-09-02, 98 % of the rows
PAIR_GROUPS = [0, 2, 3, 4]             # A/F, N/F, N/O, R/F
CHUNK = 1 << 24                        # rows made or summed at a time
# lineitem's row counts at TPC-H scale factors 0.01, 1, 10 and 100
SF001, SF1, SF10, SF100 = 60_175, 6_001_215, 59_986_052, 600_037_902
LAYOUT_BYTES = {("pair", False): 9.25, ("pair", True): 7.375, ("separate", False): 9.375,
                ("separate", True): 7.5, ("uncompressed", False): 38.0}


def listed():
    return [
        # The smallest query: the default placement over SF 0.01 in HBM. Latency of one call.
        {"name": "query_sf001", "kind": "query", "rows": SF001, "residency": "hbm", "packing": "pair",
         "placement": "in_registers_per_thread", "pushdown": False, "cutoff": CUTOFF},
        # The reference's own mode of work: the table stays in host memory and every query streams it.
        {"name": "query_sf10_streamed", "kind": "query", "rows": SF10, "residency": "pinned", "packing": "pair",
         "placement": "in_registers_per_thread", "pushdown": False, "cutoff": CUTOFF},
        # The reference's default input: uncompressed, reference-typed columns, SF 1.
        {"name": "scan_sf1_uncompressed", "kind": "scan", "rows": SF1, "packing": "uncompressed",
         "placement": "in_registers_per_thread", "pushdown": False, "cutoff": CUTOFF},
        # The reference's compressed layout (separate flags) with filter pushdown, SF 10.
        {"name": "scan_sf10_pushdown", "kind": "scan", "rows": SF10, "packing": "separate",
         "placement": "in_registers_per_thread", "pushdown": True, "cutoff": CUTOFF},
        # A table placement other than the default one (the reference's users compare all five), SF 10.
        {"name": "scan_sf10_shared", "kind": "scan", "rows": SF10, "packing": "pair",
         "placement": "shared_mem_per_thread", "pushdown": False, "cutoff": CUTOFF},
        # The headline: one scan of SF 100 in HBM, default placement, 2-bit pair codes. The largest.
        {"name": "scan_sf100", "kind": "scan", "rows": SF100, "packing": "pair",
         "placement": "in_registers_per_thread", "pushdown": False, "cutoff": CUTOFF},
        # Group by a key of few values (cells of the shared-memory table), half of the rows passing.
        {"name": "groupkey_64", "kind": "groupkey", "rows": 100_000_003, "groups": 64, "zipf": False,
         "placement": "shared_mem_per_thread", "cutoff": 728826},
        # A few thousand keys with the skew of real keys (Zipf), an ordinary table.
        {"name": "groupkey_4096_zipf", "kind": "groupkey", "rows": SF10, "groups": 4096, "zipf": True,
         "placement": "shared_mem_per_thread", "cutoff": CUTOFF},
        # The most groups the key can have, spread evenly: nothing fits one table.
        {"name": "groupkey_65536", "kind": "groupkey", "rows": 200_000_033, "groups": 65536, "zipf": False,
         "placement": "shared_mem_per_thread", "cutoff": CUTOFF},
        # Many small and middling tables of mixed group counts in one prepared batch.
        {"name": "batch_64", "kind": "batch", "instances": 64, "min_rows": 10_000, "max_rows": 10_000_000},
        # Loading SF 1 from dbgen text that is in device memory.
        {"name": "tbl_sf1", "kind": "tbl", "rows": SF1},
        # A burst of requests at a server: half on its resident table, half on ad-hoc tables.
        {"name": "serve_64", "kind": "serve", "requests": 64, "resident_rows": SF1, "tables": 16,
         "min_rows": 100_000, "max_rows": 4_000_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "scan", "scan", "scan", "groupkey", "groupkey", "groupkey", "batch", "tbl", "serve"])
    cutoff = rng.choice([CUTOFF, CUTOFF, rng.randrange(FRAME, 730090)])
    placements = ["in_registers", "in_registers_per_thread", "local_mem", "shared_mem_per_thread", "global"]
    if kind == "query":
        residency = rng.choice(["hbm", "hbm", "pinned"])
        return {"kind": kind, "rows": _log_int(rng, 1_000, SF10), "residency": residency,
                "packing": rng.choice(["pair", "separate"]), "placement": rng.choice(placements),
                "pushdown": residency == "hbm" and rng.random() < 0.3, "cutoff": cutoff}
    if kind == "scan":
        packing = rng.choice(["pair", "pair", "separate", "separate", "uncompressed"])
        placement = rng.choice(placements + ["in_registers_per_thread"] * 4)
        top = SF100 if (packing, placement) == ("pair", "in_registers_per_thread") else SF10
        return {"kind": kind, "rows": _log_int(rng, 10_000, top if packing != "uncompressed" else SF10 // 2),
                "packing": packing, "placement": placement,
                "pushdown": packing != "uncompressed" and rng.random() < 0.3, "cutoff": cutoff}
    if kind == "groupkey":
        groups = _log_int(rng, 2, 65536)
        placement = "in_registers_per_thread" if groups <= 8 and rng.random() < 0.7 else "shared_mem_per_thread"
        return {"kind": kind, "rows": _log_int(rng, 100_000, 200_000_000), "groups": groups,
                "zipf": rng.random() < 0.4, "placement": placement, "cutoff": cutoff}
    if kind == "batch":
        low = _log_int(rng, 1_000, 50_000)
        return {"kind": kind, "instances": rng.randrange(4, 65), "min_rows": low,
                "max_rows": _log_int(rng, 8 * low, 10_000_000)}
    if kind == "tbl":
        return {"kind": kind, "rows": _log_int(rng, 10_000, SF1)}
    return {"kind": "serve", "requests": rng.randrange(8, 65), "resident_rows": _log_int(rng, 100_000, SF1),
            "tables": rng.randrange(2, 17), "min_rows": 50_000, "max_rows": _log_int(rng, 200_000, 4_000_000)}


# ---------------------------------------------------------------------------------------------
# Tables
# ---------------------------------------------------------------------------------------------

def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _rows(n, gen):
    """n lineitem rows: ship (days since 1992-01-01), quantity, discount, tax, price, group."""
    def uniform(lo, hi, dtype):
        return torch.randint(lo, hi, (n,), generator=gen, device="cuda", dtype=dtype)
    ship = uniform(0, LAST_ORDER + 1, torch.int16) + uniform(1, 122, torch.int16)
    receipt = ship + uniform(1, 31, torch.int16)
    quantity = uniform(1, 51, torch.uint8)
    price = uniform(90_000, 209_900, torch.int32) * quantity
    returned = uniform(0, 2, torch.uint8) * 2                       # A or R
    rf = torch.where(receipt <= CURRENT_DAY, returned, torch.ones_like(returned))
    group = rf * 2 + (ship > CURRENT_DAY).to(torch.uint8)
    return {"ship": ship, "quantity": quantity, "discount": uniform(0, 11, torch.uint8),
            "tax": uniform(0, 9, torch.uint8), "price": price, "group": group}


def _pack(codes, bits, out, row0):
    """codes (uint8, fewer than 2^bits) into the LSB-first bit container `out` (bytes) from row0 on."""
    per = 8 // bits
    pad = (-len(codes)) % per
    if pad:
        codes = torch.cat([codes, codes.new_zeros(pad)])
    c = codes.view(-1, per)
    b = c[:, 0].clone()
    for i in range(1, per):
        b |= c[:, i] << (bits * i)
    out[row0 // per:row0 // per + len(b)] = b


def _zipf_keys(n, groups, gen):
    p = 1.0 / np.arange(1, groups + 1, dtype=np.float64)
    cdf = torch.from_numpy(np.cumsum(p) / p.sum()).cuda()
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    return torch.searchsorted(cdf, u).clamp_(max=groups - 1).to(torch.int32)


def _chunks(rows, seed, salt=0, groups=0, zipf=False):
    """The table in chunks: (first row, columns), with a key column when groups > 0."""
    gen = _generator(seed, salt)
    for r0 in range(0, rows, CHUNK):
        n = min(CHUNK, rows - r0)
        t = _rows(n, gen)
        if groups:
            t["key"] = (_zipf_keys(n, groups, gen) if zipf else
                        torch.randint(0, groups, (n,), generator=gen, device="cuda", dtype=torch.int32))
        yield r0, t


class _Table:
    """Compressed (or reference-typed) device columns as a user holds them, and their C view."""

    def __init__(self, case, seed, packing, salt=0, rows=0, groups=0, zipf=False, filter_words=False):
        n = rows or case["rows"]
        self.rows, self.keys = n, None
        words = (n + 127) // 128 * 4

        def column(dtype, length=n):
            return torch.zeros(length, dtype=dtype, device="cuda")
        if packing == "uncompressed":
            c = {"shipdate": column(torch.int32), "discount": column(torch.int64),
                 "extendedprice": column(torch.int64), "tax": column(torch.int64), "quantity": column(torch.int64),
                 "returnflag": column(torch.uint8), "linestatus": column(torch.uint8)}
            letters = torch.tensor([ord("A"), ord("N"), ord("R")], dtype=torch.uint8, device="cuda")
            for r0, t in _chunks(n, seed, salt):
                s = slice(r0, r0 + len(t["ship"]))
                c["shipdate"][s] = t["ship"].to(torch.int32) + FRAME
                c["discount"][s] = t["discount"].to(torch.int64)
                c["extendedprice"][s] = t["price"].to(torch.int64)
                c["tax"][s] = t["tax"].to(torch.int64)
                c["quantity"][s] = t["quantity"].to(torch.int64) * 100
                c["returnflag"][s] = letters[(t["group"] >> 1).long()]
                c["linestatus"][s] = torch.where((t["group"] & 1) != 0, ord("O"), ord("F")).to(torch.uint8)
            self.view = _lib.Columns(*(c[k].data_ptr() for k in ["shipdate", "discount", "extendedprice", "tax",
                                                                 "quantity", "returnflag", "linestatus"]))
        else:
            c = {"shipdate": column(torch.int16), "discount": column(torch.uint8),
                 "extendedprice": column(torch.int32), "tax": column(torch.uint8), "quantity": column(torch.uint8)}
            if packing == "pair":
                c["flags"] = column(torch.uint8, 8 * words)
            elif packing == "separate":
                c["returnflag"], c["linestatus"] = column(torch.uint8, 8 * words), column(torch.uint8, 4 * words)
            if filter_words:
                c["filter"] = column(torch.int32, words)
            if groups:
                self.keys = column(torch.int32)
            for r0, t in _chunks(n, seed, salt, groups, zipf):
                s = slice(r0, r0 + len(t["ship"]))
                c["shipdate"][s], c["discount"][s], c["tax"][s] = t["ship"], t["discount"], t["tax"]
                c["extendedprice"][s], c["quantity"][s] = t["price"], t["quantity"]
                if packing == "pair":
                    code = (t["group"] + 1) >> 1                     # groups 0, 2, 3, 4 -> codes 0, 1, 2, 2
                    _pack(torch.where(t["group"] == 4, 3, code).to(torch.uint8), 2, c["flags"], r0)
                elif packing == "separate":
                    _pack(t["group"] >> 1, 2, c["returnflag"], r0)
                    _pack(t["group"] & 1, 1, c["linestatus"], r0)
                if groups:
                    self.keys[s] = t["key"]
            self.view = _lib.CompressedColumns()
            for k, v in c.items():
                setattr(self.view, k, v.data_ptr())
            self.view.flag_packing = _lib.FLAGS_SEPARATE if packing == "separate" else _lib.FLAGS_PAIR_2BIT
            self.view.num_pair_codes = 4
            for i in range(4):
                self.view.pair_group[i] = PAIR_GROUPS[i]
        self.columns = c


def _sums(groups, index_of, chunks, cutoff):
    """[groups][6][low, high 64 bits] exact sums of the passing rows, in 64-bit integers."""
    low = torch.zeros(6, groups, dtype=torch.int64, device="cuda")
    high = torch.zeros_like(low)
    for _, t in chunks:
        keep = t["ship"].to(torch.int32) <= cutoff - FRAME
        g = t[index_of][keep].long()
        quantity, d, x, p = (t[k][keep].long() for k in ["quantity", "discount", "tax", "price"])
        dp = (100 - d) * p
        for a, v in enumerate([torch.ones_like(p), quantity * 100, p, d, dp, dp * (100 + x)]):
            low[a].scatter_add_(0, g, v & 0xFFFFFFFF)
            high[a].scatter_add_(0, g, v >> 32)
    t = (low >> 32) + high
    out = torch.stack([((t & 0xFFFFFFFF) << 32) | (low & 0xFFFFFFFF), t >> 32], dim=2)
    return out.permute(1, 0, 2).contiguous()


# ---------------------------------------------------------------------------------------------
# dbgen text
# ---------------------------------------------------------------------------------------------

_INSTRUCT = ["DELIVER IN PERSON", "COLLECT COD", "NONE", "TAKE BACK RETURN"]
_MODE = ["REG AIR", "AIR", "RAIL", "SHIP", "TRUCK", "MAIL", "FOB"]


def _text_chunk(row0, t, gen):
    """dbgen's lineitem lines of one chunk as a uint8 tensor."""
    n = len(t["ship"])
    chars, keep = [], []

    def put(c, k=None):
        chars.append(c.to(torch.uint8).view(n, -1))
        keep.append(torch.ones_like(chars[-1], dtype=torch.bool) if k is None else k.view(n, -1).expand_as(chars[-1]))

    def literal(s):
        put(torch.tensor(list(s.encode()), dtype=torch.uint8, device="cuda").expand(n, -1))

    def number(v, width, least=1):
        v = v.long()
        for i in reversed(range(width)):
            put(v // 10 ** i % 10 + 48, None if i < least else v >= 10 ** i)

    def choice(words):
        width = max(map(len, words))
        table = torch.tensor([list(w.encode().ljust(width, b"\0")) for w in words], dtype=torch.uint8, device="cuda")
        w = table[torch.randint(0, len(words), (n,), generator=gen, device="cuda")]
        put(w, None)
        keep[-1] = w != 0

    def date(day):
        d = np.datetime64("1992-01-01") + np.arange(int(day.max()) + 1)
        s = np.char.encode(np.datetime_as_string(d, unit="D")).view(np.uint8).reshape(-1, 10)
        put(torch.from_numpy(s.copy()).cuda()[day.long()])

    def uniform(lo, hi):
        return torch.randint(lo, hi, (n,), generator=gen, device="cuda")

    row = torch.arange(row0, row0 + n, device="cuda")
    for v, width in [(row // 4 + 1, 9), (uniform(1, 200_001), 6), (uniform(1, 10_001), 5), (row % 4 + 1, 1),
                     (t["quantity"], 2)]:
        number(v, width)
        literal("|")
    price = t["price"].long()
    number(price // 100, 6)
    literal(".")
    number(price % 100, 2, 2)
    literal("|0.")
    number(t["discount"], 2, 2)
    literal("|0.")
    number(t["tax"], 2, 2)
    literal("|")
    put(torch.tensor(list(b"ANR"), dtype=torch.uint8, device="cuda")[(t["group"] >> 1).long()])
    literal("|")
    put(torch.tensor(list(b"FO"), dtype=torch.uint8, device="cuda")[(t["group"] & 1).long()])
    literal("|")
    for day in [t["ship"], t["ship"] + 30, t["ship"] + uniform(1, 31).to(torch.int16)]:
        date(day)
        literal("|")
    choice(_INSTRUCT)
    literal("|")
    choice(_MODE)
    literal("|")
    letters = torch.randint(97, 123, (n, 43), generator=gen, device="cuda", dtype=torch.uint8)
    put(letters)
    keep[-1] = torch.arange(43, device="cuda").view(1, -1) < uniform(10, 44).view(-1, 1)
    literal("|\n")
    return torch.cat(chars, 1)[torch.cat(keep, 1)]


def _text(case, seed):
    gen = _generator(seed, 7)
    parts = []
    for r0, t in _chunks(case["rows"], seed):
        for a in range(0, len(t["ship"]), 1 << 20):
            parts.append(_text_chunk(r0 + a, {k: v[a:a + (1 << 20)] for k, v in t.items()}, gen))
    return torch.cat(parts)


def _line_bytes(rows):
    """Mean bytes of a line: fixed parts, the digits of the numbers, the words, the comment."""
    fixed = 16 + 1 + 1.82 + 3 + 7.3 + 8 + 2 + 30 + 12.25 + 4.14 + 26.5 + 7.0
    return fixed + max(1.0, math.log10(max(rows // 4, 1)) + 0.89)


# ---------------------------------------------------------------------------------------------
# Batches and servers
# ---------------------------------------------------------------------------------------------

def _instances(case):
    """(rows, groups, cutoff) of every instance: rows spread over the logarithm of the range."""
    n = case["instances"]
    lo, hi = math.log(case["min_rows"]), math.log(case["max_rows"])
    order = [(i * 37) % n if math.gcd(37, n) == 1 else i for i in range(n)]
    return [(int(math.exp(lo + (hi - lo) * order[i] / max(n - 1, 1))) | 1, [4, 64, 1024][i % 3],
             [CUTOFF, 728826][i // 3 % 2]) for i in range(n)]


class _Batch:
    def __init__(self, case, seed):
        self.tables, spec = [], _instances(case)
        self.out = torch.zeros(sum(g for _, g, _ in spec), 6, 2, dtype=torch.int64, device="cuda")
        c = (_lib.BatchInstance * len(spec))()
        base = 0
        for i, (rows, groups, cutoff) in enumerate(spec):
            t = _Table(case, seed, "none", salt=i + 1, rows=rows, groups=groups)
            self.tables.append(t)
            c[i].cols, c[i].keys, c[i].rows = t.view, t.keys.data_ptr(), rows
            c[i].cutoff_day, c[i].num_groups = cutoff, groups
            c[i].aggregates = self.out.data_ptr() + 96 * base
            base += groups
        self.handle = ctypes.c_void_p()
        opts = _lib.BatchOpts(1, 0, 0, 0, None)
        torch.cuda.synchronize()
        _lib.check(q.lib().q1_batch_create(c, len(spec), ctypes.byref(opts), _stream(), ctypes.byref(self.handle)))

    def __del__(self):
        if getattr(self, "handle", None):
            torch.cuda.synchronize()
            q.lib().q1_batch_destroy(self.handle)


class _Server:
    def __init__(self, case, seed):
        o = _lib.ServerOpts()
        q.lib().q1_server_opts_default(ctypes.byref(o))
        o.seed, o.resident_rows = seed, case["resident_rows"]
        o.hbm_budget_bytes, o.max_adhoc_rows, o.max_inflight = 2 << 30, case["max_rows"] | 1, 256
        self.handle = ctypes.c_void_p()
        _lib.check(q.lib().q1_server_open(ctypes.byref(o), ctypes.byref(self.handle)))
        n, lo, hi = case["tables"], math.log(case["min_rows"]), math.log(case["max_rows"])
        r = np.random.default_rng(seed)
        self.requests = []
        for i in range(case["requests"]):
            keys = bool(i // 2 % 2)
            cutoff = int(r.integers(729906, 730090))
            groups = 64 if keys else 0
            grouping = _lib.GROUP_KEYS if keys else _lib.GROUP_FLAGS
            if i % 2:
                k = int(r.integers(0, n))   # which table of the pool; its rows and its seed follow
                rows = int(math.exp(lo + (hi - lo) * k / max(n - 1, 1))) | 1
                self.requests.append(_lib.Request(_lib.REQ_ADHOC, grouping, groups, cutoff, rows, seed + 1000 + k))
            else:
                self.requests.append(_lib.Request(_lib.REQ_RESIDENT, grouping, groups, cutoff, 0, 0))

    def __del__(self):
        if getattr(self, "handle", None):
            q.lib().q1_server_close(self.handle)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# ---------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "query":
        s["ctx"] = q.Q1Context()
        s["ctx"].generate(seed, case["rows"], layout="compressed", packing=case["packing"],
                          residency=case["residency"])
        s["params"] = q.Q1Params(hash_table_placement=case["placement"], apply_compression=True,
                                 use_filter_pushdown=case["pushdown"], num_query_execution_runs=1,
                                 cutoff_day=case["cutoff"])
    elif kind == "scan":
        s["table"] = _Table(case, seed, case["packing"], filter_words=case["pushdown"])
        s["out"] = torch.zeros(6, 6, 2, dtype=torch.int64, device="cuda")
    elif kind == "groupkey":
        s["table"] = _Table(case, seed, "none", groups=case["groups"], zipf=case["zipf"])
        s["out"] = torch.zeros(case["groups"], 6, 2, dtype=torch.int64, device="cuda")
        s["scratch"] = torch.empty(q.lib().q1_groupkey_scratch_bytes(case["groups"]), dtype=torch.uint8, device="cuda")
        s["placement"] = q.placement_id(case["placement"])
    elif kind == "batch":
        s["batch"] = _Batch(case, seed)
    elif kind == "tbl":
        s["text"] = _text(case, seed)
        n = case["rows"]
        types = {"shipdate": torch.int32, "returnflag": torch.uint8, "linestatus": torch.uint8,
                 "discount": torch.int64, "tax": torch.int64, "extendedprice": torch.int64, "quantity": torch.int64}
        s["columns"] = {k: torch.zeros(n, dtype=t, device="cuda") for k, t in types.items()}
        s["view"] = _lib.ColumnsOut(*(s["columns"][k].data_ptr() for k in types))
    else:
        s["server"] = _Server(case, seed)
    torch.cuda.synchronize()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "query":
        g = state["ctx"].run(state["params"]).groups
        return np.array([[r["count"], r["sum_qty"], r["sum_base_price"], r["sum_disc"],
                          r["sum_disc_price"] >> 32, r["sum_disc_price"] & 0xFFFFFFFF,
                          r["sum_charge"] >> 32, r["sum_charge"] & 0xFFFFFFFF,
                          r["avg_qty_e4"], r["avg_price_e4"], r["avg_disc_e4"]] for r in g], dtype=np.int64)
    if kind == "scan":
        t, out = state["table"], state["out"]
        stream = torch.cuda.current_stream().cuda_stream
        out.zero_()
        if case["packing"] == "uncompressed":
            q.launch_uncompressed(case["placement"], t.view, t.rows, case["cutoff"], out.data_ptr(), stream)
        else:
            if case["pushdown"]:
                q.precompute_filter(t.view.shipdate, t.rows, case["cutoff"], t.view.filter, stream)
            q.launch_compressed(case["placement"], t.view, t.rows, case["cutoff"], case["pushdown"], out.data_ptr(),
                                stream)
        return out
    if kind == "groupkey":
        t, out = state["table"], state["out"]
        out.zero_()
        _lib.check(q.lib().q1_launch_groupkey(state["placement"], ctypes.byref(t.view), t.keys.data_ptr(),
                                              case["groups"], t.rows, case["cutoff"], None,
                                              state["scratch"].data_ptr(), out.data_ptr(), _stream()))
        return out
    if kind == "batch":
        _lib.check(q.lib().q1_batch_run(state["batch"].handle, _stream()))
        return state["batch"].out
    if kind == "tbl":
        rows = ctypes.c_uint64(0)
        _lib.check(q.lib().q1_tbl_parse_device(state["text"].data_ptr(), len(state["text"]), ctypes.byref(state["view"]),
                                               case["rows"], ctypes.byref(rows), _stream()))
        return dict(state["columns"], rows=rows.value)
    server = state["server"]
    tickets = []
    for r in server.requests:
        ticket = ctypes.c_uint64()
        _lib.check(q.lib().q1_server_submit(server.handle, ctypes.byref(r), ctypes.byref(ticket)))
        tickets.append(ticket.value)
    out = []
    for ticket in tickets:
        answer = _lib.Response()
        _lib.check(q.lib().q1_server_wait(server.handle, ticket, -1, ctypes.byref(answer)))
        _lib.check(answer.status)
        out.append(np.frombuffer(answer.aggregates, dtype=np.int64)[:answer.num_groups * 12].copy())
    return out


# ---------------------------------------------------------------------------------------------
# work / exact
# ---------------------------------------------------------------------------------------------

def work(case):
    """Columns read once and results written once; per row the predicate, the group and six sums."""
    kind = case["kind"]
    if kind == "query":
        return {"bytes": int(case["rows"] * LAYOUT_BYTES[(case["packing"], False)]) + 576, "flops": 10 * case["rows"]}
    if kind == "scan":
        per_row = LAYOUT_BYTES[(case["packing"], case["pushdown"])] + (2.125 if case["pushdown"] else 0.0)
        return {"bytes": int(case["rows"] * per_row) + 576, "flops": 10 * case["rows"]}
    if kind == "groupkey":
        return {"bytes": 13 * case["rows"] + 96 * case["groups"], "flops": 10 * case["rows"]}
    if kind == "batch":
        spec = _instances(case)
        rows = sum(r for r, _, _ in spec)
        return {"bytes": 13 * rows + 96 * sum(g for _, g, _ in spec), "flops": 10 * rows}
    if kind == "tbl":
        return {"bytes": int(case["rows"] * (_line_bytes(case["rows"]) + 38)), "flops": 0}
    lo, hi, n = math.log(case["min_rows"]), math.log(case["max_rows"]), case["tables"]
    mean = sum(math.exp(lo + (hi - lo) * k / max(n - 1, 1)) for k in range(n)) / n
    adhoc = case["requests"] // 2
    return {"bytes": int(13 * mean * adhoc) + case["requests"] * 35 * 96, "flops": int(10 * mean * adhoc)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "scan":
        return _sums(6, "group", _chunks(case["rows"], seed), case["cutoff"])
    if kind == "groupkey":
        return _sums(case["groups"], "key", _chunks(case["rows"], seed, 0, case["groups"], case["zipf"]),
                     case["cutoff"])
    if kind == "batch":
        return torch.cat([_sums(groups, "key", _chunks(rows, seed, i + 1, groups, False), cutoff)
                          for i, (rows, groups, cutoff) in enumerate(_instances(case))])
    if kind == "tbl":
        out = {k: [] for k in ["shipdate", "returnflag", "linestatus", "discount", "tax", "extendedprice", "quantity"]}
        for _, t in _chunks(case["rows"], seed):
            out["shipdate"].append(t["ship"].to(torch.int32) + FRAME)
            out["returnflag"].append(torch.tensor(list(b"ANR"), dtype=torch.uint8, device="cuda")[(t["group"] >> 1).long()])
            out["linestatus"].append(torch.tensor(list(b"FO"), dtype=torch.uint8, device="cuda")[(t["group"] & 1).long()])
            out["discount"].append(t["discount"].long())
            out["tax"].append(t["tax"].long())
            out["extendedprice"].append(t["price"].long())
            out["quantity"].append(t["quantity"].long() * 100)
        return dict({k: torch.cat(v) for k, v in out.items()}, rows=case["rows"])
    return None   # query and serve: the framework's own seeded generator makes the table
