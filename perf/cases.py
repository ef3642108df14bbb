"""Performance cases of the join engine: what a program that uses it has it do.

A case is a dict of plain values; its "kind" says what it is:

  join     a fact table joined with its dimensions on foreign keys (each fact
           row finds at most one row of a dimension), the joined rows handed
           back in columns by fact row. "form" says how it is called:
             replay  resident tables, the same query again and again (a
                     serving process; the engine replays it as a CUDA graph)
             adhoc   resident tables, graph replay off (queries that do not
                     repeat: each one is planned and launched by itself)
             host    Contest::execute on pageable host pages in and host
                     pages out (the drop-in call)
             pinned  the same with the input pages in pinned memory
  pairs    a many-to-many join over resident tables: keys repeat on both
           sides and every pair of rows comes back
  labels   exact cardinalities of every sub-plan of a query (the labels the
           learned cardinality estimator is trained on)
  fit      training of the learned estimator
  predict  its inference
  count    the row count of a two-table join, without any allocation

Tables hold INT32 or INT64 keys, INT32, INT64 or VARCHAR attributes (1 to 64
bytes, as in this repository's snowflake workload), NULL foreign keys where a
case asks for them, and uniform or Zipf-distributed foreign keys. A dimension
keeps a share of its keys, as after a filter at load time, and foreign keys
refer to all of them.

The engine returns rows in no particular order, so a pass ends the way a
program that consumes the join does: it scatters the rows' columns into
arrays indexed by the fact's row number (for pairs, by the pair's place).
"""
import ctypes
import importlib
import math
import weakref

import numpy as np
import torch

bj = importlib.import_module("contest-sigmod2025_b200")

PAGE = 8192
FULL = {bj.INT32: 1984, bj.INT64: 1007}  # rows of a full page without NULLs
TEXT = 64                                # longest VARCHAR


# ---------------------------------------------------------------------------
# Cases

def _join(name, **more):
    c = {"name": name, "kind": "join", "form": "replay", "fact": 1_000_000, "dims": 2, "dim": 100_000, "keep": 0.1,
         "nulls": 0.0, "skew": 0.0, "key": "int32", "attr": "int32", "deep": False}
    c.update(more)
    return c


def listed():
    return [
        # A point-like lookup a serving process repeats: latency and launches count.
        _join("lookup_small", fact=30_011, dims=1, dim=2_003, keep=0.5),
        # The benchmark's star shape: a large Zipf-skewed fact, selective dimensions, few rows survive.
        _join("star_large", fact=24_000_000, dims=3, dim=400_000, keep=0.02, skew=1.1),
        # The two-table benchmark shape: a large build side, 10% NULL keys, almost every row comes back.
        _join("enrich_nulls", fact=8_000_000, dims=1, dim=1_000_000, keep=1.0, nulls=0.1, attr="int64"),
        # Names looked up for the survivors of two filters: VARCHAR result pages.
        _join("names", fact=1_000_000, dims=2, dim=100_000, keep=0.1, attr="varchar"),
        # A query seen once over a snowflake schema: builds fed by probes, no replay.
        _join("snowflake_adhoc", form="adhoc", fact=600_001, dims=3, dim=60_000, keep=0.3, deep=True),
        # The contest's call on small tables: upload, page index, join, result pages back.
        _join("dropin_small", form="host", fact=60_013, dims=2, dim=6_007, keep=0.1, attr="varchar"),
        # The contest's call on a large fact table: the host link and staging count.
        _join("dropin_large", form="host", fact=12_000_000, dims=2, dim=200_000, keep=0.01, skew=1.1),
        # Keys that repeat on both sides, 64-bit: two passes over the probe, many result rows.
        {"name": "many_to_many", "kind": "pairs", "build": 300_007, "copies": 3, "probe": 2_000_003, "hit": 0.7,
         "key": "int64"},
        # Label generation for the estimator: all sub-plans of a seven-table query.
        {"name": "labels", "kind": "labels", "fact": 1_500_007, "dims": 3, "dim": 150_000, "keep": 0.3, "skew": 1.1},
        # Retraining the estimator on a corpus, and estimates for the sub-plans of a batch of queries.
        {"name": "fit", "kind": "fit", "rows": 4_000, "batch": 256, "epochs": 2},
        {"name": "predict", "kind": "predict", "rows": 6_000},
        # Counting next to another allocator's memory: the entry point that allocates nothing.
        {"name": "count_only", "kind": "count", "build": 200_003, "probe": 6_000_017, "nulls": 0.05},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["join"] * 7 + ["pairs", "labels", "fit", "predict", "count"])
    if kind == "join":
        form = rng.choice(["replay", "replay", "replay", "adhoc", "host", "pinned"])
        attr = rng.choice(["int32", "int32", "int64", "varchar"])
        key = rng.choice(["int32", "int32", "int32", "int64"])
        fact = _log(rng, 20_000, 2_000_000 if attr == "varchar" else 12_000_000 if key == "int32" else 4_000_000)
        dim = min(_log(rng, 500, 1_000_000), max(500, fact))
        dims = rng.randint(1, 4)
        deep = dims > 1 and dims < 4 and rng.random() < 0.3
        keep = math.exp(rng.uniform(math.log(0.005), 0.0))
        if attr == "varchar":
            # At most about 100,000 result rows: names are looked up for survivors, not for whole tables.
            keep = min(keep, 100_000 / fact)
        if form in ("host", "pinned"):
            keep = min(keep, 1_000_000 / fact)  # rows that travel back over the host link
        return {"kind": "join", "form": form, "fact": fact, "dims": dims, "dim": dim, "keep": round(keep, 5),
                "nulls": rng.choice([0.0, 0.0, 0.1, 0.4]), "skew": rng.choice([0.0, 1.1]), "key": key, "attr": attr,
                "deep": deep}
    if kind == "pairs":
        return {"kind": "pairs", "build": _log(rng, 1_000, 1_000_000), "copies": rng.randint(1, 5),
                "probe": _log(rng, 20_000, 2_000_000), "hit": round(rng.uniform(0.05, 1.0), 3),
                "key": rng.choice(["int32", "int64"])}
    if kind == "labels":
        return {"kind": "labels", "fact": _log(rng, 20_000, 2_000_000), "dims": rng.randint(2, 3),
                "dim": _log(rng, 1_000, 200_000), "keep": round(rng.uniform(0.05, 1.0), 3),
                "skew": rng.choice([0.0, 1.1])}
    if kind == "fit":
        return {"kind": "fit", "rows": _log(rng, 300, 8_000), "batch": rng.choice([64, 128, 256, 500]),
                "epochs": rng.randint(1, 3)}
    if kind == "predict":
        return {"kind": "predict", "rows": _log(rng, 20, 10_000)}
    return {"kind": "count", "build": _log(rng, 500, 262_144), "probe": _log(rng, 20_000, 16_000_000),
            "nulls": rng.choice([0.0, 0.05, 0.3])}


# ---------------------------------------------------------------------------
# Tables

class Pages:
    """One encoded column: the workload library's page writer (the contest's packing)."""

    def __init__(self, dtype, values=None, valid=None, offsets=None, chars=None):
        n = len(offsets) - 1 if dtype == bj.VARCHAR else len(values)
        ptr = lambda a: None if a is None else a.ctypes.data  # noqa: E731
        h = ctypes.c_void_p()
        st = bj.wlib().bjw_encode_column(dtype, n, ptr(values), ptr(valid), ptr(offsets), ptr(chars), ctypes.byref(h))
        if st != 0:
            raise bj.EngineError(st, "bjw_encode_column failed")
        self.type, self.rows, self.handle = dtype, n, h
        self.count = bj.wlib().bjw_pages_count(h)
        self.ptrs = bj.wlib().bjw_pages_ptrs(h)
        self.pinned = None
        weakref.finalize(self, bj.wlib().bjw_pages_free, h)

    def array(self):
        """The pages as one uint8 array of (count, PAGE)."""
        out = np.empty((self.count, PAGE), np.uint8)
        for i in range(self.count):
            ctypes.memmove(out[i].ctypes.data, self.ptrs[i], PAGE)
        return out

    def pin(self):
        self.pinned = torch.from_numpy(self.array()).pin_memory()
        base = self.pinned.data_ptr()
        self.ptrs = (ctypes.c_void_p * max(self.count, 1))(*[base + k * PAGE for k in range(self.count)])


class Table:
    """Columns of pages and the bj_table that names them."""

    def __init__(self, columns):
        self.columns = columns
        self.rows = columns[0].rows
        self.cols = (bj.BjColumn * len(columns))()
        self.fill()

    def fill(self):
        for s, c in zip(self.cols, self.columns):
            s.type, s.num_pages = c.type, c.count
            s.pages = ctypes.cast(c.ptrs, ctypes.POINTER(ctypes.c_void_p))
        self.struct = bj.BjTable(self.rows, len(self.columns), ctypes.cast(self.cols, ctypes.POINTER(bj.BjColumn)))

    def pin(self):
        for c in self.columns:
            c.pin()
        self.fill()


def _host(t):
    return t.cpu().numpy()


def _key_column(keys, key, valid=None):
    """Key numbers as a column: INT64 keys carry high halves from -4 to 3, as schema20w's do."""
    if key == "int64":
        k = keys.astype(np.int64)
        return Pages(bj.INT64, np.ascontiguousarray(k | ((k % 8 - 4) << 32)), valid)
    return Pages(bj.INT32, np.ascontiguousarray(keys.astype(np.int32)), valid)


def _foreign(gen, n, domain, skew):
    """n references to `domain` keys, uniform or Zipf(skew) over a random ranking."""
    if skew == 0.0:
        return torch.randint(0, domain, (n,), generator=gen, device="cuda", dtype=torch.int64)
    weight = torch.arange(1, domain + 1, device="cuda", dtype=torch.float64) ** -skew
    cdf = torch.cumsum(weight, 0)
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
    rank = torch.searchsorted(cdf, u).clamp_(max=domain - 1)
    return torch.randperm(domain, generator=gen, device="cuda")[rank]


def _attribute(gen, n, attr):
    """A payload column and, for fixed widths, its values."""
    if attr == "varchar":
        lens = _host(torch.randint(1, TEXT + 1, (n,), generator=gen, device="cuda")).astype(np.uint64)
        offsets = np.zeros(n + 1, np.uint64)
        np.cumsum(lens, out=offsets[1:])
        chars = _host(torch.randint(33, 127, (max(int(offsets[-1]), 1),), generator=gen, device="cuda",
                                    dtype=torch.uint8))
        return Pages(bj.VARCHAR, offsets=offsets, chars=chars)
    if attr == "int64":
        return Pages(bj.INT64, _host(torch.randint(0, 1 << 40, (n,), generator=gen, device="cuda")))
    return Pages(bj.INT32, _host(torch.randint(0, 1_000_000, (n,), generator=gen, device="cuda", dtype=torch.int32)))


TYPE = {"int32": bj.INT32, "int64": bj.INT64, "varchar": bj.VARCHAR}


def _domains(case):
    """(keys, kept keys) of every dimension, and of its sub-dimension in a deep case."""
    out = []
    for j in range(case["dims"]):
        keys = max(16, case["dim"] >> (2 * j))
        keep = min(1.0, case["keep"] * 3 ** j)
        sub = max(16, keys // 8)
        out.append((keys, max(1, int(keys * keep)), sub, max(1, sub * 7 // 10)))
    return out


def _star(case, seed):
    """The tables of a join or labels case, its plan, and the key numbers behind them.

    Plan: fact joined with dimension 0, 1, ...; in a deep case each dimension
    is followed by the sub-dimension it refers to. Output: the fact's row
    number, then one attribute per dimension (of its sub-dimension if deep),
    the first dimension's last."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, key, attr, deep = case["fact"], case.get("key", "int32"), case.get("attr", "int32"), case.get("deep", True)
    kt = TYPE[key]
    # Only the first dimension's attribute is of the case's type; the others' are INT32 codes.
    attrs = [attr] + ["int32"] * (case["dims"] - 1)
    doms = _domains(case)
    raw = {"fact": [], "dims": [], "subs": []}
    fact = [Pages(bj.INT32, np.arange(n, dtype=np.int32))]
    tables = [None]
    for j, (keys, kept, sub, sub_kept) in enumerate(doms):
        fk = _host(_foreign(gen, n, keys, case["skew"]))
        valid = None
        if case.get("nulls", 0.0):
            valid = _host(torch.rand(n, generator=gen, device="cuda") >= case["nulls"]).astype(np.uint8)
        fact.append(_key_column(fk, key, valid))
        own = _host(torch.randperm(keys, generator=gen, device="cuda")[:kept])
        raw["fact"].append(fk)
        raw["dims"].append(own)
        if deep:
            sfk = _host(torch.randint(0, sub, (kept,), generator=gen, device="cuda"))
            sown = _host(torch.randperm(sub, generator=gen, device="cuda")[:sub_kept])
            raw["subs"].append((sfk, sown))
            tables.append(Table([_key_column(own, key), _key_column(sfk, key)]))
            tables.append(Table([_key_column(sown, key), _attribute(gen, sub_kept, attrs[j])]))
        else:
            tables.append(Table([_key_column(own, key), _attribute(gen, kept, attrs[j])]))
    tables[0] = Table(fact)

    p = bj.Plan()
    types = [bj.INT32] + [kt] * case["dims"]
    left = p.new_scan_node(0, list(enumerate(types)))
    cur = [("id", bj.INT32)] + [("fk%d" % j, kt) for j in range(case["dims"])]
    t = 1
    for j in range(case["dims"]):
        a = TYPE[attrs[j]]
        steps = [("fk%d" % j, [("key", kt), ("sub", kt)])] + [("sub", [("key", kt), ("a%d" % j, a)])] if deep else \
                [("fk%d" % j, [("key", kt), ("a%d" % j, a)])]
        for on, cols in steps:
            right = p.new_scan_node(t, [(i, ty) for i, (_, ty) in enumerate(cols)])
            t += 1
            names = [c[0] for c in cur]
            both = cur + cols
            keep = [i for i, (nm, _) in enumerate(both) if nm != on and nm != "key"]
            left = p.new_join_node(False, left, right, names.index(on), 0, [(i, both[i][1]) for i in keep])
            cur = [both[i] for i in keep]
    # Result columns: the fact's row number and the INT32 attributes, then the first dimension's.
    first = [i for i, (nm, _) in enumerate(cur) if nm == "a0"]
    root = p.nodes[left]
    order = [i for i in range(len(cur)) if i not in first] + first
    root.output_attrs = [root.output_attrs[i] for i in order]
    p.root = left
    return tables, p, raw


class BoundPlan(bj.CPlan):
    """A plan over tables that exist already (no copies of their pages)."""

    def __init__(self, plan, tables):
        super().__init__(plan)
        self.tables = (bj.BjTable * len(tables))(*[t.struct for t in tables])
        self.owners = tables
        self.struct.num_inputs = len(tables)
        self.struct.inputs = ctypes.cast(self.tables, ctypes.POINTER(bj.BjTable))


# ---------------------------------------------------------------------------
# State

_contexts = {}


def _context(form):
    """One context per way of calling, kept for the program's life."""
    k = "adhoc" if form == "adhoc" else "main"
    if k not in _contexts:
        ctx = bj.build_context(0)
        if k == "adhoc":
            ctx.set_graphs(False)
        _contexts[k] = ctx
        _contexts[k, "stream"] = torch.cuda.ExternalStream(ctx.stream())
    return _contexts[k], _contexts[k, "stream"]


class State:
    def __init__(self, case):
        self.case = case
        self.residents = []
        weakref.finalize(self, _free, self.residents)

    def upload(self, ctx, tables):
        self.ctx = ctx
        self.residents.extend(ctx.upload(t.struct) for t in tables)


def _free(residents):
    for r in residents:
        r.free()


def _features(gen, n):
    """Feature rows as the engine writes them: two to twelve inputs of 149 values each, the rest zero."""
    used = torch.randint(2, 13, (n, 1), generator=gen, device="cuda")
    x = torch.rand((n, 12, 149), generator=gen, device="cuda") * 0.7
    x[:, :, 5:17] = (x[:, :, 5:17] > 0.6).float()  # the parent's place, one-hot in earnest
    x[:, :, 0] = 1.0
    x *= (torch.arange(12, device="cuda")[None, :] < used)[:, :, None]
    f = torch.zeros((n, bj.EST_FEATURES), device="cuda")
    f[:, :12 * 149] = x.reshape(n, -1)
    return f


def _parameters(gen):
    """Parameters of a fresh estimator: W1, b1, W2, b2, w3, b3, padding."""
    f, h = bj.EST_FEATURES, bj.EST_HIDDEN
    p = torch.zeros(bj.Estimator.num_params(), device="cuda")
    normal = lambda k, s: torch.randn(k, generator=gen, device="cuda") * s  # noqa: E731
    o = 0
    p[o:o + f * h] = normal(f * h, math.sqrt(2.0 / f))
    o += f * h + h
    p[o:o + h * h] = normal(h * h, math.sqrt(2.0 / h))
    o += h * h + h
    p[o:o + h] = normal(h, math.sqrt(1.0 / h))
    p[o + h] = 12.0
    return _host(p)


def prepare(case, seed):
    s = State(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind in ("join", "labels"):
        tables, plan, _ = _star(case, seed)
        form = case.get("form", "replay")
        ctx, s.stream = _context(form)
        if form == "pinned":
            for t in tables:
                t.pin()
        s.ctx, s.plan, s.form = ctx, BoundPlan(plan, tables), form
        if form in ("replay", "adhoc"):
            s.upload(ctx, tables)
        if kind == "labels":
            s.masks = np.array([m for m in bj.subplans(s.plan) if bin(int(m)).count("1") > 1], np.uint32)
            return s
        s.device = "cuda" if form in ("replay", "adhoc") else "cpu"
        n, attr = case["fact"], case["attr"]
        ints = 1 + case["dims"] - (attr != "int32")
        s.out = {"ints": torch.full((ints, n), -1, dtype=torch.int32, device=s.device)}
        if attr == "int64":
            s.out["wide"] = torch.full((n,), -1, dtype=torch.int64, device=s.device)
        if attr == "varchar":
            s.out["text"] = torch.zeros((n, TEXT), dtype=torch.uint8, device=s.device)
            s.places = torch.arange(TEXT, device=s.device)
            s.rows = torch.arange(n, device=s.device)
            s.pages = torch.arange(n * (TEXT + 3) // PAGE + 2, device=s.device)
            s.spare = torch.zeros(TEXT, device=s.device, dtype=torch.uint8)
    elif kind == "pairs":
        nb, npr = case["build"], case["probe"]
        distinct = max(1, nb // case["copies"])
        domain = max(distinct, int(distinct / case["hit"]))
        bkey = torch.randint(0, distinct, (nb,), generator=gen, device="cuda")
        pkey = torch.randint(0, domain, (npr,), generator=gen, device="cuda")
        pay = Pages(bj.INT32, _host(torch.randint(0, 1 << 30, (nb,), generator=gen, device="cuda", dtype=torch.int32)))
        tables = [Table([_key_column(_host(bkey), case["key"]), Pages(bj.INT32, np.arange(nb, dtype=np.int32)), pay]),
                  Table([_key_column(_host(pkey), case["key"]), Pages(bj.INT32, np.arange(npr, dtype=np.int32))])]
        p = bj.Plan()
        kt = TYPE[case["key"]]
        a = p.new_scan_node(0, [(0, kt), (1, bj.INT32), (2, bj.INT32)])
        b = p.new_scan_node(1, [(0, kt), (1, bj.INT32)])
        p.root = p.new_join_node(True, a, b, 0, 0, [(4, bj.INT32), (1, bj.INT32), (2, bj.INT32)])
        ctx, s.stream = _context("replay")
        s.plan, s.form, s.device = BoundPlan(p, tables), "replay", "cuda"
        s.upload(ctx, tables)
        # A pair's place: the pairs of the probe rows before it, then the build row's rank within its key.
        per_key = torch.bincount(bkey, minlength=domain)
        matches = per_key[pkey]
        s.first = torch.cumsum(matches, 0) - matches
        order = torch.sort(bkey, stable=True).indices
        start = torch.cumsum(per_key, 0) - per_key
        s.rank = torch.empty_like(bkey)
        s.rank[order] = torch.arange(nb, device="cuda") - start[bkey[order]]
        room = int(1.25 * npr * nb / domain) + 4096  # every seed's pairs fit
        s.out = {"ints": torch.full((3, room), -1, dtype=torch.int32, device="cuda")}
    elif kind in ("fit", "predict"):
        s.est = bj.Estimator(0, seed=1)
        s.params = _parameters(gen)
        f = _features(gen, case["rows"])
        s.features = _host(f)
        if kind == "fit":
            w = torch.randn(bj.EST_FEATURES, generator=gen, device="cuda") * 0.3
            s.targets = _host((12.0 + f @ w).clamp(0.0, 60.0))
        else:
            s.est.set_params(s.params)
    elif kind == "count":
        nb, npr = case["build"], case["probe"]
        bkey = _host(torch.randint(0, nb, (nb,), generator=gen, device="cuda", dtype=torch.int32))
        pkey = _host(torch.randint(0, 2 * nb, (npr,), generator=gen, device="cuda", dtype=torch.int32))
        valid = lambda k: None if not case["nulls"] else \
            _host(torch.rand(k, generator=gen, device="cuda") >= case["nulls"]).astype(np.uint8)  # noqa: E731
        s.build = torch.from_numpy(Pages(bj.INT32, bkey, valid(nb)).array()).cuda()
        s.probe = torch.from_numpy(Pages(bj.INT32, pkey, valid(npr)).array()).cuda()
        s.out = torch.zeros(1, dtype=torch.int64, device="cuda")
    return s


# ---------------------------------------------------------------------------
# One pass

class _Memory:
    def __init__(self, address, nbytes):
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (address, False), "version": 3}


def _result_pages(state, r):
    """The result's pages where they are, as one (pages, PAGE) tensor, and each column's number of pages."""
    page = bj.lib().bj_result_device_page if state.device == "cuda" else bj.lib().bj_result_page
    counts = [r.column_pages(c) for c in range(r.num_columns)]
    first, total = page(r.handle, 0, 0), sum(counts)
    if page(r.handle, len(counts) - 1, counts[-1] - 1) != first + (total - 1) * PAGE:
        raise RuntimeError("result pages are not back to back")
    if state.device == "cuda":
        flat = torch.as_tensor(_Memory(first, total * PAGE), device="cuda")
    else:
        flat = torch.from_numpy(np.frombuffer((ctypes.c_uint8 * (total * PAGE)).from_address(first), np.uint8))
    return flat.view(total, PAGE), counts


def _values(pages, dtype, columns, n):
    """The first n values of `columns` fixed-width columns without NULLs, (columns, n)."""
    w = pages.view(torch.int32 if dtype == bj.INT32 else torch.int64)
    return w[:, 1:1 + FULL[dtype]].reshape(columns, -1)[:, :n]


def _strings(state, pages, n):
    """The n strings of a VARCHAR column without NULLs, padded to TEXT bytes with zeros."""
    half = pages.view(torch.int16)
    rows = half[:, 0].long()
    start = rows.cumsum(0) - rows
    page = torch.repeat_interleave(rows, output_size=n)
    first = state.pages[:len(pages)] * PAGE + 4  # byte of the page's first end offset
    # A page: row count, value count, the values' end offsets (16 bits each), then their bytes.
    slot = (first // 2 - start).index_select(0, page).add_(state.rows[:n])
    end = half.reshape(-1).take(slot).long()
    begin = end.roll(1).index_fill_(0, start, 0)
    base = (first + 2 * rows).index_select(0, page).add_(begin)
    spare = torch.cat((pages.reshape(-1), state.spare))
    text = spare.unfold(0, TEXT, 1).index_select(0, base)
    return text.mul_(state.places < (end - begin)[:, None])


def _collect(state, r):
    """Scatters the result's columns (INT32 ones first, the fact's row number leading) to their rows' places."""
    n = r.num_rows
    if n == 0:
        return
    pages, counts = _result_pages(state, r)
    ints = state.out["ints"]
    k = ints.shape[0]
    v = _values(pages[:k * counts[0]], bj.INT32, k, n)
    at = v[0].long()
    if state.case["kind"] == "pairs":
        at = state.first[at] + state.rank[v[1].long()]
    ints.index_copy_(1, at, v)
    if "wide" in state.out:
        state.out["wide"].index_copy_(0, at, _values(pages[k * counts[0]:], bj.INT64, 1, n)[0])
    if "text" in state.out:
        state.out["text"].index_copy_(0, at, _strings(state, pages[k * counts[0]:], n))


def run(state):
    case = state.case
    kind = case["kind"]
    if kind in ("join", "pairs"):
        with torch.cuda.stream(state.stream):  # the result's pages are the engine's: read them in its stream's order
            if state.device == "cuda":
                r = state.ctx.execute_resident(state.plan, state.residents, bj.RESULT_DEVICE)
            else:
                r = state.ctx.execute_raw(state.plan)
            with r:
                _collect(state, r)
                return {"rows": r.num_rows, **state.out}
    if kind == "labels":
        return state.ctx.subplan_cards(state.plan, state.residents, state.masks)
    if kind == "fit":
        state.est.set_params(state.params)
        loss = state.est.train(state.features, state.targets, epochs=case["epochs"], batch=case["batch"], seed=3)
        return {"loss": loss, "params": state.est.params()}
    if kind == "predict":
        return state.est.predict(state.features)
    st = bj.lib().bj_join_count_static(
        state.build.data_ptr(), len(state.build), case["build"], state.probe.data_ptr(), len(state.probe),
        ctypes.cast(state.out.data_ptr(), ctypes.c_void_p), torch.cuda.current_stream().cuda_stream)
    if st != 0:
        raise bj.EngineError(st, "bj_join_count_static")
    return state.out


# ---------------------------------------------------------------------------
# What a pass cannot do without

def work(case):
    kind = case["kind"]
    width = {"int32": 4, "int64": 8, "varchar": 2 + TEXT / 2}
    if kind in ("join", "labels"):
        key, attr, deep = width[case.get("key", "int32")], width[case.get("attr", "int32")], case.get("deep", True)
        n = case["fact"]
        nbytes, rows = n * case["dims"] * key, n * (1.0 - case.get("nulls", 0.0)) ** case["dims"]
        for j, (keys, kept, sub, sub_kept) in enumerate(_domains(case)):
            a = attr if j == 0 else 4
            nbytes += kept * (2 * key if deep else key + a) + (sub_kept * (key + a) if deep else 0)
            rows *= kept / keys * (sub_kept / sub if deep else 1.0)
        if kind == "labels":
            return {"bytes": float(nbytes), "flops": 0.0}
        # The result's fact row numbers are read and written; its attributes written.
        return {"bytes": nbytes + rows * (8 + attr + 4 * (case["dims"] - 1)), "flops": 0.0}
    if kind == "pairs":
        key = width[case["key"]]
        pairs = case["probe"] * case["hit"] * case["copies"]
        return {"bytes": case["build"] * (key + 8) + case["probe"] * (key + 4) + pairs * 12, "flops": 0.0}
    if kind == "count":
        return {"bytes": 4.0 * (case["build"] + case["probe"]), "flops": 0.0}
    f, h, n = bj.EST_FEATURES, bj.EST_HIDDEN, case["rows"]
    products = 2.0 * n * (f * h + h * h + h)
    if kind == "predict":
        return {"bytes": 4.0 * n * f + 2.0 * (f * h + h * h), "flops": products}
    # Backward: the weight gradients of both layers and the second layer's input gradient.
    return {"bytes": 4.0 * n * f + 4.0 * (f * h + h * h), "flops": case["epochs"] * (2 * products + 2.0 * n * h * h)}


# ---------------------------------------------------------------------------
# Outputs in 64 bits (the joins' outputs are whole numbers and bytes)

def exact(case, seed):
    kind = case["kind"]
    if kind == "labels":
        _, plan, raw = _star(case, seed)
        d = case["dims"]
        masks = [int(m) for m in bj.subplans(bj.CPlan(_rows_only(plan, case))) if bin(int(m)).count("1") > 1]
        # Inputs in depth-first order: the fact, then each dimension and its sub-dimension.
        doms = _domains(case)
        out = []
        for m in masks:
            weights, total = [], None
            for j in range(d):
                has_dim, has_sub = m >> (1 + 2 * j) & 1, m >> (2 + 2 * j) & 1
                if not has_dim:
                    continue
                w = np.ones(len(raw["dims"][j]))
                if has_sub:
                    sfk, sown = raw["subs"][j]
                    w = np.bincount(sown, minlength=doms[j][2]).astype(np.float64)[sfk]
                if not m & 1:
                    total = w.sum()  # a dimension and its sub-dimension by themselves
                weights.append((j, w))
            if m & 1:
                rows = np.ones(case["fact"])
                for j, w in weights:
                    rows *= np.bincount(raw["dims"][j], weights=w, minlength=doms[j][0])[raw["fact"][j]]
                total = rows.sum()
            out.append(total)
        return np.array(out, np.float64)
    if kind == "predict":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        p = torch.from_numpy(_parameters(gen)).double().cuda()
        x = _features(gen, case["rows"]).double()
        f, h = bj.EST_FEATURES, bj.EST_HIDDEN
        o1, o2 = f * h + h, f * h + h + h * h + h
        h1 = torch.relu(x @ p[:f * h].view(f, h) + p[f * h:o1])
        h2 = torch.relu(h1 @ p[o1:o1 + h * h].view(h, h) + p[o1 + h * h:o2])
        return h2 @ p[o2:o2 + h] + p[o2 + h]
    return None


def _rows_only(plan, case):
    """The plan over tables that only have their row counts (for the sub-plans' masks)."""
    rows = [case["fact"]]
    for _, kept, _, sub_kept in _domains(case):
        rows += [kept, sub_kept]
    plan.inputs = [bj.ColumnarTable(num_rows=r, columns=[bj.Column(bj.INT32), bj.Column(bj.INT32)] +
                                    [bj.Column(bj.INT32)] * case["dims"]) for r in rows]
    return plan
