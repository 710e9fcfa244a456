"""The work that a query engine has these operators do, as cases that can be timed and compared.

A case is one query step: a hash aggregation (HashAggregationOperator, single-stage or partial +
final), a batch of small aggregation tasks (AggBatch), or a hash join (HashBuilderOperator and
LookupJoinOperator).  Columns are in HBM, as between two operators of one plan, except in the
smallest cases, which take and return host VectorBatches, and in the string case, whose batch is
uploaded first.

The operators return VectorBatches, and the order of their rows is not part of the contract.
`run` therefore returns a `Rows`: the list of the output's columns (values, then NULL mask, per
column) with the rows in sorted order, which reads them off the finished batches when it is looked
at.  How many rows come out depends on the data; `Rows` fills up to a number that holds for all
inputs of the case (with NULL zeros), and its last item is the number of rows.
"""
import math

import numpy as np
import torch

import omnioperator_gb300 as omg
from omnioperator_gb300.sizer import SizingModel

L, I, D, V = omg.LongType(), omg.IntType(), omg.DoubleType(), omg.VarcharType(24)
DEC64, DEC128 = omg.Decimal64Type(18, 2), omg.Decimal128Type(38, 2)
SUM, COUNT, COUNT_ALL = (omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_COLUMN,
                         omg.OMNI_AGGREGATION_TYPE_COUNT_ALL)
MIN, MAX, AVG = omg.OMNI_AGGREGATION_TYPE_MIN, omg.OMNI_AGGREGATION_TYPE_MAX, omg.OMNI_AGGREGATION_TYPE_AVG
JOIN_TYPES = {"inner": omg.OMNI_JOIN_TYPE_INNER, "left": omg.OMNI_JOIN_TYPE_LEFT,
              "semi": omg.OMNI_JOIN_TYPE_LEFT_SEMI, "anti": omg.OMNI_JOIN_TYPE_LEFT_ANTI}
BATCH = 4096  # rows of a host VectorBatch
DEV = "cuda"


# ---------------------------------------------------------------------------------- the cases
def listed():
    return [
        # One scan batch, host to host: what a small query or a streaming caller pays per call.
        agg("agg_scan_batch", rows=4096, groups=100, input="host"),
        # The uniform aggregation of the benchmark: 4M rows, 10,000 groups, six aggregates.
        agg("agg_uniform", rows=1 << 22, groups=10_000),
        # A report by two flag columns: a handful of groups, four partial operators and a final one,
        # as a plan over four splits runs it.
        agg("agg_few_groups", rows=(1 << 24) - 3, groups=6, key="pair_int", stages=2),
        # Skewed high-cardinality aggregation (order lines by store and item): composite key,
        # decimal SUM, COUNT(*), AVG with NULLs.
        agg("agg_zipf_pairs", rows=1 << 26, groups=50_000_000, key="pair", plan="decimal", dist="zipf"),
        # Deduplication-like group-by: about as many groups as a quarter of the rows.
        agg("agg_many_groups", rows=16_777_259, groups=4_000_000, plan="sum_count"),
        # Group-by on strings, from host data.
        agg("agg_varchar", rows=1_000_000, groups=10_000, key="varchar", plan="sum_count"),
        # Many small independent aggregations in one launch.
        {"name": "agg_tasks", "family": "tasks", "tasks": 400, "rows_min": 1000, "rows_max": 1_000_000},
        # One scan batch against a small dimension table, host to host.
        join("join_scan_batch", build=10_000, probe=4096, input="host"),
        # The star-schema probe of the benchmark: 64M rows against 1M unique dense keys.
        join("join_star", build=1 << 20, probe=1 << 26),
        # Build and probe in one query: sparse keys, up to three build rows a key, left outer.
        join("join_build_dup_left", build=1_000_002, probe=4_000_037, kind="left", key="sparse", dup=3, built="each"),
        # Two-column key and a join filter on a build column.
        join("join_pair_filter", build=1 << 20, probe=(1 << 24) + 5, key="pair", filter=True),
        # Skewed keys against a build side that no cache holds, 16 bytes of payload, hash-partitioned.
        join("join_zipf", build=1 << 24, probe=1 << 26, key="sparse", dist="zipf", payload="long2",
             strategy="hash_partitioned"),
    ]


def agg(name, rows, groups, key="long", plan="six", dist="uniform", stages=1, input="device"):
    return {"name": name, "family": "agg", "rows": rows, "groups": groups, "key": key, "plan": plan, "dist": dist,
            "stages": stages, "input": input}


def join(name, build, probe, kind="inner", key="dense", dup=1, dist="uniform", payload="int2", filter=False,
         strategy="direct", built="before", input="device"):
    return {"name": name, "family": "join", "build": build, "probe": probe, "kind": kind, "key": key, "dup": dup,
            "dist": dist, "payload": payload, "filter": filter, "strategy": strategy, "built": built, "input": input}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["agg", "agg", "agg", "tasks", "join", "join", "join"])
    if family == "tasks":
        case = {"family": "tasks", "tasks": _log_int(rng, 16, 400), "rows_min": 1000,
                "rows_max": _log_int(rng, 20_000, 1_000_000)}
    elif family == "agg":
        rows = _log_int(rng, 2000, 1 << 25)
        key = rng.choice(["long", "long", "pair_int", "pair", "varchar"])
        if key == "varchar":
            rows = min(rows, 1_000_000)
        groups = _log_int(rng, 4, max(5, min(rows, 20_000 if key == "varchar" else 8_000_000)))
        plan = rng.choice(["six", "sum_count", "decimal"])
        host = rows <= 65_536 and rng.random() < 0.5
        stages = 2 if plan == "six" and key != "varchar" and not host and rng.random() < 0.4 else 1
        case = agg("", rows, groups, key, plan, rng.choice(["uniform", "zipf"]), stages, "host" if host else "device")
    else:
        build, probe = _log_int(rng, 500, 1 << 22), _log_int(rng, 2000, 1 << 25)
        key = rng.choice(["dense", "sparse", "pair"])
        kind = rng.choice(["inner", "inner", "left", "semi", "anti"])
        dup = rng.choice([1, 1, 2, 3])
        strategy = "direct"
        payload = rng.choice(["int2", "long2"])
        if dup == 1 and kind == "inner" and key == "sparse" and probe >= 1 << 20 and rng.random() < 0.5:
            strategy = rng.choice(["hash_partitioned", "range_partitioned"])
        host = probe <= 65_536 and rng.random() < 0.5
        case = join("", build, probe, kind, key, dup, rng.choice(["uniform", "zipf"]), payload,
                    kind in ("inner", "left") and strategy == "direct" and rng.random() < 0.3, strategy,
                    rng.choice(["before", "each"]) if strategy == "direct" else "before", "host" if host else "device")
    case.pop("name", None)
    return case


# ---------------------------------------------------------------------------------- output rows
class _View:
    """A device array at an address, for torch."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3,
                                         "strides": None}


_TYPESTR = {omg.OMNI_INT: "<i4", omg.OMNI_LONG: "<i8", omg.OMNI_DOUBLE: "<f8", omg.OMNI_BOOLEAN: "|u1",
            omg.OMNI_DECIMAL64: "<i8"}


def _device_column(batch, col):
    lib = omg.lib()
    n, vec = lib.omg_batch_row_count(batch), lib.omg_batch_get(batch, col)
    t, ptr = lib.omg_vec_type(vec), lib.omg_vec_values(vec)
    if t == omg.OMNI_DECIMAL128:
        vals = torch.as_tensor(_View(ptr, (n, 2), "<i8"), device=DEV)
    else:
        vals = torch.as_tensor(_View(ptr, (n,), _TYPESTR[t]), device=DEV)
    nulls = lib.omg_vec_nulls(vec) if lib.omg_vec_has_null(vec) else None
    if not nulls:
        return vals, torch.zeros(n, dtype=torch.uint8, device=DEV)
    bits = torch.as_tensor(_View(nulls, ((n + 7) // 8,), "|u1"), device=DEV)
    mask = (bits[:, None] >> torch.arange(8, device=DEV, dtype=torch.uint8)) & 1
    return vals, mask.reshape(-1)[:n].contiguous()


def _host_column(vals, mask):
    if vals.dtype == object:  # strings: fixed-width bytes
        vals = np.array([v if v is not None else b"" for v in vals], dtype="S24").view(np.uint8).reshape(-1, 24)
    if vals.dtype == np.uint64:
        vals = vals.view(np.int64)
    return torch.from_numpy(np.ascontiguousarray(vals)), torch.from_numpy(mask.astype(np.uint8))


def _sort_words(vals):
    """The columns of 64-bit words that order `vals`."""
    if vals.dim() == 1:
        return [vals]
    return [vals[:, i] for i in range(vals.shape[1])]


def _filled(x, rows, value):
    if len(x) > rows:
        raise ValueError(f"{len(x)} rows came out, at most {rows} were expected")
    tail = torch.full((rows - len(x),) + tuple(x.shape[1:]), value, dtype=x.dtype, device=x.device)
    return torch.cat([x, tail])


class Rows(list):
    """Output batches as [values, NULL mask] * columns + [row count], sorted by the first `n_id` columns
    and filled up to `most` rows; batch k belongs to task what[k]."""

    def __init__(self, batches, n_id, most, what=None):
        super().__init__()
        self._batches, self._n_id, self._most, self._what, self._cols = batches, n_id, most, what, None

    def _read(self):
        if self._cols is not None:
            return self._cols
        lib = omg.lib()
        parts = []
        for k, b in enumerate(self._batches):
            if lib.omg_vec_is_device(lib.omg_batch_get(b, 0)):
                cols = [_device_column(b, c) for c in range(lib.omg_batch_vector_count(b))]
            else:
                cols = [_host_column(v, m) for v, m in omg.batch_to_numpy(b)]
            if self._what is not None:  # the task that a batch belongs to
                which = torch.full((len(cols[0][0]),), self._what[k], dtype=torch.int32, device=cols[0][0].device)
                cols.insert(0, (which, torch.zeros_like(which, dtype=torch.uint8)))
            parts.append(cols)
        cols = []
        for c in range(len(parts[0]) if parts else 0):
            vals, mask = torch.cat([p[c][0] for p in parts]), torch.cat([p[c][1] for p in parts])
            dead = mask.bool()
            cols.append((torch.where(dead if vals.dim() == 1 else dead[:, None], torch.zeros_like(vals), vals), mask))
        order = None
        for vals, mask in reversed(cols[: self._n_id]):
            for word in [mask] + _sort_words(vals)[::-1]:
                word = word if order is None else word[order]
                step = torch.sort(word, stable=True).indices
                order = step if order is None else order[step]
        self._cols = [_filled(x[order], self._most, i) for pair in cols for i, x in enumerate(pair)]
        self._cols.append(len(order))
        return self._cols

    def __iter__(self):
        return iter(self._read())

    def __len__(self):
        return len(self._read())

    def __getitem__(self, i):
        return self._read()[i]

    def __del__(self):
        if self._batches:
            omg.free_batches(self._batches)
            self._batches = []


class State:
    """What a program keeps between queries: factories, the build side, inputs."""

    def __init__(self, **kw):
        self.closing = []
        self.__dict__.update(kw)

    def __del__(self):
        for close in reversed(self.closing):
            close()


# ---------------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 12345)
    return g


def _codes(case_dist, rows, domain, g):
    """Row -> entity code in [0, domain): uniform, or skewed as Zipf(1.1) is (rank r drawn with probability
    proportional to r^-0.1 - (r+1)^-0.1), the ranks spread over the codes."""
    if case_dist == "uniform":
        return torch.randint(0, domain, (rows,), generator=g, device=DEV, dtype=torch.int64)
    u = torch.rand(rows, generator=g, device=DEV, dtype=torch.float64)
    out = (1 - u * (1 - (domain + 1.0) ** -0.1)).pow(-10).long().sub_(1).clamp_(0, domain - 1)
    return (out * 0x9E3779B1 + 1) % domain if math.gcd(0x9E3779B1, domain) == 1 else out


def _spread(x):
    """Codes as keys all over 63 bits (a bijection), as numbers from an outside system are."""
    x = x * 0x100000001B3 + 7
    x = x ^ ((x >> 30) & 0x3FFFFFFFF)
    x = x * -4658895280553007687
    return (x ^ ((x >> 27) & 0x1FFFFFFFFF)) & 0x7FFFFFFFFFFFFFFF


def _bitmap(mask):
    m = torch.zeros((len(mask) + 63) // 64 * 64, dtype=torch.uint8, device=DEV)
    m[: len(mask)] = mask
    w = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=DEV)
    return (m.view(-1, 8) * w).sum(1, dtype=torch.uint8)


def _words(n):
    rng = np.random.default_rng(n)
    letters = rng.integers(97, 123, (n, 16), dtype=np.uint8)
    lens = rng.integers(0, 17, n)
    return np.array([b"%07d" % i + bytes(letters[i, : lens[i]]) for i in range(n)], dtype=object)


def _agg_inputs(case, seed):
    """{"code", "keys", "vals", "nulls"}: the group code of each row, and the columns of the batch."""
    g = _gen(seed)
    rows, groups = case["rows"], case["groups"]
    code = _codes(case["dist"], rows, groups, g)
    if case["key"] == "long":
        keys = [_spread(code)]
    elif case["key"] == "pair":
        keys = [(code % 65521).to(torch.int32), _spread(code)]
    elif case["key"] == "pair_int":
        keys = [(code % 3).to(torch.int32), (code // 3).to(torch.int32)]
    else:
        keys = [code]
    if case["plan"] == "decimal":
        vals = [torch.randint(-10**9, 10**9 + 1, (rows,), generator=g, device=DEV, dtype=torch.int64),
                torch.randn(rows, generator=g, device=DEV, dtype=torch.float64)]
        nulls = [torch.rand(rows, generator=g, device=DEV) < 0.02 for _ in vals]
    else:
        vals = [torch.randint(-10**6, 10**6 + 1, (rows,), generator=g, device=DEV, dtype=torch.int64)]
        if case["plan"] == "six":
            vals.append(torch.rand(rows, generator=g, device=DEV, dtype=torch.float64))
        nulls = [None for _ in vals]
    return {"code": code, "keys": keys, "vals": vals, "nulls": nulls}


def _key_types(case):
    return {"long": [L], "pair": [I, L], "pair_int": [I, I], "varchar": [V]}[case["key"]]


def _val_types(case):
    return {"six": [L, D], "sum_count": [L], "decimal": [DEC64, D]}[case["plan"]]


def _agg_factories(case):
    kt = _key_types(case)
    k = len(kt)
    gb = list(range(k))
    if case["plan"] == "sum_count":
        return [omg.HashAggregationOperatorFactory(gb, kt, [[k], [k]], [[L], [L]], [[L], [L]], [SUM, COUNT])]
    if case["plan"] == "decimal":
        return [omg.HashAggregationOperatorFactory(gb, kt, [[k], [], [k + 1]], [[DEC64], [], [D]],
                                                   [[DEC128], [L], [D]], [SUM, COUNT_ALL, AVG])]
    funcs = [SUM, COUNT, MIN, MAX, SUM, AVG]
    cols, ins = [[k]] * 4 + [[k + 1]] * 2, [[L]] * 4 + [[D]] * 2
    if case["stages"] == 1:
        return [omg.HashAggregationOperatorFactory(gb, kt, cols, ins, [[L]] * 4 + [[D], [D]], funcs)]
    partial = omg.HashAggregationOperatorFactory(gb, kt, cols, ins, [[L]] * 4 + [[D], [D, L]], funcs,
                                                 output_partials=[True] * 6)
    merge = [[k + i] for i in range(5)] + [[k + 5, k + 6]]
    final = omg.HashAggregationOperatorFactory(gb, kt, merge, [[L]] * 4 + [[D], [D, L]], [[L]] * 4 + [[D], [D]], funcs,
                                               input_raws=[False] * 6)
    return [partial, final]


def _join_key(case, code):
    if case["key"] == "dense":
        return [code]
    if case["key"] == "sparse":
        return [_spread(code)]
    return [(code >> 10).to(torch.int32), (code & 1023).to(torch.int32)]


def _join_inputs(case, seed):
    """The build side has build // dup keys, `dup` rows each; a fifth of the probe rows match none, and
    one in a hundred has a NULL key."""
    g = _gen(seed)
    n, dup = case["probe"], case["dup"]
    keys = case["build"] // dup
    nb = keys * dup
    perm = torch.randperm(nb, generator=g, device=DEV)
    bcode = perm // dup
    if case["payload"] == "int2":
        pay = [torch.randint(-2**31, 2**31, (nb,), generator=g, device=DEV, dtype=torch.int64).to(torch.int32),
               (perm % dup).to(torch.int32)]
    else:
        pay = [torch.randint(-2**62, 2**62, (nb,), generator=g, device=DEV, dtype=torch.int64), perm % dup]
    code = _codes(case["dist"], n, keys, g)
    miss = torch.randint(keys, 2 * keys + 1, (n,), generator=g, device=DEV, dtype=torch.int64)
    code = torch.where(torch.rand(n, generator=g, device=DEV) < 0.8, code, miss)
    null = torch.rand(n, generator=g, device=DEV) < 0.01
    return {"bkey": _join_key(case, bcode), "pay": pay, "pkey": _join_key(case, code), "null": null}


def _join_types(case):
    key = [I, I] if case["key"] == "pair" else [L]
    pay = [I, I] if case["payload"] == "int2" else [L, L]
    return key, pay


# ---------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    return {"agg": _prepare_agg, "tasks": _prepare_tasks, "join": _prepare_join}[case["family"]](case, seed)


def _prepare_agg(case, seed):
    x = _agg_inputs(case, seed)
    types = _key_types(case) + _val_types(case)
    st = State(case=case, types=types, factories=_agg_factories(case), n_id=len(x["keys"]),
               most=_most_groups(case))
    st.closing += [f.close for f in st.factories]
    if case["key"] == "varchar":
        words = _words(case["groups"])
        cols = [words[x["code"].cpu().numpy()]] + [v.cpu().numpy() for v in x["vals"]]
        masks = [None] + [None if m is None else m.cpu().numpy() for m in x["nulls"]]
        st.host = omg.make_batch(types, cols, masks)
        st.closing.append(lambda h=st.host: omg.free_batch(h))
    elif case["input"] == "host":
        cols = [c.cpu().numpy() for c in x["keys"] + x["vals"]]
        masks = [None] * len(x["keys"]) + [None if m is None else m.cpu().numpy() for m in x["nulls"]]
        st.parts = [([c[s:s + BATCH] for c in cols], [None if m is None else m[s:s + BATCH] for m in masks])
                    for s in range(0, case["rows"], BATCH)]
    else:
        st.cols = x["keys"] + x["vals"]
        st.bits = [None] * len(x["keys"]) + [None if m is None else _bitmap(m) for m in x["nulls"]]
    return st


def _prepare_tasks(case, seed):
    g = _gen(seed)
    rng = np.random.default_rng(case["tasks"])
    rows = np.exp(rng.uniform(np.log(case["rows_min"]), np.log(case["rows_max"]), case["tasks"])).astype(np.int64)
    domains = np.maximum(np.exp(rng.uniform(np.log(10), np.log(np.minimum(rows, 1_000_000)))).astype(np.int64), 2)
    offs = np.concatenate([[0], np.cumsum(rows)])
    n = int(offs[-1])
    dom = torch.repeat_interleave(torch.from_numpy(domains).to(DEV), torch.from_numpy(rows).to(DEV))
    task = torch.repeat_interleave(torch.arange(case["tasks"], device=DEV), torch.from_numpy(rows).to(DEV))
    code = (torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * dom).long()
    keys = _spread(code + task * 1_000_003)
    vals = torch.randint(-10**6, 10**6 + 1, (n,), generator=g, device=DEV, dtype=torch.int64)
    fac = omg.HashAggregationOperatorFactory([0], [L], [[1], [1]], [[L], [L]], [[L], [L]], [SUM, COUNT])
    handles = [omg.wrap_device_batch([L, L], int(r), [keys.data_ptr() + 8 * int(o), vals.data_ptr() + 8 * int(o)])
               for o, r in zip(offs[:-1], rows)]
    model = SizingModel.load("omnioperator_gb300/models/agg_task_sizer.json")
    torch.cuda.synchronize()
    batch = omg.AggBatch(fac, handles, sizer=model, flags=omg.BATCH_DEVICE_OUTPUT)
    # The tasks' sizes come from the case alone, so that all seeds' outputs have the same bound.
    st = State(case=case, keys=keys, vals=vals, batch=batch, most=int(domains.sum()))
    st.closing += [fac.close, model.close, lambda: omg.free_batches(handles), batch.close]
    return st


def _prepare_join(case, seed):
    x = _join_inputs(case, seed)
    key, pay = _join_types(case)
    st = State(case=case, x=x, key=key, pay=pay, splits=None)
    if case["built"] == "before":
        st.bf, st.bop, st.pf = _build(st)
        st.closing += [st.bf.close, st.bop.delete, st.pf.close]
    if case["strategy"] == "range_partitioned":
        sample = x["pkey"][0][:: max(1, case["probe"] // 65536)].cpu().numpy()
        st.splits = omg.quantile_splits(sample, bits=12)
    if case["input"] == "host":
        cols = [c.cpu().numpy() for c in x["pkey"]]
        null = x["null"].cpu().numpy()
        st.parts = [([c[s:s + BATCH] for c in cols], [null[s:s + BATCH]] + [None] * (len(cols) - 1))
                    for s in range(0, case["probe"], BATCH)]
    else:
        st.bits = _bitmap(x["null"])
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------------- run
def run(state):
    return {"agg": _run_agg, "tasks": _run_tasks, "join": _run_join}[state.case["family"]](state)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _aggregate(factory, batches, device):
    op = factory.create_operator()
    op.set_stream(_stream())
    op.set_device_output(device)
    for b in batches:
        op.add_input(b)
    outs, _ = op.get_outputs()
    op.delete()
    return outs


def _wrap_rows(types, cols, bits, lo, hi):
    return omg.wrap_device_batch(types, hi - lo, [c.data_ptr() + lo * c.element_size() for c in cols],
                                 [None if b is None else b.data_ptr() + lo // 8 for b in bits])


def _run_agg(st):
    case = st.case
    if case["key"] == "varchar":
        return Rows(_aggregate(st.factories[0], [omg.batch_to_device(st.host)], False), st.n_id, st.most)
    if case["input"] == "host":
        batches = [omg.make_batch(st.types, cols, masks) for cols, masks in st.parts]
        return Rows(_aggregate(st.factories[0], batches, False), st.n_id, st.most)
    rows = case["rows"]
    if case["stages"] == 1:
        batch = _wrap_rows(st.types, st.cols, st.bits, 0, rows)
        return Rows(_aggregate(st.factories[0], [batch], True), st.n_id, st.most)
    cut = [rows * q // 4 // 64 * 64 for q in range(4)] + [rows]
    partials = []
    for lo, hi in zip(cut[:-1], cut[1:]):
        partials += _aggregate(st.factories[0], [_wrap_rows(st.types, st.cols, st.bits, lo, hi)], True)
    return Rows(_aggregate(st.factories[1], partials, True), st.n_id, st.most)


def _run_tasks(st):
    st.batch.run(_stream())
    outs = st.batch.outputs()
    return Rows([b for _, b in outs], 2, st.most, [t for t, _ in outs])


def _build(st):
    """HashBuilder over the build side, and the probe factory on it."""
    case, x = st.case, st.x
    types = st.key + st.pay
    nk = len(st.key)
    bf = omg.HashBuilderOperatorFactory(JOIN_TYPES[case["kind"]], types, list(range(nk)))
    bop = bf.create_operator()
    bop.set_stream(_stream())
    bop.add_input(omg.wrap_device_batch(types, len(x["pay"][0]), [c.data_ptr() for c in x["bkey"] + x["pay"]]))
    bop.get_output()
    filt = None
    if case["filter"]:  # build payload 0 >= 0
        filt = omg.Binary(omg.EXPR_GTE, omg.Field(nk + nk, st.pay[0]), omg.Literal(0, st.pay[0]))
    emits = case["kind"] in ("inner", "left")
    pf = omg.LookupJoinOperatorFactory(st.key, list(range(nk)), list(range(nk)), [nk, nk + 1] if emits else [],
                                       st.pay if emits else [], bf, filter_expr=filt)
    return bf, bop, pf


def _run_join(st):
    case, x = st.case, st.x
    each = case["built"] == "each"
    bf, bop, pf = _build(st) if each else (st.bf, st.bop, st.pf)
    op = pf.create_operator()
    op.set_stream(_stream())
    if case["input"] == "host":
        for cols, masks in st.parts:
            op.add_input(omg.make_batch(st.key, cols, masks))
    else:
        op.set_device_output(True)
        if case["strategy"] != "direct":
            op.set_join_strategy(omg.JOIN_HASH_PARTITIONED if case["strategy"] == "hash_partitioned"
                                 else omg.JOIN_RANGE_PARTITIONED, 12, st.splits)
        op.add_input(omg.wrap_device_batch(st.key, case["probe"], [c.data_ptr() for c in x["pkey"]],
                                           [st.bits.data_ptr()] + [None] * (len(st.key) - 1)))
    outs, _ = op.get_outputs()
    op.delete()
    if each:
        pf.close()
        bop.delete()
        bf.close()
    return Rows(outs, 4, _most_joined(case))  # sorted by all columns


# ---------------------------------------------------------------------------------- work, exact
def _distinct(rows, domain, dist):
    """Expected distinct codes among `rows` draws."""
    if dist == "uniform":
        return domain * -math.expm1(-rows / domain)
    edges = np.unique(np.round(np.geomspace(1, domain + 1, 4000)).astype(np.int64))
    w = np.diff(edges)
    p = -np.diff(edges ** -0.1) / w / (1 - (domain + 1.0) ** -0.1)  # a rank's mean share per interval
    return float((w * -np.expm1(-rows * p)).sum())


def _most_groups(case):
    return min(case["groups"], int(_distinct(case["rows"], case["groups"], case["dist"]) * 1.1) + 1000)


def _most_joined(case):
    n, dup = case["probe"], case["dup"]
    hits = 0.8 * 0.99 * n
    slack = 4 * math.sqrt(n) + 10
    hits, misses = int(min(n, hits + slack)), int(min(n, n - hits + slack))
    return {"inner": hits * dup, "left": hits * dup + misses, "semi": hits, "anti": misses}[case["kind"]]


def work(case):
    if case["family"] == "agg":
        kw = {"long": 8, "pair": 12, "pair_int": 8, "varchar": 7 + 8 + 4}[case["key"]]
        vw = {"six": 16, "sum_count": 8, "decimal": 16 + 0.25}[case["plan"]]
        ow = {"six": 48, "sum_count": 16, "decimal": 32}[case["plan"]]
        return {"bytes": case["rows"] * (kw + vw) + _distinct(case["rows"], case["groups"], case["dist"]) * (kw + ow),
                "flops": 0}
    if case["family"] == "tasks":
        rows, groups = 0.0, 0.0
        for u in (np.arange(64) + 0.5) / 64:  # log-uniform rows, and domains up to the rows
            r = case["rows_min"] * (case["rows_max"] / case["rows_min"]) ** u
            d = 10 * (min(r, 1e6) / 10) ** ((np.arange(64) + 0.5) / 64)
            rows += case["tasks"] / 64 * r
            groups += case["tasks"] / 64 * float((d * -np.expm1(-r / d)).mean())
        return {"bytes": rows * 16 + groups * 24, "flops": 0}
    pay = 8 if case["payload"] == "int2" else 16
    hits = 0.8 * 0.99 * case["probe"]
    out = {"inner": hits * case["dup"] * (8 + pay), "left": (hits * case["dup"] + case["probe"] - hits) * (8 + pay),
           "semi": hits * 8, "anti": (case["probe"] - hits) * 8}[case["kind"]]
    if case["filter"]:
        out = out / 2 if case["kind"] == "inner" else out
    build = case["build"] * (8 + pay) if case["built"] == "each" else 0
    return {"bytes": case["probe"] * (8 + 1 / 8) + out + build, "flops": 0}


def exact(case, seed):
    """The SUM and AVG of doubles; the other outputs are whole numbers."""
    if case["family"] != "agg" or case["plan"] == "sum_count":
        return None
    x = _agg_inputs(case, seed)
    codes, inv = torch.unique(x["code"], return_inverse=True)
    v, null = x["vals"][1], x["nulls"][1]
    live = torch.ones_like(v) if null is None else (~null).double()
    total = torch.zeros(len(codes), dtype=torch.float64, device=DEV).index_add_(0, inv, v * live)
    n = torch.zeros(len(codes), dtype=torch.float64, device=DEV).index_add_(0, inv, live)
    avg = torch.where(n > 0, total / n.clamp(min=1), torch.zeros_like(total))
    if case["key"] == "varchar":
        by = torch.arange(len(codes), device=DEV)  # the words begin with the padded code
    elif case["key"] == "long":
        by = torch.argsort(_spread(codes))
    elif case["key"] == "pair":
        by = torch.argsort(_spread(codes))
        by = by[torch.sort((codes % 65521)[by], stable=True).indices]
    else:
        by = torch.argsort((codes % 3) * (1 << 32) + codes // 3)
    k = 2 * len(x["keys"])
    total, avg = (_filled(v[by], _most_groups(case), 0) for v in (total, avg))
    if case["plan"] == "decimal":
        return [None] * (k + 4) + [avg, None, None]
    return [None] * (k + 8) + [total, None, avg, None, None]
