"""The calls whose speed matters: what programs built on this framework have
it do, from one small synchronous batch to full resident ones.

Every case goes through the package's public entry points.  Inputs come from
the framework's seeded generators (ltp_gen_ycsb, ltp_tpcc_gen), so they are a
function of the seed alone; op values and commit flags come back whole.  The
table state a pass leaves behind shows in the values of the pass after it
(every op returns its cell's value), and the insert workloads read back rows
that an earlier batch of the same pass inserted.
"""
import ctypes
import math

import numpy as np
import torch

import ltpmg_gb300 as G

M64 = (1 << 64) - 1


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A host program with a handful of transactions in hand: load, execute, results, and it waits for
        # them (the reference's per-epoch transfer / execute sequence at its smallest).  Latency.
        dict(name="call 64x10", kind="call", rows=1 << 20, txns=64, omin=10, omax=10, read=0.5, theta=0.0, rule=0,
             key32=False),
        # The same call with the smoke test's batch: 2048 x 16 under Zipf 0.99, transactions of equal length.
        dict(name="call 2048x16 zipf", kind="call", rows=1 << 20, txns=2048, omin=16, omax=16, read=0.8, theta=0.99,
             rule=0, key32=True),
        # An order-entry epoch of a small site, synchronous: int64 money, linked inserts, 64-bit results.
        dict(name="orders call", kind="orders", warehouses=2, txns=1500, batches=1, call=True),
        # The small end of the uneven-batching configuration: resident batches of 2^10..2^14 transactions with
        # 1-32 ops each, replayed from one captured graph.
        dict(name="uneven small", kind="list", rows=1 << 24, lo=1 << 10, hi=1 << 14, batches=12, omin=1, omax=32,
             read=0.7, theta=0.8, rule=0, key32=False),
        # The plain configuration: uniform keys, 2^16 x 10, resident batches in one graph.
        dict(name="plain 65536x10", kind="list", rows=1 << 20, lo=1 << 16, hi=1 << 16, batches=4, omin=10, omax=10,
             read=0.5, theta=0.0, rule=0, key32=True),
        # The priority rule (optimistic clients that re-submit what aborted), resident.
        dict(name="priority 131072x16", kind="list", rows=1 << 22, lo=1 << 17, hi=1 << 17, batches=1, omin=16, omax=16,
             read=0.8, theta=0.7, rule=1, key32=False),
        # The headline configuration: 2^20 transactions x 16 ops, Zipf 0.99 over 2^24 rows.
        dict(name="zipf 1048576x16", kind="list", rows=1 << 24, lo=1 << 20, hi=1 << 20, batches=1, omin=16, omax=16,
             read=0.8, theta=0.99, rule=0, key32=True),
        # The large end of the uneven configuration: odd sizes up to 2^20 transactions.
        dict(name="uneven large", kind="list", rows=1 << 24, lo=1 << 14, hi=900001, batches=4, omin=1, omax=32,
             read=0.7, theta=0.9, rule=0, key32=False),
        # Order entry, resident: two batches and an order-status batch over the rows just inserted.
        dict(name="orders resident", kind="orders", warehouses=8, txns=1 << 16, batches=2, call=False),
        # YCSB-E: scans of two rows, some of them over the newest rows, and an insert per transaction.
        dict(name="scans 32768x55", kind="scans", rows=1 << 20, txns=1 << 15, theta=0.99),
        # A client that streams batches from host memory through the pipeline and takes the results back.
        dict(name="pipe 6x32768x10", kind="pipe", rows=1 << 20, txns=1 << 15, batches=6, omin=10, omax=10, read=0.5,
             theta=0.6, key32=True),
        # The request-log server working off a backlog in batches of at most 4096 requests.
        dict(name="serve backlog", kind="serve", rows=1 << 22, requests=1 << 15, most=1 << 12, omin=16, omax=16,
             read=0.8, theta=0.99),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "list", "list", "list", "list", "orders", "scans", "pipe", "serve"])
    omin, omax = rng.choice([(10, 10), (16, 16), (1, 32), (4, 11), (7, 7)])
    read = rng.choice([0.5, 0.7, 0.8, 0.95])
    theta = rng.choice([0.0, 0.6, 0.8, 0.9, 0.99])
    rows = _log_int(rng, 1 << 16, 1 << 24)
    key32 = rng.random() < 0.5
    rule = 1 if rng.random() < 0.25 else 0
    if kind == "call":
        return dict(kind=kind, rows=rows, txns=_log_int(rng, 1, 1 << 14), omin=omin, omax=omax, read=read, theta=theta,
                    rule=rule, key32=key32)
    if kind == "list":
        a, b = sorted((_log_int(rng, 1 << 10, 1 << 20), _log_int(rng, 1 << 10, 1 << 20)))
        most = max(1, min(12, (14 << 20) // (b * omax)))  # no more work than the headline batch
        b = min(b, (14 << 20) // omax)
        return dict(kind=kind, rows=rows, lo=min(a, b), hi=b, batches=rng.randint(1, most), omin=omin, omax=omax,
                    read=read, theta=theta, rule=rule, key32=key32)
    if kind == "orders":
        call = rng.random() < 0.4
        return dict(kind=kind, warehouses=rng.randint(1, 8), txns=_log_int(rng, 100, 5000 if call else 100000),
                    batches=1 if call else rng.randint(1, 3), call=call)
    if kind == "scans":
        return dict(kind=kind, rows=_log_int(rng, 1 << 16, 1 << 21), txns=_log_int(rng, 1 << 9, 1 << 16), theta=theta)
    if kind == "pipe":
        return dict(kind=kind, rows=rows, txns=_log_int(rng, 1 << 10, 1 << 17), batches=rng.randint(3, 8), omin=omin,
                    omax=omax, read=read, theta=theta, key32=key32)
    most = _log_int(rng, 1 << 9, 1 << 14)
    return dict(kind="serve", rows=rows, requests=most * rng.randint(3, 9) + rng.randint(0, 500), most=most, omin=omin,
                omax=omax, read=read, theta=theta)


def _sizes(case):
    """Transactions per batch of a list: log-uniform steps from lo to hi, large and small ones in turn."""
    n, lo, hi = case["batches"], case["lo"], case["hi"]
    s = [int(round(lo * (hi / lo) ** (k / (n - 1)))) if n > 1 else hi for k in range(n)]
    return [s[k // 2] if k % 2 else s[n - 1 - k // 2] for k in range(n)]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
COLS = 10  # the YCSB table of every configuration: 10 int32 columns
ORDER_TABLES = {3: "history", 4: "new_order", 5: "order", 6: "order_line"}  # the tables that grow


def _ycsb(case, seed, b, n):
    """One batch: transactions of omin..omax ops; how long each one is goes by the case, what it does by the seed."""
    omin, omax = case["omin"], case["omax"]
    _, keys, opw = G.gen_ycsb(seed, case["rows"], COLS, omax, omax, case["read"], case["theta"], batch=b, n_txns=n)
    if case.get("key32"):
        keys = keys.astype(np.uint32)
    if omin == omax:
        return None, keys, opw, omax, None
    lens = np.random.default_rng(b).integers(omin, omax + 1, n)
    used = (np.arange(omax) < lens[:, None]).reshape(-1)
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32), keys[used], opw[used], 0, None


def _order_batch(g, b, n):
    """A batch of ltp_tpcc_gen with its mix made even: as many new-orders of every length as of any other, and as
    many payments as new-orders."""
    made = 2 * n + 200
    while True:
        tf, keys, opw, pay, _, _, pf = g.gen(b, made, with_pay_first=True)
        tf, pf, lens = tf.astype(np.int64), pf.astype(np.int64), np.diff(tf.astype(np.int64))
        kinds = [5 + 3 * lines for lines in range(5, 16)]
        share = {k: (n // 2 + i) // len(kinds) for i, k in enumerate(kinds)}
        share[7] = n - sum(share.values())
        kept = [np.flatnonzero(lens == k)[:m] for k, m in share.items()]
        if all(len(x) == m for x, m in zip(kept, share.values())):
            break
        made *= 2
    kept = np.sort(np.concatenate(kept))
    lens, slots = lens[kept], np.diff(pf)[kept]
    first, pay_first = np.concatenate([[0], np.cumsum(lens)]), np.concatenate([[0], np.cumsum(slots)])
    src = np.repeat(tf[kept] - first[:-1], lens) + np.arange(first[-1])
    pay_src = np.repeat(pf[kept] - pay_first[:-1], slots) + np.arange(pay_first[-1])
    keys, opw = keys[src].astype(np.int64), opw[src]
    keys += np.where(opw & 3 == G.OP_INSERT, np.repeat(pay_first[:-1] - pf[kept], lens), 0)
    return first.astype(np.uint32), keys.astype(np.uint64), opw, 0, pay[pay_src]


def _orders(case, seed):
    """Order-entry batches; a resident list ends with an order-status batch: every column of order and order-line
    rows that the first batch inserted."""
    g = G.Tpcc(case["warehouses"], seed=seed, items=20000)
    batches = [_order_batch(g, b, case["txns"]) for b in range(case["batches"])]
    new = [[int(((d[2] & 3 == G.OP_INSERT) & (d[2] >> 8 & 15 == t)).sum()) for t in range(9)] for d in batches]
    grow = np.sum(new, axis=0)
    if not case["call"]:
        rng = np.random.default_rng(seed)
        n = max(1, case["txns"] // 16)
        keys, opw, lens = [], [], []
        for t in (5, 6):
            cols, ins = g.table(t)[0], new[0][t]
            keys.append(np.repeat(rng.integers(0, ins, n), cols))
            opw.append(np.tile(np.arange(cols, dtype=np.uint32) << 2 | np.uint32(t << 8), n))
            lens.append(np.full(n, cols))
        tf = np.concatenate([[0], np.cumsum(np.concatenate(lens))]).astype(np.uint32)
        batches.append((tf, np.concatenate(keys).astype(np.uint64), np.concatenate(opw).astype(np.uint32), 0, None))
    return g, batches, grow


SCAN_COLS = 3


def _scans(case, seed):
    """Two batches of 9 two-row scans and one insert per transaction; an eighth of the second batch's scans read
    rows that the first one inserted."""
    n, rows = case["txns"], case["rows"]
    rng = np.random.default_rng(seed)
    out = []
    for b in range(2):
        _, k, _ = G.gen_ycsb(seed, rows, SCAN_COLS, 10, 10, 1.0, case["theta"], batch=b, n_txns=n)
        k = k.reshape(n, 10).astype(np.int64)
        first = k[:, :9].copy()
        if b:
            first = np.where(rng.random((n, 9)) < 0.125, rows + rng.integers(0, max(1, n - 1), (n, 9)), first)
        first = np.minimum(first, rows + (n - 2 if b and n > 1 else -2))
        scan = first[:, :, None] + np.arange(2)
        keys = np.concatenate([np.repeat(scan.reshape(n, 18), SCAN_COLS, axis=1),
                               np.arange(n)[:, None] * SCAN_COLS], axis=1)
        opw = np.concatenate([np.tile((np.arange(SCAN_COLS) << 2).astype(np.uint32), (n, 18)),
                              np.full((n, 1), G.OP_INSERT, np.uint32)], axis=1)
        pay = np.repeat(k[:, 9], SCAN_COLS).astype(np.int32)
        out.append((None, keys.reshape(-1).astype(np.uint32), opw.reshape(-1).astype(np.uint32), 18 * SCAN_COLS + 1, pay))
    return out


# ---------------------------------------------------------------------------
# what a program keeps
# ---------------------------------------------------------------------------
class _Device:
    """A device array as torch sees it (and the objects that keep it alive)."""

    def __init__(self, ptr, n, code, keep):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": code, "data": (ptr, False), "version": 2}


class State:
    def __init__(self):
        self.pipe = self.ingest = self.ctx = None
        self.batches = []

    def __del__(self):
        try:
            torch.cuda.synchronize()
            for x in (self.ingest, self.pipe):
                if x is not None:
                    x.close()
            for b in self.batches:
                b.free()
            if self.ctx is not None:
                self.ctx.close()
        except Exception:
            pass


_stream = None


def _the_stream():
    """The stream a program runs its work on (one for all the states that it holds)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _load(s, data, stream=None):
    for tf, keys, opw, fixed, pay in data:
        b = s.ctx.batch(len(tf) - 1 if tf is not None else len(keys) // fixed, len(keys))
        b.load(tf, keys, opw, ops_per_txn=fixed, stream=stream)
        if pay is not None:
            b.load_payload(pay, stream=stream)
        s.batches.append(b)
    s.ctx.sync(stream)


def _views(s):
    """Commit flags and op values of the resident batches, where they are."""
    out = []
    for b in s.batches:
        vals, commit = ctypes.c_void_p(), ctypes.c_void_p()
        s.ctx.check(s.ctx.L.ltp_batch_device_ptrs(b.h, None, None, None, ctypes.byref(vals), ctypes.byref(commit)))
        out.append({"commit": torch.as_tensor(_Device(commit.value, b.n_txns, "|u1", s), device="cuda"),
                    "vals": torch.as_tensor(_Device(vals.value, b.n_ops, "<i4", s), device="cuda")})
    return out


def _passes_kept(bytes_per_pass):
    """How many passes' rows an insert workload has room for before it drops them (a table's retention)."""
    return int(max(2, min(64, (2 << 30) // max(1, bytes_per_pass))))


def prepare(case, seed):
    s = State()
    s.kind = case["kind"]
    s.ctx = G.Context(rule=case.get("rule", 0))
    s.grown, s.passes, s.mode = {}, 0, G.MODE_GRAPH
    if s.kind == "orders":
        g, data, grow = _orders(case, seed)
        s.keep = _passes_kept(int(sum(int(grow[t]) * 4 * (g.table(t)[0] + 2) for t in range(9))))
        ids = g.create_tables(s.ctx, grow * s.keep)
        s.grown = {ids[t]: 0 for t in ORDER_TABLES}
        g.close()
    elif s.kind == "scans":
        data = _scans(case, seed)
        s.keep = _passes_kept(2 * case["txns"] * SCAN_COLS * 4)
        t = s.ctx.create_table(case["rows"], SCAN_COLS, rows_cap=case["rows"] + 2 * case["txns"] * s.keep)
        s.ctx.fill_seeded(t, seed)
        s.grown = {t: case["rows"]}
    else:
        t = s.ctx.create_table(case["rows"], COLS)
        s.ctx.fill_seeded(t, seed)
        if s.kind == "call":
            data = [_ycsb(case, seed, 0, case["txns"])]
        elif s.kind == "list":
            data = [_ycsb(case, seed, b, n) for b, n in enumerate(_sizes(case))]
        elif s.kind == "pipe":
            data = [_ycsb(case, seed, b, case["txns"]) for b in range(case["batches"])]
        else:
            data = [_ycsb(case, seed, 0, case["requests"])]
    s.ctx.sync()
    if s.kind == "serve":
        tf, keys, opw, fixed, _ = data[0]
        tf = np.arange(0, len(keys) + 1, fixed) if fixed else tf
        s.ingest = G.Ingest(s.ctx, tf, keys, opw, deadline_us=250, depth=3, max_txns=case["most"],
                            max_ops=case["most"] * case["omax"], keep_results=True)
        s.arrivals = np.zeros(case["requests"], np.uint64)  # all of them are waiting
    elif s.kind == "pipe":
        pin = lambda a: torch.from_numpy(np.array(a)).pin_memory()  # noqa: E731
        s.host, s.results = [], []
        for tf, keys, opw, fixed, _ in data:
            arrays = [None if a is None else pin(a) for a in (tf, keys, opw)]
            n = case["txns"]
            res = {"commit": torch.empty(n, dtype=torch.uint8, pin_memory=True),
                   "vals": torch.empty(len(keys), dtype=torch.int32, pin_memory=True)}
            s.host.append([None if a is None else a.numpy() for a in arrays] + [fixed, arrays])
            s.results.append(res)
        s.pipe = G.Pipe(s.ctx, 3, case["txns"], max(len(d[1]) for d in data))
    elif s.kind == "call" or case.get("call"):
        s.data = data[0]
        tf, keys, _, fixed, _ = data[0]
        s.batches.append(s.ctx.batch(len(tf) - 1 if tf is not None else len(keys) // fixed, len(keys)))
        s.wide = s.kind == "orders"
    else:
        _load(s, data, _the_stream())
    return s


def _make_room(s):
    """Every `keep` passes the rows that the workload inserted are dropped."""
    if s.grown:
        if s.passes == s.keep:
            torch.cuda.synchronize()
            for t, rows in s.grown.items():
                s.ctx.truncate(t, rows)
            s.passes = 0
        s.passes += 1


def run(state):
    s = state
    _make_room(s)
    if s.kind == "serve":
        s.ingest.run(s.arrivals)
        committed, _, _, _, vals = s.ingest.results(values=True)
        return {"commit": committed, "vals": vals}
    if s.kind == "pipe":
        tickets = []
        for (tf, keys, opw, fixed, _), r in zip(s.host, s.results):
            tickets.append(s.pipe.submit(tf, keys, opw, commit_out=r["commit"].numpy(), vals_out=r["vals"].numpy(),
                                         ops_per_txn=fixed))
        for t in tickets:
            s.pipe.wait(t)
        return s.results
    if hasattr(s, "data"):
        tf, keys, opw, fixed, pay = s.data
        b = s.batches[0]
        b.load(tf, keys, opw, ops_per_txn=fixed)
        if pay is not None:
            b.load_payload(pay)
        b.execute()
        commit, vals, _ = b.results64() if s.wide else b.results()
        return [{"commit": commit, "vals": vals}]
    if len(s.batches) == 1:
        s.batches[0].execute(stream=_the_stream())
    else:
        s.ctx.execute_many(s.batches, mode=s.mode, stream=_the_stream())
    return _views(s)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    k = case["kind"]
    if k == "orders":
        # per transaction 21 ops: half are new-orders (3 reads / RMWs, 2 + 10 inserts, 20 RMWs), half payments
        # (1 read, 5 RMWs, 1 insert); an order line is 15 slots, an order 7, a new-order 3, a history row 13
        n = case["txns"] * case["batches"]
        ops, rows_b = 21 * n, 4 * n * (0.5 * (10 * 15 + 7 + 3) + 0.5 * 13)
        out = 8 if case["call"] else 4
        b = ops * (8 + 4 + out) + 2 * rows_b + n * (0.5 * (20 * 12 + 8) + 0.5 * 72) + 5 * n
        if not case["call"]:
            b += 22 * max(1, case["txns"] // 16) * 20
        return {"bytes": b, "flops": 0}
    if k == "scans":
        n = 2 * case["txns"]
        return {"bytes": n * (55 * (4 + 4 + 4) + 54 * 4 + 2 * 4 * SCAN_COLS + 1), "flops": 0}
    if k == "list":
        txns, key = sum(_sizes(case)), 4 if case["key32"] else 8
    elif k == "serve":
        txns, key = case["requests"], 4
    else:
        txns, key = case["txns"] * case.get("batches", 1), 4 if case["key32"] else 8
    ops = txns * (case["omin"] + case["omax"]) / 2
    # per op its key, opword, the cell's value read, an RMW's written, the output (64 bits from the server);
    # per transaction its commit flag and, where lengths differ, its first op
    per = key + 4 + 4 + 4 * (1 - case["read"]) + (8 if k == "serve" else 4)
    return {"bytes": ops * per + txns * (1 if case["omin"] == case["omax"] else 5), "flops": 0}


# ---------------------------------------------------------------------------
# the same in plain numpy
# ---------------------------------------------------------------------------
def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _cells(seed, rows, cols, key, col):
    """Initial values of a seeded table's cells."""
    base = _mix(np.array([(seed ^ 0x5441424C45) & M64], np.uint64))
    return _mix(base + key.astype(np.uint64) * np.uint64(cols) + col.astype(np.uint64)).astype(np.uint32).view(np.int32).astype(np.int64)


class _Cells:
    """Cell values by number, for the cells that some op changed; the others come from `initial(table, key, col)`."""

    def __init__(self, initial, wide, rows):
        self.initial, self.wide, self.rows = initial, wide, dict(rows)
        self.ids, self.vals = np.zeros(0, np.int64), np.zeros(0, np.int64)

    def number(self, tb, key, col):
        return (tb << 48) | (key << 8) | col

    def get(self, cell):
        tb, key, col = cell >> 48, (cell >> 8) & ((1 << 40) - 1), cell & 255
        out = np.zeros(len(cell), np.int64)
        pos = np.searchsorted(self.ids, cell)
        known = pos < len(self.ids)
        known[known] = self.ids[pos[known]] == cell[known]
        out[known] = self.vals[pos[known]]
        for t in np.unique(tb[~known]):
            m = ~known & (tb == t)
            out[m] = self.initial(int(t), key[m], col[m])
        return out

    def put(self, cell, val):
        ids, vals = np.concatenate([cell, self.ids]), np.concatenate([val, self.vals])
        self.ids, first = np.unique(ids, return_index=True)
        self.vals = vals[first]

    def is_wide(self, cell):
        return np.isin((cell >> 48 << 8) | (cell & 255), self.wide)

    def wrap(self, cell, v):
        return np.where(self.is_wide(cell), v, v.astype(np.int32).astype(np.int64))


def _replay(tab, data, rule=0, n_cols=None):
    """One batch in serial order: (commit, op values), with the cells' new values kept in `tab`."""
    tf, keys, opw, fixed, pay = data
    n = len(keys)
    keys, w = keys.astype(np.int64), opw.astype(np.int64)
    tid = np.arange(n) // fixed if fixed else np.repeat(np.arange(len(tf) - 1), np.diff(tf.astype(np.int64)))
    n_txns = n // fixed if fixed else len(tf) - 1
    kind, col, tb = w & 3, (w >> 2) & 63, (w >> 8) & 15
    imm = np.where(kind == 1, opw.view(np.int32).astype(np.int64) >> 12, 0)
    vals, commit = np.zeros(n, np.int64), np.ones(n_txns, np.uint8)
    op = np.flatnonzero(kind < 2)
    cell = tab.number(tb[op], keys[op], col[op])
    uniq, cid = np.unique(cell, return_inverse=True)
    base = tab.get(uniq)
    if rule == 1:  # a transaction aborts when a smaller one writes a cell that it uses
        least = np.full(len(uniq), n_txns)
        wr = kind[op] == 1
        np.minimum.at(least, cid[wr], tid[op][wr])
        commit[tid[op][least[cid] < tid[op]]] = 0
        live = commit[tid[op]] == 1
        op, cid = op[live], cid[live]
        group = cid * (n_txns + 1) + tid[op]
    else:
        group = cid
    order = np.argsort(group, kind="stable")
    go, run_sum = group[order], np.cumsum(imm[op][order])
    head = np.concatenate([[True], go[1:] != go[:-1]]) if len(go) else np.zeros(0, bool)
    before = (run_sum - imm[op][order])[head]
    run_sum = run_sum - np.repeat(before, np.diff(np.append(np.flatnonzero(head), len(go))))
    v = tab.wrap(uniq[cid[order]], base[cid[order]] + run_sum)
    vals[op[order]] = v
    last = np.append(head[1:], True) if len(go) else head
    if rule == 1:  # only the smallest writer stores
        last = last & (least[cid[order]] == tid[op[order]])
    tab.put(uniq[cid[order][last]], v[last])
    for t in np.unique(tb[kind == 2]):
        ins = np.flatnonzero((kind == 2) & (tb == t))
        row = tab.rows[int(t)] + np.arange(len(ins))
        vals[ins] = row
        slot = 0
        for c in range(n_cols[int(t)]):
            wide = bool(np.isin((int(t) << 8) | c, tab.wide))
            x = pay[keys[ins] + slot].astype(np.int64)
            if wide:
                x = (pay[keys[ins] + slot + 1].astype(np.int64) << 32) | (x & 0xFFFFFFFF)
            dist = (w[ins] >> 12) & 0x3FF
            link = (dist > 0) & (col[ins] == c)
            x[link] = vals[ins[link] - dist[link]]
            cells = tab.number(np.int64(t), row, np.int64(c))
            tab.put(cells, tab.wrap(cells, x))
            slot += 2 if wide else 1
        tab.rows[int(t)] += len(ins)
    return commit, vals


def exact(case, seed):
    k = case["kind"]
    if k == "orders":
        g, data, _ = _orders(case, seed)
        shape = [g.table(t) for t in range(9)]
        cols = {(t, c): g.column(t, c).astype(np.int64) for t in range(9) if shape[t][2] for c in range(shape[t][0])}

        def initial(t, key, col):
            out = np.zeros(len(key), np.int64)
            for c in np.unique(col):
                out[col == c] = cols[t, int(c)][key[col == c]]
            return out

        wide = np.array([(t << 8) | c for t in range(9) for c in range(shape[t][0]) if (shape[t][1] >> c) & 1])
        tab = _Cells(initial, wide, {t: shape[t][2] for t in range(9)})
        out = [_replay(tab, d, n_cols={t: shape[t][0] for t in range(9)}) for d in data]
        return [{"commit": c, "vals": v if case["call"] else v.astype(np.int32)} for c, v in out]
    if k == "serve":
        data = [_ycsb(case, seed, 0, case["requests"])]
    elif k == "scans":
        data = _scans(case, seed)
    elif k == "list":
        data = [_ycsb(case, seed, b, n) for b, n in enumerate(_sizes(case))]
    else:
        data = [_ycsb(case, seed, b, case["txns"]) for b in range(case.get("batches", 1))]
    n_cols = SCAN_COLS if k == "scans" else COLS
    if sum(len(d[1]) for d in data) > 20 << 20:
        return None
    tab = _Cells(lambda t, key, col: _cells(seed, case["rows"], n_cols, key, col), np.zeros(0, np.int64), {0: case["rows"]})
    out = [_replay(tab, d, rule=case.get("rule", 0), n_cols={0: n_cols}) for d in data]
    if k == "serve":
        return {"commit": out[0][0], "vals": out[0][1]}
    return [{"commit": c, "vals": v.astype(np.int32)} for c, v in out]
