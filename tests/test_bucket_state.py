"""GPU: what the bucket path keeps from batch to batch (which of its counters
are clean, the stamps) when the cell space grows: a table created after one or
two batches, then a batch of no more ops, against the oracle's replay --
values, commits, row counts, tables and statistics."""
import numpy as np
import pytest

import ltpmg_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SPACE = 1 << 20  # rows of the first table, one column


def reads_and_adds(rng, cells):
    add = rng.random(len(cells)) < 0.5
    imm = np.where(add, rng.integers(-(1 << 19), 1 << 19, len(cells)), 0)
    opw = (add.astype(np.uint32) | ((imm & 0xFFFFF).astype(np.uint32) << np.uint32(12))).astype(np.uint32)
    return cells.astype(np.uint64), opw


def batch_of(kind, n, rng):
    """(keys, opwords, payload) of n ops."""
    cells = rng.integers(0, SPACE, n)
    if kind == "one_cell":  # too long a bucket above 32,767 ops
        cells[:] = 77
    elif kind == "frequent":  # many buckets with a frequent cell
        cells[: n // 4] = rng.integers(0, SPACE, 40)[rng.integers(0, 40, n // 4)]
        cells = cells[rng.permutation(n)]
    keys, opw = reads_and_adds(rng, cells)
    pay = None
    if kind == "inserts":
        at = np.sort(rng.choice(n, n // 10, replace=False))
        keys[at] = np.arange(len(at))
        opw[at] = G.opword(G.OP_INSERT, 0)
        pay = rng.integers(-(1 << 31), 1 << 31, len(at)).astype(np.int32)
    elif kind == "malformed":
        keys[n // 2] = SPACE + (1 << 30)
    return keys, opw, pay


@pytest.mark.parametrize("before", [1, 2])
@pytest.mark.parametrize("first,n1,second,n2", [
    ("inserts", 600, "inserts", 500),
    ("inserts", 20000, "inserts", 15000),
    ("inserts", 20000, "inserts", 1500),
    ("frequent", 1500001, "uniform", 20000),
    ("one_cell", 200000, "uniform", 20000),
    ("malformed", 20000, "uniform", 20000),
    ("malformed", 20000, "inserts", 1500),
    ("uniform", 700001, "uniform", 700001),
])
def test_table_created_between_batches(lib, first, n1, second, n2, before):
    rng = np.random.default_rng(n1 + n2 + before)
    made = [(first,) + batch_of(first, n1, rng) for _ in range(before)] + [(second,) + batch_of(second, n2, rng)]
    room = sum(0 if m[3] is None else len(m[3]) for m in made)
    with G.Context(device=0) as ctx:
        t = ctx.create_table(SPACE, 1, rows_cap=SPACE + max(room, 1))
        ctx.fill_seeded(t, 5)
        tab = np.zeros((1, SPACE + max(room, 1)), np.int32)
        tab[:, :SPACE] = ctx.download(t)
        tabs = [(tab, SPACE, 0)]
        for j, (kind, keys, opw, pay) in enumerate(made):
            if j == before:
                ctx.create_table(1 << 16, 3)
                tabs.append((np.zeros((3, 1 << 16), np.int32), 1 << 16, 0))
            b = ctx.batch(len(keys), len(keys))
            b.load(None, keys, opw, ops_per_txn=1)
            if pay is not None:
                b.load_payload(pay)
            b.execute()
            if kind == "malformed":  # refused as a whole; its status is not looked at
                continue
            commit, vals, st = b.results()
            tf = np.arange(len(keys) + 1, dtype=np.uint32)
            tabs, rc, ro = O.replay_tables(0, tabs, tf, keys, opw, pay)
            assert np.array_equal(commit, rc) and np.array_equal(vals, ro.astype(np.int32))
            assert ctx.table_rows(t) == tabs[0][1]
            cells = keys[(opw & 3) != G.OP_INSERT]
            assert st.touched_words == len(np.unique(cells // 32))
        assert np.array_equal(ctx.download(t), tabs[0][0][:, :tabs[0][1]])
