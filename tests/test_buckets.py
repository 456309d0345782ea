"""GPU: batches executed by buckets of cells (ordered rule), at the sizes
where the split can go wrong -- one block's batch and one op more, tile and
chunk edges, buckets longer than a chunk, more distinct cells than the
shared-memory hash holds, buckets left to the conflict-word path -- against
the oracle's serial replay, values, commits, tables and statistics."""
import numpy as np
import pytest

import ltpmg_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib_loaded():
    return G.load()


MIX_INVERSE = pow(0x9E3779B1, -1, 1 << 32)  # of the multiplier that picks a cell's bucket


def cells_of(pattern, n, space, rng):
    """n cell numbers out of [0, space), space a power of two."""
    if pattern == "one_cell":
        return np.full(n, space // 3)
    if pattern == "uniform":
        return rng.integers(0, space, n)
    if pattern == "skewed":
        return np.minimum(rng.zipf(1.2, n) - 1, space - 1)
    if pattern == "hot_and_cold":  # a quarter of the ops on three cells
        return np.where(rng.random(n) < 0.25, rng.integers(0, 3, n) * 1001, rng.integers(0, space, n))
    # one bucket: consecutive hashes, every cell about twice
    j = rng.integers(0, max(1, min(n // 2, space // 64)), n)
    return ((j * MIX_INVERSE) % space).astype(np.int64)


def statistics(cells, add, word):
    """(contended ops, contended cells, touched words)"""
    u, inv, cnt = np.unique(cells, return_inverse=True, return_counts=True)
    con = (cnt > 1) & (np.bincount(inv, weights=add, minlength=len(u)) > 0)
    return int(cnt[con].sum()), int(con.sum()), len(np.unique(u // word))


@pytest.mark.parametrize("n_ops", [1, 33, 1024, 1025, 4096, 4097, 8193, 32768, 32769, 81921, 163841, 700001])
@pytest.mark.parametrize("pattern", ["one_cell", "uniform", "skewed", "hot_and_cold", "one_bucket"])
def test_sizes_and_patterns(lib_loaded, n_ops, pattern):
    rng = np.random.default_rng(n_ops + len(pattern))
    space = 1 << 20
    cells = cells_of(pattern, n_ops, space, rng)
    add = rng.random(n_ops) < 0.4
    imm = np.where(add, rng.integers(-(1 << 19), 1 << 19, n_ops), 0)
    opw = (add.astype(np.uint32) | ((imm & 0xFFFFF).astype(np.uint32) << np.uint32(12))).astype(np.uint32)
    keys = cells.astype(np.uint64)
    tf = np.unique(np.concatenate([[0, n_ops], rng.integers(0, n_ops + 1, n_ops // 5)])).astype(np.uint32)
    with G.Context(device=0) as ctx:
        t = ctx.create_table(space, 1)
        ctx.fill_seeded(t, 9)
        ref = O.table_init(9, space, 1)
        b = ctx.batch(len(tf) - 1, n_ops)
        for k in (keys, keys.astype(np.uint32)):
            b.load(tf, k, opw)
            b.execute()
            commit, vals, st = b.results()
            ref, rc, ro = O.replay(0, ref, tf, keys, opw)
            assert np.array_equal(commit, rc[:len(tf) - 1]) and np.array_equal(vals, ro)
            assert (st.contended_ops, st.contended_cells, st.touched_words) == statistics(cells, add, 32)
        assert np.array_equal(ctx.download(t), ref)


# Contended ops of a block around the edges between comparing them all, by
# classes of slots, and sorting them; buckets that are executed first (more of
# them than the list holds, some of them the first buckets anyway).
@pytest.mark.parametrize("n_ops,n_hot,each", [
    (1000, 1, 63), (1000, 2, 33), (2048, 8, 250), (2048, 1, 257), (2000, 1000, 2), (40000, 300, 40),
    (40000, 100, 256), (40000, 60, 257), (150000, 40000, 3), (700001, 1, 3000), (700001, 31, 2500),
    (700001, 33, 2000), (700001, 90, 2600)])
def test_frequent_cells(lib_loaded, n_ops, n_hot, each):
    rng = np.random.default_rng(n_ops + n_hot)
    space = 1 << 20
    # every other hot cell in a bucket of its own from the first on, the others anywhere
    h = np.where(np.arange(n_hot) % 2 == 0, np.arange(n_hot) // 2 * (space // 608 + 1) % space, rng.integers(0, space, n_hot))
    hot = (h * MIX_INVERSE) % space
    cells = np.concatenate([np.repeat(hot, each), rng.integers(0, space, n_ops)])[:n_ops]
    cells = cells[rng.permutation(n_ops)]
    add = rng.random(n_ops) < 0.5
    imm = np.where(add, rng.integers(-(1 << 19), 1 << 19, n_ops), 0)
    opw = (add.astype(np.uint32) | ((imm & 0xFFFFF).astype(np.uint32) << np.uint32(12))).astype(np.uint32)
    tf = np.unique(np.concatenate([[0, n_ops], rng.integers(0, n_ops + 1, n_ops // 5)])).astype(np.uint32)
    with G.Context(device=0) as ctx:
        t = ctx.create_table(space, 1)
        ctx.fill_seeded(t, 9)
        ref = O.table_init(9, space, 1)
        b = ctx.batch(len(tf) - 1, n_ops)
        for _ in range(2):
            b.load(tf, cells.astype(np.uint64), opw)
            b.execute()
            commit, vals, st = b.results()
            ref, rc, ro = O.replay(0, ref, tf, cells.astype(np.uint64), opw)
            assert np.array_equal(commit, rc[:len(tf) - 1]) and np.array_equal(vals, ro)
            assert (st.contended_ops, st.contended_cells, st.touched_words) == statistics(cells, add, 32)
        assert np.array_equal(ctx.download(t), ref)


@pytest.mark.parametrize("n_txns", [40, 300, 2500, 30000])
@pytest.mark.parametrize("mode", [G.lib.MODE_STREAM, G.lib.MODE_GRAPH])
def test_inserts_links_and_int64(lib_loaded, n_txns, mode):
    """Two order-entry batches back to back (int64 cells, linked inserts):
    one block's batch, a few buckets, many insert tiles."""
    g = G.Tpcc(1, seed=n_txns, customers=300, items=2000)
    made = [g.gen(k, n_txns) for k in range(2)]
    with G.Context(device=0) as ctx:
        ids = g.create_tables(ctx, sum(m[5] for m in made))
        bs = []
        for tf, keys, opw, pay, _, _ in made:
            b = ctx.batch(n_txns, len(keys))
            b.load(tf, keys, opw)
            b.load_payload(pay)
            bs.append(b)
        ctx.execute_many(bs, mode=mode)
        got = [b.results64() for b in bs]
        finals = [ctx.download(t) for t in ids]
    tabs = []
    for k in range(9):
        n_cols, mask, r0 = g.table(k)
        tabs.append((g.initial(k, r0 + int(made[0][5][k] + made[1][5][k])), r0, mask))
    for m, (commit, vals, st) in zip(made, got):
        after, rc, ro = O.replay_tables(0, tabs, *m[:4])
        assert np.array_equal(commit, rc) and np.array_equal(vals, ro)
        tabs = [(a[0], a[1], tabs[k][2]) for k, a in enumerate(after)]
    for k in range(9):
        assert np.array_equal(finals[k], tabs[k][0][:, :tabs[k][1]]), k


@pytest.mark.parametrize("n_ops", [600, 3000, 20000])
def test_refused_batches_change_nothing(lib_loaded, n_ops):
    """A malformed op, and inserts beyond the table's room, fail the batch
    before any of its ops takes effect; the next batch is unaffected."""
    rng = np.random.default_rng(n_ops)
    keys = rng.integers(0, 1 << 12, n_ops).astype(np.uint64)
    opw = np.full(n_ops, G.opword(G.OP_ADD, 0, imm=5), np.uint32)
    with G.Context(device=0) as ctx:
        t = ctx.create_table(1 << 12, 2, rows_cap=(1 << 12) + 3)
        ctx.fill_seeded(t, 3)
        ref = ctx.download(t)
        b = ctx.batch(n_ops, n_ops)
        bad = keys.copy()
        bad[n_ops - 7] = 1 << 12
        b.load(None, bad, opw, ops_per_txn=1)
        b.execute()
        with pytest.raises(G.LtpError, match=f"index {n_ops - 7} "):
            b.finish()
        assert np.array_equal(ctx.download(t), ref)
        k2, w2 = keys.copy(), opw.copy()
        w2[10:14] = G.opword(G.OP_INSERT, 0)
        k2[10:14] = 0
        b.load(None, k2, w2, ops_per_txn=1)
        b.load_payload(np.zeros(2, np.int32))
        b.execute()
        with pytest.raises(G.LtpError) as e:
            b.finish()
        assert e.value.status == G.lib.LTP_E_CAPACITY
        assert ctx.table_rows(t) == 1 << 12 and np.array_equal(ctx.download(t), ref)
        b.load(None, keys, opw, ops_per_txn=1)
        b.execute()
        _, vals, _ = b.results()
        ref, _, ro = O.replay(0, ref, np.arange(n_ops + 1, dtype=np.uint32), keys, opw)
        assert np.array_equal(vals, ro) and np.array_equal(ctx.download(t), ref)


@pytest.mark.parametrize("n_txns", [1, 700, 1024, 5000])
def test_rows_of_every_width(lib_loaded, n_txns):
    """Inserts into tables of 1 to 64 columns, int32 and int64, linked and
    not, in batches whose new rows need one staging or several."""
    rng = np.random.default_rng(n_txns)
    shapes = [(64, 0), (3, 0b010), (64, (1 << 64) - 1), (1, 0), (17, 1 << 16)]  # columns, int64 ones
    slots = [c + bin(m).count("1") for c, m in shapes]
    t = rng.integers(0, len(shapes), n_txns)
    t[: n_txns // 2] = 2  # the widest rows, together
    col = np.array([rng.integers(0, shapes[x][0]) for x in t])
    link = rng.random(n_txns) < 0.5
    first = np.concatenate([[0], np.cumsum(np.array(slots)[t])])
    # a transaction: one read-modify-write of table 0, one insert that may take its output
    keys = np.stack([rng.integers(0, 50, n_txns), first[:-1]], axis=1).reshape(-1).astype(np.uint64)
    add = [G.opword(G.OP_ADD, int(c), 0, int(v)) for c, v in zip(rng.integers(0, 64, n_txns), rng.integers(-99, 99, n_txns))]
    ins = [G.opword(G.OP_INSERT, int(c), int(x), int(li)) for c, x, li in zip(col, t, link)]
    opw = np.stack([add, ins], axis=1).reshape(-1).astype(np.uint32)
    pay = rng.integers(-(1 << 31), 1 << 31, int(first[-1])).astype(np.int32)
    tf = np.arange(0, 2 * n_txns + 1, 2, dtype=np.uint32)
    rows = [50 + int((t == k).sum()) for k in range(len(shapes))]
    with G.Context(device=0) as ctx:
        for k, (c, m) in enumerate(shapes):
            ctx.create_table(50, c, rows_cap=rows[k], wide=[j for j in range(c) if m >> j & 1])
            ctx.fill_seeded(k, 11)
        tabs = [(np.concatenate([ctx.download(k), np.zeros((c, rows[k] - 50), np.int64 if m else np.int32)], axis=1), 50, m)
                for k, (c, m) in enumerate(shapes)]
        b = ctx.batch(n_txns, len(keys))
        b.load(tf, keys, opw)
        b.load_payload(pay)
        b.execute()
        _, vals, _ = b.results64()
        finals = [ctx.download(k) for k in range(len(shapes))]
    after, _, ro = O.replay_tables(0, tabs, tf, keys, opw, pay)
    assert np.array_equal(vals, ro)
    for k in range(len(shapes)):
        assert np.array_equal(finals[k], after[k][0][:, :after[k][1]]), k


@pytest.mark.parametrize("n_txns,reads", [(1, 700), (12, 700), (700, 700), (4000, 600), (300, 4)])
def test_few_rows_per_op(lib_loaded, n_txns, reads):
    """Inserts, linked and not, among many reads (both shapes of the insert
    kernel; insert tiles with no insert, one and a few)."""
    rng = np.random.default_rng(n_txns)
    shapes = [(64, (1 << 64) - 1), (3, 0), (17, 1 << 16)]
    slots = np.array([c + bin(m).count("1") for c, m in shapes])
    t = rng.integers(0, len(shapes), n_txns)
    link = rng.random(n_txns) < 0.5
    first = np.concatenate([[0], np.cumsum(slots[t])])
    kinds = rng.integers(0, 50, (n_txns, reads + 1)).astype(np.uint64)
    keys = np.concatenate([kinds, first[:-1, None].astype(np.uint64)], axis=1).reshape(-1)
    opw = np.full((n_txns, reads + 2), G.opword(G.OP_READ, 5, 0), np.uint32)
    opw[:, reads] = [G.opword(G.OP_ADD, 7, 0, int(v)) for v in rng.integers(-99, 99, n_txns)]
    opw[:, reads + 1] = [G.opword(G.OP_INSERT, 2, int(x), int(li)) for x, li in zip(t, link)]
    opw = opw.reshape(-1)
    pay = rng.integers(-(1 << 31), 1 << 31, int(first[-1])).astype(np.int32)
    assert (len(pay) < len(opw) // 4) == (reads > 100)
    tf = np.arange(0, len(opw) + 1, reads + 2, dtype=np.uint32)
    rows = [50 + int((t == k).sum()) for k in range(len(shapes))]
    with G.Context(device=0) as ctx:
        for k, (c, m) in enumerate(shapes):
            ctx.create_table(50, c, rows_cap=rows[k], wide=[j for j in range(c) if m >> j & 1])
            ctx.fill_seeded(k, 11)
        tabs = [(np.concatenate([ctx.download(k), np.zeros((c, rows[k] - 50), np.int64 if m else np.int32)], axis=1), 50, m)
                for k, (c, m) in enumerate(shapes)]
        b = ctx.batch(n_txns, len(keys))
        b.load(tf, keys, opw)
        b.load_payload(pay)
        b.execute()
        _, vals, _ = b.results64()
        finals = [ctx.download(k) for k in range(len(shapes))]
    after, _, ro = O.replay_tables(0, tabs, tf, keys, opw, pay)
    assert np.array_equal(vals, ro)
    for k in range(len(shapes)):
        assert np.array_equal(finals[k], after[k][0][:, :after[k][1]]), k
