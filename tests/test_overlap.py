"""GPU: batches beside long-running kernels of other streams.  A sleeping
one-thread kernel takes a warp of one SM; batches on the context's stream have
to complete while it sleeps, those that go to the skew fallback too, and with
the oracle's results."""
import time

import numpy as np
import pytest

import ltpmg_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SPACE = 1 << 20


@pytest.mark.parametrize("sleepers", [1, 24])  # (torch keeps 32 streams)
@pytest.mark.parametrize("n_ops,pattern", [
    (1500, "uniform"), (20000, "uniform"), (100000, "uniform"), (100000, "inserts"), (100000, "one_cell"),
    (100000, "one_cell_inserts"), (700001, "one_cell")])
@pytest.mark.parametrize("mode", [G.lib.MODE_STREAM, G.lib.MODE_GRAPH])
def test_batches_complete_beside_a_sleeping_kernel(lib, n_ops, pattern, sleepers, mode):
    import torch

    rng = np.random.default_rng(n_ops + sleepers)
    cells = rng.integers(0, SPACE, n_ops)
    if pattern.startswith("one_cell"):
        cells[rng.random(n_ops) < 0.9] = 4242
    add = rng.random(n_ops) < 0.5
    imm = np.where(add, rng.integers(-(1 << 19), 1 << 19, n_ops), 0)
    opw = (add.astype(np.uint32) | ((imm & 0xFFFFF).astype(np.uint32) << np.uint32(12))).astype(np.uint32)
    keys, pay = cells.astype(np.uint64), None
    if pattern.endswith("inserts"):
        at = np.sort(rng.choice(n_ops, n_ops // 10, replace=False))
        keys[at] = np.arange(len(at))
        opw[at] = G.opword(G.OP_INSERT, 0)
        pay = rng.integers(-(1 << 31), 1 << 31, len(at)).astype(np.int32)
    runs = 2  # one alone, one beside the sleepers
    cap = SPACE + (0 if pay is None else runs * len(pay))
    tf = np.arange(n_ops + 1, dtype=np.uint32)
    side = [torch.cuda.Stream() for _ in range(sleepers)]
    with G.Context(device=0) as ctx:
        t = ctx.create_table(SPACE, 1, rows_cap=cap)
        ctx.fill_seeded(t, 5)
        tab = np.zeros((1, cap), np.int32)
        tab[:, :SPACE] = ctx.download(t)
        tabs = [(tab, SPACE, 0)]
        b = ctx.batch(n_ops, n_ops)
        b.load(None, keys, opw, ops_per_txn=1)
        if pay is not None:
            b.load_payload(pay)
        stream = torch.cuda.ExternalStream(ctx.stream)
        for s in side:
            with torch.cuda.stream(s):
                torch.cuda._sleep(1000)
        for k in range(runs):
            if k:  # about 0.25 s at the highest clock
                for s in side:
                    with torch.cuda.stream(s):
                        torch.cuda._sleep(500_000_000)
                time.sleep(0.002)
            ctx.execute_many([b], mode=mode)
            done = torch.cuda.Event()
            done.record(stream)
            done.synchronize()
            assert not k or not any(s.query() for s in side), "the batch waited for the sleeping kernels"
            torch.cuda.synchronize()
            commit, vals, _ = b.results()
            tabs, rc, ro = O.replay_tables(0, tabs, tf, keys, opw, pay)
            assert np.array_equal(commit, rc) and np.array_equal(vals, ro.astype(np.int32))
            assert ctx.table_rows(t) == tabs[0][1]
        assert np.array_equal(ctx.download(t), tabs[0][0][:, :tabs[0][1]])
