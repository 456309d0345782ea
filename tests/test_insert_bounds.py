"""Inserts whose payload row does not lie in the batch's payload, keys near
2^64 among them (key + row width wraps there): the predicate against 128-bit
arithmetic and the oracle's check (CPU, compiled here), and the refusal of
such a batch on every route a batch takes on the GPU."""
import os
import subprocess

import numpy as np
import pytest

import ltpmg_gb300 as G
import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
TOP = (1 << 64) - 1


def test_predicate_equals_128_bit_arithmetic(tmp_path):
    exe = str(tmp_path / "bounds_check")
    subprocess.run(["g++", "-std=c++17", "-O2", os.path.join(HERE, "bounds", "bounds_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.parametrize("threads", [0, 2])
@pytest.mark.parametrize("key", [4, 7, TOP, TOP - 1, TOP - 2])
def test_oracle_refuses_rows_outside_the_payload(key, threads):
    tab, ins = np.zeros((3, 8), np.int32), np.array([O.opword(2, 0, 0, 0)], np.uint32)
    tf, pay = np.array([0, 1], np.uint32), np.arange(6, dtype=np.int32)
    with pytest.raises(ValueError):
        O.replay_tables(0, [(tab, 1)], tf, np.array([key], np.uint64), ins, pay, threads=threads)
    after, _, _ = O.replay_tables(0, [(tab, 1)], tf, np.array([3], np.uint64), ins, pay, threads=threads)
    assert after[0][0][:, 1].tolist() == [3, 4, 5]


# one block's batch, split, by conflict words (both rules, and every mode that has its own kernels)
@pytest.mark.gpu
@pytest.mark.parametrize("n_ops,rule,mode", [
    (500, 0, "single"), (20000, 0, "single"), (20000, 0, G.MODE_GRAPH), ((2 << 20) + 5, 0, "single"),
    (20000, 1, "single"), (20000, 0, G.MODE_PERSISTENT), (20000, 1, G.MODE_PERSISTENT)])
def test_rows_outside_the_payload_are_refused(lib, n_ops, rule, mode):
    rows, slots = 64, 5  # two int32 columns, one of them int64 beside a third: 1 + 2 + 2 slots
    rng = np.random.default_rng(n_ops + rule)
    good = rng.integers(0, rows, n_ops).astype(np.uint64)
    opw = np.full(n_ops, G.opword(G.OP_READ, 0), np.uint32)
    pay = rng.integers(-(1 << 31), 1 << 31, 4 * slots).astype(np.int32)
    at = n_ops - 3
    opw[at] = G.opword(G.OP_INSERT, 0)
    good[at] = 3 * slots
    with G.Context(device=0, rule=rule) as ctx:
        t = ctx.create_table(rows, 3, rows_cap=rows + 8, wide=[1, 2])
        ctx.fill_seeded(t, 2)
        before = ctx.download(t)
        b = ctx.batch(n_ops, n_ops)
        for key in (TOP, TOP - 1, TOP - slots + 1, TOP - slots, 1 << 32, (1 << 32) - slots, 4 * slots, 3 * slots + 1):
            keys = good.copy()
            keys[at] = key
            b.load(None, keys, opw, ops_per_txn=1)
            b.load_payload(pay)
            if mode == "single":
                b.execute()
            else:
                ctx.execute_many([b], mode=mode)
            with pytest.raises(G.LtpError) as e:
                b.finish()
            assert e.value.status == G.lib.LTP_E_BADARG and f"index {at} " in str(e.value)
            assert ctx.table_rows(t) == rows and np.array_equal(ctx.download(t), before)
        b.load(None, good, opw, ops_per_txn=1)
        b.load_payload(pay)
        b.execute()
        _, vals, _ = b.results()
        assert vals[at] == rows
        x = pay[3 * slots:].view(np.uint32).astype(np.int64)
        want = [pay[3 * slots], (x[2] << 32) | x[1], (x[4] << 32) | x[3]]
        got = ctx.download(t)
        assert np.array_equal(got[:, :rows], before) and got[:, rows].tolist() == want
