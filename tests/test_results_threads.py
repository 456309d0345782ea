"""GPU: threads that take the results of different batches of one context at
the same time each get their own batch's."""
import threading

import numpy as np
import pytest

import ltpmg_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ops", [1500, 60000])  # one copy back; a copy per array
@pytest.mark.parametrize("wide", [False, True])
def test_results_of_two_batches_from_two_threads(lib, n_ops, wide):
    with G.Context(device=0) as ctx:
        ctx.create_table(2 * n_ops, 1, wide=[0] if wide else [])
        batches = []
        for j in range(2):
            b = ctx.batch(n_ops, n_ops)
            keys = np.arange(n_ops, dtype=np.uint64) + n_ops * j
            b.load(None, keys, np.full(n_ops, G.opword(G.OP_ADD, 0, imm=j + 1), np.uint32), ops_per_txn=1)
            b.execute()
            batches.append(b)
        ctx.sync()
        wrong, failed = [0, 0], []

        def fetch(j):
            try:
                for _ in range(4000):
                    commit, vals, st = batches[j].results64() if wide else batches[j].results()
                    wrong[j] += not (commit.all() and np.all(vals == j + 1) and st.ops == n_ops)
            except Exception as e:  # shown below
                failed.append(e)

        threads = [threading.Thread(target=fetch, args=(j,)) for j in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed and wrong == [0, 0]


@pytest.mark.parametrize("n_ops", [700, 60000, 400000])  # one copy back, a copy per array, more than the staging holds
def test_first_and_later_results_of_a_context_agree(lib, n_ops):
    with G.Context(device=0) as ctx:
        ctx.create_table(n_ops, 2)
        ctx.fill_seeded(0, 3)
        want = ctx.download(0)[0]
        b = ctx.batch(n_ops, n_ops)
        b.load(None, np.arange(n_ops, dtype=np.uint64), np.full(n_ops, G.opword(G.OP_ADD, 0, imm=7), np.uint32), ops_per_txn=1)
        for k in range(4):
            b.execute()
            commit, vals, st = b.results()
            assert commit.all() and st.committed == n_ops and np.array_equal(vals, want + np.int32(7 * (k + 1)))
