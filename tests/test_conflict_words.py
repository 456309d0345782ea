"""GPU: the conflict-word kernels under the ordered rule at sizes that go by
buckets of cells otherwise.  Every context here is tuned to
LTP_TUNE_CONFLICT_WORDS in all size buckets, and the suites' own tests of
tilings, tile edges, word widths, batch modes, the pipeline and inserts run on
it: their oracle, their tolerance (none)."""
import numpy as np
import pytest

import ltpmg_gb300 as G
import oracle as O

from test_buckets import (test_few_rows_per_op, test_frequent_cells, test_inserts_links_and_int64,  # noqa: F401
                          test_refused_batches_change_nothing, test_rows_of_every_width, test_sizes_and_patterns)
from test_gpu_parity import (lib_loaded, test_32_bit_keys, test_dense_batches_build_no_list_and_recover_from_errors,  # noqa: F401
                             test_edge_cases, test_fixed_length_path, test_insert_capacity_and_payload_errors,
                             test_inserts_scattered_payload_rows, test_inserts_two_tables_sequence,
                             test_multi_batch_modes, test_pipeline_replays_captured_graphs, test_seeded_sequences,
                             test_tile_boundaries_and_adversarial_keys, test_tuning_variants,
                             test_word_widths_alternate_on_one_context)
from test_insert_bounds import test_rows_outside_the_payload_are_refused  # noqa: F401
from test_tpcc import small, test_tpcc_sequence_matches_oracle, test_tpcc_sequence_with_64_cell_words  # noqa: F401
from test_wide import (test_repeated_cells_in_one_transaction_and_int32_wrap,  # noqa: F401
                       test_wide_columns_and_links_match_oracle)
from test_word_range import (test_batches_on_part_of_a_multi_table_context,  # noqa: F401
                             test_insert_slots_from_mark_counts_every_tiling)

pytestmark = pytest.mark.gpu

WORDS = G.lib.TUNE_CONFLICT_WORDS


@pytest.fixture(autouse=True)
def conflict_words(request, monkeypatch):
    """Contexts are created with the flag, and keep it when a test tunes them."""
    if request.function.__module__ == __name__:
        return
    init, put, get = G.Context.__init__, G.Context.set_tuning, G.Context.get_tuning

    def set_tuning(self, bucket, block, ipt, word_bits=32, flags=0):
        put(self, bucket, block, ipt, word_bits, flags | WORDS)

    def get_tuning(self, bucket):
        block, ipt, word_bits, flags = get(self, bucket)
        return block, ipt, word_bits, flags & ~WORDS

    def create(self, *a, **k):
        init(self, *a, **k)
        for bucket in range(64):
            set_tuning(self, bucket, *get_tuning(self, bucket))

    monkeypatch.setattr(G.Context, "__init__", create)
    monkeypatch.setattr(G.Context, "set_tuning", set_tuning)
    monkeypatch.setattr(G.Context, "get_tuning", get_tuning)


@pytest.mark.parametrize("mode", ["single", G.MODE_GRAPH])
def test_the_flag_chooses_the_path_from_batch_to_batch(lib, mode):
    """On, off, on: values and table equal the replay, and only the
    conflict-word path spends time on ids."""
    n, space = 1 << 20, 1 << 22
    rng = np.random.default_rng(4)
    keys = rng.integers(0, space, n).astype(np.uint64)
    opw = np.where(rng.random(n) < 0.5, G.opword(G.OP_ADD, 0, imm=3), G.opword(G.OP_READ, 0)).astype(np.uint32)
    tf = np.arange(n + 1, dtype=np.uint32)
    with G.Context(device=0, stage_timing=True) as ctx:
        ctx.create_table(space, 1)
        ctx.fill_seeded(0, 9)
        ref = O.table_init(9, space, 1)
        b = ctx.batch(n, n)
        b.load(None, keys, opw, ops_per_txn=1)
        ids_ms = {0: [], WORDS: []}
        for flags in (0, WORDS, 0, WORDS, WORDS, 0):
            ctx.set_tuning(20, 512, 4, flags=flags)
            assert ctx.get_tuning(20) == (512, 4, 32, flags)
            if mode == "single":
                b.execute()
            else:
                ctx.execute_many([b], mode=mode)
            commit, vals, st = b.results()
            ref, rc, ro = O.replay(0, ref, tf, keys, opw)
            assert np.array_equal(commit, rc) and np.array_equal(vals, ro)
            ids_ms[flags].append(st.ms_stage[1])
        assert np.array_equal(ctx.download(0), ref)
        assert min(ids_ms[WORDS]) > 2 * max(ids_ms[0]) > 0


def test_unknown_flags_are_refused(lib):
    with G.Context(device=0) as ctx:
        with pytest.raises(G.LtpError):
            ctx.set_tuning(5, 512, 4, flags=4)
