"""The autotuner's choice between the buckets of cells and the conflict-word
kernels, for ordered-rule batches that can go either way.  CPU: a stand-in
timer; GPU: a uniform batch and one with very frequent cells."""
import numpy as np
import pytest

import ltpmg_gb300.autotune as AT
from ltpmg_gb300 import lib as L

WORDS, PRE = L.TUNE_CONFLICT_WORDS, L.TUNE_MARK_PRECHECK


class FakeCtx:
    def __init__(self, rule):
        self.rule, self.tuning, self.calls = rule, {}, []

    def set_tuning(self, bucket, block, ipt, word_bits=32, flags=0):
        self.tuning[bucket] = (block, ipt, word_bits, flags)
        self.calls.append((block, ipt, word_bits, flags))


class FakeBatch:
    def __init__(self, n_ops):
        self.n_ops = n_ops

    def execute(self):
        pass

    def finish(self):
        pass


def tune(monkeypatch, rule, n_ops, cost):
    ctx = FakeCtx(rule)
    monkeypatch.setattr(AT, "_time_batch", lambda c, b, reps, copies=1: cost(*c.tuning[AT.bucket_of(b.n_ops)]))
    return ctx, AT.tune_tiles(ctx, FakeBatch(n_ops), reps=1)


def words_cost(block, ipt, wb, flags):
    return 1.0 + (block != 256) * 0.2 + (ipt != 2) * 0.1 + (wb == 64) * 0.5 - bool(flags & PRE) * 0.05


@pytest.mark.parametrize("n_ops", [20000, 1 << 20, 2 << 20])
def test_buckets_are_kept_when_faster(monkeypatch, n_ops):
    ctx, ch = tune(monkeypatch, L.RULE_ORDERED, n_ops, lambda *t: words_cost(*t) if t[3] & WORDS else 0.5)
    assert ch["name"] == "buckets" and (ch["word_bits"], ch["flags"], ch["ms"]) == (32, 0, 0.5)
    assert ctx.tuning[ch["bucket"]] == (ch["block"], ch["ipt"], 32, 0)
    # by buckets once; everything else by conflict words
    assert [c for c in ctx.calls[:-1] if not c[3] & WORDS] == [(512, 4, 32, 0)]
    assert sorted(ch["candidates"])[-1] == "buckets" and all(k.endswith("+words") for k in ch["candidates"] if k != "buckets")


def test_conflict_words_are_kept_when_faster(monkeypatch):
    ctx, ch = tune(monkeypatch, L.RULE_ORDERED, 1 << 20, lambda *t: words_cost(*t) if t[3] & WORDS else 1.5)
    assert ch["name"] == "256x2+precheck+words" and ch["ms"] == 0.95
    assert ctx.tuning[20] == (256, 2, 32, PRE | WORDS) == AT.parse_choice(ch["name"])


@pytest.mark.parametrize("rule,n_ops,cells", [(L.RULE_PRIORITY, 1 << 20, 0), (L.RULE_ORDERED, (2 << 20) + 1, 0),
                                              (L.RULE_ORDERED, 1 << 20, (1 << 32) + 1)])
def test_batches_that_cannot_go_by_buckets(monkeypatch, rule, n_ops, cells):
    monkeypatch.setattr(FakeCtx, "cells", cells, raising=False)
    ctx, ch = tune(monkeypatch, rule, n_ops, words_cost)
    assert ch["name"] == "256x2+precheck" and ch["flags"] == PRE
    assert not any(c[3] & WORDS for c in ctx.calls) and "buckets" not in ch["candidates"]


def test_names_round_trip():
    for t in [(512, 4, 32, 0), (512, 2, 64, PRE), (128, 1, 32, WORDS), (256, 8, 64, PRE | WORDS)]:
        assert AT.parse_choice(AT.choice_name(*t)) == t
    assert AT.parse_choice("buckets")[2:] == (32, 0)


def test_refine_keeps_the_path_of_its_candidates(monkeypatch):
    choice = {"bucket": 20, "candidates": {"buckets": 1.0, "256x2+precheck+words": 1.1, "256x2+words": 1.2, "512x4+words": 1.3}}
    seen = []

    def fake_list(ctx, batches, reps, mode=L.MODE_GRAPH):
        seen.append(ctx.tuning[20])
        return {(512, 4, 32, 0): 2.0, (256, 2, 32, WORDS): 1.9, (256, 2, 32, WORDS | PRE): 1.8}[ctx.tuning[20]]

    monkeypatch.setattr(AT, "_time_list", fake_list)
    ctx = FakeCtx(L.RULE_ORDERED)
    out = AT.refine_pipeline(ctx, [FakeBatch(1 << 20)], choice)
    assert seen == [(512, 4, 32, 0), (256, 2, 32, WORDS), (256, 2, 32, WORDS | PRE)]
    assert out["name"] == "256x2+precheck+words" and ctx.tuning[20] == (256, 2, 32, WORDS | PRE)


@pytest.mark.gpu
@pytest.mark.parametrize("hot", [False, True])
def test_tuned_path_of_a_real_batch(lib, hot):
    import ltpmg_gb300 as G

    n, space = 655360, 1 << 20
    rng = np.random.default_rng(7)
    cells = rng.integers(0, space, n)
    if hot:  # a twentieth of the ops on one cell
        cells[rng.random(n) < 0.05] = 99
    opw = np.where(rng.random(n) < 0.5, G.opword(G.OP_ADD, 0, imm=1), G.opword(G.OP_READ, 0)).astype(np.uint32)
    with G.Context(device=0) as ctx:
        ctx.create_table(space, 1)
        b = ctx.batch(n, n)
        b.load(None, cells.astype(np.uint32), opw, ops_per_txn=1)
        ch = AT.tune_tiles(ctx, b, reps=5, copies=4)
        assert ctx.cells == space
        assert (ch["name"] != "buckets") == hot == bool(ctx.get_tuning(ch["bucket"])[3] & WORDS)
