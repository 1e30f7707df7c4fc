"""Which kernel a prefill projection takes and in which order it sums K (host arithmetic of the library, no GPU): row
shards sum as the whole tensor does, and from 129 tokens on every kernel sums in order into one accumulator, so that
outputs do not depend on how rows or tokens are dealt out."""
import random

import pytest


def _order(plan):
    # what the sums of a token depend on: tile_cols decides which tokens share a tile, and so its partial accumulators
    return (plan["split"], plan["accumulators"], plan["tile_cols"] if plan["accumulators"] > 1 else None)


def test_order_of_summation_does_not_depend_on_the_shard(engine):
    rng = random.Random(7)
    splits = set()
    for _ in range(3000):
        m, k = int(2 ** rng.uniform(0, 12.5)), 64 * int(2 ** rng.uniform(0, 7.5))
        n, world = rng.randint(1, 32768), rng.choice([1, 2, 3, 8])
        whole = engine.gemm_plan(m, n, k, rows_aligned=rng.random() < 0.5)
        splits.add(whole["split"])
        for r in range(world):
            _, rows = engine.shard_range(n, r, world)
            if rows == 0:
                continue
            shard = engine.gemm_plan(m, rows, k, n_total=n, gather=rng.random() < 0.5, rows_aligned=rng.random() < 0.5)
            assert _order(shard) == _order(whole), (m, n, k, world, r)
        if m > 128:
            assert whole["split"] == 1 and whole["accumulators"] == 1, (m, n, k)
    assert splits == {1, 2, 4, 8}


def test_more_token_tiles_than_a_grid_has_rows(engine):
    """Rows that are not aligned keep off the kernel of CTA pairs, but not where the other one cannot be launched."""
    assert not engine.gemm_plan(65535 * 128, 200, 64, rows_aligned=False)["pairs"]
    assert engine.gemm_plan(65535 * 128 + 1, 200, 64, rows_aligned=False)["pairs"]


def test_plan_rejects(engine):
    for args in ((0, 128, 128, 64), (8, 0, 128, 64), (8, 256, 128, 64), (8, 128, 128, 100)):
        with pytest.raises(engine.Q35bError):
            engine.gemm_plan(args[0], args[1], args[3], n_total=args[2])
