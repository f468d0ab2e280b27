"""The default schedule on both sides of its rule (leaf size, bucket size and number of keys) gives the products of the
level schedule, and every lag of the work queue's order gives them too."""
import pytest

import shockhash_b200 as shg

pytestmark = pytest.mark.gpu


def products(r):
    out = [a.tobytes() for a in (r.descriptors, r.bucket_size_acc, r.bucket_pos_acc, r.ribbon_keys, r.ribbon_bits)]
    r.free()
    return out


@pytest.mark.parametrize("leaf,bucket,n", [(24, 2000, 600_000), (25, 200, 600_000), (25, 199, 600_000), (25, 200, 599_999),
                                           (30, 1000, 1_499_999), (30, 1000, 1_500_000), (64, 512, 600_001), (64, 511, 600_001)])
def test_default_schedule_around_its_rule(engine, leaf, bucket, n):
    keys = shg.keys_mt19937_64(leaf + n, n)
    assert products(engine.build_u64(shg.SHOCKHASH2, leaf, keys, bucket)) == \
        products(engine.build_u64(shg.SHOCKHASH2, leaf, keys, bucket, mode=shg.MODE_LEVELS))


def test_queue_lags():
    keys = shg.keys_mt19937_64(9, 150_000)
    eng = shg.Engine(0)
    want = products(eng.build_u64(shg.SHOCKHASH2, 24, keys, 2000, mode=shg.MODE_LEVELS))
    for lag in (0, 1, 3, 64):
        for blocks in (0, 1):
            eng.set_tuning(shg.SHOCKHASH2, 24, queue_lag_rounds=lag, leaf_blocks_per_sm=blocks)
            assert products(eng.build_u64(shg.SHOCKHASH2, 24, keys, 2000, mode=shg.MODE_QUEUE)) == want
    eng.close()
