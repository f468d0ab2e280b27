"""Batches whose requests take different routes: the partition's shared launch (blocks of 1,280 keys or more) or, from
500,000 keys on, launches of their own; host keys staged in 2 MB pieces that cross requests. Every request's
products are those of building it alone."""
import numpy as np
import pytest

import shockhash_b200 as shg

pytestmark = pytest.mark.gpu


def products(r):
    out = [a.tobytes() for a in (r.descriptors, r.bucket_size_acc, r.bucket_pos_acc, r.ribbon_keys, r.ribbon_bits)]
    r.free()
    return out


@pytest.mark.parametrize("sizes", [
    (1279, 1280, 1281, 1, 0, 2560), (499_999, 500_000, 500_001, 3), (500_000, 0, 520_000), (0, 0), (5, 600_000, 0, 7),
    (3, 300_000, 262_144, 5, 262_139, 40_000, 299_999)])  # 757,760 keys and more: several keys' chunks per block
def test_requests_of_any_size_equal_building_alone(engine, sizes):
    keys = shg.keys_mt19937_64(sum(sizes), sum(sizes))
    sets = np.split(keys, np.cumsum(sizes)[:-1])
    batch = engine.build_batch_u64(shg.SHOCKHASH2, 20, sets, 300)
    got = [products(r) for r in batch]
    for k, g in zip(sets, got):
        assert g == products(engine.build_u64(shg.SHOCKHASH2, 20, k, 300))


def test_shards_among_whole_requests(engine):
    n, nb = 400_000, 2000
    first, second = (np.random.default_rng(i).integers(0, 2**64, size=n, dtype=np.uint64) for i in (1, 2))
    bucket = np.array([(int(f) * nb) >> 64 for f in first])
    ranges = [(0, 3), (3, 900), (900, 901), (901, 2000)]
    items = [{"first": first[m], "second": second[m], "nb_global": nb, "b0": a, "b1": b}
             for a, b in ranges for m in [(bucket >= a) & (bucket < b)]]
    items.insert(2, {"keys": shg.keys_mt19937_64(5, 130_000)})
    got = [products(r) for r in engine.build_batch_items(shg.SHOCKHASH2, 20, items, 200)]
    for it, g in zip(items, got):
        if "keys" in it:
            r = engine.build_u64(shg.SHOCKHASH2, 20, it["keys"], 200)
        else:
            r = engine.build_shard_hash128(shg.SHOCKHASH2, 20, it["first"], it["second"], nb, it["b0"], it["b1"], 200)
        assert g == products(r)


@pytest.mark.parametrize("n", [786_431, 786_432, 786_433, 1_048_577])  # 6 MB: pageable arrays are staged from here on
def test_pageable_array_around_the_staging_threshold(engine, n):
    import torch
    keys = shg.keys_mt19937_64(n, n)
    d = torch.from_numpy(keys.view(np.int64)).to("cuda")
    want = products(engine.build_u64_device(shg.SHOCKHASH2, 20, d.data_ptr(), n, 300))
    assert products(engine.build_u64(shg.SHOCKHASH2, 20, keys, 300)) == want
