"""A build that fails (device memory runs out, a trial limit is reached) leaves nothing behind: the engine's next
builds, larger and smaller ones, give the products of a fresh engine."""
import pytest

import shockhash_b200 as shg

pytestmark = pytest.mark.gpu


def products(r):
    out = [a.tobytes() for a in (r.descriptors, r.bucket_size_acc, r.bucket_pos_acc, r.ribbon_keys, r.ribbon_bits)]
    r.free()
    return out


def test_engine_goes_on_after_failed_builds():
    import torch
    sets = [shg.keys_mt19937_64(60 + i, n) for i, n in enumerate((70_000, 3_000, 150_000))]
    big = [shg.keys_mt19937_64(70 + i, 6_000_000) for i in range(2)]
    fresh = shg.Engine(0)
    want = [products(r) for r in fresh.build_batch_u64(shg.SHOCKHASH2, 24, sets, 100)]
    fresh.close()
    eng = shg.Engine(0)
    products(eng.build_u64(shg.SHOCKHASH2, 24, sets[1], 100))
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - (200 << 20)), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(shg.ShgError):
            eng.build_batch_u64(shg.SHOCKHASH2, 24, big, 100)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert products(eng.build_u64(shg.SHOCKHASH2, 24, sets[1], 100)) == want[1]
    for k in sets[:2]:
        with pytest.raises(shg.ShgError) as err:
            eng.build_u64(shg.SHOCKHASH2, 24, k, 100, max_trials=1)
        assert "trial" in str(err.value)
    assert [products(r) for r in eng.build_batch_u64(shg.SHOCKHASH2, 24, sets, 100)] == want
    for k, w in zip(sets, want):
        assert products(eng.build_u64(shg.SHOCKHASH2, 24, k, 100)) == w
    eng.close()


@pytest.mark.parametrize("mode", [shg.MODE_LEVELS, shg.MODE_QUEUE, shg.MODE_PIPELINED])
def test_larger_build_follows_a_failed_one(mode):
    # the engine's pinned buffers grow (and are given back) right after builds that stopped half way
    eng, other = shg.Engine(0), shg.Engine(0)
    for i, n in enumerate((500, 20_000, 200_000)):
        first, second = (shg.keys_mt19937_64(80 + 2 * i + j, n) for j in (0, 1))
        with pytest.raises(shg.ShgError):
            eng.build_hash128(shg.SHOCKHASH2, 24, first, second, 100, mode=mode, max_trials=1)
        keys = shg.keys_mt19937_64(90 + i, 4 * n)
        assert products(eng.build_u64(shg.SHOCKHASH2, 24, keys, 100, mode=mode)) == products(other.build_u64(shg.SHOCKHASH2, 24, keys, 100))
    eng.close()
    other.close()
