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
