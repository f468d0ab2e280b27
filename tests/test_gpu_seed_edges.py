"""Split and leaf searches over keys whose low 30 bits run over within the first seeds of a search:
the staged form of a key (shg_common.cuh, SeedKey) holds only until then, so these builds take the
plain round and stage their keys again. Compared bit for bit with the oracle."""
import numpy as np
import pytest

import shockhash_b200 as shg

pytestmark = pytest.mark.gpu

# start seeds of tree depths 0..4 and of SIMDShockHash's fixed entries 17, 18, 19 (ShockHash.h:47-49)
START = {0: 0x106393c187cae21a, 1: 0x6453cec3f7376937, 2: 0x643e521ddbd2be98, 3: 0x3740c6412f6572cb, 4: 0x717d47562f1ce470,
         17: 0x1ea2099d1fafae7f, 18: 0x425c8a06fbaaa815, 19: 0xcd4216006c74052a}


def edge_keys(seed, n, levels, reach):
    """Distinct second halves: each, plus the start seed of one of `levels`, is 1..reach short of a
    multiple of 2^30 (or of 2^32 for one in four), so that some searched seed carries out of the low bits."""
    rng = np.random.default_rng(seed)
    out = set()
    while len(out) < n:
        short = int(rng.integers(1, reach + 1))
        bits = 32 if rng.random() < 0.25 else 30
        top = int(rng.integers(0, 2**(64 - bits)))
        lv = levels[int(rng.integers(len(levels)))]
        out.add(((top << bits) - short - START[lv]) % 2**64)
    second = np.array(sorted(out), dtype=np.uint64)
    rng.shuffle(second)
    return rng.integers(0, 2**64, size=n, dtype=np.uint64), second


@pytest.mark.parametrize("variant,leaf,bucket,levels", [
    (shg.SHOCKHASH2, 64, 2000, (0, 1, 2, 3)), (shg.SHOCKHASH2, 33, 500, (0, 1, 2, 3)), (shg.SHOCKHASH2, 100, 1000, (0, 1, 2)),
    (shg.SHOCKHASH2, 2, 5, (0, 1, 2)), (shg.SHOCKHASH, 30, 2000, (0, 1, 2, 3, 4)), (shg.SHOCKHASH, 8, 100, (0, 1, 2, 3)),
    (shg.SHOCKHASH, 33, 300, (0, 1, 2, 3)), (shg.SIMDSHOCKHASH, 30, 1000, (0, 1, 17, 18, 19))])
@pytest.mark.parametrize("reach", [40, 3000])
def test_low_bits_run_over(engine, port, variant, leaf, bucket, levels, reach):
    first, second = edge_keys(leaf * 7 + reach, 3 * bucket + 77, levels, reach)
    r = engine.build_hash128(variant, leaf, first, second, bucket)
    p = port.build_hash(variant, leaf, first, second, bucket)
    assert np.array_equal(r.descriptors, p.desc)
    assert np.array_equal(r.bucket_pos_acc, p.pos_acc)
    assert np.array_equal(r.ribbon_keys, p.ribbon_keys)
    assert np.array_equal(r.ribbon_bits, p.ribbon_bits)


def test_low_bits_run_over_rotation(engine):
    # the oracle has no rotation fitting: the structure has to be a minimal perfect hash for its host query
    first, second = edge_keys(5, 3000, (0, 1, 2, 3, 4), 3000)
    r = engine.build_hash128(shg.SHOCKHASH_ROTATION, 30, first, second, 2000, query=True)
    assert np.array_equal(np.sort(r._mphf.query_hash(first, second)), np.arange(3000, dtype=np.uint64))
