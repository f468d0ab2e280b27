"""Trees of small nodes: split levels whose searches expect too few seeds for several blocks per node, and levels of up to
128 keys per node, which take blocks of half the threads (around the sizes where that changes), against the oracle."""
import numpy as np
import pytest

import shockhash_b200 as shg
from conftest import unique_u64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [shg.SHOCKHASH, shg.SHOCKHASH2, shg.SIMDSHOCKHASH])
@pytest.mark.parametrize("leaf,bucket,n", [(2, 7, 400), (2, 2000, 5000), (8, 200, 3000), (8, 3000, 127), (8, 3000, 128), (8, 3000, 129),
                                           (12, 3000, 257), (16, 1000, 9000)])
def test_small_nodes_match_the_oracle(engine, port, variant, leaf, bucket, n):
    rng = np.random.default_rng(leaf * bucket + n)
    first, second = rng.integers(0, 2**64, size=n, dtype=np.uint64), unique_u64(rng, n)
    p = port.build_hash(variant, leaf, first, second, bucket)
    for mode in (shg.MODE_LEVELS, shg.MODE_PIPELINED):
        r = engine.build_hash128(variant, leaf, first, second, bucket, mode=mode)
        assert np.array_equal(r.descriptors, p.desc)
        assert np.array_equal(r.ribbon_keys, p.ribbon_keys) and np.array_equal(r.ribbon_bits, p.ribbon_bits)
        r.free()
