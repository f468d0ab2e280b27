"""Engines in several threads of one process launch the same kernels side by side, over nodes, buckets and
key sets of different sizes: every build succeeds and gives the products that it gives alone. (A kernel's
shared-memory limit belongs to the kernel on the device, not to a thread's launch.)"""
import threading

import numpy as np
import pytest

import shockhash_b200 as shg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,variant,tuning", [(shg.MODE_LEVELS, shg.SHOCKHASH2, {}), (shg.MODE_LEVELS, shg.SIMDSHOCKHASH, {}),
                                                 (shg.MODE_QUEUE, shg.SHOCKHASH2, {"split_seeds_per_lane": 4})])
def test_builds_of_different_sizes_side_by_side(mode, variant, tuning):
    leaf = 32 if variant == shg.SHOCKHASH2 else 20
    shapes = [(2900, 2000), (40_000, 2000), (30_000, 100), (90, 100)]  # keys, bucket size
    keys = [shg.keys_mt19937_64(50 + i, n) for i, (n, _) in enumerate(shapes)]

    def products(r):
        return [a.tobytes() for a in (r.descriptors, r.bucket_size_acc, r.bucket_pos_acc, r.ribbon_keys, r.ribbon_bits)]

    def build(eng, i):
        r = eng.build_u64(variant, leaf, keys[i], shapes[i][1], mode=mode)
        out = products(r)
        r.free()
        return out

    engines = [shg.Engine(0) for _ in range(3)]
    for e in engines:
        e.set_tuning(variant, leaf, **tuning)
    alone = [build(engines[0], i) for i in range(len(shapes))]
    errors = []

    def worker(t):
        order = np.random.default_rng(t).integers(0, len(shapes), size=80)
        try:
            for i in order:
                if build(engines[t], i) != alone[i]:
                    errors.append(f"thread {t}: products of set {i} differ")
        except Exception as ex:  # noqa: BLE001 - reported by the assertion below
            errors.append(f"thread {t}: {ex!r}")

    threads = [threading.Thread(target=worker, args=(t,)) for t in range(len(engines))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e in engines:
        e.close()
    assert not errors, errors[:5]
