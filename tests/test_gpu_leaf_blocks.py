"""Leaf searches by a block per leaf and by a warp per leaf (the number of leaves of a launch decides)
give the same seeds and bits: one call over many leaves against calls over a few of them, which the
golden leaf fixtures and the oracle cover."""
import numpy as np
import pytest

import shockhash_b200 as shg
from conftest import unique_u64

pytestmark = pytest.mark.gpu


def offsets(sizes):
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


@pytest.mark.parametrize("sizes,many,few", [((65, 66, 71, 72), 30_000, 40), ((57, 63, 64, 64, 61, 9), 900, 500)])
def test_bipartite_block_and_warp_search_agree(engine, port, sizes, many, few):
    rng = np.random.default_rng(sum(sizes))
    m = np.array([sizes[i % len(sizes)] for i in range(many)])
    keys = unique_u64(rng, int(m.sum()))
    off = offsets(m)
    seeds, bits = engine.sh2_construct_leaves(keys, off)
    for a in (0, many - few):
        lo, hi = int(off[a]), int(off[a + few])
        s, b = engine.sh2_construct_leaves(keys[lo:hi], off[a:a + few + 1] - off[a])
        assert np.array_equal(s, seeds[a:a + few]) and np.array_equal(b, bits[lo:hi])


def test_bipartite_block_keys_with_little_room(engine):
    # low 30 bits about to run over: the staged keys are good for a few raw seeds only
    rng = np.random.default_rng(3)
    m, n = 64, 40
    keys = (unique_u64(rng, m * n) | np.uint64(0x3fffffff)) - rng.integers(0, 300, size=m * n).astype(np.uint64)
    assert len(np.unique(keys)) == m * n
    off = offsets([m] * n)
    s, b = engine.sh2_construct_leaves(keys, off)  # a block per leaf
    rep = 20  # the same leaves among others: a warp per leaf
    s2, b2 = engine.sh2_construct_leaves(np.tile(keys, rep), offsets([m] * (n * rep)))
    assert np.array_equal(np.tile(s, rep), s2) and np.array_equal(np.tile(b, rep), b2)


@pytest.mark.parametrize("leaf,n", [(30, 400_000), (24, 300_000)])
def test_original_block_and_warp_search_agree(engine, leaf, n):
    # many buckets take a warp per leaf, a shard of them a block per leaf
    rng = np.random.default_rng(leaf)
    first, second = rng.integers(0, 2**64, size=n, dtype=np.uint64), unique_u64(rng, n)
    nb = (n + 1999) // 2000
    whole = engine.build_hash128(shg.SHOCKHASH, leaf, first, second, 2000)
    keys, bits, acc = whole.ribbon_keys.copy(), whole.ribbon_bits.copy(), whole.bucket_size_acc.copy()
    b1 = 3
    inside = np.array([(int(f) * nb) >> 64 < b1 for f in first])
    part = engine.build_shard_hash128(shg.SHOCKHASH, leaf, first[inside], second[inside], nb, 0, b1, 2000)
    assert np.array_equal(part.bucket_size_acc, acc[:b1 + 1])
    k = len(part.ribbon_keys)
    assert np.array_equal(part.ribbon_keys, keys[:k]) and np.array_equal(part.ribbon_bits, bits[:k])


def second_halves(rng, n, kind):
    """Distinct second halves: all even, all odd, or short of where their low 30 bits run over under a
    start seed of depths 0..3 (ShockHash.h:47-49)."""
    if kind == "over":
        start = np.array([0x106393c187cae21a, 0x6453cec3f7376937, 0x643e521ddbd2be98, 0x3740c6412f6572cb], dtype=np.uint64)
        short = rng.integers(1, 3000, size=n).astype(np.uint64) + start[rng.integers(0, 4, size=n)]
        out = (unique_u64(rng, n) & ~np.uint64(0x3fffffff)) - short
    else:
        out = (unique_u64(rng, n) & ~np.uint64(1)) | np.uint64(kind == "odd")
    assert len(np.unique(out)) == n
    return out


@pytest.mark.parametrize("kind", ["even", "odd", "over"])
@pytest.mark.parametrize("leaf", [34, 35, 40])
def test_original_seed_pairs_block_search(engine, port, leaf, kind):
    # leaves of 34 keys or more, a block per leaf: the first sieve takes seeds in pairs
    rng = np.random.default_rng(leaf)
    n = 1000 + leaf // 2
    first, second = rng.integers(0, 2**64, size=n, dtype=np.uint64), second_halves(rng, n, kind)
    r, p = engine.build_hash128(shg.SHOCKHASH, leaf, first, second, 500), port.build_hash(shg.SHOCKHASH, leaf, first, second, 500)
    assert np.array_equal(r.descriptors, p.desc)
    assert np.array_equal(r.ribbon_keys, p.ribbon_keys) and np.array_equal(r.ribbon_bits, p.ribbon_bits)


@pytest.mark.parametrize("kind", ["even", "odd", "over"])
def test_original_seed_pairs_warp_search(engine, kind):
    # many leaves of 30 keys (a warp per leaf, seeds in pairs) against a few of them (a block, single seeds)
    rng = np.random.default_rng(30)
    n, nb, b1 = 400_000, 200, 3
    first, second = rng.integers(0, 2**64, size=n, dtype=np.uint64), second_halves(rng, n, kind)
    whole = engine.build_hash128(shg.SHOCKHASH, 30, first, second, 2000)
    keys, bits = whole.ribbon_keys.copy(), whole.ribbon_bits.copy()
    inside = np.array([(int(f) * nb) >> 64 < b1 for f in first])
    part = engine.build_shard_hash128(shg.SHOCKHASH, 30, first[inside], second[inside], nb, 0, b1, 2000)
    k = len(part.ribbon_keys)
    assert np.array_equal(part.ribbon_keys, keys[:k]) and np.array_equal(part.ribbon_bits, bits[:k])


@pytest.mark.parametrize("leaf,n", [(2, 90), (3, 91), (31, 700), (32, 700), (41, 300), (48, 200)])
def test_original_pseudoforest_word_sizes(engine, port, leaf, n):
    # the peeling's words and keys per lane change at 32 and 41 keys
    rng = np.random.default_rng(leaf)
    first, second = rng.integers(0, 2**64, size=n, dtype=np.uint64), unique_u64(rng, n)
    r, p = engine.build_hash128(shg.SHOCKHASH, leaf, first, second, 200), port.build_hash(shg.SHOCKHASH, leaf, first, second, 200)
    assert np.array_equal(r.descriptors, p.desc)
    assert np.array_equal(r.ribbon_keys, p.ribbon_keys) and np.array_equal(r.ribbon_bits, p.ribbon_bits)


@pytest.mark.parametrize("leaf", [2, 31, 32, 40, 41])
def test_rotation_pseudoforest_word_sizes(engine, leaf):
    # the oracle has no rotation fitting: the structure has to be a minimal perfect hash for its host query
    rng = np.random.default_rng(leaf)
    n = 40 * leaf + 3
    first, second = rng.integers(0, 2**64, size=n, dtype=np.uint64), unique_u64(rng, n)
    r = engine.build_hash128(shg.SHOCKHASH_ROTATION, leaf, first, second, 500, query=True)
    assert np.array_equal(np.sort(r._mphf.query_hash(first, second)), np.arange(n, dtype=np.uint64))
