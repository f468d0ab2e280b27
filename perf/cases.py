"""The calls whose speed this framework is measured by, each through its public entry points.

A case is one call as a program that uses the framework makes it: a construction from keys that
are already on the GPU or in host memory, a batch of constructions as the build service issues
them, queries of a whole key set on the GPU, or a retrieval structure built and queried there. The
configurations (class, leaf size, bucket size, kind of keys) are those of the benchmark and the
tests. Every output is an array of whole numbers; the keys are made from the case's seed.

The engine is the process's default one, as for the class interface: its buffers grow once and are
used again from call to call, over inputs that change.
"""
import math

import numpy as np
import torch

import shockhash_b200 as shg

VARIANTS = {"shockhash2": shg.SHOCKHASH2, "shockhash": shg.SHOCKHASH, "rotation": shg.SHOCKHASH_ROTATION,
            "simd": shg.SIMDSHOCKHASH}

# Multiply, shift, xor and add steps of one key hash under one search seed.
_OPS_PER_EVALUATION = 20


def listed():
    return [
        # the smallest serving request (1,000 keys, one bucket): latency, launches and host work
        {"name": "sh2_l64_host_1k", "kind": "build", "cls": "shockhash2", "leaf": 64, "bucket": 2000, "n": 1000, "keys": "host"},
        # a small set of odd size with a ragged last bucket: fewer tree nodes than the GPU has SMs
        {"name": "sh2_l64_host_30k", "kind": "build", "cls": "shockhash2", "leaf": 64, "bucket": 2000, "n": 30011, "keys": "host"},
        # an ordinary set, keys already on the GPU
        {"name": "sh2_l64_device_1M", "kind": "build", "cls": "shockhash2", "leaf": 64, "bucket": 2000, "n": 1000003,
         "keys": "device"},
        # the largest: above the benchmark's 10M keys, where the partition takes its other path
        {"name": "sh2_l64_device_20M", "kind": "build", "cls": "shockhash2", "leaf": 64, "bucket": 2000, "n": 20000003,
         "keys": "device"},
        # what the build service hands to the engine at once: many requests of very different sizes
        {"name": "sh2_l64_batch_48", "kind": "batch", "cls": "shockhash2", "leaf": 64, "bucket": 2000, "requests": 48, "n": 1000000},
        # original ShockHash over printable strings in host memory (the 1M-string configuration)
        {"name": "sh1_l30_strings_1M", "kind": "build", "cls": "shockhash", "leaf": 30, "bucket": 2000, "n": 1000000,
         "keys": "strings"},
        # the space-saving setting of the original ShockHash: nearly all of the time is leaf search
        {"name": "sh1_l40_device_1M", "kind": "build", "cls": "shockhash", "leaf": 40, "bucket": 2000, "n": 1000000, "keys": "device"},
        # rotation fitting, the original class's faster option
        {"name": "rotation_l30_device_2M", "kind": "build", "cls": "rotation", "leaf": 30, "bucket": 2000, "n": 2000000,
         "keys": "device"},
        # the SIMD benchmark's format
        {"name": "simd_l30_device_2M", "kind": "build", "cls": "simd", "leaf": 30, "bucket": 2000, "n": 2000000, "keys": "device"},
        # the flat class over strings of Zipf-distributed length, with its host query object
        {"name": "flat_k100_strings_500k", "kind": "flat", "k": 100, "n": 500000},
        # operator() for every key of a structure, keys and answers on the GPU
        {"name": "query_device_10M", "kind": "query", "cls": "shockhash2", "leaf": 64, "bucket": 2000, "n": 10000000, "compact": False},
        # the compact retrieval structure: built from a retrieval input on the GPU, every key queried
        {"name": "retrieval_device_2M", "kind": "retrieval", "n": 2000000},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randrange(2)


def draw(rng):
    """One more case of the same ranges: sizes log-uniform, the classes' usual leaf sizes and buckets."""
    kind = rng.choice(["shockhash2", "shockhash2", "shockhash2", "batch", "shockhash", "rotation", "simd", "flat", "query",
                       "retrieval"])
    bucket = rng.choice([500, 1000, 1500, 2000, 2000])
    if kind == "shockhash2":
        return {"kind": "build", "cls": kind, "leaf": rng.choice([33, 48, 64, 64, 64]), "bucket": bucket,
                "n": _log_size(rng, 1000, 20000000), "keys": rng.choice(["host", "device", "device"])}
    if kind == "batch":
        return {"kind": "batch", "cls": "shockhash2", "leaf": rng.choice([48, 64, 64]), "bucket": bucket,
                "requests": rng.randrange(2, 64), "n": _log_size(rng, 100000, 4000000)}
    if kind == "shockhash":
        leaf = rng.choice([30, 30, 33, 40])
        return {"kind": "build", "cls": kind, "leaf": leaf, "bucket": bucket, "keys": rng.choice(["strings", "device"]),
                "n": _log_size(rng, 1000, 1000000 if leaf == 40 else 4000000)}
    if kind in ("rotation", "simd"):
        return {"kind": "build", "cls": kind, "leaf": rng.choice([30, 30, 33]), "bucket": bucket, "n": _log_size(rng, 1000, 4000000),
                "keys": rng.choice(["host", "device"])}
    if kind == "flat":
        return {"kind": "flat", "k": rng.choice([64, 100, 100]), "n": _log_size(rng, 5000, 500000)}
    if kind == "query":
        return {"kind": "query", "cls": "shockhash2", "leaf": rng.choice([48, 64]), "bucket": bucket, "n": _log_size(rng, 10000, 10000000),
                "compact": rng.random() < 0.5}
    return {"kind": "retrieval", "n": _log_size(rng, 1000, 8000000)}


# ---------------------------------------------------------------------------------------- keys
def _signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _u64_keys(n, seed, salt=0):
    """n distinct, well mixed 64-bit keys on the GPU (a bijection of consecutive numbers), as int64."""
    base = (seed * 0x9E3779B97F4A7C15 + salt * 0xD1B54A32D192ED03 + 0x632BE59BD9B4E019) % (1 << 64)
    x = torch.arange(n, dtype=torch.int64, device="cuda") + _signed(base)
    for mul, shift in ((0xBF58476D1CE4E5B9, 29), (0x94D049BB133111EB, 32), (0xD6E8FEB86659FD93, 30)):
        x ^= (x >> shift) & ((1 << (64 - shift)) - 1)
        x *= _signed(mul)
    x ^= (x >> 31) & ((1 << 33) - 1)
    return x


def _host_u64(n, seed, salt=0):
    return _u64_keys(n, seed, salt).cpu().numpy().view(np.uint64)


def _strings(n, seed, zipf):
    """n distinct strings as (bytes, offsets): 16 to 40 printable bytes, or 8 to 200 bytes of Zipf(1.1) length."""
    rng = np.random.default_rng(seed)
    if zipf:
        lengths = np.arange(8, 201)
        p = (lengths - 7.0) ** -1.1
        length = rng.choice(lengths, size=n, p=p / p.sum())
    else:
        length = rng.integers(16, 41, size=n)
    offsets = np.zeros(n + 1, np.uint64)
    np.cumsum(length, out=offsets[1:], dtype=np.uint64)
    data = rng.integers(33, 127, size=int(offsets[-1]), dtype=np.uint8)
    # the string's number in its first five characters (base 94) keeps the short ones distinct
    number, start = np.arange(n, dtype=np.int64), offsets[:-1].astype(np.int64)
    for i in range(5):
        data[start + i] = 33 + number % 94
        number //= 94
    return data.tobytes(), offsets


def _request_sizes(case):
    """Sizes of a batch's requests: log-uniform over a factor of a thousand, their sum about n."""
    rng = np.random.default_rng([case["requests"], case["n"]])
    w = np.exp(rng.uniform(0.0, math.log(1000.0), size=case["requests"]))
    return np.maximum(1000, (case["n"] * w / w.sum()).astype(np.int64)).tolist()


# ------------------------------------------------------------------------------------- a case
def prepare(case, seed):
    state = {"case": case, "engine": shg.default_engine()}
    kind = case["kind"]
    if kind == "build":
        if case["keys"] == "device":
            state["keys"] = _u64_keys(case["n"], seed)
        elif case["keys"] == "host":
            state["keys"] = _host_u64(case["n"], seed)
        else:
            state["keys"] = _strings(case["n"], seed, zipf=False)
    elif kind == "batch":
        state["keys"] = [_host_u64(n, seed, salt=i + 1) for i, n in enumerate(_request_sizes(case))]
    elif kind == "flat":
        state["keys"] = _strings(case["n"], seed, zipf=True)
    elif kind == "query":
        keys = _u64_keys(case["n"], seed)
        torch.cuda.synchronize()
        built = state["engine"].build_u64_device(VARIANTS[case["cls"]], case["leaf"], keys.data_ptr(), case["n"], case["bucket"])
        state.update(keys=keys, answers=torch.empty_like(keys), mphf=shg.DeviceMphf(built, compact=case["compact"]))
        built.free()
    else:
        keys = _u64_keys(case["n"], seed)
        state.update(keys=keys, bits=((keys >> 17) & 1).to(torch.uint8), answers=torch.empty(case["n"], dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    return state


def _whole(a, least, most):
    """The array `a`, whose length depends on the keys, in two parts of lengths that do not: its first
    `least` entries as they lie, and the rest in `most - least` entries filled up with zeros."""
    rest = np.zeros(most - least, a.dtype)
    rest[:len(a) - least] = a[least:]
    return a[:least], rest


def _products(r, n):
    # at most one key per bucket has no retrieval bit; descriptors take 1/4 to 8 bits per key
    few = max(0, n - r.nbuckets)
    return {"descriptors": _whole(r.descriptors, n // 256, n // 8 + 64), "bucket_size_acc": r.bucket_size_acc,
            "bucket_pos_acc": r.bucket_pos_acc, "ribbon_keys": _whole(r.ribbon_keys, few, n),
            "ribbon_bits": _whole(r.ribbon_bits, few, n)}


def _batch_products(rs, n):
    """The products of all requests of a batch, field by field."""
    out = {}
    for field, most in (("descriptors", n // 8 + 64 * len(rs)), ("bucket_size_acc", None), ("bucket_pos_acc", None),
                        ("ribbon_keys", n), ("ribbon_bits", n)):
        parts = [getattr(r, field) for r in rs]
        whole = np.empty(most or sum(map(len, parts)), parts[0].dtype)
        at = sum(map(len, parts))
        np.concatenate(parts, out=whole[:at])
        whole[at:] = 0
        out[field] = whole
    return out


def run(state):
    case, engine, keys = state["case"], state["engine"], state["keys"]
    kind = case["kind"]
    state.pop("result", None)  # the products of the call before, as a program that builds again drops them
    if kind == "build":
        variant, leaf, bucket = VARIANTS[case["cls"]], case["leaf"], case["bucket"]
        if case["keys"] == "device":
            r = engine.build_u64_device(variant, leaf, keys.data_ptr(), keys.numel(), bucket)
        elif case["keys"] == "host":
            r = engine.build_u64(variant, leaf, keys, bucket)
        else:
            r = engine.build_strings(variant, leaf, keys, bucket)
        state["result"] = r
        return _products(r, case["n"])
    if kind == "batch":
        rs = engine.build_batch_u64(VARIANTS[case["cls"]], case["leaf"], keys, case["bucket"])
        state["result"] = rs
        return _batch_products(rs, sum(map(len, keys)))
    if kind == "flat":
        f = engine.build_flat_strings(case["k"], keys)
        state["result"] = f
        buckets, n = f.nbuckets, case["n"]
        return {"thresholds_and_seeds": f.thresholds_and_seeds, "fallback_seed_buckets": _whole(f.fallback_seed_buckets, 0, buckets),
                "fallback_seeds": _whole(f.fallback_seeds, 0, buckets), "free_positions": _whole(f.free_positions, 0, n),
                "ribbon_keys": f.ribbon_keys, "ribbon_bits": f.ribbon_bits}
    if kind == "query":
        state["mphf"].query_u64_device(keys.data_ptr(), keys.numel(), state["answers"].data_ptr())
        return state["answers"]
    r = shg.Retrieval.build_device(engine, keys.data_ptr(), state["bits"].data_ptr(), case["n"])
    r.query_device(keys.data_ptr(), case["n"], state["answers"].data_ptr())
    state["result"] = r
    level_buckets, solutions, thresholds = r.arrays()
    most = case["n"] // 200 + 64
    return {"answers": state["answers"], "level_buckets": _whole(level_buckets, 0, 64), "solutions": _whole(solutions, 0, 4 * most),
            "thresholds": _whole(thresholds, 0, most)}


# ---------------------------------------------------------------------------------- their work
def _trials(parts):
    """Expected seeds until m keys fall into parts of exactly these sizes."""
    m = sum(parts)
    log_p = math.lgamma(m + 1) + sum(q * math.log(q / m) - math.lgamma(q + 1) for q in parts if q)
    return math.exp(-log_p)


def _split_evaluations(m, leaf, lower, upper):
    """Expected key hashes of the splits of one bucket of m keys, and the sizes of its leaves."""
    if m <= leaf:
        return 0.0, [m] if m > 1 else []
    if m > upper:
        half = (m // 2 + upper - 1) // upper * upper
        parts = [half, m - half]
    else:
        unit = lower if m > lower else leaf
        parts = [unit] * (m // unit) + ([m % unit] if m % unit else [])
    evaluations, leaves = m * _trials(parts), []
    for part in parts:
        e, l = _split_evaluations(part, leaf, lower, upper)
        evaluations += e
        leaves += l
    return evaluations, leaves


def _evaluations_per_key(case):
    """Expected key hashes per key of a construction that tries its seeds in order."""
    leaf, m = case["leaf"], min(case["bucket"], case["n"])
    if case["cls"] == "shockhash2":
        lower, upper = 4 * leaf, 12 * leaf
    else:
        lower = leaf * (4 if leaf > 24 else 2)
        upper = lower * (3 if leaf > 24 else 2)
    evaluations, leaves = _split_evaluations(m, leaf, lower, upper)
    for size in leaves:
        if case["cls"] == "shockhash2":  # pairs of candidates, themselves pairs of raw seeds
            evaluations += size * (math.e / 2) ** (size / 4)
            continue
        trials = max(1.0, (math.e / 2) ** size / (0.8 * math.sqrt(size)))
        if case["cls"] == "rotation":  # a seed stands for `size` rotations
            trials = max(1.0, trials / size)
        evaluations += size * trials
    return evaluations / m


def work(case):
    n, kind = case["n"], case["kind"]
    if kind in ("build", "batch"):
        key_bytes = {"strings": 28 + 8}.get(case.get("keys"), 8)
        return {"bytes": n * (key_bytes + 9), "flops": n * _evaluations_per_key(case) * _OPS_PER_EVALUATION}
    if kind == "flat":  # one bipartite leaf of k keys per bucket
        return {"bytes": n * (34 + 8 + 9 + 8 // case["k"]), "flops": n * (math.e / 2) ** (case["k"] / 4) * _OPS_PER_EVALUATION}
    if kind == "query":
        return {"bytes": n * 16, "flops": n * 3 * _OPS_PER_EVALUATION}
    return {"bytes": n * 10 + n // 4, "flops": n * 2 * _OPS_PER_EVALUATION}


def exact(case, seed):
    """None: every output is a whole number (there is no value in 64-bit floating point to compare with)."""
    return None
