"""Host-key entry points given memory that is not plain host memory: managed and pinned arrays build the same
products, and a device address either does too or is refused (the staging threads never read it)."""
import ctypes

import numpy as np
import pytest

import shockhash_b200 as shg

pytestmark = pytest.mark.gpu
N = 1_000_000  # 8 MB: above the staging threshold of a single array


def products(r):
    out = [a.tobytes() for a in (r.descriptors, r.bucket_size_acc, r.bucket_pos_acc, r.ribbon_keys, r.ribbon_bits)]
    r.free()
    return out


def build_at(engine, address, n):
    p, res = engine.params(shg.SHOCKHASH2, 20, 300, shg.MODE_DEFAULT, 0), shg._Result()
    st = shg.lib().shg_build_u64(engine._h, ctypes.byref(p), ctypes.c_void_p(address), n, ctypes.byref(res))
    return engine._finish(p, st, res, False)


def build_batch_at(engine, parts):
    p, R = engine.params(shg.SHOCKHASH2, 20, 300, shg.MODE_DEFAULT, 0), len(parts)
    ptrs, ns, outs = (ctypes.c_void_p * R)(*[a for a, _ in parts]), np.array([n for _, n in parts], dtype=np.uint64), (shg._Result * R)()
    st = shg.lib().shg_build_batch_u64(engine._h, ctypes.byref(p), ptrs, shg._ptr(ns), R, outs)
    return [engine._finish(p, st, o, False) for o in outs]


@pytest.fixture(scope="module")
def keys():
    return shg.keys_mt19937_64(3, N)


@pytest.fixture(scope="module")
def want(engine, keys):
    return products(engine.build_u64(shg.SHOCKHASH2, 20, keys, 300))


def test_managed_memory(engine, keys, want):
    rt = ctypes.CDLL("libcudart.so.12")
    p = ctypes.c_void_p()
    assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(8 * N), 1) == 0
    try:
        ctypes.memmove(p, keys.ctypes.data, 8 * N)
        assert products(build_at(engine, p.value, N)) == want
        whole, few = build_batch_at(engine, [(p.value, N), (keys.ctypes.data, 5000)])
        assert products(whole) == want and products(few) == products(engine.build_u64(shg.SHOCKHASH2, 20, keys[:5000], 300))
    finally:
        rt.cudaFree(p)


def test_pinned_memory(engine, keys, want):
    import torch
    t = torch.from_numpy(keys.view(np.int64)).pin_memory()
    assert products(build_at(engine, t.data_ptr(), N)) == want


@pytest.mark.parametrize("batch", [False, True])
def test_device_address(engine, keys, want, batch):
    import torch
    d = torch.from_numpy(keys.view(np.int64)).to("cuda")
    torch.cuda.synchronize()
    try:
        r = build_batch_at(engine, [(d.data_ptr(), N), (d.data_ptr(), 20_000)])[0] if batch else build_at(engine, d.data_ptr(), N)
    except shg.ShgError:
        r = None
    if r is not None:
        assert products(r) == want
    assert products(engine.build_u64(shg.SHOCKHASH2, 20, keys, 300)) == want  # the engine goes on working
