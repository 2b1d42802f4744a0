"""Scratch of the single-grid transforms of pencils longer than 4096 points:
the grid's size, and an eighth more only where FP32c windows hand chunk heads
on and the memory is there."""
import ctypes

import pytest

from paliwa_gb300 import _lib
from test_zz_no_alloc import DevicePool

pytestmark = pytest.mark.gpu


class PoolProps(ctypes.Structure):  # cuda.h: CUmemPoolProps
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int),
                ("location_type", ctypes.c_int), ("location_id", ctypes.c_int),
                ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


def hierarchize(grid, level, lmin, stream):
    _lib.check(_lib.load().paliwa_gb_hierarchize(
        grid.data_ptr(), _lib.F32C, len(level), _lib.i64(level),
        _lib.i64(lmin), _lib.i64(level), _lib.BIORTHOGONAL,
        stream.cuda_stream))


@pytest.mark.parametrize("level, lmin, heads", [
    ((3, 15), (1, 1), False),   # the last axis
    ((13, 2), (1, 1), False),   # rows of 16 bytes
    ((17, 5), (1, 1), False),   # 2^17 points
    ((13, 8), (9, 1), False),   # four levels: none for the heads
    ((13, 8), (8, 1), True),
    ((16, 5), (1, 1), True),
])
def test_heads_are_allocated_only_where_used(level, lmin, heads):
    import torch
    grid = torch.rand([1 << l for l in level], device="cuda")
    s = torch.cuda.Stream()
    pool = DevicePool()
    torch.cuda.synchronize()
    pool.reset()
    hierarchize(grid, level, lmin, s)
    s.synchronize()
    nbytes = 4 * grid.numel()
    assert pool.high() == nbytes + (nbytes // 8 if heads else 0)


def test_transform_without_memory_for_the_heads():
    """A memory pool that holds the halo buffer, but not the heads too."""
    import torch
    level, lmin = (14, 12), (0, 0)
    a = torch.rand([1 << l for l in level], device="cuda")
    b = a.clone()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    hierarchize(a, level, lmin, s)
    s.synchronize()
    cu = DevicePool().cu
    dev, old, pool = ctypes.c_int(), ctypes.c_void_p(), ctypes.c_void_p()
    assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuDeviceGetMemPool(ctypes.byref(old), dev) == 0
    # CU_MEM_ALLOCATION_TYPE_PINNED, no export handle, CU_MEM_LOCATION_TYPE_DEVICE
    props = PoolProps(1, 0, 1, 0, None, 4 * a.numel())
    assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    try:
        assert cu.cuDeviceSetMemPool(dev, pool) == 0
        hierarchize(b, level, lmin, s)
        s.synchronize()
    finally:
        assert cu.cuDeviceSetMemPool(dev, old) == 0
        assert cu.cuMemPoolDestroy(pool) == 0
    # FP32c rounds in the same places with heads and without.
    assert torch.equal(a, b)


@pytest.mark.parametrize("dtype, level", [
    ("float32", (13, 8)),
    ("float32", (14, 10)),  # 64 MiB: the heads end with the array behind it
    ("float64", (13, 8)),
])
@pytest.mark.parametrize("direction", [1, -1])
def test_noalloc_windows_in_rows_of_128_bytes(dtype, level, direction):
    """The allocation-free transform on the 512-point windows (FP32c: with
    heads), against the allocating entry points, twice: the array keeps the
    last call's contents."""
    import torch
    lib = _lib.load()
    code = _lib.F32C if dtype == "float32" else _lib.F64
    fn = (lib.paliwa_gb_hierarchize if direction > 0
          else lib.paliwa_gb_dehierarchize)
    a = torch.rand([1 << l for l in level], device="cuda",
                   dtype=getattr(torch, dtype))
    b, before = a.clone(), a.clone()
    lv, lmin = _lib.i64(level), _lib.i64((0,) * len(level))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(2):
        _lib.check(lib.paliwa_gb_transform_noalloc(
            a.data_ptr(), code, 2, lv, lmin, lv, _lib.BIORTHOGONAL, direction,
            s.cuda_stream))
        _lib.check(fn(b.data_ptr(), code, 2, lv, lmin, lv, _lib.BIORTHOGONAL,
                      s.cuda_stream))
        s.synchronize()
        assert not torch.equal(a, before)
        assert torch.equal(a, b)
        before.copy_(a)
        torch.cuda.synchronize()


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_windows_of_a_batch_in_one_launch(dtype, oracle_mod):
    """512-point windows of several grids in one job list, and on the
    per-thread-copy kernels."""
    import numpy as np
    import torch
    from paliwa_gb300 import ct
    levels = [(13, 8), (15, 5), (14, 7), (13, 9)]
    top = (15, 9)
    rng = np.random.default_rng(5)
    hosts = [rng.uniform(-1, 1, [1 << l for l in lv]).astype(dtype)
             for lv in levels]
    grids = [torch.from_numpy(h).cuda() for h in hosts]
    batch = ct.Batch(grids, levels, (0, 0), top, "biorthogonal", groups=1)
    for forward in (True, False):
        run = oracle_mod.hierarchize
        want = [run(h.copy(), lv, (0, 0), lv, "biorthogonal", forward=forward)
                for h, lv in zip(hosts, levels)]
        for tma in (True, False):
            batch.use_tma(tma)
            for g, h in zip(grids, hosts):
                g.copy_(torch.from_numpy(h))
            batch.hierarchize() if forward else batch.dehierarchize()
            torch.cuda.synchronize()
            batch.status()
            for g, w in zip(grids, want):
                assert np.array_equal(g.cpu().numpy(), w), (forward, tma)
