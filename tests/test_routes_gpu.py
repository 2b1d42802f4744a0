"""Calls for which a newer route is the slower way: the kernels of a call, as
the nodes of its capture."""
import ctypes

import pytest

import paliwa_gb300 as pg

pytestmark = pytest.mark.gpu


def kernels(call):
    """Names of the kernel nodes that call(stream) adds to a capture."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    s = torch.cuda.Stream()
    call(s)  # what a first call sets up is not part of it
    torch.cuda.synchronize()
    graph, n = ctypes.c_void_p(), ctypes.c_size_t()
    h = ctypes.c_void_p(s.cuda_stream)
    # CU_STREAM_CAPTURE_MODE_RELAXED
    assert cu.cuStreamBeginCapture_v2(h, 2) == 0
    call(s)
    assert cu.cuStreamEndCapture(h, ctypes.byref(graph)) == 0
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    names = []
    for node in map(ctypes.c_void_p, nodes):
        kind = ctypes.c_int()
        assert cu.cuGraphNodeGetType(node, ctypes.byref(kind)) == 0
        if kind.value != 0:  # CU_GRAPH_NODE_TYPE_KERNEL
            continue
        # CUDA_KERNEL_NODE_PARAMS_v2: func first, kern after extents,
        # shared memory and two pointers
        params, name = (ctypes.c_uint64 * 16)(), ctypes.c_char_p()
        assert cu.cuGraphKernelNodeGetParams_v2(node, params) == 0
        if params[0]:
            assert cu.cuFuncGetName(ctypes.byref(name),
                                    ctypes.c_void_p(params[0])) == 0
        else:
            assert cu.cuKernelGetName(ctypes.byref(name),
                                      ctypes.c_void_p(params[7])) == 0
        names.append(name.value.decode())
    assert cu.cuGraphDestroy(graph) == 0
    return names


def launches(call):
    return len(kernels(call))


@pytest.mark.parametrize("level, dim, first, count, levels, want", [
    # few columns: a launch per pass
    ((13,), 0, 100, 4609, (13,), 2),
    ((2, 13), 1, 0, 4096, (13, 12), 4),
    # columns for every SM, a short stretch: one launch
    ((8, 8, 7), 0, 16, 160, (8, 7, 6, 5), 1),
    ((6, 6, 8), 2, 16, 160, (8, 7, 6, 5), 1),
])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_pass_list_launches(dtype, level, dim, first, count, levels, want):
    import torch
    shape = [1 << l for l in level]
    shape[dim] = count
    front = [0] * len(level)
    front[dim] = first
    x = torch.zeros(shape, dtype=getattr(torch, dtype), device="cuda")
    filters = pg.lifting_wavelet_filter_offsets_and_coefficients[
        "biorthogonal"]
    assert launches(lambda s: pg.transform_in_window(
        x, dim, level, level, levels, filters, front, stream=s)) == want


@pytest.mark.parametrize("level, want", [
    # a chunk of 32 points along some axis, or of 16 along one of two
    ((5, 5), 2), ((3, 6), 2), ((6, 5), 2), ((5, 4), 2), ((3, 3, 5), 3),
    # shorter chunks, more axes or tiny grids
    ((6, 3), 1), ((4, 4), 1), ((4, 4, 3), 1), ((2, 2, 2, 4), 1),
])
@pytest.mark.parametrize("forward", [True, False])
def test_small_double_grids_launches(level, want, forward):
    import torch
    x = torch.zeros([1 << l for l in level], dtype=torch.float64,
                    device="cuda")
    zero = (0,) * len(level)
    fn = pg.hierarchize if forward else pg.dehierarchize
    assert launches(lambda s: fn(x, level, zero, level, "biorthogonal",
                                 stream=s)) == want


@pytest.mark.parametrize("dtype, level, dim, tma", [
    # few points in pencils of 2, or of 4 floats: no TMA launch
    ("float32", (8, 1, 5), 1, False), ("float32", (8, 2, 5), 1, False),
    ("float32", (12, 2), 1, False), ("float32", (13, 2, 3), 1, False),
    ("float64", (8, 1, 5), 1, False), ("float64", (8, 1, 1), 1, False),
    # longer pencils, or many points
    ("float32", (8, 3, 5), 1, True), ("float32", (12, 2, 6), 1, True),
    ("float32", (12, 1, 7), 1, True), ("float64", (8, 2, 5), 1, True),
    ("float64", (12, 1, 7), 1, True),
])
def test_callers_filters_on_short_pencils(dtype, level, dim, tma):
    import torch
    x = torch.zeros([1 << l for l in level], dtype=getattr(torch, dtype),
                    device="cuda")
    filters = [(1, (-0.4, 1.0, -0.6)), (0, (0.3, 1.0, 0.2))]
    names = kernels(lambda s: pg.transform_in(
        x, dim, level, level, range(level[dim], 0, -1), filters, stream=s))
    assert len(names) == 1
    assert ("twide" in names[0]) == tma, names


def test_small_stages_of_a_batch_share_launches(oracle_mod):
    """Stages too small for two forms of the TMA wide kernel that fall back to
    one kernel run in one launch of it."""
    import numpy as np
    import torch
    from paliwa_gb300 import ct
    levels, lmin = [(3, 2), (5, 2)], (0, 2)
    rng = np.random.default_rng(1)
    hosts = [rng.uniform(-1, 1, [1 << l for l in lv]) for lv in levels]
    grids = [torch.from_numpy(h).cuda() for h in hosts]
    batch = ct.Batch(grids, levels, lmin, (5, 2), "biorthogonal", groups=1,
                     slabs=False)
    assert len(batch.profile(True)[2]) == 1
    for g, h in zip(grids, hosts):
        g.copy_(torch.from_numpy(h))
    batch.hierarchize()
    torch.cuda.synchronize()
    for g, h, lv in zip(grids, hosts, levels):
        want = oracle_mod.hierarchize(h.copy(), lv, lmin, lv, "biorthogonal")
        assert np.array_equal(g.cpu().numpy(), want)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_one_axis_grids_in_slab_launches(dtype):
    """A slab launch where it saves launches (code 1024), not for a lone grid
    with one axis."""
    import torch
    from paliwa_gb300 import ct
    levels = [(9,), (8,), (10,)]
    grids = [torch.zeros(1 << lv[0], dtype=getattr(torch, dtype),
                         device="cuda") for lv in levels]
    kinds = [ct.Batch(grids[:n], levels[:n], (0,), (10,), "biorthogonal",
                      groups=1).profile(True)[2] for n in (1, 3)]
    assert len(kinds[0]) == 1 and kinds[0] != [1024]
    assert kinds[1] == [1024]
