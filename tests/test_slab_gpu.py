"""The slab kernel: every level of a grid's trailing axes in one pass
(paliwa_gb300/csrc/slab.cuh), in batches.

Its results are the per-axis plan's bits (the same updates in the same
order), so every case compares a batch planned with slab launches against
the same batch planned axis by axis -- FP64, FP32 and FP32-compensated,
both directions -- and FP64 also against the oracle. The bounded waits of
the kernel report no timeout.
"""
import itertools

import numpy as np
import pytest

from paliwa_gb300 import ct as pct

pytestmark = pytest.mark.gpu

WAVELETS = ["hat", "biorthogonal", "fullweighting"]


def oracle():
    import oracle as O
    O.build()
    return O


def scheme(ndim, top, qmax, lmin=1):
    return [l for q in range(qmax + 1)
            for l in itertools.product(range(lmin, top + 1), repeat=ndim)
            if sum(l) == top - q]


def run_pair(levels, lmin, lmax, wavelet, dtype, compensated, seed):
    import torch
    rng = np.random.default_rng(seed)
    host = [rng.uniform(-1, 1, 1 << sum(l)) for l in levels]
    out = []
    for slabs in (True, False):
        buf, views = pct.packed_grids(levels, dtype)
        for v, h in zip(views, host):
            v.copy_(torch.from_numpy(h.astype(np.float64)).to(dtype))
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        bt = pct.Batch(views, levels, lmin, lmax, wavelet,
                       compensated=compensated, slabs=slabs)
        bt.hierarchize(s)
        s.synchronize()
        f = buf.clone()
        bt.dehierarchize(s)
        s.synchronize()
        bt.status()
        esz = buf.element_size()
        starts = [(v.data_ptr() - buf.data_ptr()) // esz for v in views]
        out.append((f, buf.clone(), starts))
        # The kernels of the forward plan (this runs it once more, after
        # the results were taken).
        _, _, kernels = bt.profile(forward=True, stream=s)
        s.synchronize()
        bt.status()
        out[-1] += (kernels,)
        bt.close()
    return host, out


@pytest.mark.parametrize("dtype_name", ["f64", "f32", "f32c"])
@pytest.mark.parametrize("case", [(3, 10, 2), (4, 12, 3), (5, 11, 2),
                                  (6, 12, 2), (2, 14, 2)])
def test_slab_plan_equals_per_axis_plan(dtype_name, case):
    import torch
    ndim, top, qmax = case
    levels = scheme(ndim, top, qmax)
    lmin, lmax = (1,) * ndim, (top,) * ndim
    dtype = torch.float64 if dtype_name == "f64" else torch.float32
    for w, wavelet in enumerate(WAVELETS):
        host, ((f1, b1, v1, k1), (f2, b2, _, k2)) = run_pair(
            levels, lmin, lmax, wavelet, dtype, dtype_name == "f32c",
            100 * ndim + top + w)
        assert pct.SLAB_KERNEL in k1 and pct.SLAB_KERNEL not in k2
        assert torch.equal(f1, f2), (case, wavelet)
        assert torch.equal(b1, b2), (case, wavelet)
        if dtype_name == "f64" and w == 1:
            O = oracle()
            for i in range(0, len(levels), max(1, len(levels) // 40)):
                lv = levels[i]
                off = v1[i]  # the grid's first element in the buffer
                got = f1[off:off + (1 << sum(lv))].cpu().numpy()
                want = O.hierarchize(
                    host[i].reshape([1 << l for l in lv]).copy(), lv, lmin,
                    lmax, wavelet).reshape(-1)
                assert np.array_equal(got, want), (case, lv)


def test_slab_lmin_zero_and_single_tile_grids():
    """Grids of one tile or less (down to 1 KB), minimum level 0 and axes
    of a single point."""
    import torch
    levels = [(0, 3, 5), (2, 0, 6), (1, 1, 7), (3, 4, 1), (5, 5, 0),
              (2, 2, 4), (4, 6, 2), (1, 7, 7)]
    lmin, lmax = (0, 0, 0), (7, 7, 7)
    for dtype, comp in ((torch.float64, False), (torch.float32, True)):
        host, ((f1, b1, _, k1), (f2, b2, _, _)) = run_pair(
            levels, lmin, lmax, "biorthogonal", dtype, comp, 5)
        assert pct.SLAB_KERNEL in k1
        assert torch.equal(f1, f2)
        assert torch.equal(b1, b2)


@pytest.mark.parametrize("mode", ["f64", "f32", "f32c"])
@pytest.mark.parametrize("level,lmin", [
    ((4, 4), (0, 0)), ((5, 3), (1, 0)), ((3, 3, 3), (0, 0, 0)),
    ((2, 2, 2, 2, 2, 2), (0,) * 6), ((4, 0, 5, 3), (0, 0, 1, 0)),
    ((6, 5, 5), (0, 0, 0)), ((7, 1, 6, 6), (1, 1, 1, 1)),
    ((3, 13), (0, 0)), ((2, 2, 2), (0, 0, 0)), ((1,) * 13, (0,) * 13),
    ((0, 4, 5), (0, 4, 0))])
def test_single_grids_with_slab_launches(mode, level, lmin):
    """hierarchize and dehierarchize of one grid whose trailing axes may go in
    one slab launch: whole grids of one tile and of many, leading axes before
    the slab, grids under one box, more axes than a slab job holds, axes with
    nothing to do; a grid that starts on no 128-byte row goes axis by axis."""
    import paliwa_gb300 as pg
    import torch
    import oracle as O
    from compensated import hierarchize as model
    dtype = np.float64 if mode == "f64" else np.float32
    rng = np.random.default_rng(len(level))
    x = rng.uniform(-1, 1, [1 << l for l in level]).astype(dtype)
    buf = torch.empty(x.size + 4, dtype=getattr(torch, x.dtype.name),
                      device="cuda")
    for offset in (0, 4):
        g = buf[offset:offset + x.size]
        for wavelet in ("hat", "biorthogonal"):
            for forward in (True, False):
                g.copy_(torch.from_numpy(x.reshape(-1)))
                f = pg.hierarchize if forward else pg.dehierarchize
                f(g, level, lmin, level, wavelet, compensated=mode == "f32c")
                torch.cuda.synchronize()
                if mode == "f32c":
                    want = model(x, level, lmin, wavelet, forward)
                else:
                    o = O.hierarchize if forward else O.dehierarchize
                    want = o(x.copy(), level, lmin, level, wavelet)
                got = g.cpu().numpy().reshape(x.shape)
                if mode == "f32c" and max(level) > 12:
                    # Windows round between their stages, which the model
                    # does not describe: the error bound of FP32c against
                    # the FP64 oracle instead.
                    o = O.hierarchize if forward else O.dehierarchize
                    want = o(x.astype(np.float64), level, lmin, level,
                             wavelet)
                    assert np.max(np.abs(got - want)) <= \
                        1e-6 * np.max(np.abs(want))
                    continue
                assert np.array_equal(got, want)


@pytest.mark.parametrize("dtype_name", ["f32", "f32c"])
@pytest.mark.parametrize("level", [
    (5, 6), (6, 6), (11, 1), (6, 5, 1), (1, 1, 10), (4, 8, 1), (5, 7, 2),
    (12, 1, 2), (3, 3, 2, 2, 2), (1, 0, 12), (7, 6, 0), (9, 2, 4)])
def test_pairs_of_floats_equal_the_per_axis_plan(dtype_name, level):
    """Axes worked in pairs of adjacent inner indices: tiles of 2^11 points
    (no pairs) and from 2^12, inner extents from one pair up, pencils of one
    chunk, of chunks in one warp and of chunks that meet at barriers; bit for
    bit the axis-by-axis plan, which holds no pairs in a slab."""
    import torch
    lmin = (0,) * len(level)
    for w, wavelet in enumerate(WAVELETS):
        _, out = run_pair([level], lmin, level, wavelet, torch.float32,
                          dtype_name == "f32c", w)
        (f1, b1, _, kernels), (f2, b2, _, _) = out
        assert 1024 in kernels
        assert torch.equal(f1, f2) and torch.equal(b1, b2)


def test_pairs_only_where_tiles_are_large_enough():
    """A launch of small and large tiles: the small grids go through the
    kernel that works in pairs as well, with the same bits."""
    import torch
    levels = [(3, 2, 2), (6, 6, 3), (2, 5, 4), (5, 5, 5)]
    for compensated in (False, True):
        _, out = run_pair(levels, (0,) * 3, (6,) * 3, "biorthogonal",
                          torch.float32, compensated, 5)
        (f1, b1, _, _), (f2, b2, _, _) = out
        assert torch.equal(f1, f2) and torch.equal(b1, b2)


@pytest.mark.parametrize("dtype_name", ["f64", "f32", "f32c"])
def test_one_axis_of_a_single_tile_in_the_slab_launch(dtype_name):
    """Grids of one tile with one axis to transform go in the slab launch of
    the others, leading, middle and last axis alike, up to a whole tile; a
    kernel chosen for their tuning class takes them out again. The bits are
    the axis-by-axis plan's."""
    import torch
    top = 12 if dtype_name == "f64" else 13
    levels = [(top, 0, 0), (0, top, 0), (0, 0, top), (9, 0, 1), (1, 8, 1),
              (0, 2, 8), (4, 3, 3)]
    lmin = [0, 0, 0]
    dtype = torch.float64 if dtype_name == "f64" else torch.float32
    for w, wavelet in enumerate(WAVELETS):
        _, out = run_pair(levels, lmin, (top,) * 3, wavelet, dtype,
                          dtype_name == "f32c", w)
        (f1, b1, _, kernels), (f2, b2, _, _) = out
        # (long FP32c pencils are windows that round in between)
        assert 1024 in kernels
        assert set(kernels) == {1024} or dtype_name == "f32c"
        assert torch.equal(f1, f2) and torch.equal(b1, b2)
    buf, views = pct.packed_grids(levels, dtype)
    buf.copy_(torch.from_numpy(
        np.random.default_rng(7).uniform(-1, 1, buf.numel())))
    start = buf.clone()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    bt = pct.Batch(views, levels, lmin, (top,) * 3, "hat",
                   compensated=dtype_name == "f32c")
    bt.hierarchize(s)
    s.synchronize()
    want = buf.clone()
    code, _, names, chosen = next(
        (r for r in bt.tuning(True) if len(r[2]) > 1), (None,) * 4)
    if code is None:  # one kernel applies to every class
        assert dtype_name != "f64"
        bt.close()
        return
    bt.set_tuning({code: next(n for n in names if n != chosen)}, True)
    _, _, kernels = bt.profile(forward=True, stream=s)
    assert set(kernels) != {1024}
    s.synchronize()
    buf.copy_(start)
    torch.cuda.synchronize()
    bt.hierarchize(s)
    s.synchronize()
    assert torch.equal(buf, want)
    bt.close()
