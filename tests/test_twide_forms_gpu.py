"""Single grids on the TMA wide kernel at the edges of its forms, bit for bit
against the oracle (FP64, FP32) and the compensated model: every pencil length
it takes along strided axes of several inner extents and the last axis, fewer
columns than a tile holds, partial last tiles, and grids that start on no
16-byte boundary (which keep the per-thread-copy kernels)."""
import numpy as np
import pytest

import paliwa_gb300 as pg

pytestmark = pytest.mark.gpu

WAVELETS = ["hat", "biorthogonal", "fullweighting"]


def want(x, level, lmin, wavelet, forward, mode):
    import oracle as O
    from compensated import hierarchize as model
    if mode == "f32c":
        return model(x, level, lmin, wavelet, forward)
    f = O.hierarchize if forward else O.dehierarchize
    return f(x.copy(), level, lmin, level, wavelet)


@pytest.mark.parametrize("mode", ["f64", "f32", "f32c"])
@pytest.mark.parametrize("log2_n", range(1, 13))
def test_every_pencil_length_and_inner_extent(mode, log2_n):
    import torch
    rng = np.random.default_rng(log2_n)
    dtype = np.float64 if mode == "f64" else np.float32
    wavelet = WAVELETS[log2_n % 3]
    for inner in (0, 1, 2, 3, 4, 6, 9):
        for outer in (0, 1, 3, 5):
            if outer + inner + log2_n > 18 or (outer > 3 and inner > 4):
                continue
            level, lmin = (outer, log2_n, inner), (outer, 0, inner)
            n = 1 << sum(level)
            x = rng.uniform(-1, 1, [1 << l for l in level]).astype(dtype)
            for offset in (0, 1) if inner in (0, 2) else (0,):
                buf = torch.empty(n + 1, device="cuda",
                                  dtype=getattr(torch, x.dtype.name))
                g = buf[offset:offset + n]
                for forward in (True, False):
                    g.copy_(torch.from_numpy(x.reshape(-1)))
                    f = pg.hierarchize if forward else pg.dehierarchize
                    f(g, level, lmin, level, wavelet,
                      compensated=mode == "f32c")
                    torch.cuda.synchronize()
                    got = g.cpu().numpy().reshape(x.shape)
                    exp = want(x, level, lmin, wavelet, forward, mode)
                    assert np.array_equal(got, exp), (level, offset, forward)


@pytest.mark.parametrize("mode", ["f64", "f32", "f32c"])
def test_more_tiles_than_resident_ctas(mode):
    """Enough tiles that every CTA's buffers cycle several times."""
    import torch
    rng = np.random.default_rng(3)
    dtype = np.float64 if mode == "f64" else np.float32
    for level in ((9, 5, 10), (12, 6, 5), (13, 10), (4, 10, 10)):
        dim = 1
        lmin = tuple(0 if d == dim else l for d, l in enumerate(level))
        x = rng.uniform(-1, 1, [1 << l for l in level]).astype(dtype)
        g = torch.from_numpy(x).cuda()
        pg.hierarchize(g, level, lmin, level, "biorthogonal",
                       compensated=mode == "f32c")
        torch.cuda.synchronize()
        exp = want(x, level, lmin, "biorthogonal", True, mode)
        assert np.array_equal(g.cpu().numpy(), exp), level


FILTERS = {
    # four passes, no coefficient a power of two
    "cdf97": [(1, (-1.586134342, 1.0, -1.586134342)),
              (0, (-0.05298011854, 1.0, -0.05298011854)),
              (1, (0.8829110762, 1.0, 0.8829110762)),
              (0, (0.4435068522, 1.0, 0.4435068522))],
    # powers of two, asymmetric, a middle coefficient other than 1
    "exact": [(0, (0.5, 2.0, -0.25)), (1, (0.0, 1.0, 0.125))],
    "scaled": [(1, (0.3, 1.2, -0.7))],
}


@pytest.mark.parametrize("mode", ["f64", "f32"])
@pytest.mark.parametrize("name", sorted(FILTERS))
def test_callers_filters_over_ordered_levels(mode, name):
    """transform_in over the level ranges of hierarchize_in and
    dehierarchize_in (whole and partial) with a caller's filters, for every
    form of the TMA wide kernel, against the oracle."""
    import torch
    import oracle as O
    dtype = np.float64 if mode == "f64" else np.float32
    rng = np.random.default_rng(29)
    for level in ((3, 2, 4), (2, 4, 6), (4, 5, 3), (3, 6, 4), (2, 8, 5),
                  (1, 9, 4), (1, 10, 3), (0, 11, 3), (6, 3), (5, 5), (4, 9),
                  (2, 10), (1, 12), (4, 7, 1), (13,), (12,)):
        dim = len(level) - 1 if len(level) < 3 else 1
        top = level[dim]
        for levels in (range(top, 0, -1), range(1, top + 1),
                       range(top, max(0, top - 2), -1), [top],
                       range(max(1, top - 2), top + 1)):
            levels = list(levels)
            x = rng.uniform(-1, 1, [1 << l for l in level]).astype(dtype)
            g = torch.from_numpy(x).cuda()
            pg.transform_in(g, dim, level, level, levels, FILTERS[name])
            torch.cuda.synchronize()
            exp = O.transform_in(x.copy(), level, level, dim, levels,
                                 FILTERS[name])
            assert np.array_equal(g.cpu().numpy(), exp), (level, levels)


@pytest.mark.parametrize("mode", ["f64", "f32"])
@pytest.mark.parametrize("level,lmin", [
    ((2, 13, 5), 0), ((2, 14, 4), 9), ((0, 15, 6), 3), ((1, 17, 4), 0),
    ((3, 13, 3), 0), ((15, 5), 11), ((14, 4), 0)])
def test_long_strided_pencils(mode, level, lmin):
    """Pencils of more than 4096 points: windows in the boxed form (rows of
    128 bytes and more; narrower ones on the staged kernel), with short last
    segments and partial level ranges."""
    import torch
    dim = 0 if len(level) == 2 else 1
    lo = tuple(lmin if d == dim else l for d, l in enumerate(level))
    dtype = np.float64 if mode == "f64" else np.float32
    rng = np.random.default_rng(sum(level))
    x = rng.uniform(-1, 1, [1 << l for l in level]).astype(dtype)
    for wavelet in WAVELETS:
        for forward in (True, False):
            g = torch.from_numpy(x).cuda()
            f = pg.hierarchize if forward else pg.dehierarchize
            f(g, level, lo, level, wavelet)
            torch.cuda.synchronize()
            exp = want(x, level, lo, wavelet, forward, mode)
            assert np.array_equal(g.cpu().numpy(), exp), (wavelet, forward)


@pytest.mark.parametrize("mode", ["f64", "f32", "f32c"])
@pytest.mark.parametrize("level", [(9, 15), (9, 17)])
def test_pencils_spread_over_pages(mode, level):
    """512-point pencils of 64 MB and more: the boxed form for floats."""
    import torch
    dtype = np.float64 if mode == "f64" else np.float32
    if mode == "f64" and sum(level) > 24:
        pytest.skip("the doubles' form does not depend on the span")
    rng = np.random.default_rng(7)
    x = rng.uniform(-1, 1, [1 << l for l in level]).astype(dtype)
    lo = (0, level[1])
    for forward in (True, False):
        g = torch.from_numpy(x).cuda()
        f = pg.hierarchize if forward else pg.dehierarchize
        f(g, level, lo, level, "biorthogonal", compensated=mode == "f32c")
        torch.cuda.synchronize()
        exp = want(x, level, lo, "biorthogonal", forward, mode)
        assert np.array_equal(g.cpu().numpy(), exp), forward


@pytest.mark.parametrize("level,lmin", [
    ((13, 7), 0), ((15, 5), 3), ((16, 5), 11), ((14, 8), 10), ((2, 13, 6), 0),
    ((13, 8), 12)])
def test_long_compensated_pencils(level, lmin):
    """FP32c pencils of 2^13 to 2^16 points in the boxed windows, whose heads
    go to the coarse levels unrounded and are rounded where the staged
    kernel's windows end: the bits of that plan (a batch's), forward and
    inverse."""
    import torch
    from paliwa_gb300 import ct as pct
    dim = 0 if len(level) == 2 else 1
    lo = tuple(lmin if d == dim else l for d, l in enumerate(level))
    rng = np.random.default_rng(sum(level))
    x = rng.uniform(-1, 1, 1 << sum(level)).astype(np.float32)
    for wavelet in WAVELETS:
        for forward in (True, False):
            g = torch.from_numpy(x).cuda()
            f = pg.hierarchize if forward else pg.dehierarchize
            f(g, level, lo, level, wavelet, compensated=True)
            b = torch.from_numpy(x).cuda()
            batch = pct.Batch([b], [level], lo, level, wavelet,
                              compensated=True)
            (batch.hierarchize if forward else batch.dehierarchize)()
            torch.cuda.synchronize()
            assert torch.equal(g, b), (wavelet, forward)
            batch.close()
