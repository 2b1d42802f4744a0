"""Combine and restrict on either side of their choice of kernels, against the
oracle bit for bit."""
import numpy as np
import pytest

from paliwa_gb300 import ct as pct
from test_routes_gpu import kernels

pytestmark = pytest.mark.gpu


def run(levels, dtype):
    """(kernel names of combine, of restrict) of random grids, after checking
    the results."""
    import torch
    import oracle as O
    nd = len(levels[0])
    lmax = tuple(max(l[d] for l in levels) for d in range(nd))
    rng = np.random.default_rng(17)
    coeffs = [float(c) for c in rng.integers(-3, 4, len(levels))]
    xs = [rng.uniform(-1, 1, [1 << l for l in lv]).astype(dtype)
          for lv in levels]
    gs = [torch.from_numpy(x.copy()).cuda() for x in xs]
    ct = pct.CombinationTechnique(gs, levels, coeffs, lmax)
    offsets, total = O.sparse_offsets(O.kept_subspaces(levels))
    sparse = torch.empty(total, dtype=torch.float64, device="cuda")
    names = [kernels(lambda s: ct.combine(sparse, stream=s))]
    ct.combine(sparse)
    want = O.combine_sparse(xs, levels, coeffs, offsets, total)
    torch.cuda.synchronize()
    assert np.array_equal(sparse.cpu().numpy(), want)
    names.append(kernels(lambda s: ct.restrict(sparse, stream=s)))
    for g, x in zip(gs, xs):
        g.copy_(torch.from_numpy(x))
    ct.restrict(sparse)
    torch.cuda.synchronize()
    for g, x, lv in zip(gs, xs, levels):
        exp = O.restrict_sparse(x.copy(), lv, want, offsets)
        assert np.array_equal(g.cpu().numpy(), exp), lv
    ct.close()
    return names


@pytest.mark.parametrize("dtype, levels, launches", [
    ("float32", [(8, 8), (9, 7), (7, 9)], 1),      # 2^15 points and more
    ("float32", [(9, 9), (9, 9), (10, 8)], 2),     # 2^18
    ("float32", [(16, 1), (16, 1), (15, 0)], 2),   # 2^17 in rows of two
    ("float32", [(12, 1), (12, 1), (13, 0)], 1),
    ("float32", [(12,), (12,), (13,)], 1),
    ("float64", [(9, 9), (9, 9), (10, 8)], 1),
    ("float64", [(14,), (13,)], 1),
])
def test_restrict_converts_in_a_launch_of_its_own_from_2_17_points(
        dtype, levels, launches):
    assert len(run(levels, dtype)[1]) == launches


@pytest.mark.parametrize("dtype, levels, direct", [
    ("float64", [(9, 9), (9, 9), (10, 8)], True),      # 2^18 in 3 grids
    ("float64", [(8, 8), (9, 7), (7, 9)], False),      # 2^15
    ("float64", [(9, 9)] * 20, False),                 # 20 grids
    ("float32", [(9, 9), (9, 9), (10, 8)], False),
    ("float32", [(10, 10), (10, 10), (11, 9)], True),  # 2^20
    ("float64", [(18,), (18,)], True),
    ("float64", [(5, 2, 4, 6), (5, 2, 4, 6), (4, 2, 5, 6)], True),
])
def test_combine_of_few_grids_walks_the_lists(dtype, levels, direct):
    names = run(levels, dtype)[0]
    assert len(names) == 1
    assert ("ct_combine_direct" in names[0]) == direct, names
