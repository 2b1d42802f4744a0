"""Combine and restrict at the edges of their work split, against the oracle
bit for bit: subspaces of one point and of more than one CTA's points, grid
lists longer than a staged batch, last axes of one and two points, grids
smaller than and not a multiple of a restrict unit, unaligned grids, one to
nine dimensions."""
import numpy as np
import pytest

from paliwa_gb300 import ct as pct

pytestmark = pytest.mark.gpu


def schemes():
    rng = np.random.default_rng(5)
    rand = lambda n, nd, top: [tuple(int(v) for v in rng.integers(0, top, nd))
                               for _ in range(n)]
    return {
        "1d": [(0,), (1,), (2,), (13,), (12,), (13,)],
        "last-axis-short": [(6, 0), (6, 1), (7, 0), (5, 2), (6, 2), (8, 1)],
        "large": [(9, 9), (10, 8), (8, 10), (9, 8), (11, 3)],
        "long-lists": rand(700, 2, 4),
        "3d": rand(90, 3, 6),
        "5d": rand(60, 5, 4),
        "9d": rand(40, 9, 2),
    }


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("name", ["1d", "last-axis-short", "large",
                                  "long-lists", "3d", "5d", "9d"])
@pytest.mark.parametrize("aligned", [True, False])
def test_combine_restrict_match_oracle(name, dtype, aligned):
    import torch
    import oracle as O
    levels = schemes()[name]
    nd = len(levels[0])
    lmax = tuple(max(l[d] for l in levels) for d in range(nd))
    rng = np.random.default_rng(17)
    coeffs = [float(c) for c in rng.integers(-3, 4, len(levels))]
    xs = [rng.uniform(-1, 1, [1 << l for l in lv]).astype(dtype)
          for lv in levels]
    hold, gs = [], []
    for x in xs:  # unaligned: one element past an allocation's start
        buf = torch.empty(x.size + 1, dtype=getattr(torch, dtype),
                          device="cuda")
        hold.append(buf)
        g = buf[:x.size] if aligned else buf[1:]
        g.copy_(torch.from_numpy(x.reshape(-1)))
        gs.append(g)
    ct = pct.CombinationTechnique(gs, levels, coeffs, lmax)
    subs, _ = ct.subspaces()
    assert subs == O.kept_subspaces(levels)
    offsets, total = O.sparse_offsets(subs)
    sparse = ct.combine()
    torch.cuda.synchronize()
    want = O.combine_sparse(xs, levels, coeffs, offsets, total)
    assert np.array_equal(sparse.cpu().numpy(), want)
    ct.restrict(sparse)
    torch.cuda.synchronize()
    for g, x, lv in zip(gs, xs, levels):
        exp = O.restrict_sparse(x.copy(), lv, want, offsets)
        assert np.array_equal(g.cpu().numpy().reshape(x.shape), exp), lv
    ct.close()


def test_combine_of_special_values():
    """Zeros of both signs, subnormals, the largest float, infinities and NaN
    widen exactly: FP32 grids against numpy's float64 sums."""
    import torch
    vals = np.array([0.0, -0.0, 1e-45, -1e-45, 1.17549421e-38, 1.17549435e-38,
                     3.4028235e38, -3.4028235e38, np.inf, -np.inf, np.nan,
                     1.0, -1.5, 1e-40, 6.0, 2.0 ** -126], np.float32)
    gs = [torch.from_numpy(v.copy()).cuda() for v in (vals, vals[::-1])]
    ct = pct.CombinationTechnique(gs, [(4,), (4,)], [1.0, -2.0], (4,))
    import oracle as O
    offsets, total = O.sparse_offsets(O.kept_subspaces([(4,), (4,)]))
    with np.errstate(invalid="ignore"):
        want = O.combine_sparse([vals, vals[::-1]], [(4,), (4,)], [1.0, -2.0],
                                offsets, total)
    got = ct.combine().cpu().numpy()
    assert np.array_equal(got, want, equal_nan=True)
    ct.close()
