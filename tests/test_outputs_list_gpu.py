"""The restricted-output and bounds-checked transforms where one launch holds
the whole pass list, at the edges of that rule: stretches of the axis that
fit with 32, few or too few columns, columns that fill no whole group, single
columns, lists too long for one launch, the contiguous axis and windows that
wrap around the period. Bit for bit against the oracle over the whole
buffer."""
import numpy as np
import pytest

import oracle
import restricted as R
from paliwa_gb300 import transform as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("level,dim,first,count,nlevels,npass", [
    ((8, 3, 4), 0, 100, 60, 4, 2),     # 32 columns
    ((7, 1, 5), 1, 1, 1, 1, 1),        # a single pass
    ((11, 3), 0, 1900, 700, 5, 2),     # few columns, wrapping outputs
    ((3, 12), 1, 4000, 300, 3, 2),     # the contiguous axis, wrapping
    ((13, 2), 0, 5, 8000, 2, 2),       # too long for shared memory
    ((9,), 0, 300, 100, 4, 2),         # one column
    ((6, 5), 0, 10, 20, 4, 9),         # nine filters
    ((9, 2), 0, 10, 20, 8, 7),         # 56 passes
    ((6, 3, 3), 1, 6, 4, 3, 2),        # whole window, wrapping cone
])
def test_pass_lists(dtype, level, dim, first, count, nlevels, npass):
    import torch
    rng = np.random.default_rng(sum(level) + npass)
    filters = (oracle.FORWARD["biorthogonal"] if npass == 2 else
               [(q % 2, (0.25, 1.0 if q % 3 else 0.5, -0.125))
                for q in range(npass)])
    levels = list(range(level[dim], level[dim] - nlevels, -1))
    shape = [1 << l for l in level]
    front = [0] * len(level)
    ofront, oext = [0] * len(level), list(shape)
    ofront[dim], oext[dim] = first, count
    for d in range(len(level)):
        if d != dim and shape[d] > 2:  # a column group left unfilled
            oext[d] = shape[d] - 1
    x = rng.uniform(-1, 1, shape).astype(dtype)
    g = torch.from_numpy(x).cuda()
    outputs = (ofront, oext, [1] * len(level))
    T.transform_outputs(g, dim, level, level, levels, filters, outputs,
                        window_front=front)
    torch.cuda.synchronize()
    want = x.copy()
    R.transform_outputs(want, front, level, level, dim, levels, filters,
                        *outputs)
    assert np.array_equal(g.cpu().numpy(), want)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("extents,front,dim", [
    ((100, 5, 9), (20, 1, 0), 0), ((256, 3), (0, 0), 0), ((3, 200), (1, 40), 1),
    ((1, 7), (3, 0), 0), ((2000, 3), (7, 0), 0)])
def test_windows(dtype, extents, front, dim):
    import torch
    level = tuple(max(3, int(f + e - 1).bit_length())
                  for f, e in zip(front, extents))
    rng = np.random.default_rng(sum(extents))
    x = rng.uniform(-1, 1, extents).astype(dtype)
    for levels in (list(range(level[dim], 0, -1)), [level[dim], 1, 2]):
        for filters in (oracle.FORWARD["fullweighting"],
                        [(0, (0.3, 1.0, -0.7)), (1, (0.5, 1.5, 0.25))]):
            g = torch.from_numpy(x).cuda()
            T.transform_in_window(g, dim, level, level, levels, filters,
                                  front)
            torch.cuda.synchronize()
            want = oracle.transform_in_window(x.copy(), level, level, front,
                                              dim, levels, filters)
            assert np.array_equal(g.cpu().numpy(), want), levels
