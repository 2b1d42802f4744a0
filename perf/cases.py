"""What this framework's users run, as measurable cases.

Kinds of case and what each stands for:

* ``grid``: one field kept as a full grid. A pass takes one nodal field to
  its hierarchical coefficients (``hierarchize``) and one set of coefficients
  back to nodal values (``dehierarchize``), in place, as a solver that
  switches representation does every step. The two buffers change places
  after each pass, so the values stay bounded over any number of passes.
* ``axis``: ``transform_in`` with a filter table of the caller's own (the
  four-pass CDF 9/7 lifting of JPEG 2000) along one axis, there and back.
* ``outputs``: ``transform_outputs`` on a slab with its ghost layers in a
  window buffer: the finest levels of the slab's points, after the ghost
  layers have been filled (a copy, as a halo exchange would deliver them).
* ``batch``: every component grid of a combination scheme forward, and every
  grid of a second set of coefficients back (``ct.Batch``), the step of a
  time-dependent combination technique.
* ``ct``: the combination itself: ``combine`` of all component grids into the
  sparse grid and ``restrict`` of the combined coefficients into every grid.
* ``driver``: the whole serial pipeline: new nodal values, forward of every
  component grid, combine, scatter onto the full grid, inverse of the full
  grid.

Sizes and wavelets are those of the benchmark's workloads and of the tests:
2D 64 x 64 hat, 512^3 CDF (2,2), 32^4 x 16^2 hat, the 4D scheme
|l|_1 = 20 - q and the 6D scheme |l|_1 = 16 - q, long pencils of 2^13 to 2^17
points, 3D schemes scattered onto a full grid.
"""
import itertools
import math

import numpy as np
import torch

import paliwa_gb300 as pg
from paliwa_gb300 import ct as pct

DEVICE = "cuda"

# CDF 9/7 (Daubechies and Sweldens, "Factoring wavelet transforms into lifting
# steps", 1998, without the final scaling): (offset, (c0, c1, c2)).
CDF97 = [(1, (-1.586134342, 1.0, -1.586134342)),
         (0, (-0.05298011854, 1.0, -0.05298011854)),
         (1, (0.8829110762, 1.0, 0.8829110762)),
         (0, (0.4435068522, 1.0, 0.4435068522))]
CDF97_INVERSE = [(o, (-a, b, -c)) for o, (a, b, c) in reversed(CDF97)]

# The wavelets' lifting tables, for the work counts and the 64-bit values.
FORWARD = {"hat": [(1, (-0.5, 1.0, -0.5))],
           "biorthogonal": [(1, (-0.5, 1.0, -0.5)), (0, (0.25, 1.0, 0.25))],
           "fullweighting": [(0, (0.25, 0.5, 0.25)), (1, (-0.5, 1.0, -0.5))]}
INVERSE = {"hat": [(1, (0.5, 1.0, 0.5))],
           "biorthogonal": [(0, (-0.25, 1.0, -0.25)), (1, (0.5, 1.0, 0.5))],
           "fullweighting": [(1, (0.5, 1.0, 0.5)), (0, (-0.5, 2.0, -0.5))]}


def listed():
    return [
        # The smallest field of the tests: two launches' worth of latency.
        dict(name="grid-2d-64-hat-f64", kind="grid", level="6,6", lmin=0,
             wavelet="hat", dtype="f64"),
        # The 3D workload in the compensated mode and in plain double.
        dict(name="grid-3d-512-f32c", kind="grid", level="9,9,9", lmin=0,
             wavelet="biorthogonal", dtype="f32c"),
        dict(name="grid-3d-512-f64", kind="grid", level="9,9,9", lmin=0,
             wavelet="biorthogonal", dtype="f64"),
        # The 6D workload in plain single precision.
        dict(name="grid-6d-hat-f32", kind="grid", level="5,5,5,5,4,4", lmin=0,
             wavelet="hat", dtype="f32"),
        # A strongly anisotropic field: pencils longer than one tile.
        dict(name="grid-2d-long-f32c", kind="grid", level="15,10", lmin=1,
             wavelet="fullweighting", dtype="f32c"),
        # A caller's own filters along the middle axis of a field.
        dict(name="axis-cdf97-f32", kind="axis", level="8,9,8", dim=1,
             dtype="f32"),
        # A slab of 100 planes with 30 ghost planes on either side.
        dict(name="outputs-slab-f64", kind="outputs", level="9,8,7", dim=0,
             first=77, count=100, nlevels=4, wavelet="biorthogonal",
             dtype="f64"),
        # Combination schemes: the 4D and 6D workloads in the compensated
        # mode, a smaller one in double, and one of a few tiny grids.
        dict(name="batch-4d-20-f32c", kind="batch", ndim=4, level_sum=20,
             lmin=1, wavelet="biorthogonal", dtype="f32c"),
        dict(name="batch-6d-16-f32c", kind="batch", ndim=6, level_sum=16,
             lmin=1, wavelet="biorthogonal", dtype="f32c"),
        dict(name="batch-4d-17-f64", kind="batch", ndim=4, level_sum=17,
             lmin=1, wavelet="hat", dtype="f64"),
        # The combination of the 4D scheme's grids.
        dict(name="ct-4d-19-f32", kind="ct", ndim=4, level_sum=19, lmin=1,
             dtype="f32"),
        # The whole pipeline on a 3D scheme with a 2^24-point full grid.
        dict(name="driver-3d-10-f64", kind="driver", ndim=3, level_sum=10,
             lmin=1, wavelet="biorthogonal", dtype="f64"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, total, parts, lowest, highest):
    """`parts` levels of sum `total`, each in [lowest, highest]."""
    while True:
        out = [lowest] * parts
        left = total - lowest * parts
        while left > 0:
            d = rng.randrange(parts)
            step = min(left, rng.randint(1, 3), highest - out[d])
            out[d] += step
            left -= step
            if all(x >= highest for x in out):
                break
        if left == 0:
            return out


def draw(rng):
    kind = rng.choice(["grid", "grid", "axis", "outputs", "batch", "batch",
                       "ct", "driver"])
    wavelet = rng.choice(["hat", "biorthogonal", "fullweighting"])
    dtype = rng.choice(["f32", "f32c", "f64"])
    if kind == "grid":
        nd = rng.randint(1, 6)
        most = min(26 if dtype == "f64" else 27, 17 * nd)
        total = rng.randint(min(10, most), most)
        level = _split(rng, total, nd, 1, 17)
        return dict(kind=kind, level=",".join(map(str, level)),
                    lmin=rng.randint(0, 1), wavelet=wavelet, dtype=dtype)
    if kind == "axis":
        nd = rng.randint(2, 4)
        level = _split(rng, rng.randint(14, 25), nd, 1, 12)
        return dict(kind=kind, level=",".join(map(str, level)),
                    dim=rng.randrange(nd), dtype=rng.choice(["f32", "f64"]))
    if kind == "outputs":
        dim = rng.randrange(3)
        level = [rng.randint(5, 8) for _ in range(3)]
        level[dim] = rng.randint(8, 10)
        nlevels = rng.randint(1, 4)
        n = 1 << level[dim]
        count = _log_uniform(rng, 1, n - 4 * (2 << nlevels))
        return dict(kind=kind, level=",".join(map(str, level)), dim=dim,
                    first=rng.randrange(n), count=count, nlevels=nlevels,
                    wavelet=wavelet, dtype=rng.choice(["f32", "f64"]))
    if kind == "driver":
        nd = rng.randint(2, 3)
        total = rng.randint(6, 12) if nd == 2 else rng.randint(6, 10)
        return dict(kind=kind, ndim=nd, level_sum=total, lmin=1,
                    wavelet=wavelet, dtype=dtype)
    # Schemes of up to 2^28 points and 4,000 grids.
    tops = {2: 18, 3: 18, 4: 18, 5: 17, 6: 14}
    nd = rng.randint(2, 6)
    total = rng.randint(nd + 3, tops[nd])
    if kind == "ct":
        return dict(kind=kind, ndim=nd, level_sum=total, lmin=1,
                    dtype=rng.choice(["f32", "f64"]))
    return dict(kind=kind, ndim=nd, level_sum=total, lmin=1, wavelet=wavelet,
                dtype=dtype)


# ---------------------------------------------------------------------------
# inputs


def _torch_dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _levels(case):
    return [int(x) for x in case["level"].split(",")]


def _scheme(case):
    nd, top = case["ndim"], case["level_sum"]
    levels, coeffs = pct.combination_scheme(nd, top, None, case["lmin"])
    lmax = (top - (nd - 1) * case["lmin"],) * nd
    return levels, coeffs, (case["lmin"],) * nd, lmax


class _Fields:
    """Seeded fields on grids of any level: a smooth product of parabolas
    with exponential decay plus noise (nodal values), and noise that falls
    off with the hierarchical level along each axis (coefficients)."""

    def __init__(self, seed, ndim):
        self.rng = np.random.default_rng(seed)
        self.rates = self.rng.uniform(0.0, 2.0, ndim)
        self.gen = torch.Generator(device=DEVICE)
        self.gen.manual_seed(int(seed))
        self.cache = {}

    def _axis(self, dim, level, smooth):
        key = (dim, level, smooth)
        if key not in self.cache:
            n = 1 << level
            k = np.arange(n)
            if smooth:
                x = k / n
                v = 4 * x * (1 - x) * np.exp(-self.rates[dim] * x) + 0.1
            else:
                low = np.where(k > 0, k & -k, n)  # 2^(level - own level)
                v = np.sqrt(low / n)
            self.cache[key] = torch.from_numpy(v).to(DEVICE)
        return self.cache[key]

    def _product(self, level, smooth):
        out = None
        for d, l in enumerate(level):
            v = self._axis(d, l, smooth)
            out = v if out is None else (out[:, None] * v).reshape(-1)
        return out

    def noise(self, n):
        return torch.rand(n, generator=self.gen, dtype=torch.float32,
                          device=DEVICE).sub_(0.5)

    def nodal(self, view, level):
        p = self._product(level, True)
        view.copy_(p.add_(self.noise(p.numel()), alpha=1e-3))

    def coefficients(self, view, level):
        p = self._product(level, False)
        view.copy_(p.mul_(self.noise(p.numel())))


def _packed(levels, case):
    buf, views = pct.packed_grids(levels, _torch_dtype(case), DEVICE)
    buf.zero_()
    return buf, views


def _window(case):
    """Outputs [first, first + count) along dim, with a ghost layer of the
    stencil's reach (passes * distance per level, up to the next level) on
    either side; the window may wrap around the period."""
    level, dim = _levels(case), case["dim"]
    ghost = len(FORWARD[case["wavelet"]]) * ((1 << case["nlevels"]) - 1)
    n = 1 << level[dim]
    extent = min(n, case["count"] + 2 * ghost)
    lo = ghost if extent == case["count"] + 2 * ghost else 0
    front = [0] * len(level)
    front[dim] = (case["first"] - lo) % n if extent < n else 0
    shape = [1 << l for l in level]
    shape[dim] = extent
    return front, shape


def _inputs(case, seed):
    """The values a pass starts from, as tensors of the case's type."""
    kind = case["kind"]
    if kind in ("grid", "axis"):
        level = _levels(case)
        f = _Fields(seed, len(level))
        a, b = (torch.empty([1 << l for l in level],
                            dtype=_torch_dtype(case), device=DEVICE)
                for _ in range(2))
        f.nodal(a.view(-1), level)
        f.coefficients(b.view(-1), level)
        return a, b
    if kind == "outputs":
        level = _levels(case)
        front, shape = _window(case)
        whole = torch.empty([1 << l for l in level],
                            dtype=_torch_dtype(case), device=DEVICE)
        _Fields(seed, len(level)).nodal(whole.view(-1), level)
        at = [(torch.arange(e, device=DEVICE) + s) % (1 << l)
              for s, e, l in zip(front, shape, level)]
        return whole[torch.meshgrid(*at, indexing="ij")].contiguous()
    levels = _scheme(case)[0]
    f = _Fields(seed, case["ndim"])
    if kind == "batch":
        sets = [_packed(levels, case) for _ in range(2)]
        for fill, (_, views) in zip((f.nodal, f.coefficients), sets):
            for v, l in zip(views, levels):
                fill(v, l)
        return sets
    buf, views = _packed(levels, case)
    fill = f.coefficients if kind == "ct" else f.nodal
    for v, l in zip(views, levels):
        fill(v, l)
    return buf, views


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "stream": torch.cuda.Stream()}
    if kind in ("grid", "axis"):
        a, b = _inputs(case, seed)
        level = _levels(case)
        state.update(nodal=a, hier=b, level=level,
                     lmin=[min(case.get("lmin", 0), l) for l in level])
    elif kind == "outputs":
        x = _inputs(case, seed)
        front, _ = _window(case)
        level, dim = _levels(case), case["dim"]
        first, extents = [0] * len(level), [1 << l for l in level]
        first[dim], extents[dim] = case["first"], case["count"]
        state.update(x=x, buf=torch.empty_like(x), front=front, level=level,
                     levels=list(range(level[dim],
                                       level[dim] - case["nlevels"], -1)),
                     outputs=(first, extents, [1] * len(level)))
    elif kind == "batch":
        levels, _, lmin, lmax = _scheme(case)
        for name, (buf, views) in zip(("nodal", "hier"), _inputs(case, seed)):
            state[name] = (buf, pct.Batch(views, levels, lmin, lmax,
                                          case["wavelet"],
                                          compensated=case["dtype"] == "f32c"))
    else:
        levels, coeffs, lmin, lmax = _scheme(case)
        buf, views = _inputs(case, seed)
        state.update(buf=buf, lmax=lmax)
        state["ct"] = pct.CombinationTechnique(views, levels, coeffs, lmax)
        state["sparse"] = torch.empty(state["ct"].npoints,
                                      dtype=torch.float64, device=DEVICE)
        if kind == "driver":
            state.update(x=buf.clone(), lmin=lmin,
                         full=torch.empty([1 << l for l in lmax],
                                          dtype=torch.float64, device=DEVICE),
                         batch=pct.Batch(views, levels, lmin, lmax,
                                         case["wavelet"],
                                         compensated=case["dtype"] == "f32c"))
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    with torch.cuda.stream(state["stream"]):
        if kind == "grid":
            a, b, level = state["nodal"], state["hier"], state["level"]
            comp = case["dtype"] == "f32c"
            pg.hierarchize(a, level, state["lmin"], level, case["wavelet"],
                           compensated=comp)
            pg.dehierarchize(b, level, state["lmin"], level, case["wavelet"],
                             compensated=comp)
            state["nodal"], state["hier"] = b, a
            return {"hier": a, "nodal": b}
        if kind == "axis":
            a, b, level = state["nodal"], state["hier"], state["level"]
            dim = case["dim"]
            down = list(range(level[dim], 0, -1))
            pg.transform_in(a, dim, level, level, down, CDF97)
            pg.transform_in(b, dim, level, level, down[::-1], CDF97_INVERSE)
            state["nodal"], state["hier"] = b, a
            return {"hier": a, "nodal": b}
        if kind == "outputs":
            state["buf"].copy_(state["x"])
            pg.transform_outputs(state["buf"], case["dim"], state["level"],
                                 state["level"], state["levels"],
                                 FORWARD[case["wavelet"]], state["outputs"],
                                 window_front=state["front"])
            return {"window": state["buf"], "outputs": _slab(case,
                                                             state["buf"])}
        if kind == "batch":
            a, b = state["nodal"], state["hier"]
            a[1].hierarchize()
            b[1].dehierarchize()
            state["nodal"], state["hier"] = b, a
            return {"hier": a[0], "nodal": b[0]}
        if kind == "ct":
            state["ct"].combine(state["sparse"])
            state["ct"].restrict(state["sparse"])
            return {"sparse": state["sparse"], "grids": state["buf"]}
        state["buf"].copy_(state["x"])
        state["batch"].hierarchize()
        state["ct"].combine(state["sparse"])
        state["ct"].scatter(state["sparse"], state["full"])
        pg.dehierarchize(state["full"], state["lmax"], state["lmin"],
                         state["lmax"], case["wavelet"])
        return {"grids": state["buf"], "sparse": state["sparse"],
                "full": state["full"]}


def _slab(case, window):
    """The output points of a window buffer along the transformed axis."""
    front, shape = _window(case)
    dim = case["dim"]
    n = 1 << _levels(case)[dim]
    at = (case["first"] - front[dim]) % n
    if at + case["count"] <= shape[dim]:
        return window.narrow(dim, at, case["count"])
    k = (torch.arange(case["count"], device=window.device) + at) % n
    return window.index_select(dim, k)


# ---------------------------------------------------------------------------
# the work a pass cannot do without


def _updates(level, lmin):
    """Lifting updates of one pass per point-axis, summed over the axes: the
    levels of an axis update n / 2, n / 4, ... points of each pencil."""
    n = 1 << sum(level)
    return sum(n * (1 - 2.0 ** -(l - m)) for l, m in zip(level, lmin))


def work(case):
    kind, size = case["kind"], 8 if case["dtype"] == "f64" else 4
    passes = len(FORWARD[case["wavelet"]]) if "wavelet" in case else 4
    if kind in ("grid", "axis"):
        level = _levels(case)
        lmin = [min(case.get("lmin", 0), l) for l in level]
        if kind == "axis":
            lmin = [0 if d == case["dim"] else l
                    for d, l in enumerate(level)]
        n = 1 << sum(level)
        return {"bytes": 2 * 2 * n * size,
                "flops": 2 * 4 * passes * _updates(level, lmin)}
    if kind == "outputs":
        _, shape = _window(case)
        n = math.prod(shape)
        out = n // shape[case["dim"]] * case["count"]
        return {"bytes": 2 * n * size, "flops": 4 * passes * out}
    levels, _, lmin, lmax = _scheme(case)
    n = sum(1 << sum(l) for l in levels)
    lift = sum(4 * passes * _updates(l, lmin) for l in levels)
    if kind == "batch":
        return {"bytes": 2 * 2 * n * size, "flops": 2 * lift}
    sparse = int(_Sparse(levels).npoints)
    if kind == "ct":
        return {"bytes": 2 * n * size + 8 * sparse, "flops": 2 * n}
    full = 1 << sum(lmax)
    return {"bytes": 2 * n * size + 8 * sparse + 8 * full,
            "flops": lift + 2 * n + 4 * passes * _updates(lmax, lmin)}


# ---------------------------------------------------------------------------
# the same values in 64 bits, from plain torch


def _lift(x, dim, shifts, filters):
    """Lifting passes along `dim` of a periodic float64 tensor, in place."""
    v = x.movedim(dim, -1)
    for sh in shifts:
        s = 1 << sh
        for offset, (c0, c1, c2) in filters:
            even, odd = v[..., 0::2 * s], v[..., s::2 * s]
            if offset == 1:
                me, lo, up = odd, even, torch.roll(even, -1, -1)
            else:
                me, lo, up = even, torch.roll(odd, 1, -1), odd
            me.copy_(c0 * lo + c1 * me + c2 * up)
    return x


def _transform(x, level, lmin, wavelet, forward, cache):
    """hierarchize / dehierarchize of a flat float64 grid; axes of up to 64
    points by their transform matrix."""
    filters = (FORWARD if forward else INVERSE)[wavelet]
    x = x.reshape([1 << l for l in level])
    for d, (l, m) in enumerate(zip(level, lmin)):
        if l == m:
            continue
        shifts = list(range(l - m)) if forward else list(range(l - m))[::-1]
        if l > 6:
            x = _lift(x.contiguous(), d, shifts, filters)
            continue
        key = (l, m, forward)
        if key not in cache:
            cache[key] = _lift(torch.eye(1 << l, dtype=torch.float64,
                                         device=x.device), 0, shifts, filters)
        outer = math.prod(x.shape[:d])
        x = torch.matmul(cache[key], x.reshape(outer, 1 << l, -1)).reshape(
            x.shape)
    return x.reshape(-1)


class _Sparse:
    """Sparse-grid layout of a scheme: the hierarchical subspaces held by
    more than one grid in lexicographic order, each stored densely."""

    def __init__(self, levels):
        nd = len(levels[0])
        top = [max(l[d] for l in levels) for d in range(nd)]
        count = np.zeros([t + 1 for t in top], dtype=np.int32)
        for l in levels:
            count[tuple(slice(0, x + 1) for x in l)] += 1
        size = np.ones_like(count, dtype=np.int64)
        for d in range(nd):
            ext = np.array([1] + [1 << (s - 1) for s in range(1, top[d] + 1)])
            size *= ext.reshape([-1 if e == d else 1 for e in range(nd)])
        kept = np.where(count > 1, size, 0).reshape(-1)
        first = np.cumsum(kept) - kept
        self.npoints = int(kept.sum())
        self.first = np.where(kept > 0, first, -1)
        self.shape = count.shape

    def index(self, level, first):
        """Sparse point of every point of a grid (-1: in no kept subspace);
        `first` is self.first on the device."""
        sub = None
        place = size = torch.zeros((), dtype=torch.int64, device=first.device)
        size = size + 1
        for d in range(len(level) - 1, -1, -1):
            l = level[d]
            k = np.arange(1 << l)
            low = np.where(k > 0, k & -k, 1 << l)
            s = np.array([l - int(v).bit_length() + 1 for v in low])
            j = np.where(s > 0, k // (2 * low), 0)
            ext = np.where(s > 0, 1 << np.maximum(s - 1, 0), 1)
            s, j, ext = (torch.from_numpy(v).to(first.device)
                         for v in (s, j, ext))
            stride = math.prod(self.shape[d + 1:])
            if sub is None:
                sub, place, size = s * stride, j, ext
            else:
                place = (j[:, None] * size + place).reshape(-1)
                sub = (s[:, None] * stride + sub).reshape(-1)
                size = (ext[:, None] * size).reshape(-1)
        base = first[sub]
        return torch.where(base >= 0, base + place, base)


def _combined(views, levels, coeffs):
    """(sparse values, [(kept points, their sparse points) of each grid])."""
    layout = _Sparse(levels)
    first = torch.from_numpy(layout.first).to(DEVICE)
    sparse = torch.zeros(layout.npoints, dtype=torch.float64, device=DEVICE)
    for v, l, c in zip(views, levels, coeffs):
        at = layout.index(l, first)
        kept = at >= 0
        sparse[at[kept]] += c * v.double()[kept]
    return sparse, layout, first


def _scattered(sparse, levels, lmax):
    layout = _Sparse(levels)
    full = torch.zeros([1 << l for l in lmax], dtype=torch.float64,
                       device=DEVICE)
    first = layout.first.reshape(layout.shape)
    for s in itertools.product(*[range(n) for n in layout.shape]):
        if first[s] < 0:
            continue
        shape = [1 << (x - 1) if x else 1 for x in s]
        at = tuple(slice(1 << (l - x), None, 2 << (l - x)) if x
                   else slice(0, 1) for x, l in zip(s, lmax))
        begin = int(first[s])
        full[at] = sparse[begin:begin + math.prod(shape)].reshape(shape)
    return full


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    cache = {}
    if kind in ("grid", "axis"):
        level = _levels(case)
        a, b = (v.double() for v in x)
        if kind == "axis":
            down = list(range(level[case["dim"]]))
            return {"hier": _lift(a, case["dim"], down, CDF97),
                    "nodal": _lift(b, case["dim"], down[::-1],
                                   CDF97_INVERSE)}
        lmin = [min(case["lmin"], l) for l in level]
        return {name: _transform(v.reshape(-1), level, lmin, case["wavelet"],
                                 forward, cache).reshape(v.shape)
                for name, v, forward in (("hier", a, True),
                                         ("nodal", b, False))}
    if kind == "outputs":
        # The window taken as a period of its own: its outermost points get
        # other neighbours, which the ghost layer keeps from the outputs.
        dim = case["dim"]
        n = x.shape[dim]
        unit = 1 << case["nlevels"]
        front, _ = _window(case)
        pad = front[dim] % unit  # keeps the window's place on the lattice
        shape = list(x.shape)
        shape[dim] = -(-(pad + n) // unit) * unit
        whole = n == 1 << _levels(case)[dim]
        y = x.double() if whole else torch.zeros(shape, dtype=torch.float64,
                                                 device=DEVICE)
        if not whole:
            y.narrow(dim, pad, n).copy_(x)
        _lift(y, dim, range(case["nlevels"]), FORWARD[case["wavelet"]])
        y = y if whole else y.narrow(dim, pad, n)
        return {"window": None, "outputs": _slab(case, y)}
    levels, coeffs, lmin, lmax = _scheme(case)
    if kind == "batch":
        out = {}
        for name, (buf, views), forward in zip(("hier", "nodal"), x,
                                               (True, False)):
            y = buf.double()
            base = buf.data_ptr()
            for v, l in zip(views, levels):
                at = (v.data_ptr() - base) // buf.element_size()
                part = y.narrow(0, at, v.numel())
                part.copy_(_transform(part.clone(), l, lmin, case["wavelet"],
                                      forward, cache))
            out[name] = y
        return out
    buf, views = x
    y = buf.double()
    base = buf.data_ptr()
    parts = [y.narrow(0, (v.data_ptr() - base) // buf.element_size(),
                      v.numel()) for v in views]
    if kind == "driver":
        for part, l in zip(parts, levels):
            part.copy_(_transform(part.clone(), l, lmin, case["wavelet"], True,
                                  cache))
        sparse = _combined(parts, levels, coeffs)[0]
        full = _scattered(sparse, levels, lmax)
        return {"grids": y, "sparse": sparse,
                "full": _transform(full.reshape(-1), lmax, lmin,
                                   case["wavelet"], False,
                                   cache).reshape(full.shape)}
    sparse, layout, first = _combined(parts, levels, coeffs)
    for part, l in zip(parts, levels):
        at = layout.index(l, first)
        part.copy_(torch.where(at >= 0, sparse[at.clamp(min=0)], part))
    return {"sparse": sparse, "grids": y}
