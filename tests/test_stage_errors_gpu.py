"""Reports of a bounded wait that gave up in a single-grid transform: on the
stream it ran on, before the next call there queues anything. The words that
the kernels set are set from the host here."""
import ctypes

import pytest

import paliwa_gb300 as pg
from paliwa_gb300 import _lib

pytestmark = pytest.mark.gpu

# Grids whose axes take several launches, of the TMA wide kernel among them.
GRIDS = [("float32", (11, 11), False), ("float64", (1, 14, 2), False),
         ("float32", (13, 8), True)]


def error_word(stream):
    fn = _lib.load()._ZN3pgb16stage_error_wordEP11CUstream_st
    fn.restype = ctypes.POINTER(ctypes.c_uint)
    fn.argtypes = [ctypes.c_void_p]
    return fn(stream.cuda_stream)


def entry_points(level, compensated):
    """name -> call on (grid, stream); one sequence of levels each."""
    lmin = (0,) * len(level)
    axis = max(range(len(level)), key=level.__getitem__)
    code = {"float64": _lib.F64, "float32": _lib.F32}

    def noalloc(x, s):
        dtype = _lib.F32C if compensated else code[str(x.dtype)[6:]]
        _lib.check(_lib.load().paliwa_gb_transform_noalloc(
            x.data_ptr(), dtype, len(level), _lib.i64(level), _lib.i64(lmin),
            _lib.i64(level), _lib.BIORTHOGONAL, 1, s.cuda_stream))

    filters = pg.lifting_wavelet_filter_offsets_and_coefficients[
        "biorthogonal"]
    return {
        "hierarchize": lambda x, s: pg.hierarchize(
            x, level, lmin, level, "biorthogonal", compensated=compensated,
            stream=s),
        "hierarchize_in": lambda x, s: pg.hierarchize_in(
            x, axis, level, lmin, level, "biorthogonal",
            compensated=compensated, stream=s),
        "transform_in": lambda x, s: pg.transform_in(
            x, axis, level, level, range(level[axis], 0, -1), filters,
            compensated=compensated, stream=s),
        "noalloc": noalloc,
    }


@pytest.mark.parametrize("dtype, level, compensated", GRIDS)
@pytest.mark.parametrize("name", ["hierarchize", "hierarchize_in",
                                  "transform_in", "noalloc"])
def test_next_call_on_the_stream_reports(name, dtype, level, compensated):
    import torch
    call = entry_points(level, compensated)[name]
    x = torch.rand([1 << l for l in level], device="cuda",
                   dtype=getattr(torch, dtype))
    want, got, other = x.clone(), x.clone(), x.clone()
    ran, elsewhere = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    call(want, ran)
    ran.synchronize()
    assert not torch.equal(want, x)
    error_word(ran)[0] = 1
    # Another stream's transform runs, and leaves the report alone.
    call(other, elsewhere)
    elsewhere.synchronize()
    assert torch.equal(other, want)
    # The stream's own is turned away before it queues anything ...
    with pytest.raises(pg.DeviceTimeout):
        call(got, ran)
    ran.synchronize()
    assert torch.equal(got, x)
    # ... once.
    call(got, ran)
    pg.synchronize(ran)
    assert torch.equal(got, want)


def test_synchronize_reports_its_stream():
    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.rand(1 << 11, 1 << 11, device="cuda")
    torch.cuda.synchronize()
    pg.hierarchize(x, (11, 11), (0, 0), (11, 11), "hat", stream=a)
    error_word(a)[0] = 1
    pg.synchronize(b)
    with pytest.raises(pg.DeviceTimeout):
        pg.synchronize(a)
    pg.synchronize(a)
    with torch.cuda.stream(a):  # the current stream
        error_word(a)[0] = 1
        with pytest.raises(pg.DeviceTimeout):
            pg.synchronize()


def test_captured_transforms_report_on_any_stream():
    import torch
    x = torch.rand(1 << 11, 1 << 11, device="cuda")
    want = x.clone()
    pg.hierarchize(want, (11, 11), (0, 0), (11, 11), "hat")
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    own = ctypes.addressof(error_word(s).contents)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        pg.hierarchize(x, (11, 11), (0, 0), (11, 11), "hat", stream=s)
        word = error_word(s)
    assert ctypes.addressof(word.contents) != own
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, want)
    word[0] = 1
    with pytest.raises(pg.DeviceTimeout):
        pg.hierarchize(x, (11, 11), (0, 0), (11, 11), "hat", stream=other)
    other.synchronize()
    assert torch.equal(x, want)
    word[0] = 1
    with pytest.raises(pg.DeviceTimeout):
        pg.synchronize(other)
    pg.synchronize(other)
