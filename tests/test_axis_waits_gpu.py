"""GPU tests of what the one-axis-per-launch kernels (fft_axis.cuh) wait for:
their own copies and the launches around them."""
import pytest

from test_axis_gpu import _make, _noalloc, _rel, _tol

pytestmark = pytest.mark.gpu


def _launch(describe, name):
    """The numbers of one axis launch in Plan.describe(): {"grid": ..., "nbuf": ...}."""
    part = describe.split(name + "{")[1].split("}")[0]
    return {k: int(v) for k, v in (w.split("=") for w in part.split()) if v.isdigit()}


# FP64 rows of even Nh and FP32 rows of Nh a multiple of 4 lie padded in shared memory and are stored one by one;
# 54675 and 15015 rows leave a last tile of a few rows, which takes the place of a whole one
@pytest.mark.parametrize("grid, dt, nbuf", [((225, 243, 126), "float", 2), ((225, 243, 126), "double", 2),
                                            ((105, 143, 910), "float", 1), ((105, 143, 882), "double", 1)], ids=str)
def test_inverse_rows_refilled_by_a_partial_last_tile(cuda, grid, dt, nbuf, monkeypatch):
    import torch
    import gpu_fft_b200 as g

    monkeypatch.setenv("GPUFFT_GENERIC_ONLY", "1")
    p = g.Plan(*grid, dt)
    w = 16 if dt == "float" else 8
    z = _launch(p.describe(), "axisZ")
    rows = grid[0] * grid[1]
    assert z["nbuf"] == nbuf
    assert rows % w and -(-rows // w) > z["nbuf"] * z["grid"]  # the last tile refills a buffer
    s = _make(grid, dt, 12)
    want = s.clone()
    _noalloc(g, grid, dt, False, want)
    nz = grid[2]
    first = None
    for _ in range(8):
        a = s.clone()
        p.c2r(a)
        if first is None:
            assert _rel(a[..., :nz], want[..., :nz]) < _tol(grid, dt)
            first = a
        assert torch.equal(a, first)
    p.check()


@pytest.mark.parametrize("dt", ["float", "double"])
@pytest.mark.parametrize("which", [1, 2], ids=["rows", "columns"])
def test_axis_wait_runs_out_and_reports(cuda, which, dt, monkeypatch):
    """The copies of the row or the column tiles are waited for 16 bytes too
    long, with a 20 ms limit: the launches end, plan_check reports it, and the
    device stays usable."""
    import time

    import torch
    import gpu_fft_b200 as g

    grid = (32, 100, 100)
    monkeypatch.setenv("GPUFFT_GENERIC_ONLY", "1")
    f = _make(grid, dt, 13)
    for forward in (True, False):
        monkeypatch.setenv("GPUFFT_AXIS_UNREACHABLE", str(which))
        monkeypatch.setenv("GPUFFT_AXIS_WAIT_MS", "20")
        p = g.Plan(*grid, dt)
        monkeypatch.delenv("GPUFFT_AXIS_UNREACHABLE")
        monkeypatch.delenv("GPUFFT_AXIS_WAIT_MS")
        a = f.clone()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        (p.r2c if forward else p.c2r)(a)
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 1.0
        with pytest.raises(g.GpuFFTError, match="ERR_CUDA"):
            p.check()
        p.close()
    q = g.Plan(*grid, dt)
    a, want = f.clone(), f.clone()
    q.r2c(a)
    _noalloc(g, grid, dt, True, want)
    assert _rel(a, want) < _tol(grid, dt)
    q.check()


@pytest.mark.parametrize("before", ["kernel", "copy", "other stream", "transform"])
@pytest.mark.parametrize("n, dt", [(32, "float"), (64, "float"), (100, "float"), (128, "float"), (100, "double")])
def test_launches_of_a_transform_keep_their_order(cuda, n, dt, before):
    """A transform's first launch may start while what is before it in the
    stream drains, and its kernels let the next one in early: the field written
    immediately before (by a kernel, a copy, another stream's kernel, or the
    inverse transform of another plan) and read immediately after, many times
    without a pause on a stream of its own, gives the bits of calls waited for."""
    import torch
    import gpu_fft_b200 as g

    grid = (n, n, n)
    p, q = g.Plan(*grid, dt), g.Plan(*grid, dt)
    src = [_make(grid, dt, s) for s in (1, 2)]
    f, out, want = torch.empty_like(src[0]), torch.empty_like(src[0]), []
    for x in src:
        f.copy_(x)
        torch.cuda.synchronize()
        if before == "transform":
            q.c2r(f)
            torch.cuda.synchronize()
        p.r2c(f)
        torch.cuda.synchronize()
        want.append(f.clone())
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    here, there = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(here):
        for k in range(200):
            x = src[k % 2]
            if before == "other stream":
                there.wait_stream(here)
                with torch.cuda.stream(there):
                    torch.mul(x, 1.0, out=f)
                here.wait_stream(there)
            elif before == "copy":
                f.copy_(x)
            else:
                torch.mul(x, 1.0, out=f)
            if before == "transform":
                q.c2r(f)
            p.r2c(f)
            torch.mul(f, 1.0, out=out)
            wrong += (out != want[k % 2]).any()
    torch.cuda.synchronize()
    assert wrong.item() == 0
