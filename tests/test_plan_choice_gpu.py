"""GPU tests of which kernels a plan runs."""
import ctypes

import pytest

from test_axis_gpu import _make, _noalloc, _rel, _tol

pytestmark = pytest.mark.gpu


def _wisdom(g, tmp_path, grid, a, b):
    """Plans of the grid (FP32) made from now on are tuned to candidates a and b."""
    import torch

    dev = torch.cuda.get_device_name(0).replace(" ", "_")
    major, minor = torch.cuda.get_device_capability(0)
    path = tmp_path / "w.txt"
    path.write_text(f"{dev}_sm{major * 10 + minor} 0 {grid[0]} {grid[1]} {grid[2]} {a} {b} 0\n")
    g.wisdom_load(str(path))


def test_a_plan_adopts_the_choice_of_no_registered_kernel(cuda, tmp_path):
    """A batch tunes one plan of each grid and the others adopt its choice, also
    where that is the one-axis kernels for both passes (candidates -1, -1)."""
    import torch
    import gpu_fft_b200 as g

    grid = (24, 512, 256)  # (512 x 128 planes: the queue form by default)
    p = g.Plan(*grid, "float")
    assert "fastA{kind=2 " in p.describe()
    _wisdom(g, tmp_path, grid, -1, -1)
    q = g.Plan(*grid, "float")
    assert "tuned=1 candA=-1 candB=-1" in q.describe() and "fastA" not in q.describe()
    adopt = g.load_library()["_ZN6gpufft10plan_adoptEPNS_4PlanEPKS0_"]  # gpufft::plan_adopt(Plan *, const Plan *)
    adopt.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    assert adopt(p.handle, q.handle) == 0
    assert p.describe() == q.describe()
    a = _make(grid, "float", 5)
    b = a.clone()
    p.r2c(a)
    q.r2c(b)
    assert torch.equal(a, b)


@pytest.mark.parametrize("grid, runs, tables", [((108, 512, 256), {"fastA", "axisX"}, 108 * 8),
                                                ((384, 512, 512), {"fastA", "fastB"}, 0),
                                                ((48, 360, 480), {"axisZ", "axisY", "fastB"}, (360 + 240 + 2 * 121) * 8),
                                                ((54, 54, 54), {"fastA", "fastB"}, 0),
                                                ((96, 96, 96), {"axisZ", "axisY", "fastB"}, (96 + 48 + 2 * 25) * 8),
                                                ((96, 192, 160), {"axisX", "axisY", "axisZ"}, (96 + 192 + 80 + 2 * 41) * 8)],
                         ids=str)
def test_a_plan_makes_and_names_only_what_it_runs(cuda, grid, runs, tables):
    """Default plans in FP32: no tables for an axis that a registered kernel
    takes, and no registered kernel beside the one-axis kernels that replace it."""
    import gpu_fft_b200 as g

    d = g.Plan(*grid, "float").describe()
    assert {k for k in ("fastA", "fastB", "axisX", "axisY", "axisZ") if k + "{" in d} == runs, d
    assert (f" axisTables={tables}" in d) if tables else ("axisTables" not in d), d


@pytest.mark.parametrize("grid, dt", [((64, 64, 64), "float"), ((128, 128, 128), "float"), ((512, 512, 512), "float"),
                                      ((256, 128, 64), "float"), ((128, 128, 128), "double")], ids=str)
def test_registered_kernels_agree_with_the_runtime_radix_kernels(cuda, grid, dt, monkeypatch):
    """The registered kernels of both passes, named (a default plan may take
    the one-axis kernels), against gpufft_exec_noalloc, which runs the
    runtime-radix kernels."""
    import torch
    import gpu_fft_b200 as g

    monkeypatch.setenv("GPUFFT_VARIANT_A", "0")
    monkeypatch.setenv("GPUFFT_VARIANT_B", "0")
    p = g.Plan(*grid, dt)
    d = p.describe()
    assert "fastA{" in d and "fastB{" in d and "axis" not in d
    a = _make(grid, dt, 3)
    for forward in (True, False):
        b = a.clone()
        (p.r2c if forward else p.c2r)(a)
        _noalloc(g, grid, dt, forward, b)
        x, y = (a, b) if forward else (a[..., :grid[2]], b[..., :grid[2]])
        assert _rel(x, y) < _tol(grid, dt)
        a = b
