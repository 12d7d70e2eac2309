"""GPU tests of the one-axis-per-launch kernels (fft_axis.cuh), the general
path: both directions against the plain runtime-radix kernels (which
gpufft_exec_noalloc still runs) and R2C against the FP64 oracle, at the sizes
where their tiles, copies and stages change form."""
import math
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu

# (grid, what it reaches)
GRIDS = [
    ((16, 16, 32), "smallest lengths; one whole tile and one left-over column per plane"),
    ((30, 18, 26), "m = 13: too short, the plain kernels"),
    ((18, 16, 40), "fewer columns than a tile in some groups"),
    ((27, 25, 98), "odd lengths; even row pitch (Nh = 50)"),
    ((27, 25, 96), "odd Ny, odd Nh: the odd rows' parity changes from plane to plane"),
    ((21, 20, 60), "even Ny, odd Nh: every other row 8 bytes off"),
    ((20, 21, 126), "Nh = 64: no left-over columns"),
    ((33, 26, 44), "factors of 11 and 13: run-time radices"),
    ((35, 24, 128), "m = 64: left-over columns of every plane"),
    ((343, 18, 36), "three stages"),
    ((16, 490, 36), "three stages along y"),
    ((16, 18, 980), "three stages along z"),
    ((1000, 16, 36), "three stages, two tile buffers do not fit in FP64"),
    ((1024, 20, 36), "longest two-stage length, one tile buffer in FP32"),
    ((36, 1024, 40), "the same along y"),
    ((18, 20, 1024), "longest row with kernels of its own"),
    ((18, 20, 1280), "m = 640: run-time radices"),
    ((243, 250, 84), "many tiles per CTA"),
]


def _make(grid, dt, seed):
    import torch

    nx, ny, nz = grid
    rd = torch.float32 if dt == "float" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.full((nx, ny, 2 * (nz // 2 + 1)), 3.0, dtype=rd, device="cuda")  # (the padding is not zero)
    f[:, :, :nz] = torch.randn((nx, ny, nz), generator=gen, dtype=rd, device="cuda")
    return f


def _noalloc(g, grid, dt, forward, f):
    import torch

    code = 0 if dt == "float" else 1
    rc = g.load_library().gpufft_exec_noalloc(*grid, code, 1 if forward else 0, f.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0, g.load_library().gpufft_last_error()


def _tol(grid, dt):
    # rounding of each of ~log2 N butterfly levels adds up in quadrature; 4 unit roundoffs a level for both sides
    return 4 * (2.0 ** -24 if dt == "float" else 2.0 ** -53) * math.sqrt(math.log2(np.prod(grid)))


def _rel(a, b):
    return ((a - b).double().norm() / b.double().norm()).item()


@pytest.mark.parametrize("dt", ["float", "double"])
@pytest.mark.parametrize("grid", [c[0] for c in GRIDS], ids=lambda c: "x".join(map(str, c)))
def test_axis_kernels_match_plain_kernels(oracle, cuda, grid, dt, monkeypatch):
    import torch
    import gpu_fft_b200 as g

    monkeypatch.setenv("GPUFFT_GENERIC_ONLY", "1")  # the general path, also where specialised kernels exist
    p = g.Plan(*grid, dt)
    nx, ny, nz = grid
    tol = _tol(grid, dt)
    f = _make(grid, dt, 7)
    a, b = f.clone(), f.clone()
    p.r2c(a)
    _noalloc(g, grid, dt, True, b)
    assert _rel(a, b) < tol
    if nx * ny * nz < 3e6:
        want = oracle.c_r2c(f.cpu().numpy().astype(np.float64), nx, ny, nz)
        got = a.cpu().numpy().view(np.complex64 if dt == "float" else np.complex128).reshape(want.shape)
        assert oracle.rel_l2(got, want) < tol
    # C2R of a spectrum that is not Hermitian in the bins kz = 0 and Nz/2 (their imaginary parts do not count)
    s = torch.randn(f.shape, dtype=f.dtype, device="cuda", generator=torch.Generator(device="cuda").manual_seed(8))
    a, b = s.clone(), s.clone()
    p.c2r(a)
    _noalloc(g, grid, dt, False, b)
    assert _rel(a[..., :nz], b[..., :nz]) < tol
    assert (a[..., nz:] == 0).all()


@pytest.mark.parametrize("grid", [(21, 20, 60), (27, 25, 96), (20, 21, 126), (16, 18, 980)],
                         ids=lambda c: "x".join(map(str, c)))
def test_axis_kernels_on_fields_8_bytes_off(cuda, grid, monkeypatch):
    """FP32 fields need only 8-byte alignment: the same results as on an
    aligned field, bit for bit, and nothing written around the field."""
    import torch
    import gpu_fft_b200 as g

    monkeypatch.setenv("GPUFFT_GENERIC_ONLY", "1")
    p = g.Plan(*grid, "float")
    f = _make(grid, "float", 9)
    n = f.numel()
    for op in (p.r2c, p.c2r):
        a = f.clone()
        op(a)
        big = torch.full((n + 8,), 5.0, device="cuda")
        off = big[2:2 + n].view(f.shape)
        off.copy_(f)
        assert off.data_ptr() % 16 == 8
        op(off)
        assert torch.equal(off, a)
        assert (big[:2] == 5).all() and (big[2 + n:] == 5).all()


@pytest.mark.parametrize("dt", ["float", "double"])
@pytest.mark.parametrize("grid", [(27, 25, 96), (33, 20, 60), (343, 18, 36)], ids=lambda c: "x".join(map(str, c)))
def test_axis_epilogue(cuda, grid, dt, monkeypatch):
    """Scale and 2/3-rule mask fused into the x axis: the separate steps' results, bit for bit."""
    import torch
    import gpu_fft_b200 as g

    monkeypatch.setenv("GPUFFT_GENERIC_ONLY", "1")
    p = g.Plan(*grid, dt)
    nx, ny, nz = grid
    f = _make(grid, dt, 11)
    a, b = f.clone(), f.clone()
    p.r2c(a)
    p.r2c(b, scale=0.25, dealias=True)
    spec = a.view(torch.complex64 if dt == "float" else torch.complex128) * 0.25
    for axis, n in ((0, nx), (1, ny)):
        k = torch.arange(n, device="cuda")
        spec[(slice(None),) * axis + (3 * torch.minimum(k, n - k) > n,)] = 0
    spec[..., 3 * torch.arange(nz // 2 + 1, device="cuda") > nz] = 0
    assert torch.equal(b.view(spec.dtype), spec)
    c, d = f.clone(), f.clone()
    p.c2r(c)
    p.c2r(d, scale=0.5)  # (a power of two: exact)
    assert torch.equal(d, c * 0.5)
