"""The work that programs have this framework do, as cases that can be timed and checked.

A case is a dict of plain values:

  kind   "pair": one forward and one normalised inverse transform, each in place on a field of its own -- what a
         solver's step or a filter asks for.  The two fields change places after each pass, so that every pass
         transforms a real field and a spectrum of the same size as the first one did.
         "products": the nonlinear terms of a pseudo-spectral step.  The six products of three velocity components are
         written into padded fields and transformed forward by one batch call, replayed as a CUDA graph.
  nx, ny, nz   the grid (kz fastest); nz is even, every axis a product of 2, 3, 5, 7, 11 and 13
  dtype        "float" or "double"
  dealias      (pair) whether the forward transform applies the 2/3 rule, as pseudo-spectral solvers have it

Sizes run from 32 to 1024 points an axis, in single precision up to 1024^3 and in double up to half of that.
"""
from __future__ import annotations

import math

import torch

import gpu_fft_b200 as gf

REAL = {"float": torch.float32, "double": torch.float64}
COMPLEX = {"float": torch.complex64, "double": torch.complex128}
PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))  # the products u_i u_j, i <= j


def _pair(name, nx, ny, nz, dtype="float", dealias=False):
    return {"name": name, "kind": "pair", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "dealias": dealias}


def listed():
    return [
        # the smallest grid of a mixed request stream: launches and host work count
        _pair("f32_32", 32, 32, 32),
        # a small grid that is no power of two, as parameter studies use
        _pair("f32_100", 100, 100, 100),
        # the known-answer grid of the test program
        _pair("f32_128", 128, 128, 128),
        # one step of a pseudo-spectral solver at moderate resolution, with the 2/3 rule
        _pair("f32_256_dealias", 256, 256, 256, dealias=True),
        # the nonlinear products of such a step, one batch call
        {"name": "products_256", "kind": "products", "nx": 256, "ny": 256, "nz": 256, "dtype": "float"},
        # the headline grid
        _pair("f32_512", 512, 512, 512),
        # the drop-in's double precision
        _pair("f64_512", 512, 512, 512, "double"),
        # a channel: three different powers of two
        _pair("f32_1024x512x256", 1024, 512, 256),
        # mixed radices 2, 3, 5
        _pair("f32_384x360x480", 384, 360, 480),
        # ragged sizes with factors of 5 and 7, whose rows are no multiple of anything convenient
        _pair("f32_420x378x500", 420, 378, 500),
        # the same in double precision, with odd Nx and Ny
        _pair("f64_225x243x350", 225, 243, 350, "double"),
        # the largest grid
        _pair("f32_1024", 1024, 1024, 1024),
    ]


def _smooth(n, primes):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo, hi, primes, even=False):
    """A size in [lo, hi] of the given prime factors, spread over the logarithm."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    sizes = [n for n in range(32, 1025) if lo <= n <= hi and _smooth(n, primes) and not (even and n % 2)]
    return min(sizes, key=lambda n: abs(math.log(n / want)))


def draw(rng):
    dtype = "double" if rng.random() < 0.3 else "float"
    # most programs choose sizes of small factors; some have 7, 11 or 13 among them
    primes = rng.choice(((2, 3, 5), (2, 3, 5), (2, 3, 5), (2, 3, 5, 7), (2, 3, 5, 7), (2, 3, 5, 7, 11, 13)))
    cells = 1024 ** 3 if dtype == "float" else 1024 ** 3 // 2
    if rng.random() < 0.15:
        n = _size(rng, 64, 320, primes, even=True)
        return {"kind": "products", "nx": n, "ny": n, "nz": n, "dtype": dtype}
    while True:
        if rng.random() < 0.5:  # a cube
            n = _size(rng, 32, 1024, primes, even=True)
            nx, ny, nz = n, n, n
        else:  # a box of moderate proportions
            base = math.exp(rng.uniform(math.log(45), math.log(720)))
            lo, hi = max(32, 0.6 * base), min(1024, 1.6 * base)
            nx, ny = _size(rng, lo, hi, primes), _size(rng, lo, hi, primes)
            nz = _size(rng, lo, hi, primes, even=True)
        if nx * ny * nz < cells:
            break
    return {"kind": "pair", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "dealias": rng.random() < 0.25}


def _inputs(case, seed):
    """The case's fields, from the seed alone: i.i.d. N(0,1) values at the grid points."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dt = REAL[case["dtype"]]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def normal():
        return torch.randn((nx, ny, nz), generator=g, device="cuda", dtype=dt)

    if case["kind"] == "products":
        return [normal() for _ in range(3)]
    real = torch.zeros(gf.field_shape(nx, ny, nz), device="cuda", dtype=dt)
    real[..., :nz] = normal()
    spec = torch.fft.rfftn(normal()).contiguous()  # the spectrum of another real field
    return real, spec


class _Pair:
    def __init__(self, case, seed):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.real, self.spec = _inputs(case, seed)
        self.plan = gf.Plan(nx, ny, nz, case["dtype"])
        self.scale = 1.0 / (nx * ny * nz)
        self.dealias = case["dealias"]
        self.cdtype, self.rdtype = COMPLEX[case["dtype"]], REAL[case["dtype"]]

    def run(self):
        a, b = self.real, self.spec
        if self.dealias:
            self.plan.r2c(a, dealias=True)
        else:
            self.plan.r2c(a)
        self.plan.c2r(b, scale=self.scale)
        self.real, self.spec = b.view(self.rdtype) if b.is_complex() else b, a
        return {"spectrum": a if a.is_complex() else a.view(self.cdtype), "field": self.real}


class _Products:
    def __init__(self, case, seed):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.u = _inputs(case, seed)
        shape = gf.field_shape(nx, ny, nz)
        self.fields = [torch.zeros(shape, device="cuda", dtype=REAL[case["dtype"]]) for _ in PAIRS]
        self.inner = [f[..., :nz] for f in self.fields]
        self.out = [f.view(COMPLEX[case["dtype"]]) for f in self.fields]
        n = len(PAIRS)
        self.batch = gf.Batch([(nx, ny, nz)] * n, ["r2c"] * n, case["dtype"], schedule="branches", branches=4)

    def run(self):
        for (i, j), f in zip(PAIRS, self.inner):
            torch.mul(self.u[i], self.u[j], out=f)
        self.batch.exec(self.fields, graph=True)
        return self.out


def prepare(case, seed):
    return _Products(case, seed) if case["kind"] == "products" else _Pair(case, seed)


def run(state):
    return state.run()


def work(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    real = 4 if case["dtype"] == "float" else 8
    spectrum = nx * ny * (nz // 2 + 1) * 2 * real
    one = 2.5 * n * math.log2(n)  # operations of one real transform
    if case["kind"] == "products":
        return {"bytes": 3 * n * real + len(PAIRS) * spectrum, "flops": len(PAIRS) * (n + one)}
    return {"bytes": 2 * (n * real + spectrum), "flops": 2 * one}


def exact(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] == "products":
        u = [v.double() for v in _inputs(case, seed)]
        # the products are rounded to the fields' precision before they are transformed
        return [torch.fft.rfftn((u[i] * u[j]).to(REAL[case["dtype"]]).double()) for i, j in PAIRS]
    real, spec = _inputs(case, seed)
    out = torch.fft.rfftn(real[..., :nz].double())
    if case["dealias"]:
        for axis, n in enumerate((nx, ny)):
            k = torch.arange(n, device="cuda")
            drop = 3 * torch.minimum(k, n - k) > n
            out[(slice(None),) * axis + (drop,)] = 0
        out[..., 3 * torch.arange(nz // 2 + 1, device="cuda") > nz] = 0
    field = torch.zeros(real.shape, device="cuda", dtype=torch.float64)
    del real
    field[..., :nz] = torch.fft.irfftn(spec.to(torch.complex128), s=(nx, ny, nz))
    return {"spectrum": out, "field": field}
