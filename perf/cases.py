"""Performance cases of the pencil FFT library, through its public plan API.

Each case is one pass a user's program makes over a field it already holds on
the GPU: a transform forward and back, the gradient of a spectral loss, a
ragged batch, a layout change.  ``listed`` names the cases that are tracked,
``draw`` makes further ones over the same ranges, ``prepare`` / ``run`` build
and execute one, ``work`` counts what the pass cannot do without and ``exact``
gives the outputs in 64-bit arithmetic from torch alone.
"""

from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pencil-rs_b200"))

import pencil_b200 as pb  # noqa: E402
from pencil_b200 import autograd as pba  # noqa: E402
from pencil_b200 import workloads  # noqa: E402

REAL = {"f32": torch.float32, "f64": torch.float64}
COMPLEX = {"f32": torch.complex64, "f64": torch.complex128}
R2R_KINDS = ("DctI", "DctII", "DctIII", "DctIV", "DstI", "DstII", "DstIII", "DstIV", "Dht")


def _case(name, family, dtype, shape, grid, extra="", kinds="", permute=True, count=0, seed=0):
    c = {"family": family, "dtype": dtype, "shape": shape, "grid": grid, "extra": extra, "kinds": kinds,
         "permute": permute, "count": count, "shapes_seed": seed}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a vector field on a thin grid, where launches and host work are all there is
        _case("c2c_f32_24x20x18", "c2c", "f32", "24x20x18", "2x3", extra="2"),
        # the small double-precision solver grid of the basic configuration
        _case("c2c_f64_64cube", "c2c", "f64", "64x64x64", "2x2"),
        # the headline field of a turbulence-sized solver: real input, half spectrum, back
        _case("r2c_f32_512cube", "r2c", "f32", "512x512x512", "4x8"),
        # wall-bounded vector field: cosine, sine and Hartley axes on real data
        _case("r2r_f32_3x256x384x320", "r2r", "f32", "256x384x320", "2x3", extra="3", kinds="DctII,DstI,Dht"),
        # the same axes through the mixed plan, complex data in double precision
        _case("mixed_c128_3x256x384x320", "mixed", "f64", "256x384x320", "2x3", extra="3", kinds="DctII,DstI,Dht"),
        # training step through the transform: gradient of a spectral loss, and a Poisson solve
        _case("grad_r2c_f32_384cube", "grad", "f32", "384x384x384", "4x8"),
        # many independent grids of uneven shapes, forward and back in one launch
        _case("batch_c2c_f32_64grids", "batch", "f32", "32..256", "1x1", count=64, seed=4),
        # prime extents (a cell-centred 256 grid plus one)
        _case("r2c_f32_512x257x257", "r2c", "f32", "512x257x257", "4x8"),
        # odd extents 255 = 3*5*17 in double precision
        _case("r2c_f64_255cube", "r2c", "f64", "255x255x255", "2x2"),
        # memory order kept by the caller (permute_dims = false): strided lines
        _case("c2c_f32_384cube_unpermuted", "c2c", "f32", "384x384x384", "4x8", permute=False),
        # a large image or hologram: two axes, long lines
        _case("c2c_f32_4096x4096", "c2c", "f32", "4096x4096", "8"),
        # the layout change alone, on the spectrum of the headline field
        _case("transpose_c64_512x512x257", "transpose", "f32", "512x512x257", "4x8"),
    ]


def _smooth(n, primes=(2, 3, 5, 7)):
    """The number of the form prod(p^e) nearest to n."""
    for d in range(n):
        for m in (n + d, n - d):
            r = m
            for p in primes:
                while r > 1 and r % p == 0:
                    r //= p
            if m >= 1 and r == 1:
                return m
    return n


def _draw_length(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    how = rng.random()
    if how < 0.2:
        return 1 << max(3, round(math.log2(n)))
    if how < 0.6:
        return _smooth(n)
    if how < 0.8:  # even grids with one factor of 11 or 13
        return max(11, _smooth(n, (2, 3, 5, 7, 11, 13)))
    return n if n <= 1024 else _smooth(n)


def draw(rng):
    family = rng.choice(["c2c", "c2c", "r2c", "r2c", "r2r", "r2r", "mixed", "grad", "batch", "transpose"])
    dtype = rng.choice(["f32", "f32", "f64"])
    if family == "batch":
        return _case(None, "batch", "f32", "32..256", rng.choice(["1x1", "2x2"]), count=rng.randint(4, 48),
                     seed=rng.randint(5, 10 ** 6))
    long_max = 1024 if family in ("r2r", "mixed") else 4096
    if rng.random() < 0.25 and family != "grad":
        dims, lo, hi = 2, 64, long_max
    else:
        dims, lo, hi = 3, 16, 512
    if family == "grad":
        dtype = "f32"
    limit = 2 ** 26 if dtype == "f32" else 2 ** 24
    extra = rng.choice([1, 1, 1, 2, 3, 8]) if family != "grad" else 1
    while True:
        shape = [_draw_length(rng, lo, hi) for _ in range(dims)]
        if 2 ** 12 <= math.prod(shape) * extra <= limit:
            break
    grid = rng.choice(["1x1", "2x2", "2x3", "4x8"] if dims == 3 else ["1", "4", "8"])
    kinds = ""
    if family in ("r2r", "mixed"):
        pool = R2R_KINDS + (("Fft", "Fft") if family == "mixed" else ())
        kinds = ",".join(rng.choice(pool) for _ in shape)
    permute = family in ("grad", "transpose") or rng.random() < 0.75
    return _case(None, family, dtype, "x".join(map(str, shape)), grid, extra=str(extra) if extra > 1 else "",
                 kinds=kinds, permute=permute)


# ---------------------------------------------------------------- geometry
def _ints(text):
    return tuple(int(t) for t in text.split("x")) if text else ()


def _batch_shapes(case):
    n = case["count"]
    return workloads.ragged_batch(seed=case["shapes_seed"], count=n, with_extra=n // 4)


def _layout(glob, grid, dec, perm):
    """Global [extra, spatial...] tensor -> the ranks' local arrays one after
    another: grid axis t splits spatial axis dec[t] at floor(n*c/P), local
    arrays are [extra, spatial axes in the order perm]."""
    n = glob.dim() - 1
    parts = []
    for r in range(math.prod(grid)):
        sl, q = [slice(None)] * (n + 1), r
        for t in reversed(range(len(grid))):
            c, q = q % grid[t], q // grid[t]
            ext = glob.shape[1 + dec[t]]
            sl[1 + dec[t]] = slice(ext * c // grid[t], ext * (c + 1) // grid[t])
        parts.append(glob[tuple(sl)].permute([0] + [1 + a for a in perm]).reshape(-1))
    return torch.cat(parts)


def _input_layout(glob, case):
    grid = _ints(case["grid"])
    return _layout(glob, grid, range(len(grid)), range(glob.dim() - 1))


def _output_layout(glob, case):
    grid, n = _ints(case["grid"]), glob.dim() - 1
    perm = list(reversed(range(n))) if case["permute"] else list(range(n))
    return _layout(glob, grid, [t + 1 for t in range(len(grid))], perm)


def _extra_count(case):
    return math.prod(_ints(case["extra"])) if case["extra"] else 1


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _field(shape, dtype, gen, uniform=False):
    if uniform:
        return torch.rand(shape, dtype=dtype, device="cuda", generator=gen).mul_(2).sub_(1)
    return torch.randn(shape, dtype=dtype, device="cuda", generator=gen)


def _inputs(case, seed):
    """The global input field(s), made from the seed alone."""
    gen = _generator(seed)
    if case["family"] == "batch":
        return [_field((math.prod(e),) + s, torch.complex64, gen) for s, e in _batch_shapes(case)]
    shape = (_extra_count(case),) + _ints(case["shape"])
    if case["family"] in ("r2c", "r2r", "grad"):
        return _field(shape, REAL[case["dtype"]], gen, uniform=case["family"] == "r2c")
    return _field(shape, COMPLEX[case["dtype"]], gen)


def _plan(case):
    topo = pb.MpiTopology(_ints(case["grid"]))
    shape, extra = _ints(case["shape"]), _ints(case["extra"])
    layout = pb.DistributedLayout(case["permute"])
    family, dtype = case["family"], case["dtype"]
    if family == "c2c":
        return pb.C2cPlan.from_shape(topo, shape, extra, layout=layout, dtype=COMPLEX[dtype])
    if family in ("r2c", "grad"):
        return pb.R2cPlan.from_shape(topo, shape, extra, layout=layout, dtype=REAL[dtype])
    kinds = case["kinds"].split(",")
    if family == "r2r":
        return pb.R2rPlan.from_shape(topo, shape, extra, kinds, layout=layout, dtype=REAL[dtype])
    return pb.MixedC2cPlan.from_shape(topo, shape, extra, kinds, layout=layout, dtype=COMPLEX[dtype])


def prepare(case, seed):
    x = _inputs(case, seed)
    if case["family"] == "batch":
        topo = pb.MpiTopology(_ints(case["grid"]))
        plans = [pb.C2cPlan.from_shape(topo, s, e, dtype=torch.complex64) for s, e in _batch_shapes(case)]
        batch = pb.PlanBatch(plans)
        # one allocation for all spectra and one for all results, a slice per grid
        sizes = [p.info.output_elems for p in plans]
        spectra = torch.zeros(sum(sizes), dtype=torch.complex64, device="cuda")
        back = torch.zeros(sum(sizes), dtype=torch.complex64, device="cuda")
        buffers = [[_input_layout(g, case) for g in x], list(spectra.split(sizes)), list(back.split(sizes))]
        return {"family": "batch", "batch": batch, "plans": plans, "buffers": buffers, "spectra": spectra,
                "back": back, "workspace": batch.allocate_workspace()}
    if case["family"] == "transpose":
        topo = pb.MpiTopology(_ints(case["grid"]))
        pencils, _ = pb.route_pencils(topo, _ints(case["shape"]))
        plan = pb.AllToAllvTransposePlan(pencils[-2], pencils[-1], _extra_count(case), dtype=COMPLEX[case["dtype"]])
        grid, n = _ints(case["grid"]), x.dim() - 1
        src = _layout(x, grid, list(pencils[-2].decomposition), list(pencils[-2].permutation))
        return {"family": "transpose", "plan": plan, "src": src, "dst": torch.empty_like(src)}
    plan = _plan(case)
    state = {"family": case["family"], "plan": plan, "src": _input_layout(x, case)}
    if case["family"] == "grad":
        state["src"].requires_grad_(True)
    else:
        state.update(spectrum=plan.allocate_output(), back=plan.allocate_input(),
                     workspace=plan.allocate_workspace())
    return state


def run(state):
    family = state["family"]
    if family == "batch":
        state["batch"].execute(state["buffers"], state["workspace"])
        return [state["spectra"], state["back"]]
    plan, src = state["plan"], state["src"]
    if family == "transpose":
        plan.execute(src, state["dst"])
        return state["dst"]
    if family == "grad":
        spectrum = pba.forward(plan, src)
        weighted = pba.spectral_multiply(plan, spectrum, "k2")
        loss = torch.sum((spectrum.conj() * weighted).real)
        (grad,) = torch.autograd.grad(loss, src)
        potential = pba.inverse(plan, pba.spectral_multiply(plan, spectrum.detach(), "poisson"))
        return {"loss": loss.detach(), "grad": grad, "potential": potential}
    plan.forward(src, state["spectrum"], workspace=state["workspace"])
    plan.inverse(state["spectrum"], state["back"], workspace=state["workspace"])
    return [state["spectrum"], state["back"]]


# ---------------------------------------------------------------- work
def work(case):
    """Bytes read and written once each, and 5 N log2 N operations per complex
    transform of N points (half for real data)."""
    if case["family"] == "batch":
        b = f = 0
        for s, e in _batch_shapes(case):
            n = math.prod(s) * math.prod(e)
            b += 4 * n * 8
            f += 2 * 5 * n * math.log2(math.prod(s))
        return {"bytes": b, "flops": f}
    shape, extra = _ints(case["shape"]), _extra_count(case)
    real = 4 if case["dtype"] == "f32" else 8
    n = math.prod(shape) * extra
    half = n // shape[-1] * (shape[-1] // 2 + 1)
    f = 5 * n * math.log2(math.prod(shape))
    family = case["family"]
    if family == "transpose":
        return {"bytes": 2 * n * 2 * real, "flops": 0}
    if family == "r2c":
        return {"bytes": 2 * (n * real + half * 2 * real), "flops": f}
    if family == "r2r":
        return {"bytes": 4 * n * real, "flops": f}
    if family == "grad":
        # the field in, the gradient and the potential out; forward, adjoint and inverse transforms
        return {"bytes": 3 * n * real, "flops": 1.5 * f + 12 * half}
    return {"bytes": 4 * n * 2 * real, "flops": 2 * f}


# ---------------------------------------------------------------- exact values
def _r2r_axis(x, dim, kind):
    """FFTW's unnormalised real-to-real transform of one axis in 64 bits: the
    samples with their mirror images at positions of an m-point DFT."""
    n = x.shape[dim]
    if kind == "Fft":
        return torch.fft.fft(x, dim=dim)
    if kind == "Dht":
        f = torch.fft.fft(x, dim=dim)
        g = torch.roll(torch.flip(f, (dim,)), 1, dim)  # index -k
        h = (f + g) / 2 + 1j * (f - g) / 2
        return h if x.is_complex() else h.real
    j = torch.arange(n, device=x.device)
    sine, odd = kind.startswith("Dst"), {"DctI": (2 * (n - 1), j, j), "DctII": (4 * n, 2 * j + 1, j),
                                         "DctIII": (4 * n, j, 2 * j + 1), "DctIV": (8 * n, 2 * j + 1, 2 * j + 1),
                                         "DstI": (2 * (n + 1), j + 1, j + 1), "DstII": (4 * n, 2 * j + 1, j + 1),
                                         "DstIII": (4 * n, j + 1, 2 * j + 1),
                                         "DstIV": (8 * n, 2 * j + 1, 2 * j + 1)}[kind]
    m, pos, out = odd
    moved = x.movedim(dim, -1)
    flat = moved.reshape(-1, n)
    res = torch.empty_like(flat)
    mirror = (m - pos) % m
    keep = mirror != pos
    rows = max(1, 2 ** 27 // m)
    for a in range(0, flat.shape[0], rows):
        v = flat[a:a + rows]
        if kind == "DstIII":
            v = v.clone()
            v[:, n - 1] /= 2
        ext = torch.zeros((v.shape[0], m), dtype=v.dtype, device=v.device)
        ext[:, pos] = v
        ext[:, mirror[keep]] = -v[:, keep] if sine else v[:, keep]
        f = torch.fft.fft(ext)[:, out]
        if sine:
            f = 1j * f
        res[a:a + rows] = f if x.is_complex() else f.real
    return res.reshape(moved.shape).movedim(-1, dim)


def _wavenumbers(shape, device):
    """|k|^2 on the half spectrum of a real field of this shape, signed integer
    wave numbers."""
    n = len(shape)
    k2 = torch.zeros((), dtype=torch.float64, device=device)
    for a, ext in enumerate(shape):
        k = torch.arange(ext // 2 + 1 if a == n - 1 else ext, dtype=torch.float64, device=device)
        if a != n - 1:
            k = torch.where(2 * k > ext, k - ext, k)
        k2 = k2 + (k * k).reshape([-1 if i == a else 1 for i in range(n)])
    return k2


def exact(case, seed):
    x = _inputs(case, seed)
    family = case["family"]
    if family == "batch":
        wide = [g.to(torch.complex128) for g in x]
        return [torch.cat([_output_layout(torch.fft.fftn(g, dim=(1, 2, 3)), case) for g in wide]),
                torch.cat([_input_layout(g, case) for g in wide])]
    dims = tuple(range(1, x.dim()))
    if family == "transpose":
        return _output_layout(x, case)
    x = x.to(torch.complex128 if x.is_complex() else torch.float64)
    if family == "grad":
        shape = _ints(case["shape"])
        k2 = _wavenumbers(shape, x.device)
        u = x[0].requires_grad_(True)
        spec = torch.fft.rfftn(u)
        loss = torch.sum(k2 * (spec.real ** 2 + spec.imag ** 2))
        (grad,) = torch.autograd.grad(loss, u)
        mult = torch.where(k2 > 0, -1 / k2.clamp(min=1), torch.zeros_like(k2))
        pot = torch.fft.irfftn(spec.detach() * mult, s=shape)
        return {"loss": loss.detach(), "grad": _input_layout(grad[None], case),
                "potential": _input_layout(pot[None], case)}
    if family == "c2c":
        spec = torch.fft.fftn(x, dim=dims)
    elif family == "r2c":
        spec = torch.fft.rfftn(x, dim=dims)
    else:
        spec = x
        for d, kind in zip(dims, case["kinds"].split(",")):
            spec = _r2r_axis(spec, d, kind)
    return [_output_layout(spec, case), _input_layout(x, case)]
