"""Timed cases of the transforms: what programs that use this package have it do.

A case is a dict of plain values:

  kind       "type1" (points to modes), "type2" (modes to points), "pair" (the
             forward type 2 and the adjoint type 1 of one iteration of an
             image reconstruction, each with a plan of its own on one point
             set), "type3" (sources to targets), "uneven" (many small type-1
             problems executed together)
  call       "execute": the plan holds its sorted points (iterative methods,
             repeated frames on one trajectory); "encode": sort and execute
             (particles that move, a new trajectory every time)
  modes      modes per axis as text, axis 0 first ("64x64"); type 3: bounds
             of the targets, +-, the sources lie in [-1, 1]
  points, targets, batch, eps, precision ("f32" / "f64"), sigma, isign, order
  spread     "uniform", "clustered" (8 centres, standard deviation 0.01) or
             "radial" (3D spokes through the origin, jittered by 1e-3)

Strengths and modes have N(0, 1) real and imaginary parts. Df64 is left out: it
is the reference's replacement for a missing f64, and its plans run the f64
pipeline between two conversions.
"""

from __future__ import annotations

import math

import torch

import wgpunufft_b200 as w

FFT_ORDER = w.ModeOrder.FFT
CENTERED = w.ModeOrder.CENTERED


def _case(kind, call, modes, points, eps, spread="uniform", batch=1, precision="f32", isign=1, order=CENTERED,
          sigma=2.0, targets=0, **more):
    return dict(kind=kind, call=call, modes=modes, points=points, eps=eps, spread=spread, batch=batch,
                precision=precision, isign=isign, order=order, sigma=sigma, targets=targets, **more)


def listed():
    return [
        # Smallest calls: launches and latency. A resampled 1D signal, new sample times on every call.
        _case("type2", "encode", "1000", 20_011, 1e-6, name="signal_1d_t2"),
        # A small image grid on prepared points: the plain method of the package's own benchmark.
        _case("type1", "execute", "64x64", 100_000, 1e-6, name="small_2d_t1"),
        # Gridding of a large image from many samples, uniform and crowded, in the two directions.
        _case("type1", "execute", "1024x1024", 10_000_000, 1e-5, name="uniform_2d_t1"),
        _case("type2", "execute", "1024x1024", 10_000_000, 1e-5, spread="clustered", name="clustered_2d_t2"),
        # Moving points on a grid of no power of two: sorted and transformed on every call.
        _case("type1", "encode", "750x486", 3_000_017, 1e-6, spread="clustered", order=FFT_ORDER, isign=-1,
              name="moving_2d_t1"),
        # Volumes from a radial trajectory (4096 spokes of 12207 samples): the largest calls.
        _case("type1", "execute", "256x256x256", 4096 * 12207, 1e-5, spread="radial", name="radial_3d_t1"),
        _case("type2", "execute", "256x256x256", 4096 * 12207, 1e-5, spread="radial", name="radial_3d_t2"),
        # Many vectors (frames, coils, right-hand sides) on one point set, forward and adjoint.
        _case("pair", "execute", "512x512", 2_000_000, 1e-6, batch=64, name="batched_2d_pair"),
        # Double precision, forward and adjoint.
        _case("pair", "execute", "512x512", 2_000_000, 1e-9, precision="f64", name="double_2d_pair"),
        # A few coils on a ragged volume at a loose tolerance, one iteration of a reconstruction.
        _case("pair", "execute", "100x90x72", 1_000_003, 1e-3, batch=4, isign=-1, name="coils_3d_pair"),
        # Nonuniform to nonuniform in double precision.
        _case("type3", "execute", "200x200x200", 1_000_000, 1e-9, precision="f64", targets=1_000_000,
              name="scattered_3d_t3"),
        # Many independent problems of uneven sizes in one execution.
        _case("uneven", "execute", "", 64, 1e-6, spread="mixed", name="uneven_t1"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choices(["type1", "type2", "pair", "type3", "uneven"], [5, 5, 3, 2, 1])[0]
    if kind == "uneven":
        return _case("uneven", "execute", "", rng.randint(8, 96), 1e-6, spread="mixed")
    if kind == "type3":
        dims = rng.choice([1, 2, 3])
        precision = rng.choice(["f32", "f64"])
        top = {1: 3000, 2: 250, 3: 60}[dims]
        bounds = "x".join(str(_log_int(rng, 12, top)) for _ in range(dims))
        return _case("type3", "execute", bounds, _log_int(rng, 5_000, 400_000),
                     rng.choice([1e-4, 1e-6] if precision == "f32" else [1e-6, 1e-9, 1e-11]), precision=precision,
                     isign=rng.choice([1, -1]), targets=_log_int(rng, 5_000, 300_000))
    dims = rng.choices([1, 2, 3], [2, 5, 4])[0]
    low, high = {1: (200, 200_000), 2: (40, 1024), 3: (20, 160)}[dims]
    modes = [_log_int(rng, low, high) for _ in range(dims)]
    if rng.random() < 0.3:
        modes = [min(high, 1 << max(4, int(round(math.log2(n))))) for n in modes]
    precision = rng.choices(["f32", "f64"], [3, 1])[0]
    eps = rng.choice([1e-3, 1e-4, 1e-5, 1e-6] if precision == "f32" else [1e-6, 1e-9, 1e-12])
    sigma = 1.5 if eps == 1e-3 and rng.random() < 0.3 else 2.0
    spread = rng.choice(["uniform", "clustered"] + (["radial"] if dims == 3 else []))
    batch = rng.choices([1, rng.randint(2, 7), rng.choice([16, 64])], [6, 2, 1 if dims < 3 else 0])[0]
    count = 1
    for n in modes:
        count *= n
    # From sparse sets to several points per mode, within the work of the largest listed case.
    top = min(12.0 * count, 8e6, 2.5e9 / (_width(eps, sigma) ** dims * batch * (8 if precision == "f64" else 1)))
    points = _log_int(rng, max(2_000, min(0.1 * count, top / 4)), max(4_000, top))
    return _case(kind, rng.choice(["execute", "execute", "encode"]), "x".join(map(str, modes)), points, eps,
                 spread=spread, batch=batch, precision=precision, isign=rng.choice([1, -1]),
                 order=rng.choice([CENTERED, FFT_ORDER]), sigma=sigma)


# ---------------------------------------------------------------------------
# Inputs, from the seed alone.

def _shape(case):
    return tuple(int(n) for n in case["modes"].split("x"))


def _real(case):
    return torch.float32 if case["precision"] == "f32" else torch.float64


def _complex(case):
    return torch.complex64 if case["precision"] == "f32" else torch.complex128


def _precision(case):
    return w.Precision.F32 if case["precision"] == "f32" else w.Precision.F64


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _points(spread, count, dims, dtype, g):
    two_pi = 2.0 * math.pi

    def uniform(*size):
        return torch.rand(size, generator=g, device="cuda", dtype=torch.float64)

    def normal(*size):
        return torch.randn(size, generator=g, device="cuda", dtype=torch.float64)

    if spread == "uniform":
        p = uniform(count, dims) * two_pi - math.pi
    elif spread == "clustered":
        centres = uniform(8, dims) * two_pi - math.pi
        which = torch.randint(0, 8, (count,), generator=g, device="cuda")
        p = centres[which] + 0.01 * normal(count, dims)
        p = torch.remainder(p + math.pi, two_pi) - math.pi
    else:
        # As many spokes as samples per spoke allow, at most 4096; the last spoke may be cut.
        spokes = min(4096, max(1, int(math.isqrt(count))))
        per = -(-count // spokes)
        v = normal(spokes, 3)
        v = v / v.norm(dim=1, keepdim=True)
        r = torch.linspace(-math.pi, math.pi, per + 1, device="cuda", dtype=torch.float64)[:-1]
        p = (v[:, None, :] * r[None, :, None]).reshape(-1, 3)[:count]
        p = p + (uniform(*p.shape) * 2e-3 - 1e-3)
        p = torch.clamp(p, -math.pi, math.pi - 1e-6)
    return p.to(dtype).contiguous()


def _values(batch, count, dtype, g):
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    return torch.complex(torch.randn((batch, count), generator=g, device="cuda", dtype=real),
                         torch.randn((batch, count), generator=g, device="cuda", dtype=real))


def _uneven(count):
    """(modes, points, spread) of `count` problems: half 2D and half 3D, points log-uniform in [1e3, 1e6]."""
    shapes = {2: [(64, 64), (128, 128), (256, 256)], 3: [(32, 32, 32), (64, 64, 64)]}
    problems = []
    for k in range(count):
        dims = 2 + k % 2
        points = int(round(10 ** (3.0 + 3.0 * ((k * 0.6180339887) % 1.0))))
        problems.append((shapes[dims][(k // 2) % len(shapes[dims])], points, ("uniform", "clustered")[(k // 4) % 2]))
    return problems


def _inputs(case, seed):
    """Points and inputs of a case: a dict, or a list of dicts for uneven problems."""
    g = _generator(seed)
    if case["kind"] == "uneven":
        return [dict(modes=modes, points=_points(spread, count, len(modes), torch.float32, g),
                     strengths=_values(1, count, torch.complex64, g))
                for modes, count, spread in _uneven(case["points"])]
    shape, batch = _shape(case), case["batch"]
    if case["kind"] == "type3":
        bounds = torch.tensor(shape, dtype=torch.float64, device="cuda")
        sources = torch.rand((case["points"], len(shape)), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        targets = (torch.rand((case["targets"], len(shape)), generator=g, device="cuda", dtype=torch.float64) * 2 - 1)
        # f32 roundings stay within the plan's intervals: the draws stop a little short of them.
        return dict(sources=(sources * (1 - 1e-6)).to(_real(case)).contiguous(),
                    targets=(targets * bounds * (1 - 1e-6)).to(_real(case)).contiguous(),
                    strengths=_values(batch, case["points"], _complex(case), g))
    made = dict(points=_points(case["spread"], case["points"], len(shape), _real(case), g))
    if case["kind"] != "type2":
        made["strengths"] = _values(batch, case["points"], _complex(case), g)
    if case["kind"] != "type1":
        made["coefficients"] = _values(batch, math.prod(shape), _complex(case), g)
    return made


# ---------------------------------------------------------------------------
# The calls.

def prepare(case, seed):
    made = _inputs(case, seed)
    kind = case["kind"]
    if kind == "uneven":
        plans, outputs = [], []
        for problem in made:
            plan = w.NufftPlan.type1_gpu(w.NufftConfig(problem["modes"], case["eps"]))
            plan.set_points_gpu(problem["points"])
            plans.append(plan)
            outputs.append(torch.empty((1, math.prod(problem["modes"])), dtype=torch.complex64, device="cuda"))
        return dict(kind=kind, batch=w.NufftBatch(plans), strengths=[p["strengths"] for p in made], outputs=outputs,
                    made=made)
    state = dict(kind=kind, call=case["call"], batch=case["batch"], **made)
    shape = _shape(case)
    if kind == "type3":
        config = w.NufftType3Config(((-1.0, 1.0),) * len(shape), tuple((-float(b), float(b)) for b in shape),
                                    eps=case["eps"], isign=case["isign"], batch=case["batch"],
                                    precision=_precision(case))
        state["plan"] = w.NufftType3Plan(config)
        state["plan"].set_points_gpu(made["sources"], made["targets"])
        state["values"] = torch.empty((case["batch"], case["targets"]), dtype=_complex(case), device="cuda")
        return state
    config = w.NufftConfig(shape, case["eps"], isign=case["isign"], mode_order=case["order"], sigma=case["sigma"],
                           batch=case["batch"], precision=_precision(case))
    if kind != "type1":
        state["type2"] = w.NufftPlan.type2_gpu(config)
        state["values"] = torch.empty((case["batch"], case["points"]), dtype=_complex(case), device="cuda")
    if kind != "type2":
        state["type1"] = w.NufftPlan.type1_gpu(config.with_isign(-case["isign"]) if kind == "pair" else config)
        state["modes"] = torch.empty((case["batch"], math.prod(shape)), dtype=_complex(case), device="cuda")
    if case["call"] == "execute":
        for plan in ("type1", "type2"):
            if plan in state:
                state[plan].set_points_gpu(made["points"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "uneven":
        state["batch"].execute(state["strengths"], state["outputs"])
        return state["outputs"]
    if kind == "type3":
        state["plan"].execute_gpu_batch(state["batch"], state["strengths"], state["values"])
        return state["values"]
    outputs = {}
    if "type2" in state:
        if state["call"] == "encode":
            state["type2"].encode_type2_gpu(state["points"], state["coefficients"], state["values"])
        else:
            state["type2"].execute_type2_gpu(state["coefficients"], state["values"])
        outputs["values"] = state["values"]
    if "type1" in state:
        if state["call"] == "encode":
            state["type1"].encode_type1_gpu(state["points"], state["strengths"], state["modes"])
        else:
            state["type1"].execute_type1_gpu(state["strengths"], state["modes"])
        outputs["modes"] = state["modes"]
    return outputs


# ---------------------------------------------------------------------------
# What a pass cannot do without, and what its outputs may differ by.

def _width(eps, sigma):
    if sigma == 2.0:
        return max(2, math.ceil(math.log10(10.0 / eps) - 1e-12))
    return max(2, math.ceil(math.log(1.0 / eps) / (math.pi * math.sqrt(1.0 - 1.0 / sigma))))


def _transform_work(shape, points, batch, eps, sigma, scalar, directions=1):
    """Coordinates, values and modes once; window sums (a complex value times a real weight, added) and the FFT."""
    dims, modes = len(shape), math.prod(shape)
    fine = math.prod(sigma * n for n in shape)
    per = points * dims * scalar + batch * (points + modes) * 2 * scalar
    flops = batch * (4.0 * points * _width(eps, sigma) ** dims + 5.0 * fine * math.log2(max(fine, 2)))
    return directions * per, directions * flops


def work(case):
    scalar = 4 if case["precision"] == "f32" else 8
    if case["kind"] == "uneven":
        total = [_transform_work(modes, count, 1, case["eps"], 2.0, 4)
                 for modes, count, _ in _uneven(case["points"])]
        return {"bytes": float(sum(t[0] for t in total)), "flops": float(sum(t[1] for t in total))}
    shape = _shape(case)
    if case["kind"] == "type3":
        dims, width = len(shape), _width(case["eps"], case["sigma"])
        # The outer grid spans the product of the intervals; the inner transform oversamples it once more.
        outer = [max(2 * width, 2 * case["sigma"] / math.pi * b + width + 1) for b in shape]
        fine = math.prod(2.0 * n for n in outer)
        values = case["batch"] * (case["points"] + case["targets"])
        return {"bytes": float((case["points"] + case["targets"]) * dims * scalar + values * 2 * scalar),
                "flops": 4.0 * values * width ** dims + case["batch"] * 5.0 * fine * math.log2(fine)}
    total = _transform_work(shape, case["points"], case["batch"], case["eps"], case["sigma"], scalar,
                            2 if case["kind"] == "pair" else 1)
    return {"bytes": float(total[0]), "flops": float(total[1])}


def tolerance(case):
    # Rounding of the data type; the windows' own error (eps) is the same for every implementation of them. Measured:
    # f32 with the points in another order 1.7e-7 to 4.3e-7, and sums in split products against plain f32 1.1e-6;
    # f64 in another order 8e-15, with window offsets of 1e-13 cells on the longest axes.
    return {"rel": 5e-6} if case["precision"] == "f32" else {"rel": 1e-12}


# ---------------------------------------------------------------------------
# Direct sums in 64 bits.

# Complex multiply-adds of a direct sum that stay well under 20 seconds: as
# matrix products over one axis, and (type 3) one exponential per term.
_MOST_PRODUCTS = 8e13
_MOST_TERMS = 6e10


def _phases(points, n, order, isign):
    """exp(i isign k x) of every point and mode of one axis, (points, modes)."""
    index = torch.arange(n, device="cuda", dtype=torch.float64)
    if order == CENTERED:
        k = index - n // 2
    else:
        k = torch.where(index < (n + 1) // 2, index, index - n)
    angle = isign * points[:, None].to(torch.float64) * k[None, :]
    return torch.polar(torch.ones_like(angle), angle)


def _chunk(shape, batch):
    outer = math.prod(shape[1:])
    return max(32, min(65536, int(6e8 // (16 * (batch * outer + sum(shape))))))


def _exact_type1(shape, points, strengths, order, isign):
    batch, outer = strengths.shape[0], math.prod(shape[1:])
    total = torch.zeros((batch, outer, shape[0]), dtype=torch.complex128, device="cuda")
    step = _chunk(shape, batch)
    for first in range(0, points.shape[0], step):
        p = points[first:first + step]
        left = strengths[:, first:first + step].to(torch.complex128)[:, None, :]
        for axis in range(1, len(shape)):
            e = _phases(p[:, axis], shape[axis], order, isign).T  # (modes, points)
            left = (e[None, :, None, :] * left[:, None, :, :]).reshape(batch, -1, p.shape[0])
        total += torch.matmul(left, _phases(p[:, 0], shape[0], order, isign))
    return total.reshape(batch, -1)


def _exact_type2(shape, points, coefficients, order, isign):
    batch, outer = coefficients.shape[0], math.prod(shape[1:])
    grid = coefficients.to(torch.complex128).reshape(batch * outer, shape[0])
    values = torch.empty((batch, points.shape[0]), dtype=torch.complex128, device="cuda")
    step = _chunk(shape, batch)
    for first in range(0, points.shape[0], step):
        p = points[first:first + step]
        part = torch.matmul(grid, _phases(p[:, 0], shape[0], order, isign).T.contiguous())
        for axis in range(1, len(shape)):
            e = _phases(p[:, axis], shape[axis], order, isign).T
            part = (part.reshape(-1, shape[axis], p.shape[0]) * e[None]).sum(1)
        values[:, first:first + step] = part.reshape(batch, -1)
    return values


def _exact_type3(sources, targets, strengths, isign):
    values = torch.empty((strengths.shape[0], targets.shape[0]), dtype=torch.complex128, device="cuda")
    s, c = sources.to(torch.float64), strengths.to(torch.complex128)
    step = max(1, int(4e7 // sources.shape[0]))
    for first in range(0, targets.shape[0], step):
        angle = isign * (targets[first:first + step].to(torch.float64) @ s.T)
        values[:, first:first + step] = c @ torch.polar(torch.ones_like(angle), angle).T
    return values


def exact(case, seed):
    kind, batch = case["kind"], case["batch"]
    if kind == "type3":
        if float(case["points"]) * case["targets"] > _MOST_TERMS:
            return None
        made = _inputs(case, seed)
        return _exact_type3(made["sources"], made["targets"], made["strengths"], case["isign"])
    if kind == "uneven":
        return [_exact_type1(p["modes"], p["points"], p["strengths"], CENTERED, 1) for p in _inputs(case, seed)]
    shape = _shape(case)
    directions = 2 if kind == "pair" else 1
    if float(directions) * batch * case["points"] * math.prod(shape) > _MOST_PRODUCTS:
        return None
    made = _inputs(case, seed)
    outputs = {}
    if kind != "type1":
        outputs["values"] = _exact_type2(shape, made["points"], made["coefficients"], case["order"], case["isign"])
    if kind != "type2":
        isign = -case["isign"] if kind == "pair" else case["isign"]
        outputs["modes"] = _exact_type1(shape, made["points"], made["strengths"], case["order"], isign)
    return outputs
