"""Spreading and interpolation by matrix products over strips of support starts.

f32 results are compared with the f64 plan of the same tolerance, which uses
the same window up to its Horner rows below 0.05 eps, so the difference is
f32 rounding and at most a few such rows: window weights, strengths and sums
carry a few units of 2^-24 each and the split products drop terms of 2^-22
(together below 16 x 2^-23), and 0.2 eps stands for the rows. f64 results are
compared with the direct sums at the reference's 20 eps (2D) and 32 eps (3D).
"""

import numpy as np
import pytest

from oracle import gpu_direct, native

pytestmark = pytest.mark.gpu

F32_ROUNDING = 16 * 2.0**-23


def points_of(rng, kind, count, fine):
    """f32-exact points: uniform, crowded in one cell's neighbourhood, or on and beside the grid's edges."""
    dims = len(fine)
    p = rng.uniform(-np.pi, np.pi, (count, dims))
    if kind == "crowded":
        p[: count // 2] = rng.uniform(-0.2, 0.2, (count // 2, dims))
    elif kind == "edges":
        cell = 2.0 * np.pi / np.asarray(fine)
        near = -np.pi + cell * rng.integers(-3, 4, (count, dims))
        p = np.where(rng.random((count, dims)) < 0.5, np.remainder(near + np.pi, 2 * np.pi) - np.pi, p)
        p[0] = np.nan  # out of reach: weighs zero
    return p.astype(np.float32)


def transform(w, kind, n_modes, eps, precision, batch, points, inputs, outputs):
    import torch

    real, cplx = ((torch.float32, torch.complex64) if precision == w.Precision.F32
                  else (torch.float64, torch.complex128))
    plan = w.NufftPlan(kind, w.NufftConfig(n_modes, eps, batch=batch, precision=precision))
    out = torch.empty((batch, outputs), dtype=cplx, device="cuda")
    plan.encode_gpu(torch.from_numpy(points).to("cuda", real), torch.from_numpy(inputs).to("cuda", cplx), out)
    plan.synchronize()
    return plan, out.cpu().numpy()


def values(rng, batch, count):
    return (rng.standard_normal((batch, count)) + 1j * rng.standard_normal((batch, count))).astype(np.complex64)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("eps", [1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("n_modes, count, spread, batch", [
    ((16, 16, 16), 9, "uniform", 1),           # fewer points than a chunk
    ((16, 16, 16), 40_000, "uniform", 1),      # one tile deep along z
    ((21, 19, 33), 60_001, "crowded", 3),      # ragged tiles, parts of one tile
    ((8, 40, 13), 30_003, "edges", 2),         # windows that wrap, a point out of reach
])
def test_f32_3d_differs_from_f64_by_rounding(kind, eps, n_modes, count, spread, batch):
    import wgpunufft_b200 as w

    rng = np.random.default_rng(11)
    points = points_of(rng, spread, count, [2 * n for n in n_modes])
    total = int(np.prod(n_modes))
    inputs = values(rng, batch, count if kind == 1 else total)
    outputs = total if kind == 1 else count
    plan, got = transform(w, kind, n_modes, eps, w.Precision.F32, batch, points, inputs, outputs)
    plan64, want = transform(w, kind, n_modes, eps, w.Precision.F64, batch, points, inputs, outputs)
    # Support starts at exact cell boundaries may round to either side.
    assert plan.kernel_width() == plan64.kernel_width()
    if spread == "edges":
        assert rel(got, want) < 32 * eps
    else:
        assert rel(got, want) < F32_ROUNDING + 0.2 * eps


@pytest.mark.parametrize("n_modes, count, spread, batch", [
    ((32, 32), 7, "uniform", 1),             # below the density of the rows
    ((64, 64), 100_000, "uniform", 1),       # whole tiles, rows longer than a chunk
    ((75, 41), 9_001, "uniform", 3),         # ragged tiles, rows shorter than a chunk
    ((50, 300), 200_003, "crowded", 1),      # parts of one tile, rows of thousands of points
    ((33, 90), 20_003, "edges", 2),          # windows that wrap, a point out of reach
])
def test_f32_2d_rows_differ_from_f64_by_rounding(n_modes, count, spread, batch):
    import wgpunufft_b200 as w

    eps = 1e-6  # width 7
    rng = np.random.default_rng(13)
    points = points_of(rng, spread, count, [2 * n for n in n_modes])
    inputs = values(rng, batch, count)
    total = int(np.prod(n_modes))
    plan, got = transform(w, 1, n_modes, eps, w.Precision.F32, batch, points, inputs, total)
    _, want = transform(w, 1, n_modes, eps, w.Precision.F64, batch, points, inputs, total)
    assert plan.kernel_width() == 7
    assert rel(got, want) < (20 * eps if spread == "edges" else F32_ROUNDING + 0.2 * eps)


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("eps", [1e-4, 1e-8, 1e-9, 1e-12, 1e-14])  # widths 5, 9, 10, 13, 15
@pytest.mark.parametrize("n_modes, count, spread", [
    ((40, 30), 5, "uniform"),
    ((40, 30), 20_003, "crowded"),
    ((9, 70), 6_001, "edges"),
    ((12, 14, 10), 20_001, "uniform"),
    ((30, 8, 9), 6_003, "edges"),
    ((15, 16, 17), 30_001, "crowded"),   # several parts of one tile
])
def test_f64_matches_direct_sums(kind, eps, n_modes, count, spread):
    import wgpunufft_b200 as w

    rng = np.random.default_rng(12)
    points = points_of(rng, spread, count, [2 * n for n in n_modes]).astype(np.float64)
    total = int(np.prod(n_modes))
    inputs = values(rng, 1, count if kind == 1 else total).astype(np.complex128)
    _, got = transform(w, kind, n_modes, eps, w.Precision.F64, 1, points, inputs, total if kind == 1 else count)
    reach = np.isfinite(points).all(axis=1)
    if kind == 1:
        want = native.direct_type1(points[reach], inputs[0][reach], n_modes)[0]
    else:
        want = np.zeros(count, dtype=np.complex128)
        want[reach] = native.direct_type2(points[reach], inputs[0], n_modes)[0]
    bound = max((20 if len(n_modes) == 2 else 32) * eps, 2e-13)  # 2e-13: rounding of the sums and the FFT
    assert rel(got[0], want) < bound


def test_bin_offsets_across_long_empty_stretches():
    """Two crowds a few cells wide: all other bins of the grid are empty."""
    import torch

    import wgpunufft_b200 as w
    from tests.test_gpu_type12 import oracle_order

    rng = np.random.default_rng(14)
    points = np.concatenate([rng.normal(-1.0, 0.01, (70_001, 2)), rng.normal(2.0, 0.01, (80_002, 2))]).astype(np.float32)
    plan = w.NufftPlan.type1_gpu(w.NufftConfig((300, 200), 1e-5))
    plan.set_points_gpu(torch.from_numpy(points).cuda())
    perm, offsets = plan.bin_order()
    ref_perm, ref_offsets, *_ = oracle_order(points, plan.fine_grid_shape(), 1e-5, 1)
    assert np.array_equal(perm.numpy(), ref_perm)
    assert np.array_equal(offsets.numpy(), ref_offsets)


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])  # widths 2 to 7
@pytest.mark.parametrize("batch", [1, 3, 18])
@pytest.mark.parametrize("n_modes, spread", [((40, 30), "crowded"), ((9, 70), "edges"), ((300, 200), "uniform")])
def test_batched_2d_type2_strips_match_the_gather(eps, batch, n_modes, spread):
    """The strips, asked for by the tensor-core method, against the CUDA-core
    kernels on the same windows: rounding of both (F32_ROUNDING) apart."""
    import torch

    import wgpunufft_b200 as w

    rng = np.random.default_rng(15)
    count = 5_003
    points = torch.from_numpy(points_of(rng, spread, count, [2 * n for n in n_modes])).cuda()
    inputs = torch.from_numpy(values(rng, batch, int(np.prod(n_modes)))).cuda()

    def run(method):
        plan = w.NufftPlan.type2_gpu(w.NufftConfig(n_modes, eps, batch=batch, spread_method=method))
        out = torch.empty((batch, count), dtype=torch.complex64, device="cuda")
        plan.encode_type2_gpu(points, inputs, out)
        first = out.clone()
        plan.execute_type2_gpu(inputs, out)
        plan.synchronize()
        assert torch.equal(first.view(torch.int32), out.view(torch.int32))
        return out.cpu().numpy()

    assert rel(run(w.SpreadMethod.TENSOR_CORES), run(w.SpreadMethod.CUDA_CORES)) < F32_ROUNDING


@pytest.mark.parametrize("tile", [1, 2, 4, 64])
def test_2d_f64_strips_of_every_tuned_tile(tile):
    """Tiles from one start up: the records' counters then outgrow the tile's cells."""
    import wgpunufft_b200 as w
    from wgpunufft_b200 import _native

    eps, n_modes, count = 1e-4, (12, 17), 900  # width 5
    rng = np.random.default_rng(16)
    points = points_of(rng, "crowded", count, [2 * n for n in n_modes]).astype(np.float64)
    inputs = values(rng, 2, count).astype(np.complex128)
    override = _native.library().b200nufft_tuning_override
    override(_native.Tuning(tile, 0, 0, 0))
    try:
        _, got = transform(w, 1, n_modes, eps, w.Precision.F64, 2, points, inputs, int(np.prod(n_modes)))
    finally:
        override(None)
    for b in range(2):
        assert rel(got[b], native.direct_type1(points, inputs[b], n_modes)[0]) < 20 * eps


@pytest.mark.parametrize("eps, n_modes", [(1e-4, (32, 30, 28)), (1e-5, (32, 30, 28)), (1e-6, (32, 30, 28)),
                                          (1e-6, (128, 100))])
def test_f32_products_lose_no_share_of_one_signed_sums(eps, n_modes):
    """Positive strengths against the CUDA-core kernels, which round every sum:
    the modes agree on average. Truncated products alone leave them 2^-24 / (2
    ln 2) = 4.3e-8 smaller (measured 3.7e-8 to 4.1e-8); the mean of 8 draws
    varies by 1e-9 to 3e-9, and half the loss stands for its mantissas."""
    import torch

    import wgpunufft_b200 as w

    shares = []
    for seed in range(8):
        rng = np.random.default_rng(100 + seed)
        count = 600_000
        points = torch.from_numpy((rng.normal(0.0, 0.3, (count, len(n_modes)))).astype(np.float32)).cuda()
        strengths = torch.from_numpy((rng.uniform(0.5, 1.0, (1, count)) + 0j).astype(np.complex64)).cuda()
        outs = []
        for method in (w.SpreadMethod.AUTO, w.SpreadMethod.CUDA_CORES):
            plan = w.NufftPlan.type1_gpu(w.NufftConfig(n_modes, eps, spread_method=method))
            out = torch.empty((1, int(np.prod(n_modes))), dtype=torch.complex64, device="cuda")
            plan.encode_type1_gpu(points, strengths, out)
            plan.synchronize()
            outs.append(out.to(torch.complex128))
        got, want = outs
        shares.append(float((got * want.conj()).real.sum() / (want.abs() ** 2).sum()) - 1.0)
    assert abs(np.mean(shares)) < 2e-8


@pytest.mark.parametrize("eps", [1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12, 1e-13, 1e-14])
@pytest.mark.parametrize("n_modes, spread", [((70, 90), "uniform"), ((12, 150), "edges")])
def test_2d_f64_values_do_not_depend_on_the_other_points(eps, n_modes, spread):
    """A few scattered points, which each lane of a warp gathers, and the same
    points among many, which go through the products: the same bits."""
    import torch

    import wgpunufft_b200 as w

    rng = np.random.default_rng(17)
    few = points_of(rng, spread, 401, [2 * n for n in n_modes]).astype(np.float64)
    many = rng.uniform(-np.pi, np.pi, (90_000, 2))
    inputs = torch.from_numpy(values(rng, 6, int(np.prod(n_modes))).astype(np.complex128)).cuda()

    def run(points):
        plan = w.NufftPlan.type2_gpu(w.NufftConfig(n_modes, eps, batch=6, precision=w.Precision.F64))
        out = torch.empty((6, len(points)), dtype=torch.complex128, device="cuda")
        plan.encode_type2_gpu(torch.from_numpy(points).cuda(), inputs, out)
        plan.synchronize()
        return out

    alone = run(few)
    among = run(np.concatenate([few, many]))[:, : len(few)].contiguous()
    assert torch.equal(torch.view_as_real(alone), torch.view_as_real(among))


@pytest.mark.parametrize("eps", [1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12, 1e-13, 1e-14])
@pytest.mark.parametrize("n_modes", [(40, 50), (400, 400)])  # one kernel; a kernel for sparse tiles, one for others
def test_2d_f64_sparse_and_crowded_tiles(eps, n_modes):
    """Scattered points and a few crowds in one set, three vectors."""
    import wgpunufft_b200 as w

    rng = np.random.default_rng(18)
    fine = np.asarray([2 * n for n in n_modes])
    count = int(fine.prod()) // 160
    crowds = [c + 2 * np.pi / fine * rng.normal(0.0, 6.0, (600, 2)) for c in ((0.0, 0.0), (-np.pi, 2.0))]
    points = np.concatenate([rng.uniform(-np.pi, np.pi, (count, 2)), *crowds])
    points = np.remainder(points + np.pi, 2 * np.pi) - np.pi
    inputs = values(rng, 3, len(points)).astype(np.complex128)
    plan, got = transform(w, 1, n_modes, eps, w.Precision.F64, 3, points, inputs, int(np.prod(n_modes)))
    want = gpu_direct.direct_type1(points, inputs, n_modes)
    for b in range(3):
        assert rel(got[b], want[b]) < max(20 * eps, 2e-13)


@pytest.mark.parametrize("eps, tile", [(1e-6, (18, 10, 10)), (1e-9, (15, 15, 7)), (1e-11, (13, 13, 5))])
def test_3d_f64_crowd_where_register_tiles_meet(eps, tile):
    """All points in the bins around a corner of eight tiles, which count them all
    and spread their own: the parts stay within those reserved."""
    import wgpunufft_b200 as w

    n_modes, count = (30, 25, 20), 200_003
    rng = np.random.default_rng(19)
    fine = np.asarray([2 * n for n in n_modes])
    plan = w.NufftPlan.type1_gpu(w.NufftConfig(n_modes, eps, precision=w.Precision.F64))
    width = plan.kernel_width()
    assert tile == (24 - width + 1, (16 if width <= 9 else 24) - width + 1, 16 - width + 1)
    # Support starts (cells) within 1.5 of the corner at 2 x, 1 y and 1 z tiles.
    corner = np.asarray(tile) * (2, 1, 1)
    x = (corner + rng.uniform(-1.5, 1.5, (count, 3)) + width / 2 - fine / 2) * 2 * np.pi / fine
    points = np.remainder(x + np.pi, 2 * np.pi) - np.pi
    inputs = values(rng, 2, count).astype(np.complex128)
    _, got = transform(w, 1, n_modes, eps, w.Precision.F64, 2, points, inputs, int(np.prod(n_modes)))
    want = gpu_direct.direct_type1(points, inputs, n_modes)
    for b in range(2):
        assert rel(got[b], want[b]) < max(32 * eps, 2e-13)


@pytest.mark.parametrize("eps", [1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12])  # widths 5 to 13
def test_3d_f64_sparse_tiles_spread_in_shared_memory(eps):
    """One point set below the density of the register tiles, one above, on one plan."""
    import torch

    import wgpunufft_b200 as w

    n_modes = (40, 41, 38)
    rng = np.random.default_rng(20)
    plan = w.NufftPlan.type1_gpu(w.NufftConfig(n_modes, eps, batch=2, precision=w.Precision.F64))
    out = torch.empty((2, int(np.prod(n_modes))), dtype=torch.complex128, device="cuda")
    for count in (301, 12_001, 300):
        points = rng.uniform(-np.pi, np.pi, (count, 3))
        inputs = values(rng, 2, count).astype(np.complex128)
        plan.encode_type1_gpu(torch.from_numpy(points).cuda(), torch.from_numpy(inputs).cuda(), out)
        plan.synchronize()
        want = gpu_direct.direct_type1(points, inputs, n_modes)
        for b in range(2):
            assert rel(out[b].cpu().numpy(), want[b]) < max(32 * eps, 2e-13)


@pytest.mark.parametrize("eps", [1e-5, 1e-6])  # widths 6 and 7
@pytest.mark.parametrize("n_modes, count, spread, batch", [
    ((32, 32, 32), 262_144, "uniform", 1),
    ((21, 19, 33), 250_001, "crowded", 3),
    ((8, 40, 13), 250_003, "edges", 2),
])
def test_f32_3d_values_of_many_points_differ_from_f64_by_rounding(eps, n_modes, count, spread, batch):
    """Point sets large enough for the strips (interp_strips_chosen), in both precisions."""
    import wgpunufft_b200 as w

    rng = np.random.default_rng(21)
    points = points_of(rng, spread, count, [2 * n for n in n_modes])
    inputs = values(rng, batch, int(np.prod(n_modes)))
    _, got = transform(w, 2, n_modes, eps, w.Precision.F32, batch, points, inputs, count)
    _, want = transform(w, 2, n_modes, eps, w.Precision.F64, batch, points, inputs, count)
    assert rel(got, want) < (32 * eps if spread == "edges" else F32_ROUNDING + 0.2 * eps)


@pytest.mark.parametrize("eps", [1e-1, 1e-3, 1e-4, 1e-6])  # widths 2, 4, 5, 7
@pytest.mark.parametrize("capacity, active", [(16, 16), (20, 5), (48, 18), (48, 48)])
@pytest.mark.parametrize("n_modes, count", [((64, 64), 2_000), ((64, 64), 33_000), ((300, 200), 9_000)])
def test_batched_2d_type2_of_either_kernel_matches_the_bins(eps, capacity, active, n_modes, count):
    """16 to 63 vectors, point sets on both sides of the rule: against the CUDA-core kernels."""
    import torch

    import wgpunufft_b200 as w

    rng = np.random.default_rng(22)
    points = torch.from_numpy(points_of(rng, "uniform", count, [2 * n for n in n_modes])).cuda()
    inputs = torch.from_numpy(values(rng, active, int(np.prod(n_modes)))).cuda()

    def run(method):
        plan = w.NufftPlan.type2_gpu(w.NufftConfig(n_modes, eps, batch=capacity, spread_method=method))
        plan.set_points_gpu(points)
        out = torch.empty((active, count), dtype=torch.complex64, device="cuda")
        plan.execute_type2_gpu_batch(active, inputs, out)
        plan.synchronize()
        return out.cpu().numpy()

    assert rel(run(w.SpreadMethod.AUTO), run(w.SpreadMethod.CUDA_CORES)) < F32_ROUNDING


def test_override_sets_the_batch_of_type2_strips():
    """tensor_min_batch of an override decides for 16 to 63 vectors too: the
    same bits as the plan that is asked for the kernel."""
    import torch

    import wgpunufft_b200 as w
    from wgpunufft_b200 import _native

    n_modes, count, batch = (64, 64), 30_000, 32  # eps 1e-3: bins by the rule
    rng = np.random.default_rng(23)
    points = torch.from_numpy(points_of(rng, "uniform", count, [128, 128])).cuda()
    inputs = torch.from_numpy(values(rng, batch, 64 * 64)).cuda()
    override = _native.library().b200nufft_tuning_override

    def run(method, least=0):
        if least:
            override(_native.Tuning(0, 0, 0, least))
        try:
            plan = w.NufftPlan.type2_gpu(w.NufftConfig(n_modes, 1e-3, batch=batch, spread_method=method))
            out = torch.empty((batch, count), dtype=torch.complex64, device="cuda")
            plan.encode_type2_gpu(points, inputs, out)
            plan.synchronize()
        finally:
            override(None)
        return out.view(torch.int32)

    strips, bins = run(w.SpreadMethod.TENSOR_CORES), run(w.SpreadMethod.CUDA_CORES)
    assert not torch.equal(strips, bins)
    assert torch.equal(run(w.SpreadMethod.AUTO), bins)
    assert torch.equal(run(w.SpreadMethod.AUTO, 16), strips)
    assert torch.equal(run(w.SpreadMethod.AUTO, 33), bins)


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("n_modes, count", [((33, 21), 9_001), ((14, 11, 13), 12_001)])
@pytest.mark.parametrize("width", range(5, 17))
def test_f64_vectors_of_a_batch_are_those_of_single_calls(kind, n_modes, count, width):
    """Every width's kernels, five vectors: each the bits of a call of its own,
    the last one the direct sums."""
    import wgpunufft_b200 as w

    eps = 10.0 ** (1 - width)
    rng = np.random.default_rng(24)
    points = points_of(rng, "crowded", count, [2 * n for n in n_modes]).astype(np.float64)
    total = int(np.prod(n_modes))
    inputs = values(rng, 5, count if kind == 1 else total).astype(np.complex128)
    outputs = total if kind == 1 else count
    plan, got = transform(w, kind, n_modes, eps, w.Precision.F64, 5, points, inputs, outputs)
    assert plan.kernel_width() == width
    for b in (0, 4):
        _, alone = transform(w, kind, n_modes, eps, w.Precision.F64, 1, points, inputs[b : b + 1], outputs)
        assert np.array_equal(got[b].view(np.float64), alone[0].view(np.float64))
    direct = gpu_direct.direct_type1 if kind == 1 else gpu_direct.direct_type2
    want = direct(points, inputs[4:5], n_modes)[0]
    assert rel(got[4], want) < max((20 if len(n_modes) == 2 else 32) * eps, 2e-13)


@pytest.mark.parametrize("kind, n_modes, eps, precision, batch, many, few", [
    (1, (48, 40, 44), 1e-9, "F64", 2, 60_000, 500),     # register tiles; shared-memory tiles
    (2, (48, 40, 44), 1e-9, "F64", 1, 200_000, 3_000),  # strips; the gather's order
    (2, (48, 40, 44), 1e-6, "F32", 1, 400_000, 5_000),
    (2, (100, 90), 1e-6, "F32", 16, 60_000, 2_000),     # strips; bins
    (2, (100, 90), 1e-4, "F32", 16, 100_000, 3_000),
    (1, (200, 180), 1e-9, "F64", 1, 100_000, 2_000),
    (2, (200, 180), 1e-9, "F64", 1, 300_000, 2_000),
])
def test_sparser_points_are_set_and_executed_in_a_graph(kind, n_modes, eps, precision, batch, many, few):
    """A plan that has run on many points takes fewer inside a capture, where
    nothing can be allocated, whichever kernels its rules choose for them."""
    import torch

    import wgpunufft_b200 as w

    real, cplx = (torch.float32, torch.complex64) if precision == "F32" else (torch.float64, torch.complex128)
    rng = np.random.default_rng(25)
    total = int(np.prod(n_modes))
    config = w.NufftConfig(n_modes, eps, batch=batch, precision=getattr(w.Precision, precision))

    def buffers(count):
        points = torch.from_numpy(rng.uniform(-np.pi, np.pi, (count, len(n_modes)))).to("cuda", real)
        points.clamp_(-3.1415, 3.1415)
        inputs = torch.from_numpy(values(rng, batch, count if kind == 1 else total)).to("cuda", cplx)
        return points, inputs, torch.empty((batch, total if kind == 1 else count), dtype=cplx, device="cuda")

    plan, stream = w.NufftPlan(kind, config), torch.cuda.Stream()
    points, inputs, out = buffers(few)
    with torch.cuda.stream(stream):
        plan.encode_gpu(*buffers(many), stream=stream)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            plan.encode_gpu(points, inputs, out, stream=stream)
    graph.replay()
    torch.cuda.synchronize()
    captured = out.clone()
    alone = w.NufftPlan(kind, config)
    alone.encode_gpu(points, inputs, out)
    alone.synchronize()
    assert torch.equal(torch.view_as_real(captured), torch.view_as_real(out))
    del graph
