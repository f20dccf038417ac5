"""The noisy lane walk where its chunks, lattice windows and dispatch end:
CV counts around multiples of its 16-CV chunk and past the lane groups' 128,
strands short enough that the frequency floor applies, segments longer than a
lattice window, the serial path of a workspace without the offset table, and
the Classic application after a chunked walk."""
import numpy as np
import pytest

from helpers import max_position_error

pytestmark = pytest.mark.gpu

TOL = 1e-5  # x mesh bounding-box diagonal, the generator's bar


@pytest.fixture(scope="module")
def sphere(cuda, nxg_lib):
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    w = fixtures.plain_sphere(strands=401)
    return w, build_asset(w.build_input, w.stencil_slots)


def _check(asset, params, oracle, **kw):
    import torch
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    out = generate_packed(DeviceAsset(asset), params, **kw)
    torch.cuda.synchronize()
    pts, roots, _, counts = oracle.generate(asset.buffer, params, threads=8)
    assert np.array_equal(out.roots_numpy().view(np.uint8), roots.view(np.uint8))
    assert np.array_equal(out.point_counts.cpu().numpy().view(np.uint32), counts)
    mine = out.points.cpu().numpy()
    assert max_position_error(mine, pts) <= TOL * asset.bbox_diagonal()
    assert np.abs(mine[:, 3] - pts[:, 3]).max() <= TOL * asset.bbox_diagonal()
    return mine


@pytest.mark.parametrize("preserve", [0.0, 0.5])
@pytest.mark.parametrize("cvs", [2, 3, 15, 16, 17, 18, 31, 33, 34, 47, 49, 127, 129, 161])
def test_chunk_edges(oracle, sphere, cvs, preserve):
    w, asset = sphere
    _check(asset, w.params.copy(cvs_per_strand=cvs, noise_preserve_length=preserve), oracle)


@pytest.mark.parametrize("cvs,frequency", [(7, 0.3), (40, 0.3), (40, 1.0), (5, 200.0), (40, 60.0)])
def test_frequency_floor_and_long_segments(oracle, sphere, cvs, frequency):
    """0.5 / length above the frequency (the measured base length decides),
    near it, and segments of more lattice cells than a window holds."""
    w, asset = sphere
    _check(asset, w.params.copy(cvs_per_strand=cvs, noise_frequency=frequency), oracle)


@pytest.mark.parametrize("count", [1, 33, 401])
def test_long_strands_without_a_table(oracle, sphere, count):
    """A workspace that holds the strand order alone is enough past 128 CVs
    (the serial kernel); one byte less is refused."""
    import torch
    from nanoxgen_b200._abi import ERRORS, NxgError
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    w, asset = sphere
    params = w.params.copy(cvs_per_strand=150, strand_count=count, noise_preserve_length=0.3)
    d = DeviceAsset(asset)
    up = lambda n: (n + 255) // 256 * 256
    need = 2 * up(4 * count) + up(4 * (asset.header.guide_count + 1))
    d.workspace = lambda p, n: torch.empty(need, dtype=torch.uint8, device="cuda")
    serial = generate_packed(d, params).points.cpu().numpy()
    walked = _check(asset, params, oracle)
    assert max_position_error(serial, walked) <= TOL * asset.bbox_diagonal()
    d.workspace = lambda p, n: torch.empty(need, dtype=torch.uint8, device="cuda")[:need - 1]
    with pytest.raises(NxgError) as e:
        generate_packed(d, params)
    assert e.value.code == ERRORS["WorkspaceTooSmall"]


@pytest.mark.parametrize("noise", [0.0, 0.1])
@pytest.mark.parametrize("cvs", [12, 16, 32, 33, 61, 140])
def test_classic_application(cuda, nxg_lib, sphere, cvs, noise):
    """scale about the first point, radius = 0.5 * max(width, 0) *
    radius_scale, point count 0 below a width of 1e-4, over the same strands
    without scalars (xgen_classic_runtime.cpp:1650-1678, :1827-1858); one
    rounding per coordinate operation apart."""
    import torch
    from nanoxgen_b200.classic import generate_packed_classic
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    w, asset = sphere
    d = DeviceAsset(asset)
    params = w.params.copy(cvs_per_strand=cvs, noise_amplitude=noise, noise_preserve_length=0.4)
    rng = np.random.default_rng(3)
    S = params.strand_count
    scalars = np.stack([rng.uniform(0.2, 1.5, S), rng.uniform(-0.01, 0.02, S)], 1).astype(np.float32)
    for length, width in ((True, True), (True, False), (False, True)):
        plain = generate_packed(d, params, 1.5).points.cpu().numpy().reshape(S, cvs, 4).astype(np.float64)
        out = generate_packed_classic(d, params, torch.from_numpy(scalars).cuda(), length, width, 1.5)
        got = out.points.cpu().numpy().reshape(S, cvs, 4)
        want = plain.copy()
        if length:
            want[:, :, :3] = plain[:, :1, :3] + (plain[:, :, :3] - plain[:, :1, :3]) * scalars[:, None, :1]
        if width:
            want[:, :, 3] = 0.5 * np.maximum(scalars[:, 1:], 0.0) * 1.5
        # Two roundings of coordinates of at most 2, and the plain points' own.
        assert np.abs(got[:, :, :3] - want[:, :, :3]).max() <= 4 * 2.0 ** -23
        assert np.abs(got[:, :, 3] - want[:, :, 3]).max() <= 2.0 ** -23
        dropped = scalars[:, 1] < 1e-4 if width else np.zeros(S, bool)
        counts = out.point_counts.cpu().numpy()
        assert np.array_equal(counts, np.where(dropped, 0, cvs))


@pytest.mark.parametrize("noise,strands", [(0.1, 250_000), (0.0, 800_000)])
def test_ordered_and_unordered_strands_agree(cuda, nxg_lib, noise, strands):
    """A call large enough to order its strands by guide gives the points and
    roots of its ranges, which are not ordered, bit for bit."""
    import torch
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    w = fixtures.large_sphere(strands=strands, guides=400, n_lon=60, n_rings=41)
    params = w.params.copy(noise_amplitude=noise, noise_frequency=6.0)
    d = DeviceAsset(build_asset(w.build_input, w.stencil_slots))
    full = generate_packed(d, params)
    for first, count in ((0, 70_001), (strands - 70_001, 70_001)):
        part = generate_packed(d, params, first_strand=first, count=count)
        assert torch.equal(part.points, full.points[first * 32:(first + count) * 32])
        assert torch.equal(part.roots, full.roots[first:first + count])
        assert torch.equal(part.root_uvs, full.root_uvs[first:first + count])
