"""Noisy strands whose points are rewritten once the strand is known, staged
whole (17 to 32 CVs) or in one chunk (up to 16): the ends of each stage size,
preserveLength against the C restatement, and Classic scalars with their drop
rule over the same strands without them."""
import numpy as np
import pytest
import torch

from helpers import max_position_error
from test_classic_drop_gpu import _asset, _spline_lengths

pytestmark = pytest.mark.gpu

STAGES = [2, 3, 16, 17, 23, 24, 25, 31, 32, 33]


@pytest.mark.parametrize("cvs", STAGES)
def test_preserve_length(oracle, cuda, nxg_lib, cvs):
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    asset, params, _ = _asset(32)
    params = params.copy(cvs_per_strand=cvs, noise_amplitude=0.1, noise_preserve_length=0.7, noise_frequency=3.0)
    got = generate_packed(DeviceAsset(asset), params, 1.5).points.cpu().numpy()
    want = oracle.generate(asset.buffer, params, 1.5, threads=8)[0]
    assert max_position_error(got, want) <= 1e-5 * asset.bbox_diagonal()
    assert np.abs(got[:, 3] - want[:, 3]).max() <= 1e-5 * asset.bbox_diagonal()


@pytest.mark.parametrize("preserve", [0.0, 0.5])
@pytest.mark.parametrize("moved", [False, True])
@pytest.mark.parametrize("cvs", STAGES)
def test_classic_scalars(cuda, nxg_lib, cvs, moved, preserve):
    """`moved`: the mesh deformed under guides that stay, so a strand's first
    point need not be its root."""
    from nanoxgen_b200.classic import generate_packed_classic
    from nanoxgen_b200.generator import DeformedGeometry, DeviceAsset, generate_packed
    asset, params, pos = _asset(32)
    d = DeviceAsset(asset)
    params = params.copy(cvs_per_strand=cvs, noise_amplitude=0.1, noise_preserve_length=preserve)
    S = params.strand_count
    frame = DeformedGeometry(torch.from_numpy((pos * np.float32([1.02, 0.97, 1.0])).astype(np.float32)).cuda()) \
        if moved else None
    points = generate_packed(d, params, 1.5, frame).points.cpu().numpy().reshape(S, cvs, 4).astype(np.float64)
    plain = points[..., :3]
    length = _spline_lengths(plain)
    rng = np.random.default_rng(cvs)
    scalars = np.stack([10.0 ** rng.uniform(-4.5, -3.5, S) / length,
                        np.where(rng.random(S) < 0.1, 5e-5, 0.01)], 1).astype(np.float32)
    scalars[::7, 0] = 0.0
    scalars[1::7, 0] = 1.25
    scalars[2::7, 1] = -1.0
    scaled = length * scalars[:, 0]
    # A coordinate of at most 2 is off by 2^-22, so a length by at most 2 P
    # times that; strands that near the threshold may fall on either side.
    clear = np.abs(scaled - 1e-4) > 2 * cvs * 2.0 ** -22 * scalars[:, 0] + 1e-4 * 2.0 ** -20
    assert clear.mean() > 0.95
    for by_length, by_width in ((True, True), (True, False), (False, True)):
        out = generate_packed_classic(d, params, torch.from_numpy(scalars).cuda(), by_length, by_width, 1.5, frame)
        short = (scaled if by_length else length) < 1e-4
        thin = scalars[:, 1] < 1e-4 if by_width else np.zeros(S, bool)
        np.testing.assert_array_equal(out.point_counts.cpu().numpy()[clear], np.where(short | thin, 0, cvs)[clear])
        got = out.points.cpu().numpy().reshape(S, cvs, 4)
        want = plain[:, :1] + (plain - plain[:, :1]) * scalars[:, None, :1] if by_length else plain
        # Two roundings of coordinates of at most 2, and the plain points' own.
        assert np.abs(got[..., :3] - want).max() <= 4 * 2.0 ** -23
        radius = 0.5 * np.maximum(scalars[:, 1:], 0.0) * 1.5 if by_width else points[..., 3]
        assert np.abs(got[..., 3] - radius).max() <= 2.0 ** -23


@pytest.mark.parametrize("strands,cvs", [(180_000, 24), (140_000, 32)])
def test_ordered_classic_calls(cuda, nxg_lib, strands, cvs):
    """A call large enough to take its strands in order has its ranges' points,
    which are not ordered, bit for bit."""
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    from nanoxgen_b200.classic import generate_packed_classic
    from nanoxgen_b200.generator import DeviceAsset
    w = fixtures.large_sphere(strands=strands, guides=400, n_lon=60, n_rings=41)
    params = w.params.copy(noise_frequency=6.0, cvs_per_strand=cvs, noise_preserve_length=0.3)
    d = DeviceAsset(build_asset(w.build_input, w.stencil_slots))
    scalars = torch.rand((strands, 2), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    full = generate_packed_classic(d, params, scalars)
    first, count = strands - 50_001, 50_001
    part = generate_packed_classic(d, params, scalars[first:].contiguous(), first_strand=first, count=count)
    assert torch.equal(part.points.view(count, -1), full.points.view(strands, -1)[first:])
    assert torch.equal(part.point_counts, full.point_counts[first:])
