"""The noisy lane walk on strands that turn at every CV: coils and zig-zags,
whose transported normal (generate.h:475-481) the reference renormalises at
every step, from the longest strand of the lane groups to the walk's limit and
past it."""
import numpy as np
import pytest

from helpers import max_position_error

TOL = 1e-5  # x mesh bounding-box diagonal, the generator's bar

SPACING = 0.003


def turning_curve(cvs, degrees, zigzag):
    """A root-relative curve of equal segments: a zig-zag, or a coil rising out
    of its plane by a twentieth of a segment per CV, that turns by `degrees` at
    every CV."""
    if zigzag:
        heading = np.where(np.arange(cvs - 1) % 2 == 0, 0.5, -0.5) * np.radians(degrees)
    else:
        heading = np.arange(cvs - 1) * np.radians(degrees)
    step = np.stack([np.cos(heading), np.sin(heading), np.full(cvs - 1, 0.0 if zigzag else 0.05)], 1)
    return np.concatenate([np.zeros((1, 3)), np.cumsum(SPACING * step, 0)])


def turning_asset(cvs, degrees, zigzag):
    """The plain sphere with every guide replaced by the same turning curve."""
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import AssetBuildInput, GuideSet, build_asset
    w = fixtures.plain_sphere(strands=65)
    b, g = w.build_input, w.build_input.guides
    roots = g.cvs[np.cumsum(g.cv_counts.astype(np.int64)) - g.cv_counts]
    curves = (roots[:, None] + turning_curve(cvs, degrees, zigzag)[None]).astype(np.float32).reshape(-1, 3)
    guides = GuideSet(np.full(len(roots), cvs, np.uint32), curves, g.root_normals, g.root_uvs, g.triangles,
                      g.barycentrics, g.support_radii)
    asset = build_asset(AssetBuildInput(b.positions, b.triangles, guides, b.normals, b.texcoords), w.stencil_slots)
    return asset, w.params.copy(cvs_per_strand=cvs, noise_amplitude=0.02, noise_frequency=3.0)


CASES = [(33, 45, False), (128, 60, False), (161, 30, False), (320, 45, False), (512, 40, False), (700, 20, False),
         (1024, 18, False), (1025, 45, False), (128, 120, True), (320, 60, True), (512, 90, True), (1024, 135, True)]


@pytest.mark.gpu
@pytest.mark.parametrize("preserve", [0.0, 0.5])
@pytest.mark.parametrize("cvs,degrees,zigzag", CASES)
def test_turning_strands(oracle, cuda, nxg_lib, cvs, degrees, zigzag, preserve):
    import torch
    from nanoxgen_b200.classic import generate_packed_classic
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    asset, params = turning_asset(cvs, degrees, zigzag)
    params = params.copy(noise_preserve_length=preserve)
    d = DeviceAsset(asset)
    out = generate_packed(d, params)
    scalars = torch.tensor([[1.0, 0.01]], device="cuda").repeat(params.strand_count, 1)
    scaled = generate_packed_classic(d, params, scalars, True, True)
    torch.cuda.synchronize()
    want, _, _, counts = oracle.generate(asset.buffer, params, threads=8)
    got = out.points.cpu().numpy()
    assert np.isfinite(got).all()
    assert max_position_error(got, want) <= TOL * asset.bbox_diagonal()
    # A Classic length of 1 moves a point by its own rounding only.
    assert max_position_error(scaled.points.cpu().numpy(), want) <= TOL * asset.bbox_diagonal()
    assert np.array_equal(scaled.point_counts.cpu().numpy().view(np.uint32), counts)
