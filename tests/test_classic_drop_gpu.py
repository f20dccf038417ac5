"""Classic scalars at the places the plain walk and the root gathers branch:
scaled lengths around the drop threshold (the chord test of the base step and
the sampled spline behind it), first points off the root, and mesh arrays at
odd words."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _asset(lon, rings=21, strands=401):
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200._abi import GenerationParams
    from nanoxgen_b200.asset import AssetBuildInput, build_asset
    rng = np.random.default_rng(lon)
    pos, uv, tris = fixtures.sphere_mesh(lon, rings)
    guides = fixtures.surface_guides(pos, tris, 64, 16, rng, texcoords=uv)
    params = GenerationParams(strand_count=strands, cvs_per_strand=12, seed=7, root_width=0.01, tip_width=0.001,
                              noise_amplitude=0.0, noise_frequency=8.0)
    return build_asset(AssetBuildInput(pos, tris, guides, None, uv), 4), params, pos


def _spline_lengths(p):
    """The 2P + 4 chords of the B-spline of [S, P, 3] in 64 bits, its ends extrapolated."""
    S, P, _ = p.shape
    q = np.concatenate([2 * p[:, :1] - p[:, 1:2], p, 2 * p[:, -1:] - p[:, -2:-1]], 1)
    x = np.arange(1, 2 * P + 4) / (2 * P + 4) * (P - 1)
    i = x.astype(int)
    f = (x - i)[:, None]
    w = [(1 - f) ** 3, 3 * f ** 3 - 6 * f ** 2 + 4, -3 * f ** 3 + 3 * f ** 2 + 3 * f + 1, f ** 3]
    at = sum(w[k] * q[:, i + k] for k in range(4)) / 6
    at = np.concatenate([p[:, :1], at, p[:, -1:]], 1)
    return np.linalg.norm(np.diff(at, axis=1), axis=-1).sum(1)


@pytest.mark.parametrize("moved", [False, True])
@pytest.mark.parametrize("cvs", [2, 3, 12, 32, 33, 140])
def test_drop_threshold(cuda, nxg_lib, cvs, moved):
    """`moved`: the mesh deformed under guides that stay, so a strand's first
    point need not be its root."""
    from nanoxgen_b200.classic import generate_packed_classic
    from nanoxgen_b200.generator import DeformedGeometry, DeviceAsset, generate_packed
    asset, params, pos = _asset(32)
    d, params = DeviceAsset(asset), params.copy(cvs_per_strand=cvs)
    S = params.strand_count
    frame = DeformedGeometry(torch.from_numpy((pos * np.float32([1.02, 0.97, 1.0])).astype(np.float32)).cuda()) \
        if moved else None
    plain = generate_packed(d, params, 1.0, frame).points.cpu().numpy().reshape(S, cvs, 4).astype(np.float64)[..., :3]
    length = _spline_lengths(plain)
    rng = np.random.default_rng(cvs)
    scalars = np.stack([10.0 ** rng.uniform(-4.5, -3.5, S) / length,
                        np.where(rng.random(S) < 0.1, 5e-5, 0.01)], 1).astype(np.float32)
    scalars[::7, 0] = 0.0
    out = generate_packed_classic(d, params, torch.from_numpy(scalars).cuda(), deformed=frame)
    scaled = length * scalars[:, 0]
    counts = out.point_counts.cpu().numpy()
    want = np.where((scaled < 1e-4) | (scalars[:, 1] < 1e-4), 0, cvs)
    # A coordinate of at most 2 is off by 2^-22, so a length by at most 2 P
    # times that; strands that near the threshold may fall on either side.
    clear = np.abs(scaled - 1e-4) > 2 * cvs * 2.0 ** -22 * scalars[:, 0] + 1e-4 * 2.0 ** -20
    assert clear.mean() > 0.95 and 0 < (want[clear] == 0).sum() < clear.sum()
    np.testing.assert_array_equal(counts[clear], want[clear])
    got = out.points.cpu().numpy().reshape(S, cvs, 4)[..., :3]
    moved_to = plain[:, :1] + (plain - plain[:, :1]) * scalars[:, None, :1]
    assert np.abs(got - moved_to).max() <= 4 * 2.0 ** -23  # two roundings of coordinates of at most 2


@pytest.mark.parametrize("lon", [31, 32, 33, 34])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_roots_from_arrays_at_any_word(cuda, nxg_lib, lon, shift):
    """The plain walk's and the scalar kernel's wide gathers against the noise
    walk's loads of one word, bit for bit: sections and deformed arrays that
    start at odd words."""
    from nanoxgen_b200.classic import Expression, ScalarPlan, root_scalars
    from nanoxgen_b200.generator import DeformedGeometry, DeviceAsset, generate_packed
    asset, params, pos = _asset(lon)
    d = DeviceAsset(asset)

    def off(a):
        flat = torch.empty(a.size + shift, device="cuda")
        flat[shift:] = torch.from_numpy(a.reshape(-1)).cuda()
        return flat[shift:].view(a.shape)

    normals = pos / np.linalg.norm(pos, axis=1, keepdims=True)
    frame = DeformedGeometry(off((pos * np.float32(1.1)).astype(np.float32)), off(normals.astype(np.float32)))
    for deformed in (None, frame):
        runs = [generate_packed(d, params.copy(noise_amplitude=a), 1.0, deformed).roots_numpy() for a in (0.0, 0.1)]
        assert np.array_equal(runs[0].view(np.uint8), runs[1].view(np.uint8))
        if deformed is None:
            rest = runs[0]
    plan = ScalarPlan(Expression.classic("$u", "length"), Expression.classic("$v", "width"))
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    s = root_scalars(d, params, plan, status=status)
    s = (s[0] if isinstance(s, tuple) else s).cpu().numpy()
    assert status.cpu().tolist() == [0, 0]
    np.testing.assert_array_equal(s.view(np.uint32).reshape(-1, 2), np.ascontiguousarray(rest["uv"]).view(np.uint32))
