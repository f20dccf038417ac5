"""How a call is launched: a caller's prepared order, registered tiles and the
autotuner, and ranges of a description, leave the points what they are and are
taken as the interface says."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sphere(cuda, nxg_lib):
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    from nanoxgen_b200.generator import DeviceAsset
    w = fixtures.plain_sphere(strands=2000)
    return DeviceAsset(build_asset(w.build_input, w.stencil_slots)), w.params


@pytest.mark.parametrize("noise", [0.0, 0.1])
@pytest.mark.parametrize("strands,cvs", [(33, 2), (2000, 16), (2000, 40)])
def test_a_prepared_order_is_taken(sphere, strands, cvs, noise):
    """Two-phase calls of any size generate the strands of the order that the
    workspace holds: entries past the strand count leave their strands out, the
    others have the points of a whole call."""
    import torch
    from nanoxgen_b200.generator import generate_packed, generate_packed_ordered, prepare_strand_order
    d, params = sphere
    params = params.copy(strand_count=strands, cvs_per_strand=cvs, noise_amplitude=noise)
    want = generate_packed(d, params).points.view(strands, cvs, 4)
    ws = prepare_strand_order(d, params)
    words = ws[(4 * strands + 255) // 256 * 256:].view(torch.int32)[:strands]
    order = words.clone()
    assert torch.equal(order.sort().values, torch.arange(strands, dtype=torch.int32, device="cuda"))
    words[::3] = -1
    got = torch.full_like(want, float("nan"))
    generate_packed_ordered(d, params, got.view(-1, 4), workspace=ws)
    left_out = torch.zeros(strands, dtype=torch.bool, device="cuda")
    left_out[order[::3].long()] = True
    assert bool(got[left_out].isnan().all())
    assert torch.equal(got[~left_out], want[~left_out])


@pytest.mark.parametrize("noise", [False, True])
@pytest.mark.parametrize("cvs", [2, 16, 32, 33, 64, 128])
def test_tiles_read_and_registered_again(sphere, cvs, noise):
    """The tile that is read is the one in use: registered again, points are
    the same bits (a lane-group kernel's differ), and it reads the same.  A
    lane-walk tile of any CTA size leaves the bits alone; the autotuner
    returns what it leaves in use."""
    import torch
    from nanoxgen_b200.generator import autotune, generate_packed, get_tile, set_tile
    d, params = sphere
    params = params.copy(strand_count=401, cvs_per_strand=cvs, noise_amplitude=0.1 if noise else 0.0)
    try:
        want = generate_packed(d, params).points
        builtin = get_tile(cvs, noise)
        set_tile(cvs, noise, *builtin)
        assert get_tile(cvs, noise) == builtin and builtin[0] == 1
        assert torch.equal(generate_packed(d, params).points, want)
        for block in (0, 32, 96, 1024):
            set_tile(cvs, noise, builtin[0], builtin[1], block)
            assert torch.equal(generate_packed(d, params).points, want)
        set_tile(cvs, noise, 32, 4, 64)
        assert get_tile(cvs, noise) == (32, 4, 64)
        tile, _ = autotune(d, params, torch.empty_like(want), repeats=1)
        assert get_tile(cvs, noise) == tile
    finally:
        set_tile(cvs, noise)
    assert get_tile(cvs, noise) == builtin


@pytest.mark.parametrize("cvs", [129, 200])
def test_short_ranges_of_long_strands(sphere, cvs):
    """Ranges of fewer strands than guides, past 128 CVs, have the whole
    call's points bit for bit (the walk's; the serial kernel's differ)."""
    import torch
    from nanoxgen_b200.generator import generate_packed
    d, params = sphere
    guides = d.header.guide_count
    params = params.copy(strand_count=3 * guides, cvs_per_strand=cvs)
    want = generate_packed(d, params).points.view(-1, cvs, 4)
    for first, count in ((0, guides - 1), (guides, 1), (2 * guides + 1, guides - 1)):
        got = generate_packed(d, params, first_strand=first, count=count).points.view(-1, cvs, 4)
        assert torch.equal(got, want[first:first + count])


def test_base_points_past_128_cvs(sphere):
    """The offset table samples guides for strands past 128 CVs with a fused
    multiply-add, as the serial kernel does: nearest-guide points are nearer to
    64 bits than from the reference's three roundings."""
    import torch
    from nanoxgen_b200.generator import generate_packed
    d, params = sphere
    cvs = 160
    params = params.copy(strand_count=400, cvs_per_strand=cvs, noise_amplitude=0.0, guide_support_scale=1e-6)
    out = generate_packed(d, params)
    got = out.points.cpu().numpy()[:, :3].reshape(-1, cvs, 3)
    roots = out.roots_numpy()
    g, F = d.asset.guides(), np.float32
    curves = d.asset.guide_cvs().reshape(len(g), -1, 3)
    # The nearest eligible guide, and its curve, at the strand's parameters.
    near = d.asset.stencil()[roots["triangle_index"]].astype(np.int64)
    ok = near < len(g)
    d2 = np.where(ok, ((roots["position"][:, None] - curves[np.where(ok, near, 0), 0]) ** 2).sum(-1), np.inf)
    guide = curves[near[np.arange(len(near)), d2.argmin(1)]]
    x = (np.arange(cvs, dtype=F) / F(cvs - 1)) * F(guide.shape[1] - 1)
    i = np.minimum(x.astype(np.int64), guide.shape[1] - 2)
    f = (x - i.astype(F))[None, :, None]
    a, b = guide[:, i], guide[:, i + 1]
    root = roots["position"][:, None]
    thrice = root + ((a * (F(1) - f) + b * f) - guide[:, :1])
    wide = root + (a.astype(np.float64) * (1.0 - f.astype(np.float64)) + b.astype(np.float64) * f - guide[:, :1])
    rms = lambda e: float(np.sqrt((e.astype(np.float64) ** 2).mean()))
    assert np.abs(got - wide).max() <= 8 * 2.0 ** -24 * np.abs(wide).max()
    assert rms(got - wide) < 0.97 * rms(thrice - wide)


@pytest.mark.parametrize("strands", [10, 63, 64, 100])
def test_long_strands_whatever_the_room(sphere, strands):
    """Past 128 CVs the kernel depends on the description, not on how much more
    room a workspace has than was asked for: the static scratch and a larger
    workspace give the bits of the queried one, below, at and above the 64
    guides."""
    import ctypes
    import torch
    from nanoxgen_b200 import _abi
    from nanoxgen_b200.generator import generate_packed, packed_output_descriptor
    d, params = sphere
    params = params.copy(strand_count=strands, cvs_per_strand=140)
    want = generate_packed(d, params).points
    asked = int(_abi.lib().nxg_packed_workspace_size(ctypes.byref(d.desc), ctypes.byref(params), strands))
    room = torch.empty(asked + (8 << 20), dtype=torch.uint8, device="cuda")
    frame, config = _abi.DeformedDesc(), _abi.LaunchConfig(128)
    stream = torch.cuda.current_stream().cuda_stream
    for scratch in (False, True):
        got = torch.full_like(want, float("nan"))
        call = [ctypes.byref(x) for x in (d.desc, frame, params, packed_output_descriptor(got), config)]
        if scratch:
            code = _abi.lib().nxg_generate_packed_static_scratch(*call, stream)
        else:
            code = _abi.lib().nxg_generate_packed(*call, room.data_ptr(), room.numel(), stream)
        assert code == 0
        assert torch.equal(got, want)
