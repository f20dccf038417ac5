"""The streaming passes at the ends of their tiles: the flat payload pass
(128-point tiles turned in shared memory) bit for bit against the same
operations in numpy, with misaligned arrays, tails and batch boundaries inside
a tile; and the curve-cache check's 1,024-element tiles against the host
validator."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

AFFINE = (0.98, -0.17, 0.0, 0.5, 0.17, 0.98, 0.25, -0.25, 0.0, 0.125, 1.0, 2.0)


def _transform(p, m):
    """curve_payload.cpp:127-133 in float32, one rounding per operation."""
    m = np.float32(m).reshape(3, 4)
    return np.stack([((m[r, 0] * p[:, 0] + m[r, 1] * p[:, 1]) + m[r, 2] * p[:, 2]) + m[r, 3] for r in range(3)], 1)


@pytest.mark.parametrize("identity", [True, False])
@pytest.mark.parametrize("strands,cvs,batch,samples,shift", [
    (1, 2, 65536, 1, 0), (64, 2, 7, 2, 0), (32, 4, 65536, 0, 0), (43, 3, 5, 1, 0), (1000, 13, 65536, 2, 1),
    (1000, 13, 77, 2, 0), (1024, 16, 64, 3, 0), (777, 24, 100, 1, 3), (5000, 32, 1000, 2, 0)])
def test_flat_payload_pass(cuda, nxg_lib, identity, strands, cvs, batch, samples, shift):
    from nanoxgen_b200.payload import IDENTITY, Curves, build_curve_batches
    gen = torch.Generator("cuda").manual_seed(strands * 31 + cvs)
    N = strands * cvs

    def array(n, width):  # `shift` floats off the allocation's alignment
        flat = torch.randn(n * width + shift, generator=gen, device="cuda")[shift:]
        return flat.view(n, width) if width > 1 else flat

    sets = [array(N, 3) for _ in range(samples + 1)]
    widths = array(N, 1)
    uvs = torch.rand((strands, 2), generator=gen, device="cuda")
    m = IDENTITY if identity else AFFINE
    b = build_curve_batches(Curves(sets[0], strands, cvs, None, widths, uvs),
                            [(0.5 * k, Curves(p, strands, cvs)) for k, p in enumerate(sets[1:])],
                            max_strands_per_batch=batch, transform=m, radius_scale=1.5)
    host = [p.cpu().numpy() for p in sets]
    moved = host if identity else [_transform(p, m) for p in host]
    want = np.concatenate([moved[0], (widths.cpu().numpy() * (np.float32(0.5) * np.float32(1.5)))[:, None]], 1)
    assert np.array_equal(b.points.cpu().numpy().view(np.uint32), want.view(np.uint32))
    firsts = [s * cvs for s in range(0, strands, batch)] + [N]
    assert b.batch_first_point.cpu().tolist() == firsts
    assert (b.point_counts.cpu().numpy() == cvs).all() and torch.equal(b.root_uvs, uvs)
    if samples:
        rows = np.concatenate([p[lo:hi] for lo, hi in zip(firsts, firsts[1:]) for p in moved[1:]])
        assert np.array_equal(b.motion_points.cpu().numpy().view(np.uint32), rows.view(np.uint32))


@pytest.mark.parametrize("strands", [1, 255, 1023, 1024, 1025, 5000])
def test_cache_check_tiles(cuda, nxg_lib, strands):
    """Valid caches, then one bad element at the first, last and middle index
    of each section: the device's message is the host's."""
    from nanoxgen_b200 import curve_cache as cc
    from test_curve_cache import aligned_copy, header_of, random_cache, rehash, section
    good = aligned_copy(cc.build_curve_cache(**random_cache(np.random.default_rng(strands), strands=strands, samples=2)))

    def device(blob):
        d = cc.DeviceCurveCache(blob)
        d.validate()
        return d.outcome()

    h = header_of(good)
    assert device(good) == ("", h.point_count, cc.point_checksum(good))
    points, total = h.point_count, h.point_count * 2
    for field, dtype, width, count, value in (
            ("points_offset", np.float32, 4, points, np.nan), ("texcoords_offset", np.float32, 2, points, np.inf),
            ("motion_points_offset", np.float32, 3, total, np.nan), ("patch_uvs_offset", np.float32, 2, strands, np.nan),
            ("face_uvs_offset", np.float32, 2, strands, np.inf), ("point_counts_offset", np.uint32, 1, strands, 1)):
        assert getattr(h, field)
        for i in {0, count // 2, count - 1}:
            blob = aligned_copy(good)
            section(blob, field, dtype)[i * width] = value
            rehash(blob)
            expected = cc.validate_curve_cache(blob)
            assert expected and device(blob)[0] == expected
