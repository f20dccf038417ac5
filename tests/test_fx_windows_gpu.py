"""The Classic FX pass where its branches meet: NoiseFX from moving lattice
windows against the per-CV lookups (a constant ramp as the magnitude) and a
64-bit restatement; and cLength, measured only where a program binds it,
against plans that bind it everywhere."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DOMAIN = np.array([0.419276, 0.184247, 0.805721], np.float32).astype(np.float64)


def _curves(S, P, seed=0, step=0.03):
    """Random walks (a third of them dropped already), a tenth of them far shorter than the rejection length."""
    rng = np.random.default_rng([S, P, seed])
    steps = step * (np.array([0.0, 0.0, 1.0]) + 0.5 * rng.normal(size=(S, P, 3)))
    steps[rng.random(S) < 0.1] *= 1e-5
    pts = np.empty((S, P, 4), np.float32)
    pts[..., :3] = rng.normal(size=(S, 1, 3)) + np.cumsum(steps, 1)
    pts[..., 3] = 0.01
    normals = rng.normal(size=(S, 3))
    normals = (normals / np.linalg.norm(normals, axis=1, keepdims=True)).astype(np.float32)
    tangents = rng.normal(size=(S, 3)).astype(np.float32)
    return pts, normals, tangents, np.where(rng.random(S) < 0.3, 0, P).astype(np.int32)


def _apply(curves, primitive, effects, clumps=()):
    from nanoxgen_b200 import _abi
    from nanoxgen_b200.classic import ClumpGuides, FxPlan, classic_fx_apply
    from nanoxgen_b200.generator import PackedCurves
    pts, normals, tangents, counts = curves
    S, P = pts.shape[:2]
    roots = np.zeros(S, _abi.ROOT_DTYPE)
    roots["normal"] = normals
    roots["position"] = pts[:, 0, :3]
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    c = PackedCurves(strand_count=S, cvs_per_strand=P, points=put(pts.reshape(-1, 4)),
                     roots=put(roots.view(np.int32).reshape(S, -1)),
                     root_uvs=put(np.full((S, 2), 0.5, np.float32)), point_counts=put(counts))
    status = classic_fx_apply(FxPlan(primitive, effects, 3, "description"), c, put(tangents),
                              clumps=[ClumpGuides(*g) for g in clumps])
    assert status.cpu().tolist() == [0, 0]
    return c.points.cpu().numpy().reshape(S, P, 4), c.point_counts.cpu().numpy()


def _gradient_noise(grads, p):
    """2 (noise - 0.5) in 64 bits at points [..., 3]."""
    cell = np.floor(p)
    w, i = p - cell, cell.astype(np.int64)
    v = []
    for corner in range(8):
        o = np.array([corner & 1, corner >> 1 & 1, corner >> 2])
        s = np.zeros(p.shape[:-1], np.int64)
        for k in range(3):
            s = (s * 1664525 + i[..., k] + o[k] + 1013904223) & 0xffffffff
        s ^= s >> 11
        s ^= (s << 7) & 0x9d2c5680
        s ^= (s << 15) & 0xefc60000
        s ^= s >> 18
        v.append((grads[s & 0xff] * (w - o)).sum(-1))
    a = w * w * w * (w * (w * 6.0 - 15.0) + 10.0)
    for k in range(3):
        v = [(1.0 - a[..., k]) * v[2 * j] + a[..., k] * v[2 * j + 1] for j in range(len(v) // 2)]
    return v[0]


def _noise_fx(curves, grads, frequency, magnitude, correlation):
    """apply_noise with preserveLength 0 in 64 bits; also the largest noise coordinate."""
    pts, normal, v = (a.astype(np.float64) for a in curves[:3])
    base, P = pts[..., :3], pts.shape[1]
    unit = lambda a: a / np.linalg.norm(a, axis=-1, keepdims=True)
    dot = lambda a, b: (a * b).sum(-1, keepdims=True)
    seg = np.linalg.norm(np.diff(base, axis=1), axis=-1)
    arc = np.concatenate([np.zeros_like(seg[:, :1]), np.cumsum(seg, 1)], 1)
    distance = arc * np.maximum(0.5 / arc[:, -1:], frequency)
    domain = np.repeat(((base[:, 0] + DOMAIN) * (100.0 * (1.0 - 0.01 * correlation) ** 2))[:, None], P, 1)
    n = np.stack([_gradient_noise(grads, domain + distance[..., None] * np.eye(3)[ax]) for ax in range(3)], -1)
    n *= 0.5 * magnitude
    v, tangent, out = unit(v), normal, base.copy()
    for c in range(P):
        ahead = unit(base[:, c + 1] - base[:, c]) if c + 1 < P else tangent
        axis, d = unit(np.cross(tangent, ahead) + 1e-30), np.clip(dot(tangent, ahead), -1.0, 1.0)
        turned = d * v + (1.0 - d) * dot(axis, v) * axis + np.sqrt(1.0 - d * d) * np.cross(axis, v)
        v = np.where(d < 1.0 - 5e-13, unit(turned), v)
        b = unit(np.cross(v, ahead))
        if c:
            out[:, c] += v * n[:, c, :1] + b * n[:, c, 1:2] + np.cross(b, v) * n[:, c, 2:]
        tangent = ahead
    return out, np.abs(domain).max(initial=0.0) + distance.max(initial=0.0)


@pytest.mark.parametrize("strands,cvs,frequency,correlation", [
    (1, 2, 4, 20), (33, 3, 8, 30), (500, 5, 200, 30), (500, 24, 8, 30), (500, 24, 40, 100), (500, 17, 500, 0),
    (777, 32, 3, 60), (129, 64, 20, 90)])
def test_noise_windows(cuda, nxg_lib, strands, cvs, frequency, correlation):
    """Segments of a small part of a lattice cell up to ones longer than a window (frequency 200 and 500)."""
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    w = fixtures.plain_sphere(strands=10, cvs=8)
    asset = build_asset(w.build_input, w.stencil_slots)
    grads = asset.section("noise_gradients", np.float32, 256, 3).astype(np.float64)
    curves = _curves(strands, cvs)
    noise = dict(mask="1", magnitude="0.05", magnitudeScale="1", frequency=str(frequency),
                 correlation=str(correlation), preserveLength="0")
    got, kept = _apply(curves, {"width": "0.01"}, [("noise", noise)])
    ramp, same = _apply(curves, {"width": "0.01"}, [("noise", dict(noise, magnitudeScale="rampUI(0,1,1:1,1,1)"))])
    np.testing.assert_array_equal(kept, same)
    short = np.linalg.norm(np.diff(curves[0][..., :3].astype(np.float64), axis=1), axis=-1).sum(1) < 5e-4
    np.testing.assert_array_equal(kept, np.where(short, 0, curves[3]))
    live = kept != 0
    # Both take the noise at the same coordinates: a value of at most 1 from
    # some 20 roundings of 2^-24, and the last sums at the points' size.
    size = np.abs(got[..., :3]).max()
    assert np.abs(got[live] - ramp[live])[..., :3].max(initial=0.0) <= 0.025 * 40 * 2.0 ** -24 + size * 2.0 ** -22
    # Against 64 bits: a coordinate's error (a rounding per segment of the
    # distance) times the noise's slope (below 4), and the frame's, a few
    # roundings per CV.
    want, x = _noise_fx([a[live] for a in curves], grads, frequency, 0.05, correlation)
    bound = 0.025 * (4.0 * x * (cvs + 16) * 2.0 ** -24 + cvs * 64 * 2.0 ** -24) + size * 2.0 ** -21
    assert np.abs(got[live][..., :3] - want).max(initial=0.0) <= bound


NOISE = dict(mask="1", magnitude="0.03", magnitudeScale="1", frequency="8", correlation="30", preserveLength="40")
CLUMP = dict(mask="1", clump="0.6", clumpScale="0.1", noise="0.02", noiseScale="1", noiseFrequency="6",
             noiseCorrelation="40")
READ = "+0*$cLength"


@pytest.mark.parametrize("kinds,reader", [
    (("noise",), "taper"), (("clump",), "taper"), (("cut",), None), (("clump", "cut"), "cut"),
    (("clump", "clump", "cut"), "cut"), (("noise", "clump", "cut"), "cut"), (("cut", "clump", "noise"), "noise"),
    (("clump", "noise", "clump"), "taper"), ((), "width")])
def test_clength_where_it_is_read(cuda, nxg_lib, kinds, reader):
    """A plan that binds cLength at one place gives, bit for bit, what it gives with every attribute binding it."""
    curves = _curves(700, 12, seed=len(kinds))
    rng = np.random.default_rng(7)
    pts = curves[0]
    of = rng.integers(0, 16, 700).astype(np.uint32)
    of[rng.random(700) < 0.3] = 0xFFFFFFFF
    guide = (pts[:16, :, :3] - pts[:16, :1, :3] + 0.01, curves[1][:16], curves[2][:16], rng.random((16, 2)),
             np.arange(16), of)

    def plan(extra):
        primitive = {"length": "0.8" + extra, "width": ("0.01+0.001*$cLength" if reader == "width" else "0.01") + extra,
                     "taper": ("0.5*$cLength" if reader == "taper" else "0.5") + extra, "taperStart": "0.2"}
        made = {"noise": dict(NOISE, magnitude="0.1*$cLength" if reader == "noise" else "0.03"), "clump": dict(CLUMP),
                "cut": {"amount": "0.5*$cLength" if reader == "cut" else "0.05"}}
        # (The guide noise stays as it is: bound to cLength it is not shared by a guide's strands.)
        add = lambda k, a: k == "cut" or a in ("mask", "magnitude", "clump", "clumpScale")
        return primitive, [(k, {a: v + extra if add(k, a) else v for a, v in made[k].items()}) for k in kinds]

    clumps = [guide] * kinds.count("clump")
    (a, na), (b, nb) = (_apply(curves, *plan(extra), clumps=clumps) for extra in ("", READ))
    np.testing.assert_array_equal(na, nb)
    assert 0 < (na == 12).sum() < 700
    np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
