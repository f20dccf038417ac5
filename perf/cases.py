"""The calls a user of the strand generator makes, at the sizes they make them.

Every case is a dict of plain values; ``prepare`` makes what a program has in
hand before the call (an uploaded .nxg asset, parameters, output buffers, a
Classic plan, a curve set), ``run`` is one pass through the public API and
``exact`` the same result in 64 bits from plain torch and numpy.  Grooms stand
on a displaced UV sphere, with guides along the surface normal as in
``nanoxgen_b200.fixtures``.  The mesh of a case is fixed, as a character's is;
guides, curves, deformation and the strand seed follow the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from nanoxgen_b200 import classic, curve_cache, fixtures, generator, payload
from nanoxgen_b200._abi import GenerationParams
from nanoxgen_b200.asset import AssetBuildInput, GuideSet, build_asset_device

DEVICE = "cuda"
TRANSFORM = (0.98, -0.17, 0.0, 0.5, 0.17, 0.98, 0.0, -0.25, 0.0, 0.0, 1.0, 2.0)
FX_LENGTH = "0.5*(1+0.4*noise($Prefg*6))"
FX_EFFECTS = (("noise", dict(mask="1", magnitude="0.03", magnitudeScale="1", frequency="8", correlation="30",
                             preserveLength="40")),
              ("clump", dict(mask="1", clump="0.6", clumpScale="0.1", noise="0.02", noiseScale="1",
                             noiseFrequency="6", noiseCorrelation="40")),
              ("cut", {"amount": "$cLength*0.1"}))


# ------------------------------------------------------------------- cases

def _frame(strands, cvs, noise, *, lon=400, rings=251, guides=4096, slots=8, preserve=0.0, power=2.0):
    return dict(kind="frame", strands=strands, cvs=cvs, noise=noise, lon=lon, rings=rings, guides=guides, slots=slots,
                preserve=preserve, power=power)


def listed():
    return [
        # Interactive grooming: a small patch regenerated on every stroke.
        dict(_frame(2000, 16, 0.1, lon=32, rings=33, guides=64, slots=4), name="patch_2k_x16_noise"),
        # Viewport preview of a groom, noise off (the reference's published 100,000 x 12 size).
        dict(_frame(100_000, 12, 0.0), name="preview_100k_x12"),
        # One large description at render density.
        dict(_frame(1_000_000, 32, 0.2), name="render_1m_x32_noise"),
        # Long hair: more CVs than the short-strand kernels hold, lengths preserved, odd sizes.
        dict(_frame(150_001, 61, 0.1, guides=1500, preserve=0.4), name="long_150k_x61_noise"),
        # Very long strands (braids, ropes) past 128 CVs.
        dict(_frame(20_011, 160, 0.1, guides=512, preserve=0.4, power=1.5), name="rope_20k_x160_noise"),
        # Motion blur: five shutter samples of a deforming description.
        dict(kind="motion", strands=250_000, cvs=24, noise=0.15, lon=400, rings=251, guides=2048, slots=8, samples=5,
             name="motion_250k_x24_5"),
        # A character: nine descriptions on one mesh in one frame.
        dict(kind="batch", descriptions=9, low=20_000, high=1_000_000, lon=1000, rings=251, sizes=2590,
             name="character_9"),
        # Classic length and width expressions over a dense fur.
        dict(kind="classic", strands=4_000_000, cvs=24, lon=400, rings=251, guides=4096, slots=8,
             name="fur_4m_x24_classic"),
        # Classic FX modules over a generated frame.
        dict(kind="fx", strands=500_000, cvs=24, lon=400, rings=251, guides=4096, slots=8, name="fx_500k_x24"),
        # Renderer payload of a frame with one motion sample.
        dict(kind="payload", strands=1_000_000, cvs=32, variable=False, resample=0, samples=1, batch=65536,
             name="payload_1m_x32"),
        # An ingested curve cache checked before use.
        dict(kind="cache", strands=400_000, cvs=24, name="cache_400k_x24"),
        # The stencil search of an asset build.
        dict(kind="stencil", lon=400, rings=251, guides=4096, slots=8, name="stencil_200k_tris"),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["frame"] * 8 + ["long"] * 2 + ["motion", "batch", "classic", "fx", "payload", "payload", "cache",
                                                       "stencil"])
    mesh = dict(lon=_log(rng, 24, 500), rings=_log(rng, 17, 251), guides=_log(rng, 48, 4096), slots=rng.choice([4, 8, 8]))
    if kind == "frame":
        return _frame(_log(rng, 300, 1_000_000), rng.randint(2, 32), rng.choice([0.0, round(rng.uniform(0.05, 0.2), 3)]),
                      preserve=rng.choice([0.0, 0.0, 0.4]), power=rng.choice([2.0, 2.0, 2.0, 1.5, 3.0]), **mesh)
    if kind == "long":
        cvs = rng.randint(33, 200)
        return _frame(_log(rng, 300, 9_000_000 // cvs if cvs <= 128 else 3_000_000 // cvs), cvs,
                      rng.choice([0.0, 0.1, 0.1]), preserve=rng.choice([0.0, 0.4]), power=rng.choice([2.0, 1.5]), **mesh)
    if kind == "motion":
        return dict(kind="motion", strands=_log(rng, 2000, 250_000), cvs=rng.randint(4, 32),
                    noise=rng.choice([0.0, 0.15]), samples=rng.randint(2, 5), **mesh)
    if kind == "batch":
        low = _log(rng, 500, 20_000)
        return dict(kind="batch", descriptions=rng.randint(2, 9), low=low, high=low * rng.randint(2, 20),
                    lon=mesh["lon"], rings=mesh["rings"], sizes=rng.randint(1, 10_000))
    if kind == "classic":
        return dict(kind="classic", strands=_log(rng, 2000, 4_000_000), cvs=rng.randint(4, 24), **mesh)
    if kind == "fx":
        return dict(kind="fx", strands=_log(rng, 2000, 500_000), cvs=rng.randint(5, 24), **mesh)
    if kind == "payload":
        variable = rng.random() < 0.5
        return dict(kind="payload", strands=_log(rng, 500, 600_000), cvs=rng.randint(4, 48), variable=variable,
                    resample=rng.choice([0, rng.randint(2, 40)]), samples=rng.randint(0, 2),
                    batch=rng.choice([65536, rng.randint(300, 65536)]))
    if kind == "cache":
        return dict(kind="cache", strands=_log(rng, 500, 400_000), cvs=rng.randint(4, 24))
    return dict(kind="stencil", **mesh)


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=4)
def _mesh(lon, rings):
    """Positions, uvs, triangles, vertex normals and the running share of the area of the displaced sphere."""
    pos, uv, tris = fixtures.sphere_mesh(lon, rings, fixtures.displaced_sphere_radius)
    area = np.cumsum(fixtures.triangle_areas(pos, tris))
    return pos, uv, tris, _vertex_normals(pos, tris), area / area[-1]


def _vertex_normals(pos, tris):
    p, t = pos.astype(np.float64), tris.astype(np.int64)
    n = np.cross(p[t[:, 1]] - p[t[:, 0]], p[t[:, 2]] - p[t[:, 0]])
    acc = np.stack([np.bincount(t.reshape(-1), np.repeat(n[:, k], 3), len(p)) for k in range(3)], 1)
    length = np.linalg.norm(acc, axis=1, keepdims=True)
    return np.where(length > 1e-30, acc / np.maximum(length, 1e-30), [0.0, 1.0, 0.0]).astype(np.float32)


def _guides(lon, rings, count, cvs, rng):
    """`count` guides of `cvs` CVs along the surface normal, bent a little CV by CV (a tenth of the CV spacing)."""
    pos, uv, tris, normals, share = _mesh(lon, rings)
    tri = np.minimum(np.searchsorted(share, rng.random(count)), len(tris) - 1)
    r1, r2 = np.sqrt(rng.random(count)), rng.random(count)
    b = np.stack([1.0 - r1, r1 * (1.0 - r2), r1 * r2], 1)
    at = lambda a: np.einsum("gkc,gk->gc", a.astype(np.float64)[tris[tri]], b)
    root, n = at(pos), at(normals)
    n /= np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-30)
    reach = rng.uniform(0.3, 0.6, count)[:, None, None] * np.linspace(0.0, 1.0, cvs)[None, :, None]
    curve = root[:, None] + n[:, None] * reach + rng.normal(0.0, 0.045 / max(cvs - 1, 7), (count, cvs, 3))
    curve[:, 0] = root
    return GuideSet(np.full(count, cvs, np.uint32), curve.astype(np.float32).reshape(-1, 3), n.astype(np.float32),
                    at(uv).astype(np.float32), tri.astype(np.uint32), b[:, 1:].astype(np.float32),
                    np.zeros(count, np.float32))


def _asset(lon, rings, guides, slots, cvs, rng):
    pos, uv, tris, normals, _ = _mesh(lon, rings)
    gs = _guides(lon, rings, guides, min(max(cvs, 8), 32), rng)
    return build_asset_device(AssetBuildInput(pos, tris, gs, normals, uv), slots)


def _params(case, seed, **more):
    noise = case.get("noise", 0.0)
    return GenerationParams(**{**dict(strand_count=case["strands"], cvs_per_strand=case["cvs"], seed=11 + seed % 100_003,
                                      root_width=0.02, tip_width=0.002, noise_amplitude=noise, noise_frequency=9.0,
                                      noise_preserve_length=case.get("preserve", 0.0),
                                      guide_weight_power=case.get("power", 2.0)), **more})


def _groom(case, seed):
    """(asset, parameters) of a case with one description."""
    rng = np.random.default_rng([seed, 5])
    return (_asset(case["lon"], case["rings"], case["guides"], case["slots"], case["cvs"], rng), _params(case, seed))


def _descriptions(case):
    """Per description of a frame of several: strands, CVs, guides, slots, noise, mesh."""
    rng = np.random.default_rng(case["sizes"])
    lo, hi = math.log(case["low"]), math.log(case["high"])
    counts = [int(round(math.exp(rng.uniform(lo, hi)))) for _ in range(case["descriptions"])]
    cvs = [int(rng.choice(fixtures.BATCH_CVS)) for _ in counts]
    return [dict(strands=s, cvs=p, guides=int(rng.integers(512, 2049)), slots=int(rng.choice([4, 8])),
                 noise=float(rng.uniform(0.05, 0.2)) if rng.random() < 2 / 3 else 0.0, lon=case["lon"],
                 rings=case["rings"]) for s, p in zip(counts, cvs)]


def _deformation(case, seed, asset):
    """Per shutter time: positions, normals and guide CVs moved by a sinusoid per vertex, guides with their roots."""
    rng = np.random.default_rng([seed, 6])
    pos, _, tris, _, _ = _mesh(case["lon"], case["rings"])
    phase = rng.uniform(0.0, 2.0 * math.pi, len(pos))
    direction = rng.normal(size=pos.shape)
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    g = asset.guides()
    b = np.concatenate([1.0 - g["barycentric"].sum(1, keepdims=True), g["barycentric"]], 1)
    frames = []
    for t in np.linspace(0.0, 1.0, case["samples"]):
        disp = 0.01 * np.sin(2.0 * math.pi * t + phase)[:, None] * direction
        moved = (pos + disp).astype(np.float32)
        roots = np.einsum("gkc,gk->gc", disp[tris[g["triangle_index"]]], b)
        cvs = asset.guide_cvs() + np.repeat(roots, g["cv_count"], axis=0)
        frames.append((moved, _vertex_normals(moved, tris), cvs.astype(np.float32)))
    return np.linspace(0.0, 1.0, case["samples"]).astype(np.float32), frames


def _across(n):
    """A unit tangent per normal: across the z axis, the y axis near the poles."""
    n = n.astype(np.float64)
    t = np.cross(n, np.where(np.abs(n[:, 2:]) < 0.999, [[0.0, 0.0, 1.0]], [[0.0, 1.0, 0.0]]))
    return (t / np.maximum(np.linalg.norm(t, axis=1, keepdims=True), 1e-30)).astype(np.float32)


def _clump_guides(asset, cvs):
    """The asset's own guides at `cvs` CVs, with normals, tangents and uvs."""
    g = asset.guides()
    curves = asset.guide_cvs().reshape(len(g), -1, 3)
    x = np.linspace(0.0, curves.shape[1] - 1, cvs)
    i = np.minimum(x.astype(np.int64), curves.shape[1] - 2)
    f = (x - i)[None, :, None]
    normals = np.ascontiguousarray(g["root_normal"])
    return (curves[:, i] * (1.0 - f) + curves[:, i + 1] * f).astype(np.float32), normals, _across(normals), g["root_uv"]


def _curves(case, seed):
    """A curve set on the device: per strand a count, points as a walk from a random root, widths, root uvs."""
    gen = torch.Generator(DEVICE).manual_seed(seed * 7919 + 13)
    S, P = case["strands"], case["cvs"]
    rand = lambda *shape: torch.rand(shape, generator=gen, device=DEVICE)
    counts = None
    if case["variable"]:
        counts = torch.randint(max(2, P // 2), P + 1, (S,), generator=gen, device=DEVICE, dtype=torch.int32)
    N = S * P if counts is None else int(counts.sum())
    owner = (torch.arange(N, device=DEVICE) // P if counts is None
             else torch.repeat_interleave(torch.arange(S, device=DEVICE), counts.long()))
    points = 2.0 * rand(S, 3)[owner] + 0.2 * rand(N, 3)
    sets = [points] + [points + 0.01 * (k + 1) * rand(N, 3) for k in range(case["samples"])]
    widths, uvs = 0.002 + 0.01 * rand(N), rand(S, 2)
    fixed = 0 if case["variable"] else P
    base = payload.Curves(sets[0], S, fixed, counts, widths, uvs)
    return base, [(0.25 * (k + 1), payload.Curves(p, S, fixed, counts)) for k, p in enumerate(sets[1:])]


def _root_uv_strands(S, P, rng):
    root = rng.normal(size=(S, 1, 3)).astype(np.float32)
    xyz = root + np.cumsum(rng.random((S, P, 3), dtype=np.float32) * np.float32(0.02), axis=1, dtype=np.float32)
    w = np.broadcast_to(np.linspace(0.01, 0.001, P, dtype=np.float32)[None, :, None], (S, P, 1))
    return np.concatenate([xyz, w], 2).reshape(-1, 4)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(kind=kind)
    if kind == "batch":
        rng = np.random.default_rng([seed, 5])
        parts = [(_asset(d["lon"], d["rings"], d["guides"], d["slots"], d["cvs"], rng), _params(d, seed + k))
                 for k, d in enumerate(_descriptions(case))]
        state["runner"] = generator.BatchRunner([generator.DeviceAsset(a, DEVICE) for a, _ in parts],
                                                [p for _, p in parts])
    elif kind == "payload":
        state["base"], state["samples"] = _curves(case, seed)
        state["options"] = dict(max_strands_per_batch=case["batch"], resample_cv_count=case["resample"],
                                transform=TRANSFORM)
    elif kind == "cache":
        rng = np.random.default_rng([seed, 7])
        S, P = case["strands"], case["cvs"]
        blob = curve_cache.build_curve_cache(np.full(S, P, np.uint32), _root_uv_strands(S, P, rng),
                                             patch_uvs=rng.random((S, 2), dtype=np.float32))
        state["cache"] = curve_cache.DeviceCurveCache(blob, DEVICE)
    elif kind == "stencil":
        pos, _, tris, _, _ = _mesh(case["lon"], case["rings"])
        gs = _guides(case["lon"], case["rings"], case["guides"], 2, np.random.default_rng([seed, 5]))
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)
        state["inputs"] = (put(pos), put(tris.view(np.int32)), put(gs.cvs.reshape(-1, 2, 3)[:, 0]), put(gs.root_normals))
        state["slots"] = case["slots"]
    else:
        asset, params = _groom(case, seed)
        S, P = case["strands"], case["cvs"]
        state.update(asset=generator.DeviceAsset(asset, DEVICE), params=params)
        if kind == "motion":
            times, frames = _deformation(case, seed, asset)
            put = lambda a: torch.from_numpy(a).to(DEVICE)
            state.update(times=times, frames=[generator.DeformedGeometry(*map(put, f)) for f in frames],
                         outputs=[generator.allocate_outputs(S, P, DEVICE) for _ in frames])
        else:
            state["outputs"] = dict(zip(("points", "roots", "root_uvs", "point_counts"),
                                        generator.allocate_outputs(S, P, DEVICE)))
        if kind == "classic":
            state["plan"] = classic.ScalarPlan(classic.Expression.classic(fixtures.CLASSIC_LENGTH, "length"),
                                               classic.Expression.classic(fixtures.CLASSIC_WIDTH, "width"))
        if kind == "fx":
            roots = generator.generate_packed(state["asset"], params, **state["outputs"]).roots_numpy()
            state["plan"] = classic.FxPlan(dict(length=FX_LENGTH, width=fixtures.CLASSIC_WIDTH, taper="0.6",
                                                taperStart="0.3"), FX_EFFECTS, 3, "description")
            state["plan"].upload(DEVICE)
            state["tangents"] = torch.from_numpy(_across(roots["normal"])).to(DEVICE)
            curves, normals, tangents, uvs = _clump_guides(asset, P)
            state["clumps"] = [classic.ClumpGuides(curves, normals, tangents, uvs, np.arange(len(curves)),
                                                   asset.stencil()[roots["triangle_index"], 0], device=DEVICE)]
    return state


# --------------------------------------------------------------------- run

def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["runner"].run()
        return [dict(points=c.points, counts=c.point_counts, roots=c.roots, uvs=c.root_uvs)
                for c in state["runner"].curves()]
    if kind == "payload":
        b = payload.build_curve_batches(state["base"], state["samples"], **state["options"])
        return dict(counts=b.point_counts, points=b.points, uvs=b.root_uvs, motion=b.motion_points,
                    first=b.batch_first_point, status=b.status)
    if kind == "cache":
        state["cache"].validate()
        return state["cache"].result
    if kind == "stencil":
        return generator.build_stencils(*state["inputs"], state["slots"])
    asset, params = state["asset"], state["params"]
    if kind == "motion":
        out = generator.generate_motion_packed(asset, params, state["frames"], state["times"], outputs=state["outputs"])
        return [dict(points=c.points, counts=c.point_counts, roots=c.roots, uvs=c.root_uvs) for c in out]
    more = {}
    if kind == "classic":
        more["scalars"], more["status"] = classic.root_scalars(asset, params, state["plan"])
        c = classic.generate_packed_classic(asset, params, more["scalars"], **state["outputs"])
    else:
        c = generator.generate_packed(asset, params, **state["outputs"])
    if kind == "fx":
        more["status"] = classic.classic_fx_apply(state["plan"], c, state["tangents"], clumps=state["clumps"])
    return dict(more, points=c.points, counts=c.point_counts, roots=c.roots, uvs=c.root_uvs)


# -------------------------------------------------------------------- work

def _frame_work(c):
    """Points and root records written; of the mesh what the strands touch, or all of it; guides read once.  Operations:
    the slots' weighted sum per point, with noise the frame and three gradient-noise values."""
    S, P, G = c["strands"], c["cvs"], c["guides"]
    T, V = 2 * c["lon"] * (c["rings"] - 1), (c["lon"] + 1) * c["rings"]
    mesh = min(T * (8 + 12 + 32) + V * 32, S * (8 + 12 + 32 + 96))
    each = 6 * c["slots"] + 9 + (150 if c.get("noise") else 0)
    return S * P * 16 + S * 60 + mesh + G * (56 + 12 * min(max(P, 8), 32)), S * P * each + S * 200


def work(case):
    kind = case["kind"]
    S, P = case.get("strands", 0), case.get("cvs", 0)
    if kind == "batch":
        parts = [_frame_work(d) for d in _descriptions(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "payload":
        n = S * P * (0.75 if case["variable"] else 1.0)
        m = S * case["resample"] or n
        b, f = n * (16 + 12 * case["samples"]) + m * (16 + 12 * case["samples"]) + S * 20, m * 18 * (1 + case["samples"])
    elif kind == "cache":
        b, f = S * (4 + 8) + S * P * 16, 0
    elif kind == "stencil":
        T, V = 2 * case["lon"] * (case["rings"] - 1), (case["lon"] + 1) * case["rings"]
        b, f = V * 12 + T * 44 + case["guides"] * 24, 0
    else:
        b, f = _frame_work(case)
        if kind == "motion":
            b, f = b * case["samples"], f * case["samples"]
        if kind == "classic":
            b, f = b + S * 16, f + S * 250
        if kind == "fx":
            b, f = b + S * (32 * P + 16), f + S * P * 450
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact

def _t(a):
    device = DEVICE if torch.cuda.is_available() else "cpu"
    a = np.ascontiguousarray(a)
    if a.dtype.kind == "u":
        a = a.astype(np.int64)
    t = torch.from_numpy(a.astype(np.float64) if a.dtype == np.float32 else a)
    return t.to(device)


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(v, fallback=None, least=1e-20):
    l2 = _dot(v, v)
    if fallback is None:
        fallback = torch.tensor([0.0, 1.0, 0.0], dtype=v.dtype, device=v.device)
    return torch.where(l2 > least, v / torch.sqrt(torch.clamp(l2, min=1e-60)), fallback)


def _hash32(x):
    for shift, factor in ((16, 0x7feb352d), (15, 0x846ca68b), (16, None)):
        x = x ^ (x >> shift)
        if factor:
            x = (x * (factor & 0xffff) + ((x * (factor >> 16) & 0xffff) << 16)) & 0xffffffff
    return x


def _random01(seed, strand, dim):
    return (_hash32(seed ^ _hash32((strand + 0x9e3779b9 * (dim + 1)) & 0xffffffff)) >> 8).double() / 16777216.0


def _noise(grads, p):
    """Gradient noise in [0, 1] at points [..., 3]."""
    cell = torch.floor(p)
    w, i = p - cell, cell.long()
    v = []
    for corner in range(8):
        o = torch.tensor([corner & 1, corner >> 1 & 1, corner >> 2], device=p.device)
        s = torch.zeros_like(i[..., 0])
        for k in range(3):
            s = (s * 1664525 + i[..., k] + o[k] + 1013904223) & 0xffffffff
        s = s ^ (s >> 11)
        s = s ^ ((s << 7) & 0x9d2c5680)
        s = s ^ ((s << 15) & 0xefc60000)
        s = s ^ (s >> 18)
        v.append((grads[s & 0xff] * (w - o)).sum(-1))
    a = w * w * w * (w * (w * 6.0 - 15.0) + 10.0)
    for k in range(3):
        v = [(1.0 - a[..., k]) * v[2 * j] + a[..., k] * v[2 * j + 1] for j in range(len(v) // 2)]
    return 0.5 * v[0] + 0.5


def _displace(base, normal, surface_u, domain, frequency, magnitude, grads, preserve, unit_axis):
    """The noise walk along base curves [S, P, 3]: the transported frame, the displaced points, the length rule."""
    S, P, _ = base.shape
    seg = torch.linalg.vector_norm(base[:, 1:] - base[:, :-1], dim=-1)
    arc = torch.cat([torch.zeros_like(seg[:, :1]), torch.cumsum(seg, 1)], 1)
    length = arc[:, -1:]
    f = torch.where(length > 0, torch.clamp(0.5 / torch.clamp(length, min=1e-60), min=frequency), frequency)
    distance = arc * f
    amount = []
    for axis in range(3):
        p = domain[:, None].repeat(1, P, 1)
        p[..., axis] += distance
        amount.append((_noise(grads, p) - 0.5) * magnitude)
    tangent, v, points = normal, surface_u, [base[:, 0]]
    for c in range(P):
        ahead = _unit(base[:, c + 1] - base[:, c], tangent) if c + 1 < P else tangent
        axis, d = torch.linalg.cross(tangent, ahead), _dot(tangent, ahead).clamp(-1.0, 1.0)
        l2 = _dot(axis, axis)
        if unit_axis:
            axis = axis / torch.sqrt(l2.clamp(min=1e-60))
        turned = d * v + (1.0 - d) * _dot(axis, v) * axis + torch.sqrt(1.0 - d * d) * torch.linalg.cross(axis, v)
        v = torch.where(l2 > (1e-12 if unit_axis else 0.0), _unit(turned), v)
        b = torch.linalg.cross(v, ahead)
        if unit_axis:
            b = _unit(b)
        if c:
            points.append(base[:, c] + v * amount[0][:, c, None] + b * amount[1][:, c, None] +
                          torch.linalg.cross(b, v) * amount[2][:, c, None])
        tangent = ahead
    points = torch.stack(points, 1)
    if preserve > 0.001:
        noisy = torch.linalg.vector_norm(points[:, 1:] - points[:, :-1], dim=-1).sum(1, keepdim=True)
        scale = (length * preserve + noisy * (1.0 - preserve)) / noisy.clamp(min=1e-60)
        scale = torch.where((noisy > 0) & ((noisy * (scale - 1.0)).abs() >= 1e-4), scale, 1.0)
        points = points[:, :1] + (points - points[:, :1]) * scale[..., None]
    return points


class _Exact:
    """One description in 64 bits: the asset's arrays, and strands by chunks."""

    def __init__(self, asset, params, frame=None):
        h, self.p, self.asset = asset.header, params, asset
        section = lambda name, dtype, n, w: _t(asset.section(name, dtype, n, w))
        self.rest, self.normals = _t(asset.positions()), _t(asset.normals())
        self.uv = section("texcoords", np.float32, h.vertex_count, 2)
        self.tris, self.stencil = _t(asset.triangles()), _t(asset.stencil())
        alias = asset.section("alias_table", np.uint32, h.triangle_count, 2)
        self.share, self.other = _t(alias[:, 0].copy().view(np.float32)), _t(alias[:, 1])
        self.grads = section("noise_gradients", np.float32, 256, 3)
        self.positions, cvs = self.rest, asset.guide_cvs()
        g = asset.guides()
        normals = _t(g["root_normal"])
        if frame is not None:
            self.positions, self.normals, cvs = _t(frame[0]), _t(frame[1]), frame[2]
            b = _t(g["barycentric"])
            b = torch.cat([1.0 - b.sum(1, keepdim=True), b], 1)
            normals = _unit((self.normals[self.tris[_t(g["triangle_index"])]] * b[..., None]).sum(1))
        P = params.cvs_per_strand
        curves = _t(cvs).view(len(g), -1, 3)
        self.t = torch.arange(P, device=curves.device).double() / (P - 1)
        x = self.t * (curves.shape[1] - 1)
        i = x.long().clamp(max=curves.shape[1] - 2)
        f = (x - i)[None, :, None]
        self.offsets = curves[:, i] * (1.0 - f) + curves[:, i + 1] * f - curves[:, :1]
        self.roots, self.guide_normals, self.support = curves[:, 0], normals, _t(g["support_radius"])

    def strands(self, first, end):
        """Root triangle, position, normal, uv, surface u and rest position, and base curves, of strands [first, end)."""
        p, s = self.p, torch.arange(first, end, device=self.t.device)
        T = len(self.tris)
        bucket = (_random01(p.seed, s, 0).float() * torch.tensor(float(T), device=s.device)).long().clamp(max=T - 1)
        tri = torch.where(_random01(p.seed, s, 1) < self.share[bucket], bucket, self.other[bucket])
        r1, r2 = torch.sqrt(_random01(p.seed, s, 2)), _random01(p.seed, s, 3)
        b = torch.stack([1.0 - r1, r1 * (1.0 - r2), r1 * r2], 1)[..., None]
        v = self.tris[tri]
        corner, uvs = self.positions[v], self.uv[v]
        root, n, uv = (corner * b).sum(1), _unit((self.normals[v] * b).sum(1)), (uvs * b).sum(1)
        e1, e2, d1, d2 = corner[:, 1] - corner[:, 0], corner[:, 2] - corner[:, 0], uvs[:, 1] - uvs[:, 0], uvs[:, 2] - uvs[:, 0]
        det = (d1[:, :1] * d2[:, 1:] - d1[:, 1:] * d2[:, :1])
        u = torch.where(det.abs() > 1e-12, (e1 * d2[:, 1:] - e2 * d1[:, 1:]) / torch.where(det == 0, 1.0, det), 0.0)
        u = u - n * _dot(u, n)
        z = torch.where(n[:, 2:].abs() < 0.999, torch.tensor([0.0, 0.0, 1.0], device=s.device).double(),
                        torch.tensor([0.0, 1.0, 0.0], device=s.device).double())
        u = _unit(u, _unit(torch.linalg.cross(n, z)))
        gi = self.stencil[tri]
        ok = gi < len(self.roots)
        gi = torch.where(ok, gi, 0)
        d2 = ((root[:, None] - self.roots[gi]) ** 2).sum(-1)
        ok &= (n[:, None] * self.guide_normals[gi]).sum(-1) >= p.normal_rejection_cos
        r = self.support[gi] * p.guide_support_scale
        w = torch.where(ok & (d2 < r * r), (1.0 - torch.sqrt(d2) / r).clamp(min=0.0) ** p.guide_weight_power, 0.0)
        total = w.sum(1, keepdim=True)
        nearest = torch.where(ok, d2, math.inf).argmin(1, keepdim=True)
        one = torch.zeros_like(w).scatter_(1, nearest, 1.0) * ok.any(1, keepdim=True)
        w = torch.where(total > 1e-12, w / total.clamp(min=1e-60), one)
        off = torch.zeros((len(s), len(self.t), 3), dtype=torch.float64, device=s.device)
        for j in range(gi.shape[1]):
            off += self.offsets[gi[:, j]] * w[:, j, None, None]
        lost = ((total <= 1e-12) & ~ok.any(1, keepdim=True))[..., None]
        off = torch.where(lost, n[:, None] * self.t[None, :, None], off)
        return dict(tri=tri, root=root, normal=n, uv=uv, u=u, rest=(self.rest[v] * b).sum(1),
                    base=root[:, None] + off * p.length_scale)

    def curves(self, s):
        p = self.p
        if p.noise_amplitude == 0.0:
            return s["base"]
        domain = (s["rest"] + torch.tensor([0.419276, 0.184247, 0.805721], device=self.t.device)) * \
            (100.0 * (1.0 - p.noise_correlation) ** 2)
        return _displace(s["base"], s["normal"], s["u"], domain, p.noise_frequency,
                         p.noise_mask * p.noise_amplitude * self.t, self.grads, p.noise_preserve_length, False)

    def result(self, finish=None):
        """Points with radii and uvs of every strand; `finish(strands, curves, radii)` applies what follows."""
        S, P = self.p.strand_count, self.p.cvs_per_strand
        points = torch.empty((S, P, 4), dtype=torch.float64)
        uvs = torch.empty((S, 2), dtype=torch.float64)
        more = []
        step = max(1, 3_000_000 // P)
        radii = 0.5 * (self.p.root_width * (1.0 - self.t) + self.p.tip_width * self.t)
        for first in range(0, S, step):
            end = min(S, first + step)
            s = self.strands(first, end)
            c, r = self.curves(s), radii.expand(end - first, P)
            if finish is not None:
                c, r, extra = finish(s, c, r)
                more.append(extra)
            points[first:end, :, :3], points[first:end, :, 3], uvs[first:end] = c.cpu(), r.cpu(), s["uv"].cpu()
        return dict(points=points.reshape(-1, 4), counts=None, roots=None, uvs=uvs), more


def _spline(curves, t):
    """The uniform cubic B-spline through end-extrapolated curves [S, P, 3] at parameters t [k] or [S, k]."""
    S, P, _ = curves.shape
    t = t.expand(S, -1) if t.dim() == 1 else t
    c = torch.cat([2.0 * curves[:, :1] - curves[:, 1:2], curves, 2.0 * curves[:, -1:] - curves[:, -2:-1]], 1)
    x = t * (P - 1)
    i = x.long().clamp(max=P - 2)
    f = (x - i)[..., None]
    w = ((1.0 - f) ** 3, 3.0 * f ** 3 - 6.0 * f ** 2 + 4.0, -3.0 * f ** 3 + 3.0 * f ** 2 + 3.0 * f + 1.0, f ** 3)
    at = lambda k: torch.gather(c, 1, (i + k)[..., None].expand(-1, -1, 3))
    p = sum(at(k) * w[k] for k in range(4)) / 6.0
    p = torch.where((t < 1e-7)[..., None], curves[:, :1], p)
    return torch.where((t > 1.0 - 1e-7)[..., None], curves[:, -1:], p)


def _samples(curves):
    """The 2P + 5 spline samples of the length measure, ends included, and their parameters."""
    n = 2 * curves.shape[1] + 4
    t = torch.arange(n + 1, device=curves.device).double() / n
    return _spline(curves, t), t


def _chords(samples):
    return torch.linalg.vector_norm(samples[:, 1:] - samples[:, :-1], dim=-1)


def _cut_at(lengths, amount, t):
    """The parameter where the running length reaches `amount`; the last one where it never does."""
    run = torch.cumsum(lengths, 1)
    reached = run >= amount
    k = reached.int().argmax(1, keepdim=True)
    over = (torch.gather(run, 1, k) - amount) / torch.gather(lengths, 1, k).clamp(min=1e-60)
    cut = t[k + 1] - over * (t[k + 1] - t[k])
    return torch.where(reached.any(1, keepdim=True), cut, t[-1])


def _between(value, a, b, fraction):
    axis = torch.linalg.cross(a, b)
    l2 = _dot(axis, axis)
    axis = axis / torch.sqrt(l2.clamp(min=1e-60))
    angle = torch.acos(_dot(a, b).clamp(-1.0, 1.0)) * fraction
    c, s = torch.cos(angle), torch.sin(angle)
    turned = value * c + torch.linalg.cross(axis, value) * s + axis * _dot(axis, value) * (1.0 - c)
    return torch.where(l2 >= 1e-12, turned, value)


def _clump_axes(source, normals, tangents, grads, frequency, correlation):
    """Per guide: the rebuilt CVs, their spline length, and the unit noise displacement of every CV."""
    G, P, _ = source.shape
    t = torch.arange(P, device=source.device).double() / (P - 1)
    axis = _spline(source, t)
    length = _chords(_samples(source)[0]).sum(1)
    seg = _chords(source)
    f = torch.where(seg.sum(1) > 0, torch.clamp(0.5 / seg.sum(1).clamp(min=1e-60), min=frequency), frequency)
    domain = (source[:, 0] + torch.tensor([0.419276, 0.184247, 0.805721], device=source.device)) * \
        (100.0 * (1.0 - correlation) ** 2)
    n, u = _unit(normals), _unit(tangents)
    v, ct = torch.linalg.cross(n, u), _unit(axis[:, 1] - axis[:, 0], n)
    bent = _dot(n, ct) < 0.99999
    u, v = torch.where(bent, _between(u, n, ct, 1.0), u), torch.where(bent, _between(v, n, ct, 1.0), v)
    travelled, units = torch.zeros_like(f), [torch.zeros_like(n)]
    for c in range(1, P):
        travelled = travelled + seg[:, c - 1]
        nt = _unit(axis[:, c + 1] - axis[:, c], ct) if c + 1 < P else ct
        bent = _dot(ct, nt).abs() < 0.99999
        su, sv = (torch.where(bent, _between(x, ct, nt, 0.5), x) for x in (u, v))
        shift = (travelled * f)[:, None] * torch.eye(3, dtype=torch.float64, device=source.device)[:, None]
        first, second = _noise(grads, domain + shift[0]) - 0.5, _noise(grads, domain + shift[2]) - 0.5
        units.append(su * first[:, None] + sv * second[:, None])
        u, v = (torch.where(bent, _between(x, ct, nt, 1.0), x) for x in (u, v))
        ct = nt
    return axis, length[:, None], torch.stack(units, 1)


def _exact_fx(e, asset):
    P = e.p.cvs_per_strand
    curves, normals, tangents, _ = map(_t, _clump_guides(asset, P))
    axis, target, unit = _clump_axes(curves, normals, tangents, e.grads, 6.0, 0.4)
    number = {kind: {k: float(v) for k, v in values.items() if not v.startswith("$")} for kind, values in FX_EFFECTS}
    noise, clump = number["noise"], number["clump"]
    grid = torch.arange(P, device=e.t.device).double() / (P - 1)

    def finish(s, c, _):
        scale = 0.5 * (1.0 + 0.4 * _noise(e.grads, s["root"] * 6.0))[:, None, None]
        width = 0.01 * (1.0 + 0.3 * _noise(e.grads, s["root"] * 20.0))[:, None]
        c = c[:, :1] + (c - c[:, :1]) * scale
        tangent = _t(_across(s["normal"].float().cpu().numpy()))
        domain = (c[:, 0] + torch.tensor([0.419276, 0.184247, 0.805721], device=c.device)) * \
            (100.0 * (1.0 - 0.01 * noise["correlation"]) ** 2)
        c = _displace(c, s["normal"], tangent, domain, noise["frequency"], noise["magnitude"] * noise["magnitudeScale"],
                      e.grads, 0.01 * noise["preserveLength"], True)
        g = e.stencil[s["tri"], 0]
        at, t = _samples(c)
        c = _spline(c, _cut_at(_chords(at), target[g], t) * grid)
        moved = c + (axis[g] - c) * (clump["mask"] * clump["clump"] * (1.0 - 2.0 * clump["clumpScale"])) + \
            unit[g] * (clump["mask"] * clump["noise"] * clump["noiseScale"])
        c = torch.cat([c[:, :1], moved[:, 1:]], 1)
        at, t = _samples(c)
        chords = _chords(at)
        back = _cut_at(chords.flip(1), 0.1 * chords.sum(1, keepdim=True), t)
        c = _spline(c, (1.0 - back) * grid)
        profile = torch.where(e.t > 0.3, 1.0 - 0.6 * (e.t - 0.3) / 0.7, 1.0)
        return c, 0.5 * width * profile, None

    out, _ = e.result(finish)
    return dict(out, status=None)


def _exact_classic(e):
    def finish(s, c, _):
        scale = 0.5 * (1.0 + 0.4 * _noise(e.grads, s["root"] * 6.0)) * (1.0 - s["uv"][:, 1]).clamp(0.2, 1.0)
        width = 0.01 * (1.0 + 0.3 * _noise(e.grads, s["root"] * 20.0))
        c = c[:, :1] + (c - c[:, :1]) * scale[:, None, None]
        return c, (0.5 * width)[:, None].expand(c.shape[:2]), torch.stack([scale, width], 1).cpu()

    out, more = e.result(finish)
    return dict(out, scalars=torch.cat(more), status=None)


def _exact_payload(case, seed):
    base, samples = _curves(case, seed)
    S, R = case["strands"], case["resample"]
    counts = (torch.full((S,), case["cvs"], device=DEVICE) if base.point_counts is None else base.point_counts).long()
    starts = torch.cumsum(counts, 0) - counts
    m = torch.tensor(TRANSFORM, device=DEVICE).double().view(3, 4)
    out_counts = torch.full_like(counts, R) if R else counts
    owner = torch.repeat_interleave(torch.arange(S, device=DEVICE), out_counts)
    first = torch.cumsum(out_counts, 0) - out_counts
    x = torch.arange(len(owner), device=DEVICE) - first[owner]
    last = (counts - 1)[owner]
    x = x.double() / (out_counts - 1)[owner] * last if R else x.double()
    i = torch.minimum(x.long(), last - 1)
    f = x - i

    def sampled(a):
        a = a.double().view(len(a), -1)
        lo = starts[owner] + i
        return a[lo] * (1.0 - f[:, None]) + a[lo + 1] * f[:, None]

    move = lambda a: sampled(a) @ m[:, :3].T + m[:, 3]
    points = torch.cat([move(base.points), 0.5 * sampled(base.widths)], 1)
    motion = None
    if samples:
        moved = [move(c.points) for _, c in samples]
        bounds = [int(first[b]) for b in range(0, S, case["batch"])] + [len(owner)]
        motion = torch.cat([a[lo:hi] for lo, hi in zip(bounds, bounds[1:]) for a in moved]).reshape(-1, 3).cpu()
    return dict(counts=None, points=points.cpu(), uvs=base.root_uvs.double().cpu(), motion=motion, first=None, status=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cache", "stencil"):  # whole numbers and bytes
        return None
    if kind == "payload":
        return _exact_payload(case, seed)
    if kind == "batch":
        rng = np.random.default_rng([seed, 5])
        return [_Exact(_asset(d["lon"], d["rings"], d["guides"], d["slots"], d["cvs"], rng),
                       _params(d, seed + k)).result()[0] for k, d in enumerate(_descriptions(case))]
    asset, params = _groom(case, seed)
    if kind == "motion":
        return [_Exact(asset, params, frame).result()[0] for frame in _deformation(case, seed, asset)[1]]
    e = _Exact(asset, params)
    if kind == "classic":
        return _exact_classic(e)
    if kind == "fx":
        return _exact_fx(e, asset)
    return e.result()[0]
