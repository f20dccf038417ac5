"""The stencil search over sorted guide clusters (stencil.cu) against the host
builder: guide counts around a cluster's 32 and the path's ends, ties and
penalties, wild positions (the all-pairs path), meshes whose triangles come in
no order, and flat or coincident guides."""
import numpy as np
import pytest
import torch

from nanoxgen_b200 import fixtures
from nanoxgen_b200.asset import AssetBuildInput, GuideSet, build_asset
from nanoxgen_b200.generator import build_stencils

pytestmark = pytest.mark.gpu


def _source(guides, shape, rng):
    pos, _, tris = fixtures.sphere_mesh(200, 101 if guides < 1600 else 201)
    t = rng.integers(0, len(tris), guides)
    b = rng.dirichlet([1, 1, 1], guides)
    root = np.einsum("gkc,gk->gc", pos[tris[t]].astype(np.float64), b)
    normal = root / np.linalg.norm(root, axis=1, keepdims=True)
    if shape == "shuffled":
        tris = tris[rng.permutation(len(tris))]
    elif shape == "ties":            # equal scores, every other copy penalised
        half = guides // 2
        root[half:2 * half] = root[:half]
        normal[1::2] *= -1.0
    elif shape == "flat":
        root[:, 1] = 0.0
    elif shape == "coincident":
        root[:] = root[0]
    elif shape == "wild":
        root[7] = np.nan
        root[11, 1] = np.inf
    root = root.astype(np.float32)
    if shape == "wild_mesh":
        pos = pos.copy()
        pos[5000] = np.nan
        pos[7000, 0] = 3.0e38
    if shape == "invalid":
        tris = tris.copy()
        tris[[0, 77, len(tris) - 1]] = len(pos)
    gs = GuideSet(np.full(guides, 2, np.uint32), np.stack([root, root + normal], 1).astype(np.float32).reshape(-1, 3),
                  normal.astype(np.float32), np.zeros((guides, 2), np.float32), t.astype(np.uint32),
                  b[:, 1:].astype(np.float32), np.ones(guides, np.float32))
    return pos, tris, gs


CASES = [(n, "plain", 8) for n in (639, 640, 641, 671, 672, 1600, 5120, 5121)] + \
        [(900, shape, slots) for shape in ("shuffled", "ties", "flat", "coincident", "wild", "wild_mesh", "invalid")
         for slots in (8, 3)]


@pytest.mark.parametrize("guides,shape,slots", CASES)
def test_rows_equal_the_host_builder(nxg_lib, guides, shape, slots):
    pos, tris, gs = _source(guides, shape, np.random.default_rng(guides))
    valid = (tris < len(pos)).all(1)
    host_tris = np.where(valid[:, None], tris, 0).astype(np.uint32)
    normals = np.tile(np.float32([0, 1, 0]), (len(pos), 1))
    asset = build_asset(AssetBuildInput(pos, host_tris, gs, normals, None), slots) if "wild" not in shape else None
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    roots = gs.cvs.reshape(-1, 2, 3)[:, 0]
    inputs = dev(pos), dev(tris.astype(np.uint32).view(np.int32)), dev(roots)
    if asset is not None:
        rows = build_stencils(*inputs, dev(asset.guides()["root_normal"]), slots).cpu().numpy().view(np.uint32)
        want = asset.stencil().reshape(-1, 8).copy()
        want[~valid] = 0xFFFFFFFF
        assert np.array_equal(rows, want)
        return
    # The host builder refuses wild input: the same triangles in calls small
    # enough to take all pairs.
    rows = build_stencils(*inputs, dev(gs.root_normals), slots)
    for first in range(0, len(tris), 1500):
        part = build_stencils(inputs[0], inputs[1][first:first + 1500].contiguous(), inputs[2], dev(gs.root_normals), slots)
        assert torch.equal(rows[first:first + 1500], part)
