"""The stencil search on meshes whose triangles come in no order, in scattered
patches, or in order but for a part: whichever of its searches each takes, the
rows are the ordered mesh's, and the all-pairs search's."""
import numpy as np
import pytest
import torch

from nanoxgen_b200 import fixtures
from nanoxgen_b200.generator import build_stencils

pytestmark = pytest.mark.gpu


def _order(n, how, rng):
    at = np.arange(n)
    if how == "shuffled":
        return rng.permutation(n)
    if how.startswith("patches"):
        k = int(how[7:])
        m = n // k * k
        return np.concatenate([at[:m].reshape(-1, k)[rng.permutation(m // k)].reshape(-1), at[m:]])
    part = {"first": slice(0, n // 3), "last": slice(n - n // 3, n), "ordered": slice(0, 0)}[how]
    at[part] = rng.permutation(at[part])
    return at


@pytest.mark.parametrize("guides", [700, 2048])
@pytest.mark.parametrize("how", ["ordered", "shuffled", "patches8", "patches16", "patches32", "first", "last"])
def test_rows_do_not_depend_on_the_triangle_order(cuda, nxg_lib, how, guides):
    rng = np.random.default_rng(guides)
    pos, _, tris = fixtures.sphere_mesh(200, 126)
    t = rng.integers(0, len(tris), guides)
    root = np.einsum("gkc,gk->gc", pos[tris[t]].astype(np.float64), rng.dirichlet([1, 1, 1], guides))
    normal = root / np.linalg.norm(root, axis=1, keepdims=True)
    normal[::7] *= -1.0
    order = _order(len(tris), how, rng)
    tris = tris[order].astype(np.uint32)
    broken = np.zeros(len(tris), bool)
    broken[[0, len(tris) // 2, len(tris) - 1]] = True
    tris[broken] = len(pos)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    mesh, mine = dev(pos), dev(tris.view(np.int32))
    g = dev(root.astype(np.float32)), dev(normal.astype(np.float32))
    rows = build_stencils(mesh, mine, *g)
    assert bool((rows[dev(broken)] == -1).all())
    # Calls of a few triangles take all pairs.
    for first in range(0, len(tris), 6000):
        assert torch.equal(rows[first:first + 6000], build_stencils(mesh, mine[first:first + 6000].contiguous(), *g))


@pytest.mark.parametrize("special", ["degenerate", "wild", "plain", "invalid"])
@pytest.mark.parametrize("slots", [8, 3])
def test_row_searched_by_itself(cuda, nxg_lib, special, slots):
    """In a mesh in no order the last row is searched by itself: a degenerate
    triangle (its face normal penalises half the guides), one beyond the finite
    range, an ordinary one, and one of no vertices."""
    rng = np.random.default_rng(3)
    guides = 1000
    pos, _, tris = fixtures.sphere_mesh(200, 126)
    tris = tris[rng.permutation(len(tris))].astype(np.uint32)
    pos = np.concatenate([pos, np.float32([[np.inf, 0, 0]])])
    row = len(tris) - 1
    of = {"degenerate": [7000, 7000, 7000], "wild": [len(pos) - 1, 5, 6], "plain": tris[row], "invalid": [len(pos)] * 3}
    tris[row] = of[special]
    t = rng.integers(0, row, guides)
    root = pos[tris[t]].mean(1).astype(np.float32)
    root[500:] = root[:500]
    normal = (root / np.linalg.norm(root, axis=1, keepdims=True)).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    mesh, mine, g = dev(pos), dev(tris.view(np.int32)), (dev(root), dev(normal))
    rows = build_stencils(mesh, mine, *g, slots)
    for first in range(0, len(tris), 6000):
        assert torch.equal(rows[first:first + 6000], build_stencils(mesh, mine[first:first + 6000].contiguous(), *g, slots))
