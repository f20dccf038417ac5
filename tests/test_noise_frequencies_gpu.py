"""The noisy walk below its frequency floor (the base curve is measured, from
the stage and chunk by chunk) and where segments reach over so many lattice
cells that their noise is taken directly, at the ends of its chunks and stages,
against the C restatement."""
import numpy as np
import pytest

from helpers import max_position_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cvs", [2, 15, 16, 17, 18, 24, 32, 33, 49, 130])
@pytest.mark.parametrize("cells", [None, 1.4, 1.6, 3.9, 6.0])
def test_floor_and_cells_per_segment(oracle, cuda, nxg_lib, cvs, cells):
    """`cells`: lattice cells of a segment of the longest guide; None: the floor."""
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    from nanoxgen_b200.generator import DeviceAsset, generate_packed
    w = fixtures.large_sphere(strands=333, guides=100, n_lon=40, n_rings=31)
    asset = build_asset(w.build_input, w.stencil_slots)
    curves = asset.guide_cvs().reshape(100, -1, 3)
    length = np.linalg.norm(np.diff(curves, axis=1), axis=-1).sum(1).max()
    frequency = 0.1 if cells is None else float(cells * (cvs - 1) / length)
    d = DeviceAsset(asset)
    for preserve in (0.0, 0.5):
        params = w.params.copy(cvs_per_strand=cvs, noise_frequency=frequency, noise_amplitude=0.02,
                               noise_preserve_length=preserve)
        got = generate_packed(d, params).points.cpu().numpy()
        want = oracle.generate(asset.buffer, params, threads=8)[0]
        assert max_position_error(got, want) <= 1e-5 * asset.bbox_diagonal()
