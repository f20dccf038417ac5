"""NoiseFX values that are taken CV by CV (a magnitude with a ramp, a segment
longer than a lattice window) have the reference's rounding: straight strands
along an axis, whose frame is the axes themselves and adds no rounding, against
the reference's operations in 32 bits, bit for bit."""
import numpy as np
import pytest

from test_fx_windows_gpu import _apply

pytestmark = pytest.mark.gpu
F = np.float32


def _classic_noise(grads, x, y, z):
    """xgen_classic_noise_float (xgen_classic_runtime.cpp:803-837), one rounding per operation."""
    p = [np.asarray(v, F) for v in np.broadcast_arrays(x, y, z)]
    cell = [np.floor(v) for v in p]
    w = [a - b for a, b in zip(p, cell)]
    v = []
    for corner in range(8):
        o = (corner & 1, corner >> 1 & 1, corner >> 2)
        s = np.zeros(p[0].shape, np.int64)
        for k in range(3):
            s = (s * 1664525 + cell[k].astype(np.int64) + o[k] + 1013904223) & 0xffffffff
        s ^= s >> 11
        s ^= (s << 7) & 0x9d2c5680
        s ^= (s << 15) & 0xefc60000
        s ^= s >> 18
        g = grads[s & 0xff]
        v.append((g[..., 0] * (w[0] - F(o[0])) + g[..., 1] * (w[1] - F(o[1]))) + g[..., 2] * (w[2] - F(o[2])))
    a = [t * t * t * (t * (t * F(6) - F(15)) + F(10)) for t in w]
    for k in range(3):
        v = [(F(1) - a[k]) * v[2 * j] + a[k] * v[2 * j + 1] for j in range(len(v) // 2)]
    return F(0.5) * v[0] + F(0.5)


@pytest.mark.parametrize("cvs,frequency,ramp", [(2, 8, True), (17, 8, True), (24, 40, True), (5, 500, False),
                                                (24, 700, False)])
def test_noise_taken_cv_by_cv(cuda, nxg_lib, cvs, frequency, ramp):
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    w = fixtures.plain_sphere(strands=10, cvs=8)
    grads = build_asset(w.build_input, w.stencil_slots).section("noise_gradients", F, 256, 3)
    S, step = 300, F(2.0 ** -5)
    rng = np.random.default_rng(cvs)
    root = np.zeros((S, 3), F)
    root[:, 2] = rng.integers(-4096, 4096, S) * step
    pts = np.zeros((S, cvs, 4), F)
    pts[..., :3] = root[:, None]
    pts[..., 2] += np.arange(cvs, dtype=F) * step
    pts[..., 3] = 0.01
    axis = lambda k: np.tile(np.eye(3, dtype=F)[k], (S, 1))
    noise = dict(mask="1", magnitude="0.0625", magnitudeScale="rampUI(0,1,1:1,1,1)" if ramp else "1",
                 frequency=str(frequency), correlation="50", preserveLength="0")
    got, _ = _apply((pts, axis(2), axis(0), np.full(S, cvs, np.int32)), {"width": "0.01"}, [("noise", noise)])
    scale = F(100) * (F(1) - F(50) * F(0.01)) * (F(1) - F(50) * F(0.01))
    domain = (root + np.array([0.419276, 0.184247, 0.805721], F)) * scale
    distance = np.arange(cvs, dtype=F) * step * max(F(0.5) / (F(cvs - 1) * step), F(frequency))
    at = lambda k: [domain[:, None, i] + distance if i == k else domain[:, None, i] for i in range(3)]
    l = [(_classic_noise(grads, *at(k)) - F(0.5)) * F(0.0625) for k in range(3)]
    # normal x, binormal normal x tangent = -y, and the tangent z.
    want = np.stack([l[0], -l[1], pts[..., 2] + l[2]], -1)
    want[:, 0] = pts[:, 0, :3]
    np.testing.assert_array_equal(np.abs(got[..., 0]), np.abs(want[..., 0]))
    np.testing.assert_array_equal(np.abs(got[..., 1]), np.abs(want[..., 1]))
    np.testing.assert_array_equal(got[..., 2], want[..., 2])
