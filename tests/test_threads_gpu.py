"""Calls of several host threads, each on its own stream: launches whose
shared-memory sizes differ, and tiles registered between the launches of a
call, do not disturb one another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run_threads(*bodies):
    """Runs the bodies at once; re-raises what one of them raised."""
    failed = []

    def guarded(body):
        try:
            body()
        except BaseException as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=guarded, args=(b,)) for b in bodies]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if failed:
        raise failed[0]


def test_small_and_large_calls_at_once(cuda, nxg_lib):
    """A few noisy strands (CTAs of a warp or two) beside many long ones (full
    CTAs and their longer tables), and two sizes of the stencil search: every
    call is launched and gives what it gives alone."""
    import torch
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    from nanoxgen_b200.generator import DeviceAsset, build_stencils, generate_packed
    w = fixtures.plain_sphere(strands=40_000)
    asset = build_asset(w.build_input, w.stencil_slots)
    calls = [w.params.copy(strand_count=64, cvs_per_strand=4), w.params.copy(cvs_per_strand=40),
             w.params.copy(strand_count=2000, cvs_per_strand=300)]
    meshes = []
    for guides in (700, 4096):
        m = fixtures.large_sphere(strands=1, guides=guides, n_lon=240, n_rings=121).build_input
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        g = m.guides
        roots = g.cvs[np.cumsum(g.cv_counts.astype(np.int64)) - g.cv_counts]
        meshes.append((put(m.positions), put(m.triangles.view(np.int32)), put(roots), put(g.root_normals)))

    def generating(params):
        d, stream = DeviceAsset(asset), torch.cuda.Stream()
        torch.cuda.synchronize()
        want = generate_packed(d, params).points.clone()
        torch.cuda.synchronize()

        def body():
            out = torch.empty_like(want)
            for _ in range(400):
                generate_packed(d, params, points=out, want_roots=False, stream=stream)
            stream.synchronize()
            assert torch.equal(out, want)
        return body

    def searching(mesh):
        stream = torch.cuda.Stream()
        want = build_stencils(*mesh)
        torch.cuda.synchronize()

        def body():
            out = torch.empty_like(want)
            for _ in range(100):
                build_stencils(*mesh, out=out, stream=stream)
            stream.synchronize()
            assert torch.equal(out, want)
        return body

    run_threads(*[generating(p) for p in calls], *[searching(m) for m in meshes])
