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


def test_motion_call_keeps_its_form(cuda, nxg_lib):
    """Lane-group tiles registered and withdrawn by another thread while a
    motion call is enqueued: every sample holds every strand (the lane groups
    read a strand order, which a call of this size writes only if its first
    sample takes them)."""
    import torch
    from nanoxgen_b200 import fixtures
    from nanoxgen_b200.asset import build_asset
    from nanoxgen_b200.generator import (DeformedGeometry, DeviceAsset, allocate_outputs, generate_motion_packed,
                                         set_tile)
    w = fixtures.plain_sphere(strands=3000)
    asset = build_asset(w.build_input, w.stencil_slots)
    d, params, samples = DeviceAsset(asset), w.params.copy(cvs_per_strand=24), 6
    rest = torch.from_numpy(np.ascontiguousarray(asset.positions())).cuda()
    frames = [DeformedGeometry(positions=rest * (1.0 + 0.01 * k)) for k in range(samples)]
    times = np.linspace(0.0, 1.0, samples).astype(np.float32)
    outputs = [allocate_outputs(3000, 24, "cuda") for _ in frames]
    want = [c.points.clone() for c in generate_motion_packed(d, params, frames, times, outputs=outputs)]
    torch.cuda.synchronize()
    done = threading.Event()

    def toggling():
        while not done.is_set():
            set_tile(24, True, 8, 4, 128)
            set_tile(24, True)

    def generating():
        try:
            stream = torch.cuda.Stream()
            for _ in range(300):
                with torch.cuda.stream(stream):
                    d.workspace(params, 3000).fill_(255)
                    for o in outputs:
                        o[0].fill_(float("nan"))
                    generate_motion_packed(d, params, frames, times, outputs=outputs, stream=stream)
                    # lane groups and lane walk agree to the generator's bar
                    near = [((o[0][:, :3] - p[:, :3]).norm(dim=1).max() <= 1e-5 * asset.bbox_diagonal())
                            for o, p in zip(outputs, want)]
                stream.synchronize()
                assert all(bool(n) for n in near)
        finally:
            done.set()

    try:
        run_threads(toggling, generating)
    finally:
        set_tile(24, True)
