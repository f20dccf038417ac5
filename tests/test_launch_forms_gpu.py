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
