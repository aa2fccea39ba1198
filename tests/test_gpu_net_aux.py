"""The activations that gate the data gradient may start at any element: the
same result from a view off the 16-byte boundary."""
import pytest

from test_gpu_net import _case, _conv, _pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("offset", [1, 4, 8])
def test_gating_activations_off_the_boundary(cin, cout, offset):
    import torch

    h, w = 3, 131
    x, wt, _ = _case(h, w, cin, cout, seed=offset)
    g = torch.Generator().manual_seed(cin)
    dy = torch.randn(h, w, cout, generator=g).to(torch.bfloat16).cuda()
    packed = _pack(wt, 1)
    room = torch.empty(x.numel() + offset, dtype=torch.bfloat16, device="cuda")
    moved = room[offset:].view_as(x)
    moved.copy_(x)
    assert x.data_ptr() % 16 == 0 and moved.data_ptr() % 16 == 2 * offset % 16
    assert torch.equal(_conv(dy, packed, None, cin, 2, moved, True), _conv(dy, packed, None, cin, 2, x, True))
