"""Joint bilateral upsampling of images with more block rows than a grid's y
holds (65,535 of 8 rows), through the context and the allocation-free entry."""
import ctypes

import numpy as np
import pytest

import hpm_b200 as hb
import oracle as orc
from test_gpu_jbu_edges import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [8 * 65535, 8 * 65535 + 10])
def test_jbu_of_a_tall_image(rows):
    import torch

    guide, depth, normal = _inputs(2, rows, 1, rows // 2, rows)
    normal = 0.3 * normal - np.float32([0, 0, 1])  # no sum of them comes near zero
    normal /= np.linalg.norm(normal, axis=-1, keepdims=True)
    od, on = orc.jbu(guide, depth, normal)
    with hb.Context() as ctx:
        gd, gn = ctx.jbu(guide, depth, normal)
    dev = [torch.from_numpy(a).cuda() for a in (guide, depth, normal)]
    out = torch.empty(rows, 2, device="cuda"), torch.empty(rows, 2, 3, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (*dev, *out)]
    assert hb.lib().hpm_jbu_noalloc(0, ptr[0], 2, rows, ptr[1], ptr[2], 1, rows // 2, ptr[3], ptr[4],
                                    None) == hb.HPM_OK
    torch.cuda.synchronize()
    for d, n in ((gd, gn), (out[0].cpu().numpy(), out[1].cpu().numpy())):
        np.testing.assert_allclose(d, od, rtol=1e-4, atol=1e-5)
        np.testing.assert_allclose(n, on, rtol=1e-4, atol=1e-5)
