"""Maps in and out through every kind of host memory, on both sides of the
sizes from which pageable memory is staged by threads, with lengths that leave
a last chunk short."""
import ctypes

import numpy as np
import pytest

import hpm_b200 as hb

pytestmark = pytest.mark.gpu


def _context(w, h):
    cams = np.zeros(2, hb.CAMERA_DTYPE)
    cams["K"], cams["R"] = [w, 0, w / 2, 0, w, h / 2, 0, 0, 1], np.eye(3).reshape(-1)
    cams["t"][1] = [0.1, 0, 0]
    cams["width"], cams["height"], cams["depth_min"], cams["depth_max"] = w, h, 1, 5
    ctx = hb.Context()
    ctx.set_views([np.zeros((h, w), np.float32)] * 2, cams)
    return ctx


@pytest.mark.parametrize("w,h", [(5, 3), (1021, 773), (1601, 1199)])
@pytest.mark.parametrize("memory", ["pageable", "pinned", "device", "mixed"])
def test_hypotheses_come_back_as_they_went_in(w, h, memory):
    import torch

    r = np.random.default_rng(w)
    planes, costs = (torch.from_numpy(r.random(s, np.float32)) for s in ((h, w, 4), (h, w)))
    kinds = {"pageable": "hh", "pinned": "pp", "device": "dd", "mixed": "dh"}[memory]

    def place(t, kind):
        return t.cuda() if kind == "d" else (t.pin_memory() if kind == "p" else t.clone())

    ins = [place(t, k) for t, k in zip((planes, costs), kinds)]
    outs = [place(torch.zeros_like(t), "h" if k == "d" else k) for t, k in zip((planes, costs), kinds)]
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in ins + outs]
    with _context(w, h) as ctx:
        for _ in range(2):  # the buffers are used again
            assert hb.lib().hpm_set_hypotheses(ctx.handle, ptr[0], ptr[1]) == hb.HPM_OK
            assert hb.lib().hpm_get_result(ctx.handle, ptr[2], ptr[3]) == hb.HPM_OK
            assert torch.equal(outs[0], planes) and torch.equal(outs[1], costs)
            for t in outs:
                t.zero_()
