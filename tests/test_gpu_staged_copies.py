"""Pageable maps through the pinned buffers of a context: a new context makes
none for a copy that saves less than they cost, a context that goes on copying
does, and the copies then hold whatever memory the other maps of the call lie
in."""
import ctypes

import numpy as np
import pytest

import hpm_b200 as hb
from test_gpu_host_copies import _context

pytestmark = pytest.mark.gpu

BUFFERS = 16 << 20


def _pinned():
    """Bytes of pinned buffers: shared anonymous memory, as the driver maps its
    own, or private memory of huge pages that a child does not get."""
    total, size = 0, 0
    for line in open("/proc/self/smaps"):
        key, *rest = line.split()
        if "-" in key and not key.endswith(":"):
            lo, hi = key.split("-")
            size = int(hi, 16) - int(lo, 16)
            if "/dev/zero" in line and "rw-s" in line:
                total += size
        elif key == "VmFlags:" and {"hg", "dc"} <= set(rest):
            total += size
    return total


def _hypotheses(w, h):
    r = np.random.default_rng(w)
    return r.random((h, w, 4), np.float32), r.random((h, w), np.float32)


def _warm(ctx, w, h):
    """Copies until the context has its buffers: 100 MB or more."""
    planes, costs = _hypotheses(w, h)
    for _ in range(5):
        ctx.set_hypotheses(planes, costs)


@pytest.mark.parametrize("w,h", [(1001, 1009), (1301, 1201)])
def test_a_new_context_makes_no_buffers_for_one_copy(w, h):
    planes, costs = _hypotheses(w, h)  # 20 and 31 MB
    before = _pinned()
    with _context(w, h) as ctx:
        ctx.set_hypotheses(planes, costs)
        got = ctx.get_result()
        assert _pinned() - before < BUFFERS
    assert np.array_equal(got[0], planes) and np.array_equal(got[1], costs)


def test_the_buffers_go_with_the_context():
    before = _pinned()
    for _ in range(2):
        with _context(1001, 1009) as ctx:
            _warm(ctx, 1001, 1009)
            assert _pinned() - before >= BUFFERS
        assert _pinned() <= before


@pytest.mark.parametrize("kinds", ["hh", "hd", "hp", "dh", "ph"])
def test_staged_beside_other_memory(kinds):
    import torch

    w, h = 1601, 1399  # 35.8 MB of planes, 9 MB of costs
    planes, costs = (torch.from_numpy(a) for a in _hypotheses(w, h))

    def place(t, kind):
        return t.cuda() if kind == "d" else (t.pin_memory() if kind == "p" else t.clone())

    ins = [place(t, k) for t, k in zip((planes, costs), kinds)]
    outs = [place(torch.zeros_like(t), k) for t, k in zip((planes, costs), kinds)]
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in ins + outs]
    before = _pinned()
    with _context(w, h) as ctx:
        _warm(ctx, w, h)
        assert _pinned() - before >= BUFFERS
        zero = np.zeros((h, w, 4), np.float32)
        for _ in range(2):
            ctx.set_hypotheses(zero, zero[..., 0].copy())
            assert hb.lib().hpm_set_hypotheses(ctx.handle, ptr[0], ptr[1]) == hb.HPM_OK
            assert hb.lib().hpm_get_result(ctx.handle, ptr[2], ptr[3]) == hb.HPM_OK
            assert torch.equal(outs[0].cpu(), planes) and torch.equal(outs[1].cpu(), costs)
            for t in outs:
                t.zero_()
            torch.cuda.synchronize()


def test_staged_images_beside_one_on_the_device():
    import torch

    w, h, n = 1201, 901, 6  # 26 MB
    r = np.random.default_rng(5)
    images = [(255 * r.random((h, w), np.float32)).round() for _ in range(n)]
    cams = np.zeros(n, hb.CAMERA_DTYPE)
    cams["K"], cams["R"] = [w, 0, w / 2, 0, w, h / 2, 0, 0, 1], np.eye(3).reshape(-1)
    cams["t"][:, 0] = 0.05 * np.arange(n)
    cams["width"], cams["height"], cams["depth_min"], cams["depth_max"] = w, h, 1, 5
    plane = np.zeros((h, w, 4), np.float32)
    plane[..., 2:] = [-1, 3]
    pinned = [torch.from_numpy(i).pin_memory() for i in images]
    on_device = torch.from_numpy(images[2]).cuda()
    costs = []
    for staged in (False, True):
        at = [p.data_ptr() for p in pinned]
        if staged:
            at = [i.ctypes.data for i in images]
            at[2] = on_device.data_ptr()
        with _context(w, h) as ctx:
            if staged:
                _warm(ctx, w, h)
            arr = (ctypes.c_void_p * n)(*at)
            assert hb.lib().hpm_set_views(ctx.handle, arr, ctypes.c_void_p(cams.ctypes.data), n) == hb.HPM_OK
            ctx.shape = (h, w)
            ctx.n = n
            costs.append(ctx.cost_vectors(plane))
    assert np.array_equal(costs[0], costs[1])
