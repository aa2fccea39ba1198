"""The training loss is a sum in 64 bits and a fixed order: rounded once, and
the same in every run.  Sizes of one block, of one pixel more, and of more
blocks than the threads that add them up."""
import ctypes

import pytest

import hpm_b200 as hb

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    import torch

    g = torch.Generator().manual_seed(seed)
    out = torch.randn(n, 16, generator=g).cuda()
    td = (torch.rand(n, generator=g) * 6 + 2).cuda()
    tn = torch.nn.functional.normalize(torch.randn(n, 3, generator=g), dim=1).cuda()
    tm = (torch.rand(n, generator=g) < 0.7).to(torch.uint8).cuda()
    return out, td, tn, tm, torch.empty(n, 16, dtype=torch.bfloat16, device="cuda")


def _add(inputs, loss, first=0, n=None):
    n = n or inputs[0].shape[0]
    ptr = [ctypes.c_void_p(t[first:].data_ptr()) for t in inputs]
    assert hb.lib().hpm_net_loss(*ptr[:4], n, ctypes.c_float(1.2), ctypes.c_float(9.6), ctypes.c_float(0.5),
                                 ctypes.c_float(1.0 / n), ptr[4], ctypes.c_void_p(loss.data_ptr()), None) == hb.HPM_OK


@pytest.mark.parametrize("n", [1, 256, 257, 5000])
def test_the_sum_is_rounded_once(n):
    import torch

    inputs = _inputs(n, n)
    each = torch.zeros(n, device="cuda")  # the pixels' losses, one call each
    for i in range(n):
        _add(inputs, each[i:], i, 1)
    loss = torch.zeros(1, device="cuda")
    _add(inputs, loss)
    want = float(each.double().sum())
    assert abs(float(loss) - want) <= 2.0**-24 * want  # half a unit in the last place
    assert (inputs[4][:, 4:].float() == 0).all()


@pytest.mark.parametrize("n", [120000, 200003])
def test_every_run_gives_the_same_loss(n):
    import torch

    inputs = _inputs(n, 7)
    runs = []
    for _ in range(10):
        loss = torch.zeros(1, device="cuda")
        for _ in range(3):
            _add(inputs, loss)
        runs.append(float(loss))
    assert len(set(runs)) == 1, runs
    assert (inputs[4][:, 4:].float() == 0).all()
