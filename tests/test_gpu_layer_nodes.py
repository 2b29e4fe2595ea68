"""The layer calls of the compiled extension: what makes an output require a gradient, and calls from several threads."""
import os
import subprocess
import sys

import pytest
import torch

from mappedconvolutions_b200 import nn as mnn

pytestmark = pytest.mark.gpu


def _cases():
    m = torch.rand(5, 6, 3, 2, device="cuda") * 4
    x = torch.randn(2, 4, 5, 6, device="cuda")
    return [(mnn.MappedConvolution(4, 3, 3).cuda(), (x, m)), (mnn.MappedTransposedConvolution(4, 3, 3).cuda(), (x, 7, 8, m)),
            (mnn.MappedMaxPool(3), (x, m)), (mnn.MappedAvgPool(3), (x, m)), (mnn.MappedAvgUnpool(3), (x, 7, 8, m)),
            (mnn.Resample(), (x, m[:, :, 0].contiguous(), (7, 8))), (mnn.Unresample(), (x, m[:, :, 0].contiguous()))]


@pytest.mark.parametrize("which", range(7))
def test_a_map_that_requires_a_gradient(which):
    """The output requires one too, and the map's own is undefined: a loss over frozen layers can be run backward."""
    layer, args = _cases()[which]
    layer.requires_grad_(False)
    assert not layer(*args).requires_grad
    m = next(a for a in args[1:] if isinstance(a, torch.Tensor)).requires_grad_()
    y = layer(*args)
    assert y.requires_grad
    y.backward(torch.ones_like(y))
    assert m.grad is None and args[0].grad is None


THREADS = """
import threading, time, torch
from torch.utils._python_dispatch import TorchDispatchMode
from mappedconvolutions_b200 import nn as mnn

inside, other = threading.Event(), threading.Event()

class Mode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if 'empty' in str(func) and not inside.is_set():
            n[0] += 1
            if n[0] == 2:  # the plan's buffer, after the output: this thread is building a plan
                inside.set()
                other.wait()
                time.sleep(0.5)  # the other thread now waits for the plans
        return func(*args, **(kwargs or {}))

n = [0]
x = torch.randn(2, 4, 5, 6, device='cuda')
m1, m2 = [torch.rand(5, 6, 3, 2, device='cuda') * 4 for _ in range(2)]
layer = mnn.MappedAvgUnpool(3)

def second():
    inside.wait()
    other.set()
    layer(x, 7, 8, m2)

t = threading.Thread(target=second)
t.start()
with Mode():
    layer(x, 7, 8, m1)
t.join()
torch.cuda.synchronize()
assert inside.is_set()
print('both done')
"""


def test_two_threads_while_a_plan_is_built():
    """Building a plan calls into Python (here a dispatch mode) under the plans' lock while another thread asks for a
    plan: neither may wait for the other."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", THREADS], cwd=root, capture_output=True, text=True, timeout=180)
    assert r.returncode == 0 and "both done" in r.stdout, r.stderr
