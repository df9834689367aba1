"""The helpers around launches that run on the host: views kept by the workspace, what a torch without CUDA meets."""

import os
import subprocess
import sys

import torch

from redline_b200.parts.base import Workspace


def test_workspace_keeps_a_steps_views_among_many_odd_shapes():
    """Shapes that come once (a buffer sized by a text's length) don't keep the shapes of every step out for good,
    and a view is never of a buffer that a larger one has replaced."""
    ws = Workspace(torch.device("cpu"))
    for n in range(3000, 0, -1):
        assert ws.get("odd", (n, 2), torch.float32).shape == (n, 2)
    a = ws.get("hot", (4, 8), torch.float32)
    assert ws.get("hot", (4, 8), torch.float32) is a
    assert len(ws._views) <= 1024
    b = ws.get("hot", (64, 8), torch.float32)                 # grows: the smaller shape is now a part of this one
    assert ws.get("hot", (4, 8), torch.float32).data_ptr() == b.data_ptr() != a.data_ptr()


def test_a_torch_without_cuda_imports_the_module_and_refuses_launches():
    """(In a process of its own, whose torch has lost the two functions that a CUDA build adds.)"""
    code = ("import torch\n"
            "for name in ('_cuda_getCurrentRawStream', '_cuda_getDevice'):\n"
            "    delattr(torch._C, name)\n"
            "from redline_b200.ops import kernels\n"
            "for call in (lambda: kernels.add_residual(torch.zeros(4), torch.zeros(4)), kernels._stream):\n"
            "    try:\n"
            "        call()\n"
            "    except kernels.KernelError:\n"
            "        continue\n"
            "    raise SystemExit('not refused')\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
