"""The helpers around launches that run on the host: views kept by the workspace, what a torch without CUDA meets, the
choice between two kernels."""

import os
import subprocess
import sys

import pytest
import torch

from redline_b200.ops import kernels
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


# Times on a B200 in us of launches whose two decode kernels differ by more than a tenth: sequences, kv heads, head size,
# longest and summed keys, (CTAs per row, clusters resident), the streaming or one-partition kernel, the cluster kernel.
DECODE_LAUNCHES = [
    (1, 8, 64, 16384, 16384, (8, 15), 22.6, 11.4),
    (8, 8, 64, 4096, 32768, (2, 74), 19.9, 14.5),
    (8, 8, 64, 65536, 524288, (2, 74), 183.8, 152.9),
    (1, 8, 64, 131072, 131072, (8, 15), 67.7, 53.7),
    (128, 8, 64, 8192, 589824, (1, 148), 201.0, 235.2),
    (16, 8, 64, 16384, 31744, (1, 148), 23.0, 52.3),
    (128, 8, 64, 1024, 9152, (1, 148), 12.3, 28.9),
    (8, 8, 64, 65536, 94208, (2, 74), 48.0, 100.3),
    (1, 1, 64, 65536, 65536, (8, 15), 48.0, 28.0),
    (128, 1, 64, 2048, 147456, (1, 148), 16.8, 11.8),
    (128, 1, 64, 32768, 292864, (1, 148), 28.6, 98.3),
    (8, 8, 128, 4096, 32768, (2, 74), 36.7, 25.4),
    (8, 8, 128, 65536, 294912, (2, 74), 201.0, 244.2),
    (4, 8, 128, 131072, 294912, (4, 33), 214.1, 241.8),
    (16, 8, 128, 512, 4608, (1, 148), 14.0, 9.0),
    (32, 8, 128, 8192, 24064, (1, 148), 35.1, 93.8),
    (1, 1, 128, 131072, 131072, (4, 33), 89.2, 221.7),
    (64, 1, 128, 65536, 2359296, (2, 74), 208.2, 246.1),
]


@pytest.mark.parametrize("n,kv,dim,longest,total,cluster,other_us,rows_us", DECODE_LAUNCHES)
def test_decode_kernel_choice(n, kv, dim, longest, total, cluster, other_us, rows_us):
    """Equal lengths, spread ones and one long row among short ones, up to 131,072 keys."""
    est = kernels.decode_rows_estimate(n, kv, dim, longest, total, *cluster, {64: 12, 128: 6}[dim], 148)
    assert (est < 0.0) == (rows_us < other_us)
