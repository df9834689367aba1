"""The helpers around launches that run on the host: views kept by the workspace."""

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
