"""How the layout helpers reach their kernels: `_offer` without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from quantforge_b200 import ops


@pytest.mark.parametrize("capturing", [False, True])
def test_no_context_is_created_during_a_capture(monkeypatch, capturing):
    made = []
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    monkeypatch.setattr(ops, "_ctxs", {})
    monkeypatch.setattr(ops, "_ctx", made.append)
    t = SimpleNamespace(device=SimpleNamespace(index=0))
    assert ops._offer(lambda x: None, t) is None
    assert len(made) == (0 if capturing else 1)
