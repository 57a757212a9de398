"""Views of the workspace's buffers: the same one for the same question, a new one once the buffer was replaced."""

from __future__ import annotations

import torch


def test_views_are_kept_until_their_buffer_is_replaced():
    from mini_engine_b200.engine.workspace import Workspace

    workspace = Workspace(8, device="cpu")
    first = workspace.get("a", (3, 4), torch.float32)
    assert workspace.get("a", (3, 4), torch.float32) is first and first.shape == (3, 4)
    assert workspace.get("a", (8, 4), torch.float32).data_ptr() == first.data_ptr()
    assert workspace.get("a", (3, 4), torch.int32).dtype == torch.int32
    larger = workspace.get("a", (9, 4), torch.float32)  # past the capacity: another buffer
    again = workspace.get("a", (3, 4), torch.float32)
    assert again.data_ptr() == larger.data_ptr() != first.data_ptr()
    parts = workspace.partials("p", 2, 3, 5)
    assert parts.shape == (2, 3, 5) and workspace.partials("p", 2, 3, 5) is parts
    grown = workspace.growing("g", (2, 5), torch.float32)
    workspace.growing("g", (40, 5), torch.float32)
    assert workspace.growing("g", (2, 5), torch.float32).data_ptr() != grown.data_ptr()
    workspace.frozen = True  # views of what is there may still be asked for, of any shape that fits
    assert workspace.growing("g", (3, 5), torch.float32).shape == (3, 5)
    for tokens in range(1, 200):  # steps of many token counts
        assert workspace.partials("p", 1, tokens % 16 + 1, 5).shape == (1, tokens % 16 + 1, 5)


def test_shapes_may_be_lists():
    from mini_engine_b200.engine.workspace import Workspace

    workspace = Workspace(8, device="cpu")
    assert workspace.get("a", [3, 4], torch.float32) is workspace.get("a", (3, 4), torch.float32)
    assert workspace.growing("g", [2, 5], torch.float32).shape == (2, 5)
    assert workspace.growing("g", torch.Size([2, 5]), torch.float32) is workspace.growing("g", (2, 5), torch.float32)
