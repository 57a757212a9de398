"""Named, persistent device buffers for one step's activations.

Parts ask for a buffer by name and shape; the first request allocates it at the engine's
token capacity and every later request returns a view of the same memory.  Addresses are
therefore stable from step to step, which is what lets a decode step be captured in a CUDA
graph and lets TMA descriptors of activations be made once.
"""

from __future__ import annotations

import math

import torch

from mini_engine_b200.parts.linear import partial_rows


class Workspace:
    def __init__(self, max_tokens: int, device: str | torch.device = "cuda"):
        self.max_tokens = max_tokens
        self.device = torch.device(device)
        self._buffers: dict[tuple[str, torch.dtype], torch.Tensor] = {}
        self.frozen = False  # set while a graph is captured: no new allocation may happen
        # Buffers that were replaced by larger ones.  A captured graph keeps the address of the
        # buffer it was captured with and goes on writing and reading there, so the memory must
        # neither be freed nor given to anyone else.
        self._retired: list[torch.Tensor] = []
        # The views handed out of each buffer, by how they were asked for: a step asks for some hundred, and making one
        # (two calls into torch) takes 3 us, a fifth of what the host spends on a launch.
        self._views: dict[tuple[str, torch.dtype], dict[tuple, torch.Tensor]] = {}

    def _view(self, name: str, dtype: torch.dtype, shape: tuple[int, ...], elements: int) -> torch.Tensor:
        """``shape`` at the start of the named buffer, which holds at least ``elements``."""
        shape = tuple(shape)
        flat = self._flat(name, elements, dtype)
        views = self._views.setdefault((name, dtype), {})
        if len(views) >= 64:  # steps of many token counts
            views.clear()
        view = views[shape] = flat[: math.prod(shape)].view(shape)
        return view

    def _held_view(self, name: str, dtype: torch.dtype, shape: tuple[int, ...]) -> torch.Tensor | None:
        views = self._views.get((name, dtype))
        try:
            return None if views is None else views.get(shape)
        except TypeError:  # a list; looking first would cost a step of some hundred buffers more than the exception ever does
            return views.get(tuple(shape))

    def _flat(self, name: str, elements: int, dtype: torch.dtype) -> torch.Tensor:
        key = (name, dtype)
        held = self._buffers.get(key)
        if held is None or held.numel() < elements:
            if self.frozen:
                raise RuntimeError(f"workspace buffer {name!r} would have to grow during graph capture")
            if held is not None:
                self._retired.append(held)
                self._views.pop(key, None)
            held = torch.empty(elements, dtype=dtype, device=self.device)
            self._buffers[key] = held
        return held

    def get(self, name: str, shape: tuple[int, ...], dtype: torch.dtype) -> torch.Tensor:
        """A contiguous view ``shape`` of the named buffer.  The first axis is a token count;
        the buffer is sized for ``max_tokens`` of them."""
        held = self._held_view(name, dtype, shape)
        if held is not None:
            return held
        return self._view(name, dtype, shape, max(shape[0], self.max_tokens) * math.prod(shape[1:]))

    def partials(self, name: str, splits: int, tokens: int, width: int) -> torch.Tensor:
        """``[splits, tokens, width]`` float32 for the partial sums of a split product."""
        shape = (splits, tokens, width)
        held = self._held_view(name, torch.float32, shape)
        if held is not None:
            return held
        return self._view(name, torch.float32, shape, max(partial_rows(self.max_tokens), splits * tokens) * width)

    def growing(self, name: str, shape: tuple[int, ...], dtype: torch.dtype) -> torch.Tensor:
        """A buffer of exactly ``shape`` that grows on demand instead of being sized for the
        token capacity (logits: ``[rows, vocab]`` is large and ``rows`` is usually small).  It grows
        by half at least, so that steps of ever longer prompts do not leave one buffer behind for
        every length: all that it has ever replaced is less than twice what it holds."""
        view = self._held_view(name, dtype, shape)
        if view is not None:
            return view
        elements = math.prod(shape)
        held = self._buffers.get((name, dtype))
        if held is not None and held.numel() < elements:
            self._flat(name, max(elements, held.numel() + held.numel() // 2), dtype)
        return self._view(name, dtype, shape, elements)

    def zeroed(self, name: str, count: int) -> torch.Tensor:
        """``count`` int32 values that are zero when first handed out.  Kernels that use them
        (arrival counters) leave them zero again, so they are never cleared between steps."""
        key = (name, torch.int32)
        held = self._buffers.get(key)
        if held is None or held.numel() < count:
            if self.frozen:
                raise RuntimeError(f"workspace buffer {name!r} would have to grow during graph capture")
            if held is not None:
                self._retired.append(held)
                self._views.pop(key, None)
            held = torch.zeros(max(count, 1024), dtype=torch.int32, device=self.device)
            self._buffers[key] = held
        return held[:count]

    def bytes_held(self) -> int:
        return sum(t.numel() * t.element_size() for t in [*self._buffers.values(), *self._retired])
