"""Float32 attention of decoded tokens in two kernels (scores of all tiles side by side, then softmax and values by columns): the bits of
the kernel with one warp per (token, head), with every option, and the rule that takes a step there."""

from __future__ import annotations

import pytest
import torch
from test_attention_rows_gpu import OPTIONS, both

# one key, the edges of a tile and of a step of four tiles, several steps, entries of two and three tokens
STEPS = [[(0, 1)], [(31, 1), (32, 1), (127, 1), (128, 1)], [(129, 2), (300, 1), (5, 3)]]


def few(monkeypatch, step, heads, *args, **kwargs):
    from mini_engine_b200.csrc import ops

    rows, capacity = ops.paged_attention_rows, -(-max(past + new for past, new in step) // 32) * 32

    def with_scores(q, *given, **options):
        rows(q, *given, scores=torch.full((q.shape[0], heads, capacity), float("nan"), device="cuda"), **options)

    monkeypatch.setattr(ops, "paged_attention_rows", with_scores)
    shared, alone = both(step, heads, *args, **kwargs)
    assert not shared.isnan().any() and torch.equal(shared, alone)


@pytest.mark.gpu
@pytest.mark.parametrize("step", STEPS, ids=str)
@pytest.mark.parametrize("name", sorted(OPTIONS))
def test_bits_with_every_option(monkeypatch, step, name):
    few(monkeypatch, step, 8, 2, 128, 128, 16, OPTIONS[name])


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,value_dim,page_size", [(1, 1, 20, 4, 8), (5, 1, 36, 100, 32), (4, 4, 128, 256, 16)])
@pytest.mark.parametrize("step", STEPS, ids=str)
def test_bits_at_other_head_sizes(monkeypatch, step, heads, kv_heads, dim, value_dim, page_size):
    few(monkeypatch, step, heads, kv_heads, dim, value_dim, page_size, dict(window=45))


@pytest.mark.gpu
@pytest.mark.parametrize("step", STEPS[:2], ids=str)
def test_bits_with_values_inside_the_key_rows(monkeypatch, step):
    few(monkeypatch, step, 16, 1, 576, 512, 16, dict(gate="heads"), in_keys=True)


def test_which_steps_take_the_two_kernels():
    from mini_engine_b200.csrc import ops

    take = ops.few_rows_capacity
    assert take(8, 1, 16, 8, 513, 0) == 544 and take(8, 8, 16, 8, 513, 0) == 544
    assert take(8, 9, 16, 8, 513, 0) == 0 and take(8, 1, 17, 1, 513, 0) == 0  # more rows than a block holds
    assert take(8, 1, 16, 8, 64, 0) == 0 and take(8, 1, 16, 8, 65, 0) == 96
    assert take(8, 1, 16, 8, 4096, 1024) == 1056  # keys behind the window need no room
    assert take(64, 1, 64, 8, 1 << 20, 0) == 0  # more scratch than is kept


# entries, heads, KV heads, widths, values in the keys, context, whether the two kernels were measured faster: many entries, whose blocks of value
# columns each form the softmax again; as many just under three blocks to an SM; short contexts, where the second launch decides
@pytest.mark.parametrize(
    "entries,heads,kv_heads,dim,value_dim,in_keys,context,two",
    [(8, 16, 8, 128, 128, False, 2048, True), (128, 32, 8, 128, 128, False, 2048, True), (96, 16, 2, 128, 128, False, 2048, True),
     (128, 16, 2, 128, 128, False, 2048, False), (48, 24, 4, 128, 128, False, 512, True), (64, 24, 4, 128, 128, False, 512, False),
     (8, 16, 1, 576, 512, True, 128, True), (48, 16, 1, 576, 512, True, 2048, True), (128, 16, 1, 576, 512, True, 2048, False),
     (32, 16, 2, 64, 64, False, 128, False), (32, 16, 2, 64, 64, False, 2048, True)],
)  # fmt: skip
def test_the_faster_form_is_taken(entries, heads, kv_heads, dim, value_dim, in_keys, context, two):
    from mini_engine_b200.csrc import ops

    got = ops.few_rows_capacity(entries, 1, heads, kv_heads, context, 0, entries, dim, value_dim, in_keys)
    assert got == (context if two else 0)
