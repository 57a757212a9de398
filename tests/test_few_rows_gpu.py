"""Float32 attention of decoded tokens in two kernels (scores of all tiles side by side, then softmax and values by columns): the bits of
the kernel with one warp per (token, head), with every option, and the rule that takes a step there."""

from __future__ import annotations

import pytest
import torch
from test_attention_rows_gpu import OPTIONS, both

# one key, the edges of a tile and of a step of four tiles, several steps, entries of two and three tokens
STEPS = [[(0, 1)], [(31, 1), (32, 1), (127, 1), (128, 1)], [(129, 2), (300, 1), (5, 3)]]


def few(monkeypatch, step, heads, *args, before=None, capacity=None, **kwargs):
    from mini_engine_b200.csrc import ops

    rows, capacity = ops.paged_attention_rows, capacity or -(-max(past + new for past, new in step) // 32) * 32

    def with_scores(q, k_pages, v_pages, *given, **options):
        if before is not None:
            before(q, k_pages, v_pages)
        rows(q, k_pages, v_pages, *given, scores=torch.full((q.shape[0], heads, capacity), float("nan"), device="cuda"), **options)

    monkeypatch.setattr(ops, "paged_attention_rows", with_scores)
    shared, alone = both(step, heads, *args, **kwargs)
    assert torch.equal(shared.isnan(), alone.isnan()) and torch.equal(shared.nan_to_num(3.0, 4.0, 5.0), alone.nan_to_num(3.0, 4.0, 5.0))
    assert before is not None or not shared.isnan().any()
    return shared


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


@pytest.mark.gpu
@pytest.mark.parametrize("step", [[(2047, 1), (2048, 1), (4500, 2)], [(40 * i % 700, 1) for i in range(70)]], ids=["long", "many"])
@pytest.mark.parametrize("name", ["plain", "window", "slopes_gate"])
def test_bits_of_long_contexts_and_of_many_entries(monkeypatch, step, name):
    """More keys than one round of 64 blocks of scores covers, whose shared memory is then used again; more blocks than are resident."""
    few(monkeypatch, step, 8, 4, 64, 64, 16, OPTIONS[name])


@pytest.mark.gpu
@pytest.mark.parametrize("new", [1, 2, 3])
@pytest.mark.parametrize("window", [34, 45, 64])
def test_bits_where_a_window_bounds_the_scratch(monkeypatch, new, window):
    """Entries at every place of a tile, with exactly the room that the rule asks for: the scores of one row end where the next one's begin."""
    from mini_engine_b200.csrc import ops

    step = [(200 + i, new) for i in range(32)]
    capacity = ops.few_rows_capacity(32 * new, new, 8, 2, 231 + new, window)
    assert 0 < capacity <= window + new + 62
    few(monkeypatch, step, 8, 2, 32, 32, 16, dict(window=window), capacity=capacity)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["plain", "window", "sigmoid", "sink_values_gate", "softcap"])
def test_infinities_and_nan_come_out_as_from_one_warp(monkeypatch, name):
    inf, nan = float("inf"), float("nan")

    def before(q, k_pages, v_pages):
        q[0, 5], q[2, 70] = nan, inf
        flat_k, flat_v = k_pages.view(-1, k_pages.shape[-1]), v_pages.view(-1, v_pages.shape[-1])
        rows = torch.arange(0, flat_k.shape[0], 37, device="cuda")
        flat_k[rows[0::4], 3], flat_k[rows[1::4], 9] = inf, -inf
        flat_v[rows[2::4], 1], flat_v[rows[3::4], 30] = nan, -inf

    shared = few(monkeypatch, [(129, 2), (300, 1), (5, 3), (64, 1)], 8, 2, 128, 128, 16, OPTIONS[name], before=before)
    assert shared.isnan().any() and shared.isfinite().any()


@pytest.mark.gpu
@pytest.mark.parametrize("entries,launches", [(4, 2), (300, 1)])
def test_a_step_takes_the_form_of_the_rule(entries, launches):
    """Through the entry point that the parts call, with the scratch in a workspace: eight rows an entry, few entries and many."""
    from types import SimpleNamespace

    from mini_engine_b200.csrc import ops
    from mini_engine_b200.engine.workspace import Workspace

    heads, kv_heads, dim, context, page = 16, 2, 64, 513, 16
    torch.manual_seed(entries)
    pages = -(-context // page)
    k, v = (torch.randn(entries * pages, kv_heads, page, dim, device="cuda") for _ in range(2))
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")  # noqa: E731
    ctx = SimpleNamespace(cu_tokens=ints(range(entries + 1)), positions=ints([context - 1 - i % 40 for i in range(entries)]),
                          entry_of_token=ints(range(entries)), num_entries=entries, max_query_len=1, max_context_len=context,
                          workspace=Workspace(entries, "cuda"))  # fmt: skip
    table = torch.arange(entries * pages, dtype=torch.int32, device="cuda").view(entries, pages)
    q, out, alone = (torch.randn(entries, heads * dim, device="cuda") for _ in range(3))
    given = dict(heads=heads, kv_heads=kv_heads, head_dim=dim, scale=dim**-0.5, window=0)
    before = ops.launch_count()
    ops.paged_attention(q=q, k_pages=k, v_pages=v, block_table=table, ctx=ctx, out=out, **given)
    assert ops.launch_count() - before == launches
    ops.paged_attention_generic(q, k, v, table, ctx.entry_of_token, ctx.positions, alone, **given)
    assert torch.equal(out, alone)
