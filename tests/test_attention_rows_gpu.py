"""The float32 attention whose blocks share every key among many rows gives the bits of the kernel with one warp per (token,
head), with every option, whatever the block's rows; keys that a row does not see may hold anything."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

# (past, new) of the entries: below and above 16 and 64 rows, a ragged last block, decoded tokens beside a prompt
STEPS = [[(0, 1)], [(31, 1), (32, 1), (100, 1)], [(0, 70)], [(5, 17), (60, 1), (0, 130)], [(90, 33), (250, 9)]]
OPTIONS = {
    "plain": {},
    "window": dict(window=40),
    "window_of_one": dict(window=1),
    "chunk_sink": dict(chunk=24, sink=True),
    "sink_values_gate": dict(sink_values=True, gate="elements", window=33),
    "slopes_gate": dict(slopes=True, gate="heads"),
    "softcap": dict(softcap=5.0),
    "sigmoid": dict(sigmoid_bias=True, window=50),
}


def both(step, heads, kv_heads, dim, value_dim, page_size, options, in_keys=False):
    from mini_engine_b200.csrc import ops

    generator = torch.Generator("cuda").manual_seed(heads + dim)
    rand = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    width = max(-(-(past + new) // page_size) for past, new in step)
    total = sum(-(-(past + new) // page_size) for past, new in step)
    order = torch.randperm(total + 3, generator=torch.Generator().manual_seed(1))[:total].tolist()
    k_pages = torch.full((total + 3, kv_heads, page_size, dim), float("nan"), device="cuda")
    v_pages = None if in_keys else torch.full((total + 3, kv_heads, page_size, value_dim), float("nan"), device="cuda")
    table = torch.full((len(step), width), -1, dtype=torch.int32)
    cu, positions, entry_of = [0], [], []
    for i, (past, new) in enumerate(step):
        for j in range(-(-(past + new) // page_size)):
            page = order.pop()
            table[i, j] = page
            held = min(page_size, past + new - j * page_size)  # keys behind the entry's last token stay NaN
            k_pages[page, :, :held] = rand(kv_heads, held, dim)
            if v_pages is not None:
                v_pages[page, :, :held] = rand(kv_heads, held, value_dim)
        cu.append(cu[-1] + new)
        positions += range(past, past + new)
        entry_of += [i] * new
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")  # noqa: E731
    n = cu[-1]
    ctx = SimpleNamespace(cu_tokens=ints(cu), positions=ints(positions), entry_of_token=ints(entry_of), num_entries=len(step),
                          max_query_len=max(new for _, new in step))  # fmt: skip
    given = dict(options)
    if given.get("sink_values"):
        given["sink_values"] = rand(heads)
    if given.get("slopes"):
        given["slopes"] = rand(heads).abs()
    if given.get("sigmoid_bias"):
        given["sigmoid_bias"] = rand(heads)
    if "gate" in given:
        given["gate"] = rand(n, heads * value_dim if given["gate"] == "elements" else heads)
    window = given.pop("window", 0)
    q = rand(n, heads * dim)
    shared, alone = (torch.full((n, heads * value_dim), float("nan"), device="cuda") for _ in range(2))
    table = table.cuda()
    assert ops.attention_rows_supports(q, k_pages, v_pages, shared, dim, value_dim)
    ops.paged_attention_rows(q, k_pages, v_pages, table, ctx, shared, heads, kv_heads, dim, dim**-0.5, window, value_dim=value_dim, **given)
    ops.paged_attention_generic(
        q, k_pages, v_pages, table, ctx.entry_of_token, ctx.positions, alone, heads, kv_heads, dim, dim**-0.5, window, value_dim=value_dim, **given
    )
    torch.cuda.synchronize()
    return shared, alone


@pytest.mark.parametrize("step", STEPS, ids=str)
@pytest.mark.parametrize("name", sorted(OPTIONS))
def test_bits_with_every_option(step, name):
    shared, alone = both(step, 8, 2, 128, 128, 16, OPTIONS[name])
    assert not shared.isnan().any() and torch.equal(shared, alone)


# value heads from one quad to the widest, key heads of no power of two, one head, groups that do not divide a block's rows
@pytest.mark.parametrize("heads,kv_heads,dim,value_dim,page_size", [(6, 2, 20, 4, 8), (1, 1, 64, 64, 16), (6, 1, 36, 100, 32), (4, 4, 128, 256, 16), (3, 1, 16, 512, 8)])
@pytest.mark.parametrize("step", STEPS, ids=str)
def test_bits_at_other_head_sizes(step, heads, kv_heads, dim, value_dim, page_size):
    shared, alone = both(step, heads, kv_heads, dim, value_dim, page_size, dict(window=45))
    assert not shared.isnan().any() and torch.equal(shared, alone)


@pytest.mark.parametrize("step", STEPS, ids=str)
@pytest.mark.parametrize("heads,dim,value_dim", [(16, 576, 512), (5, 48, 32)])
def test_bits_with_values_inside_the_key_rows(step, heads, dim, value_dim):
    shared, alone = both(step, heads, 1, dim, value_dim, 16, dict(gate="heads"), in_keys=True)
    assert not shared.isnan().any() and torch.equal(shared, alone)
