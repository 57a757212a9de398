"""Mixed heads of decoded tokens: the kernel that stages a tile's values in shared memory gives the bits of the one that fetches four keys
at a time, which buffers off 16 bytes still take."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# one key, a tile's edge, several tiles a warp, with and without kept keys; groups of each form and none that fills it; the narrowest rows,
# rows of no power of two, the widest; more blocks than are resident
@pytest.mark.parametrize("heads,kv_heads,vdim", [(16, 8, 128), (4, 1, 72), (8, 1, 128), (3, 3, 8), (12, 2, 40)])
@pytest.mark.parametrize("window,keep_first", [(0, 0), (70, 33)])
@pytest.mark.parametrize("contexts", [[1, 32, 33, 600], [1 + 29 * i % 300 for i in range(90)]], ids=["four", "many"])
@pytest.mark.parametrize("odd", [False, True])
def test_bits_of_both_kernels(heads, kv_heads, vdim, window, keep_first, contexts, odd):
    from mini_engine_b200.csrc import ops

    generator = torch.Generator("cuda").manual_seed(heads + vdim)
    rand = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    dim, page = 64, 16
    counts = [-(-c // page) for c in contexts]
    table, first = torch.full((len(contexts), max(counts)), -1, dtype=torch.int32), 0
    for i, count in enumerate(counts):
        table[i, :count] = torch.arange(first, first + count)
        first += count
    k_pages, v_pages = rand(first + 1, kv_heads, page, dim).bfloat16(), rand(first + 1, kv_heads, page, vdim).bfloat16()
    if odd:  # infinities and NaN among the values and, by the keys, among the scores
        values, keys = v_pages.view(-1, vdim), k_pages.view(-1, dim)
        values[5::131, 1], values[17::131, 6], values[40::131, 3] = float("inf"), float("nan"), -float("inf")
        keys[23::311, 2], keys[90::311, 7], keys[200::311, 9] = float("inf"), -float("inf"), float("nan")
    shifted = torch.empty(v_pages.numel() + 4, dtype=torch.bfloat16, device="cuda")[4:].view(v_pages.shape)  # starts on 8 bytes
    shifted.copy_(v_pages)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")  # noqa: E731
    n, stride = len(contexts), max(contexts)
    given = dict(
        q=rand(n, heads * dim).bfloat16(), k_pages=k_pages, block_table=table.cuda(), entry_of_token=ints(list(range(n))),
        positions=ints([c - 1 for c in contexts]), heads=heads, kv_heads=kv_heads, head_dim=dim, value_dim=vdim, scale=dim**-0.5, window=window,
        keep_first=keep_first, r1=rand(heads).abs(), r2=rand(heads).abs(), talk=rand(heads, heads), stride=stride,
    )  # fmt: skip
    outs = []
    for values in (v_pages, shifted):
        out = torch.full((n, heads * vdim), float("nan"), dtype=torch.bfloat16, device="cuda")
        scores, stats = torch.full((n * heads * stride,), float("nan"), device="cuda"), torch.empty(n * heads * 2, device="cuda")
        ops.mixed_attention(v_pages=values, out=out, scores=scores, stats=stats, **given)
        outs.append(out)
    torch.cuda.synchronize()
    assert torch.equal(outs[0].isnan(), outs[1].isnan()) and torch.equal(*(o.nan_to_num(3.0, 4.0, 5.0) for o in outs))
    assert odd == bool(outs[0].isnan().any())
