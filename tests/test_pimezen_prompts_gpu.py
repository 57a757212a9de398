"""The kernels that long portions of the Pimezen design take in bfloat16: mixed heads from tiles of eight tokens on tensor
cores, the gated recurrence in chunks of 16 tokens; each against float64 and beside the kernel that short portions take."""

from __future__ import annotations

import pytest
import torch

import plain_pimezen as plain
import schedules
from test_pimezen_gpu import (
    TOLERANCE, branch, compare, expected_logits, layer, load_plain, paged, plain_attention, random_ids, replay, run_attention,
)  # fmt: skip

pytestmark = pytest.mark.gpu


def inputs_of(requests, heads, kv_heads, window, keep_first, page_size, alike=False, odd=()):
    """Requests ``(past, new)`` in one step: arguments of both forms, of each alone, and float64 of all new tokens.  ``alike``: the
    heads' weights differ by about a thousandth and are mixed with signs that cancel, so that only their last bits are left.  ``odd``: values ``(request, token, KV head, column, value)``."""
    dim, dtype = 128, torch.bfloat16
    r1, r2, talk = torch.rand(heads) * 2, torch.rand(heads) + 0.1, torch.randn(heads, heads)
    if alike:
        r1, r2 = r1[:1].expand(heads).clone(), r2[:1].expand(heads).clone()
        talk = torch.stack([1.0 - 2.0 * (torch.randperm(heads) % 2) for _ in range(heads)])
    q_rows, positions, cu, tables, wants, pools = [], [], [0], [], [], []
    width = max(-(-(past + new) // page_size) for past, new in requests)
    base = 0
    for i, (past, new) in enumerate(requests):
        total = past + new
        q, k, v = (torch.randn(total, h, dim).to(dtype).float() for h in (heads, kv_heads, kv_heads))
        if alike:
            k = k[:, :1].expand(-1, kv_heads, -1).clone()
            q = torch.where(torch.rand(q.shape) < 0.05, q[:, :1] * (1 + 2.0**-7), q[:, :1]).to(dtype).float()
        for request, token, head, column, value in odd:
            if request == i:
                v[token, head, column] = value
        count = 2 * (-(-total // page_size)) + 1
        k_pages, table = paged(k, page_size, count, torch.Generator().manual_seed(i))
        v_pages, _ = paged(v, page_size, count, torch.Generator().manual_seed(i))
        row = torch.full((width,), -1, dtype=torch.int32)
        row[: len(table)] = table + base
        base += k_pages.shape[0]
        pools.append((k_pages, v_pages)), tables.append(row), q_rows.append(q[past:])
        positions += range(past, total)
        cu.append(cu[-1] + new)
        wants.append(plain_attention(q, k, v, r1, r2, talk, dim**-0.5, window, keep_first)[past:])
    cuda = lambda t, dt=None: t.to(device="cuda", dtype=dt or t.dtype).contiguous()  # noqa: E731
    n, stride = cu[-1], window + keep_first
    shared = dict(
        q=cuda(torch.cat(q_rows).view(n, -1), dtype), k_pages=cuda(torch.cat([p[0] for p in pools]), dtype),
        v_pages=cuda(torch.cat([p[1] for p in pools]), dtype), block_table=cuda(torch.stack(tables)),
        positions=torch.tensor(positions, dtype=torch.int32, device="cuda"), heads=heads, kv_heads=kv_heads, head_dim=dim,
        value_dim=dim, scale=dim**-0.5, window=window, keep_first=keep_first, r1=cuda(r1), r2=cuda(r2), talk=cuda(talk),
    )  # fmt: skip
    entry = torch.cat([torch.full((new,), i, dtype=torch.int32) for i, (_, new) in enumerate(requests)])
    cu_tokens = torch.tensor(cu, dtype=torch.int32, device="cuda")
    for_tiles = dict(cu_tokens=cu_tokens, longest=max(new for _, new in requests))
    for_rows = dict(
        entry_of_token=cuda(entry), scores=torch.full((n * heads * stride,), float("nan"), device="cuda"),
        stats=torch.empty(n * heads * 2, device="cuda"), stride=stride,
    )  # fmt: skip
    return shared, for_tiles, for_rows, torch.cat(wants).reshape(n, -1).double()


def tiles_and_rows(*args, **options):
    """The step of :func:`inputs_of` through each form; (tiles, two kernels, float64)."""
    from mini_engine_b200.csrc import ops

    shared, for_tiles, for_rows, want = inputs_of(*args, **options)
    tiles, rows = (torch.full(want.shape, float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.mixed_attention_tiles(**shared, **for_tiles, out=tiles)
    ops.mixed_attention(**shared, **for_rows, out=rows)
    torch.cuda.synchronize()
    return tiles.double().cpu(), rows.double().cpu(), want


@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 8), (16, 4)])
@pytest.mark.parametrize(
    "requests,window,keep_first,page_size",
    [
        ([(0, 9)], 5, 40, 16),  # every key kept, a second tile of one token
        ([(0, 33), (20, 8), (61, 1)], 20, 6, 16),  # window and kept keys within tiles; portion and decoded token beside a prompt
        ([(90, 47)], 33, 17, 8),
        ([(0, 130), (200, 3)], 64, 64, 32),  # kept keys fill two tiles
        ([(5, 70)], 1, 0, 16),  # a query sees itself alone
    ],
)
def test_mixed_heads_from_tiles(heads, kv_heads, requests, window, keep_first, page_size):
    torch.manual_seed(heads + window)
    tiles, rows, want = tiles_and_rows(requests, heads, kv_heads, window, keep_first, page_size)
    scale = want.norm()
    # both round the output to bfloat16 (relative 2^-9 / sqrt(3) = 1.1e-3 at most); the weights' three terms add nothing to it
    assert float((tiles - want).norm() / scale) < 2.5e-3
    assert float((tiles - want).norm()) < 1.02 * float((rows - want).norm())


@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 8), (16, 4)])
def test_mixed_heads_keep_32_bits_of_every_weight(heads, kv_heads):
    """Weights and mixing matrix are float32: where 32 nearly equal weights cancel, 17 bits of each leave an error of some
    2^-17 sqrt(32) / 2^-10 = 4e-2 of what remains, 24 bits one of 3e-4, far below the output's rounding (1.1e-3)."""
    torch.manual_seed(heads)
    tiles, rows, want = tiles_and_rows([(0, 90), (130, 21)], heads, kv_heads, 70, 6, 16, alike=True)
    scale = want.norm()
    assert float((rows - want).norm() / scale) < 2.5e-3
    assert float((tiles - want).norm()) < 1.02 * float((rows - want).norm())


@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 8), (16, 4)])
def test_values_that_are_not_finite_reach_only_the_queries_that_see_their_key(heads, kv_heads):
    """A kept key, keys inside windows and the last key of a portion, behind and ahead of queries of the same tile."""
    inf, nan = float("inf"), float("nan")
    odd = [(0, 2, 1, 3, inf), (0, 21, 0, 5, nan), (0, 21, 0, 100, -inf), (0, 27, 3, 64, inf), (0, 39, 2, 0, nan), (1, 45, 1, 127, -inf)]
    torch.manual_seed(heads)
    tiles, rows, _ = tiles_and_rows([(0, 40), (37, 12)], heads, kv_heads, 12, 6, 16, odd=odd)
    assert rows.isnan().any() and rows.isinf().any()
    assert torch.equal(tiles.isnan(), rows.isnan())
    assert torch.equal(torch.where(tiles.isinf(), tiles, 0.0), torch.where(rows.isinf(), rows, 0.0))
    finite = rows.isfinite()
    assert float((tiles - rows)[finite].norm() / rows[finite].norm()) < 2.5e-3  # both rounded to bfloat16


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,vdim", [(3, 3, 129), (4, 2, 256), (8, 2, 200), (3, 1, 64), (7, 1, 96), (8, 1, 192), (16, 2, 128)])
def test_every_form_of_the_two_kernels(heads, kv_heads, vdim, dtype):
    """Groups and value widths on both sides of the forms' bounds (2, 4 and 8 heads; 128 and 256 columns), heads that are no
    multiple of the scores fetched at a time; a long step (two warps in bfloat16) and a short one (sixteen)."""
    torch.manual_seed(heads + vdim)
    count, dim = 600, 24
    q, k, v = (torch.randn(count, h, d).to(dtype).float() for h, d in ((heads, dim), (kv_heads, dim), (kv_heads, vdim)))
    r1, r2, talk = torch.rand(heads), torch.rand(heads) + 0.1, torch.randn(heads, heads)
    want = plain_attention(q, k, v, r1, r2, talk, dim**-0.5, 50, 7)
    for positions in (list(range(count)), [0, 31, 64, 599]):
        got = run_attention(q, k, v, r1, r2, talk, dim**-0.5, 50, 7, positions, dtype)  # the one-pass form beside the two kernels
        error = float((got - want[positions]).norm() / want[positions].norm())
        assert error < (2e-6 if dtype == torch.float32 else 2.5e-3)  # sums of 57 weighted values; the output's rounding


@pytest.mark.parametrize("heads,kv_heads", [(32, 8), (16, 8), (16, 4)])
def test_each_entry_takes_one_form(heads, kv_heads):
    """With both forms in a step an entry comes from the form that its tokens and keys choose, none from both, none from neither."""
    from mini_engine_b200.csrc import ops

    window, keep_first = 500, 20
    eighths, most = ops.MIXED_TILES[kv_heads, heads // kv_heads]
    edge = -(-520 * eighths // 8)  # tokens behind a full window from which on tiles are taken
    edge = min(edge, most)
    requests = [(0, 7), (0, 8), (600, 1), (700, edge - 1), (700, edge), (3, 1), (64, 24), (30, 40)]
    shared, for_tiles, for_rows, _ = inputs_of(requests, heads, kv_heads, window, keep_first, 16)
    tokens = for_rows["entry_of_token"].shape[0]
    tiles, rows, both, fewer = (torch.full((tokens, heads * 128), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(4))
    ops.mixed_attention_tiles(**shared, **for_tiles, out=tiles)
    ops.mixed_attention(**shared, **for_rows, out=rows)
    ops.mixed_attention_tiles(**shared, **for_tiles, out=both, by_entry=True)
    ops.mixed_attention(**shared, **for_rows, out=both, besides_tiles=for_tiles["cu_tokens"])
    ops.mixed_attention(**shared, **for_rows, out=fewer, besides_tiles=for_tiles["cu_tokens"])
    begin = 0
    for past, new in requests:
        span = slice(begin, begin + new)
        in_tiles = new >= 8 and (new >= most or 8 * new >= eighths * min(past + new, window + keep_first))
        assert torch.equal(both[span], (tiles if in_tiles else rows)[span]), (past, new)
        assert torch.equal(fewer[span], torch.full_like(fewer[span], 7.0) if in_tiles else rows[span]), (past, new)
        begin += new


# Three layers of the sizes that the tile kernel is built for, with kept keys and windows shorter than the prompts.
CONFIG_TILES = {
    "architecture": "Pimezen", "vocab": 96, "width": 64, "norm": {"eps": 1e-5},
    "layers": [
        layer(branch(16, 8, 128, 128, 0.08, 40, 6), {"heads": 2, "dim": 16, "vdim": 32, "tau": 8.0, "decay_rank": 4}, 1.0, 0.7,
              {"kind": "dense", "ff": 96, "limit": 2.0}),
        layer(branch(16, 4, 128, 128, 0.08, 33, 17), {"heads": 1, "dim": 32, "vdim": 64, "tau": 4.0, "decay_rank": 2}, 0.8, 1.0, None),
        layer(branch(32, 8, 128, 128, 0.08, 70, 0), {"heads": 2, "dim": 16, "vdim": 16, "tau": 12.0, "decay_rank": 8}, 1.2, 0.5,
              {"kind": "dense", "ff": 64, "limit": 1.0}),
    ],
}  # fmt: skip


@pytest.fixture(scope="module")
def tiles_folder(tmp_path_factory):
    from mini_engine_b200.config import PimezenConfig
    from mini_engine_b200.weights import write_random_model

    folder = tmp_path_factory.mktemp("pimezen_tiles")
    write_random_model(folder, PimezenConfig.from_dict(CONFIG_TILES), seed=23, dtype=torch.bfloat16, scale=12.0)
    return folder


@pytest.fixture
def tile_calls(monkeypatch):
    """Which steps take tiles, and whether by entry."""
    from mini_engine_b200.csrc import ops

    calls, run = [], ops.mixed_attention_tiles
    monkeypatch.setattr(ops, "mixed_attention_tiles", lambda **args: (calls.append(args.get("by_entry", False)), run(**args)))
    return calls


@pytest.mark.parametrize("schedule", ["whole", "tail_one_by_one", "changing_portions", "mixed"])
def test_a_model_whose_sizes_reach_the_tiles(schedule, tiles_folder, tile_calls):
    requests = {f"r{i}": random_ids(700 + i, n, 96) for i, n in enumerate([150, 64, 17, 230, 5, 9, 90])}
    steps = getattr(schedules, schedule)(requests)
    got = replay(tiles_folder, "bfloat16", steps)
    compare(got, expected_logits(tiles_folder, requests), requests, "bfloat16")
    assert True in tile_calls if schedule == "mixed" else set(tile_calls) == {False}  # by entry beside other entries only


def test_the_tiles_through_the_engine_with_and_without_graphs(tiles_folder, tile_calls):
    """Lone prompts and second portions from captured steps (a dummy entry beside them), decoded entries beside a portion, slots
    and pages used again: every token within the tolerance of the plain logits' largest."""
    from mini_engine_b200 import EngineConfig, LLMEngine, SamplingParams

    weights, config = load_plain(tiles_folder)
    prompts = [random_ids(60 + i, n, 96) for i, n in enumerate((5, 9, 70, 130, 33, 100))]
    for graphs in (True, False):
        engine = LLMEngine.from_pretrained(
            tiles_folder, EngineConfig(block_size=16, num_blocks=96, max_model_len=256, max_num_seqs=3, max_num_batched_tokens=112,
                                       dtype=torch.bfloat16, cuda_graphs=graphs)  # fmt: skip
        )
        tile_calls.clear()
        alone = [engine.generate([prompt], SamplingParams(max_tokens=6, ignore_eos=True))[0] for prompt in prompts]
        assert (engine.stats.prompt_graph_steps > 0) == graphs
        together = engine.generate(prompts, SamplingParams(max_tokens=12, ignore_eos=True))
        assert True in tile_calls
        for prompt, tokens in [*zip(prompts, alone), *zip(prompts, together)]:
            logits = plain.forward_logits(weights, config, (prompt + tokens)[:-1])
            slack = 2 * TOLERANCE["bfloat16"] * float(logits.abs().max())
            for i, token in enumerate(tokens):
                row = logits[len(prompt) - 1 + i]
                assert float(row.max() - row[token]) <= slack, f"graphs {graphs}: token {i} of a {len(prompt)}-token prompt"


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("token", [32, 40, 63])
def test_a_value_that_is_not_finite_leaves_earlier_tokens_of_its_chunk_alone(token, value):
    """Its own column from that token on is spoilt, as token by token, and nothing else."""
    from test_pimezen_gpu import FakeContext

    from mini_engine_b200.csrc import ops

    torch.manual_seed(token)
    heads, dim, vdim, tokens, rank = 2, 64, 40, 70, 4
    columns = {"q": 0, "k": heads * dim, "v": 2 * heads * dim, "g": 2 * heads * dim + heads * vdim, "a": 2 * heads * (dim + vdim)}
    proj = torch.randn(1, tokens, columns["a"] + rank, device="cuda")
    proj[0, token, columns["v"] + vdim + 7] = value  # head 1, column 7
    a2t, bias = torch.randn(rank, heads * dim, device="cuda"), torch.randn(heads * dim, device="cuda")
    outs = []
    for chunk_min in (0, 33):
        state, out = torch.zeros(2, heads, dim, vdim, device="cuda"), torch.full((tokens, heads * vdim), 7.0, device="cuda")
        ops.gla_scan(
            proj=proj, columns=columns, a2t=a2t, a2_bias=bias, ctx=FakeContext([tokens], [0], [1]), state=state, out=out,
            prepared=torch.empty(tokens * heads * (3 * dim + vdim), device="cuda"), q_scale=1.0, tau=6.0, heads=heads, dim=dim, vdim=vdim,
            chunk_min=chunk_min, records=torch.empty(6, heads * ops.state_record_floats("gated", dim), device="cuda") if chunk_min else None,
        )  # fmt: skip
        outs.append((out.cpu().double(), state[0].cpu().double()))
    (walk, walk_state), (chunks, chunk_state) = outs
    assert not walk[token:, vdim + 7].isfinite().any()
    assert torch.equal(chunks.isfinite(), walk.isfinite()) and torch.equal(chunk_state.isfinite(), walk_state.isfinite())
    there = walk.isfinite()
    assert float((chunks - walk)[there].norm() / walk[there].norm()) < 2e-6


@pytest.mark.parametrize("heads,dim,vdim", [(2, 8, 24), (3, 64, 128), (2, 128, 128), (1, 100, 36)])
@pytest.mark.parametrize("counts,starts", [([33], [0]), ([48, 5], [7, 0]), ([1, 200, 34], [3, 0, 50])])
def test_gated_recurrence_in_chunks(heads, dim, vdim, counts, starts):
    """Entries below and above the chunks' minimum, from zero and from a held state, against the walk token by token and
    against float64; the states behind them too."""
    from test_pimezen_gpu import FakeContext

    from mini_engine_b200.csrc import ops

    torch.manual_seed(dim + len(counts))
    tokens, rank, tau = sum(counts), 4, 6.0
    widths = {"q": heads * dim, "k": heads * dim, "v": heads * vdim, "g": heads * vdim, "a": rank}
    columns, width = {}, 0
    for key, w in widths.items():
        columns[key], width = width, width + w
    proj = torch.randn(2, tokens, width)
    a2, bias = torch.randn(heads * dim, rank) * 0.5, torch.randn(heads * dim)
    slots, fresh = list(range(len(counts))), [1 if start == 0 else 0 for start in starts]
    first = torch.randn(len(counts) + 1, heads, dim, vdim)
    results = []
    for chunk_min, off in ((0, 0), (33, 0), (33, 1)):  # `off` floats: states that do not start on 16 bytes walk
        state, out = torch.empty(first.numel() + off, device="cuda")[off:].view(first.shape), torch.full((tokens, heads * vdim), float("nan"), device="cuda")
        state.copy_(first)
        prepared = torch.full((tokens * heads * (3 * dim + vdim),), float("nan"), device="cuda")
        chunks = tokens // ops.STATE_CHUNK + len(counts)
        records = torch.full((chunks, heads * ops.state_record_floats("gated", dim)), float("nan"), device="cuda")
        ops.gla_scan(
            proj=proj.cuda(), columns=columns, a2t=a2.t().contiguous().cuda(), a2_bias=bias.cuda(), ctx=FakeContext(counts, slots, fresh),
            state=state, out=out, prepared=prepared, q_scale=dim**-0.5, tau=tau, heads=heads, dim=dim, vdim=vdim,
            chunk_min=chunk_min, records=records if chunk_min else None,
        )  # fmt: skip
        torch.cuda.synchronize()
        results.append((out.cpu().double(), state.cpu().double()))
    summed = proj.double().sum(0)
    take = lambda key: summed[:, columns[key] : columns[key] + widths[key]]  # noqa: E731
    q, k, v = take("q").view(tokens, heads, dim) * dim**-0.5, take("k").view(tokens, heads, dim), take("v").view(tokens, heads, vdim)
    decay = torch.sigmoid(take("a") @ a2.double().T + bias.double()).pow(1 / tau).view(tokens, heads, dim)
    want, states, t = [], first.clone().double(), 0
    for slot, (count, start) in enumerate(zip(counts, starts)):
        s = states[slot] if start else torch.zeros(heads, dim, vdim, dtype=torch.float64)
        for _ in range(count):
            s = decay[t].unsqueeze(-1) * s + k[t].unsqueeze(-1) * v[t].unsqueeze(1)
            want.append((q[t].unsqueeze(1) @ s).reshape(-1))
            t += 1
        states[slot] = s
    want = torch.stack(want)
    (walk, walk_state), (chunked, chunk_state), (walked, walked_state) = results
    assert torch.equal(walked, walk) and torch.equal(walked_state, walk_state)
    for got, exact in ((walk, want), (chunked, want), (walk_state, states), (chunk_state, states)):
        assert float((got - exact).norm() / exact.norm()) < 2e-6  # sums of float32, up to 200 terms a state element
    # entries below the minimum walk in both
    begin = 0
    for count in counts:
        if count < 33:
            assert torch.equal(walk[begin : begin + count], chunked[begin : begin + count])
        begin += count
