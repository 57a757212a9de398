"""The float32 product on the tensor cores (three bfloat16 pieces of each operand): against float64, beside the
CUDA-core kernel's error, and the order of its sums."""

from __future__ import annotations

import pytest
import torch


def tensor_core():
    from mini_engine_b200.csrc import tensor_core as module

    return module


@pytest.mark.parametrize("outs", [1, 128, 130, 2048, 4096, 6144, 24576, 151936])
@pytest.mark.parametrize("inner", [64, 260, 1024, 4096, 12288])
def test_segments_cover_the_reduction(outs, inner):
    tc = tensor_core()
    segments = tc.split_segments(outs, inner)
    blocks = -(-inner // tc.BLOCK_K)
    per_segment = -(-blocks // segments)
    assert 1 <= segments <= 8
    assert (segments - 1) * per_segment < blocks <= segments * per_segment  # none is empty, none is missing


# tokens: one, a full and an overfull small tile, a full and an overfull large tile; outs: less than a tile, a ragged
# second tile; inner: one block, a partial block, several segments of which the last is shorter
SHAPES = [(1, 5, 64), (16, 128, 100), (17, 130, 68), (64, 200, 2048), (65, 300, 1100), (130, 520, 260), (8, 2048, 2816), (300, 4096, 1000)]


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,outs,inner", SHAPES)
def test_split_product(tokens, outs, inner):
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(3)
    x = torch.randn(tokens, inner, device="cuda") * torch.exp(2 * torch.randn(tokens, 1, device="cuda"))
    w = torch.randn(outs, inner, device="cuda")
    plan = tc.SplitPlan(w)
    simt = torch.empty(tokens, outs, device="cuda")
    ops.gemm_simt(x, w, simt)
    want = x.double() @ w.double().T

    def error(y):
        return float(((y.double() - want) / want.norm(dim=1, keepdim=True)).norm())

    out = torch.full((tokens, outs), float("nan"), device="cuda")
    tc.gemm_split(plan, x, out, (64, False))
    assert tc.take_error() == 0
    # no less exact than the fmaf chain; a quarter more for the few outputs of the small shapes
    assert error(out) <= 1.25 * error(simt)
    # the same bits with the segments in a cluster, with another token tile, and for rows of another batch
    for form in [(16, False), (16, True), (64, True), (128, plan.segments > 1)]:
        other = torch.full((tokens, outs), float("nan"), device="cuda")
        tc.gemm_split(plan, x, other, form)
        assert tc.take_error() == 0
        assert torch.equal(out, other), form
    for rows in (slice(tokens // 2, tokens // 2 + 1), slice(0, min(tokens, 16)), slice(tokens // 3, tokens)):
        part = torch.empty(len(range(*rows.indices(tokens))), outs, device="cuda")
        tc.gemm_split(plan, x[rows].clone(), part)
        assert torch.equal(part, out[rows])


# small products of more than 16 tokens, where the launch that makes pieces counts; larger ones, where weights converted once for many tokens do
@pytest.mark.parametrize(
    "tokens,outs,inner,form",
    [(17, 64, 64, (16, False)), (256, 64, 64, (16, False)), (64, 1024, 1024, (16, True)), (17, 2048, 2048, (16, True)), (128, 160, 2048, (16, True)),
     (17, 2048, 6144, (16, True)), (512, 2048, 2048, (64, False)), (512, 2048, 512, (64, False)),
     (64, 2048, 9216, (64, True)), (256, 24576, 4096, (128, False)), (8, 24576, 4096, (16, False))],
)  # fmt: skip
def test_the_form_that_was_measured_fastest_is_taken(tokens, outs, inner, form):
    tc = tensor_core()
    assert tc.split_form(tokens, outs, inner, tc.split_segments(outs, inner)) == form


def test_the_launch_that_makes_pieces_counts_in_plain_stream_order_only():
    tc = tensor_core()
    segments = tc.split_segments(2048, 2048)
    assert tc.split_form(40, 2048, 2048, segments)[0] == 16  # 17.7 us, 21.1 with 64
    segments = tc.split_segments(4096, 2048)
    assert tc.split_form(40, 4096, 2048, segments, overlapped=True) == (64, True)  # 22.1 us, 25.4 with 16


@pytest.mark.gpu
def test_infinities_and_nan_come_out_as_in_one_chain():
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(4)
    x, w = torch.randn(40, 256, device="cuda"), torch.randn(130, 256, device="cuda")
    x[3, 5], x[4, 7], w[9, 5], w[7, 3] = float("inf"), float("nan"), 1.0, -float("inf")
    x[6] *= 1e38
    x[8], w[11] = 1e-38, 1e-38
    out, want = torch.empty(40, 130, device="cuda"), torch.empty(40, 130, device="cuda")
    tc.gemm_split(tc.SplitPlan(w), x, out)
    ops.gemm_simt(x, w, want)
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    odd = torch.isinf(want)
    assert odd.any() and torch.equal(out[odd], want[odd]) and not torch.isinf(out[~odd]).any()
    small = torch.isfinite(want) & ((torch.arange(40, device="cuda")[:, None] == 8) | (torch.arange(130, device="cuda") == 11))
    small &= want.abs() < 2.0**-90  # row 8 and column 11 hold nothing else but the rows of huge and odd values
    assert small.sum() > 150 and torch.equal(out[small], want[small])  # their pieces fall under bfloat16's range: one chain


def operands(kind, tokens, outs, inner):
    normal = lambda *shape: torch.randn(*shape, device="cuda")  # noqa: E731
    x, w = normal(tokens, inner), normal(outs, inner)
    if kind == "one sign":
        return x.abs(), w.abs()
    if kind == "between 1 and 2":
        return torch.rand_like(x) + 1, torch.rand_like(w) + 1
    if kind == "largest dropped when cut":  # 1 + 2^-7 - 2^-23: all lower bits set
        return torch.full_like(x, 1 + 2.0**-7 - 2.0**-23), torch.full_like(w, 1 + 2.0**-7 - 2.0**-23)
    at = torch.randint(0, inner, (tokens,), device="cuda")
    rows = torch.arange(tokens, device="cuda")
    if kind == "one alone":
        alone = torch.zeros_like(x)
        alone[rows, at] = x[rows, at]
        return alone, w
    if kind == "one dominates":
        x[rows, at] *= 1e4
        return x, w
    if kind == "one in ten":
        x = torch.relu(x).square()
        x[:, torch.rand(inner, device="cuda") < 0.9] = 0
        return x, w
    half = inner // 2
    x[:, half : 2 * half] = x[:, :half]
    w[:, half : 2 * half] = -w[:, :half] * (1 + 1e-4 * normal(outs, half))
    return x, w  # "cancels"


KINDS = ["one sign", "between 1 and 2", "largest dropped when cut", "one alone", "one dominates", "one in ten", "cancels"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("inner", [64, 260, 2048, 12288])
def test_operands_that_do_not_average_out(kind, inner):
    """No less exact than one fmaf chain whatever the operands; a tenth more for a product that stands alone, whose dropped part
    (0.09 x 2^-24 in the mean square, 2^-24 at most) joins one rounding (2^-24 / sqrt(12) of the mean operand), and for draws."""
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(inner)
    x, w = operands(kind, 70, 300, inner)
    out, simt = torch.empty(70, 300, device="cuda"), torch.empty(70, 300, device="cuda")
    tc.gemm_split(tc.SplitPlan(w), x, out)
    ops.gemm_simt(x, w, simt)
    assert tc.take_error() == 0
    want = x.double() @ w.double().T
    error = lambda y: float((y.double() - want).norm() / want.norm())  # noqa: E731
    assert error(out) <= 1.1 * error(simt)
    # of the products' absolute sum: what is dropped, a rounding per block of 64 and at the end, truncation within a block
    size = x.double().abs() @ w.double().abs().T
    assert float(((out.double() - want).abs() / size)[size > 0].max()) <= (inner / 64 + 16) * 2.0**-24


@pytest.mark.gpu
def test_activations_off_16_bytes_and_no_tokens():
    """A product of the parts takes both: the first on CUDA cores, the second without a launch."""
    from mini_engine_b200.engine.workspace import Workspace
    from mini_engine_b200.parts.linear import Linear

    class Context:
        workspace = Workspace(8, "cuda")

    torch.manual_seed(5)
    linear = Linear(torch.randn(70, 64, device="cuda"))
    x = torch.randn(3 * 64 + 1, device="cuda")[1:].view(3, 64)
    out = linear.forward(x, Context, "out")[0].clone()
    assert torch.allclose(out.double(), x.double() @ linear.weight.double().T, rtol=1e-5, atol=1e-4)
    assert linear.forward(x[:0].clone(), Context, "out").shape == (1, 0, 70)


@pytest.mark.gpu
def test_weights_that_tma_cannot_address_are_refused_by_the_rule():
    tc = tensor_core()
    base = torch.randn(4 * 128 + 1, device="cuda")
    assert tc.split_supports(base[: 4 * 128].view(4, 128))
    assert not tc.split_supports(base[1:].view(4, 128))  # starts on 4 bytes
    assert not tc.split_supports(torch.randn(4, 130, device="cuda"))
    assert not tc.split_supports(torch.randn(4, 60, device="cuda"))
    assert not tc.split_supports(torch.randn(4, 128, device="cuda").to(torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,units,top,outs,inner", [(1, 4, 1, 64, 64), (9, 8, 2, 130, 260), (70, 5, 3, 384, 1100), (300, 8, 2, 200, 520)])
def test_grouped_product_gives_the_bits_of_each_groups_own(tokens, units, top, outs, inner):
    """Rows sorted by unit, one unit without rows, choices outside the units; runs of 16 and of 64 rows, segments side by
    side and one after the other: every row has the bits of the product of its own unit's weight alone."""
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(tokens)
    h, w = torch.randn(tokens, inner, device="cuda"), torch.randn(units, outs, inner, device="cuda")
    scores = torch.rand(tokens, units + 1)
    scores[:, min(2, units - 1)] = -1.0  # nobody's choice unless all are needed
    chosen = scores.topk(top, dim=1).indices.to(torch.int32).cuda()  # `units` itself: outside
    alone = []
    for u in range(units):
        out = torch.empty(tokens, outs, device="cuda")
        tc.gemm_split(tc.SplitPlan(w[u].clone()), h, out)
        alone.append(out)
    plan = tc.SplitPlan(w.reshape(units * outs, inner), group_rows=outs)
    for pad in (16, 64):
        capacity = -(-(tokens * top + units * (pad - 1)) // pad) * pad
        ints = lambda *shape: torch.empty(shape, dtype=torch.int32, device="cuda")  # noqa: E731
        row_of, token_of, unit_of_block = ints(tokens, top), ints(capacity), ints(capacity // pad)
        ops.sort_by_unit(chosen=chosen, units=units, pad=pad, row_of=row_of, token_of=token_of, unit_of_block=unit_of_block)
        rows = torch.empty(capacity, inner, device="cuda")
        ops.gather_rows(h, token_of, rows)
        for side_by_side in (False, True):
            out = torch.full((capacity, outs), float("nan"), device="cuda")
            tc.gemm_split_grouped(plan, rows, out, unit_of_block, pad, units, side_by_side)
            assert tc.take_error() == 0
            for t in range(tokens):
                for u, row in zip(chosen[t].tolist(), row_of[t].tolist()):
                    assert (row < 0) == (u >= units)
                    if row >= 0:
                        assert torch.equal(out[row], alone[u][t])


@pytest.mark.gpu
@pytest.mark.parametrize("side_by_side", [False, True])
def test_a_wait_that_runs_out_is_reported_and_leaves_the_device_usable(side_by_side):
    """The product with its tiles withheld: every role gives up, the CTAs of a cluster meet all the same, the error reaches the host
    once, and tensor memory is free for the next product (512 columns an SM would be gone after two leaks)."""
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(6)
    x, w = torch.randn(20, 1100, device="cuda"), torch.randn(300, 1100, device="cuda")
    plan = tc.SplitPlan(w)
    assert plan.segments > 1 and tc.take_error() == 0
    out = torch.full((20, 300), 7.0, device="cuda")
    for _ in range(8):
        tc.split_wait_probe(plan, x, out, side_by_side)
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())  # nothing is written
    with pytest.raises(ops.KernelError, match="limit of a wait"):
        ops.raise_on_device_error()
    assert tc.take_error() == 0
    for form in [(16, side_by_side), (128, True)]:
        tc.gemm_split(plan, x, out, form)
        assert float((out.double() - x.double() @ w.double().T).abs().max()) < 1e-3
    assert tc.take_error() == 0


# 128 tokens to a CTA, one segment of 65 blocks (its rings go round 32 times, the last block is partial) and eight of 24 in a cluster; 64 to a CTA with
# segments one after the other, which the rule takes for the first, and of 192 blocks in all
@pytest.mark.gpu
@pytest.mark.parametrize("tokens,outs,inner,form", [(130, 20500, 4100, (128, False)), (200, 520, 12288, (128, True)), (70, 520, 12288, (64, True))])
def test_long_reductions_give_the_same_bits_in_every_form(tokens, outs, inner, form):
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(7)
    x, w = torch.randn(tokens, inner, device="cuda"), torch.randn(outs, inner, device="cuda")
    plan = tc.SplitPlan(w)
    assert (plan.segments == 1) == (form == (128, False))
    got = []
    for chosen in (form, (64, False), form):
        got.append(torch.full((tokens, outs), float("nan"), device="cuda"))
        tc.gemm_split(plan, x, got[-1], chosen)
    assert tc.take_error() == 0
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    simt, want = torch.empty(tokens, outs, device="cuda"), x.double() @ w.double().T
    ops.gemm_simt(x, w, simt)
    error = lambda y: float((y.double() - want).norm() / want.norm())  # noqa: E731
    assert error(got[0]) <= error(simt)  # of one fmaf chain, which is twice as far off at 1,024 already


@pytest.mark.gpu
def test_products_of_many_sizes_share_the_pieces_buffer():
    """Back to back through one workspace, smaller and larger than the one before; the last two read the same rows."""
    from mini_engine_b200.engine.workspace import Workspace

    tc = tensor_core()
    torch.manual_seed(8)
    workspace = Workspace(16, "cuda")
    runs = []
    for tokens, outs, inner in [(300, 520, 1100), (17, 130, 68), (64, 2048, 2048), (130, 520, 4100), (20, 200, 12288), (300, 640, 1100)]:
        x, w = torch.randn(tokens, inner, device="cuda"), torch.randn(outs, inner, device="cuda")
        runs.append((tc.SplitPlan(w), x, torch.full((tokens, outs), float("nan"), device="cuda"), torch.empty(tokens, outs, device="cuda")))
    runs.append((runs[0][0], runs[-1][1], torch.empty(300, 520, device="cuda"), torch.empty(300, 520, device="cuda")))
    for plan, x, out, _ in runs:
        tc.gemm_split(plan, x, out, workspace=workspace)
    for plan, x, _, alone in runs:
        tc.gemm_split(plan, x, alone)
    assert tc.take_error() == 0
    for _, _, out, alone in runs:
        assert torch.equal(out, alone)


@pytest.mark.gpu
def test_grouped_product_in_runs_of_128_gives_the_bits_of_each_groups_own():
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(9)
    tokens, units, top, outs, inner, pad = 300, 5, 2, 384, 1100, 128
    h, w = torch.randn(tokens, inner, device="cuda"), torch.randn(units, outs, inner, device="cuda")
    chosen = torch.rand(tokens, units).topk(top, dim=1).indices.to(torch.int32).cuda()
    capacity = -(-(tokens * top + units * (pad - 1)) // pad) * pad
    ints = lambda *shape: torch.empty(shape, dtype=torch.int32, device="cuda")  # noqa: E731
    row_of, token_of, unit_of_block = ints(tokens, top), ints(capacity), ints(capacity // pad)
    ops.sort_by_unit(chosen=chosen, units=units, pad=pad, row_of=row_of, token_of=token_of, unit_of_block=unit_of_block)
    rows = torch.empty(capacity, inner, device="cuda")
    ops.gather_rows(h, token_of, rows)
    plan = tc.SplitPlan(w.reshape(units * outs, inner), group_rows=outs)
    assert plan.segments > 1
    out = torch.full((capacity, outs), float("nan"), device="cuda")
    tc.gemm_split_grouped(plan, rows, out, unit_of_block, pad, units, True)
    assert tc.take_error() == 0
    for u in range(units):
        alone = torch.empty(tokens, outs, device="cuda")
        tc.gemm_split(tc.SplitPlan(w[u].clone()), h, alone)
        at, place = (chosen == u).nonzero(as_tuple=True)
        assert torch.equal(out[row_of[at, place].long()], alone[at])


@pytest.mark.gpu
@pytest.mark.parametrize("tile,side_by_side", [(64, False), (64, True), (128, True)])
def test_giving_up_with_pieces_in_flight(tile, side_by_side):
    """The forms whose tokens arrive as pieces: these are on their way when every role gives up, and have landed before shared memory is
    given back.  Registers, barriers and tensor memory serve the next products."""
    from mini_engine_b200.csrc import ops

    tc = tensor_core()
    torch.manual_seed(10)
    x, w = torch.randn(150, 1100, device="cuda"), torch.randn(300, 1100, device="cuda")
    plan = tc.SplitPlan(w)
    assert plan.segments > 1 and tc.take_error() == 0
    out, want = torch.full((150, 300), 7.0, device="cuda"), torch.empty(150, 300, device="cuda")
    tc.gemm_split(plan, x, want, (16, False))
    for _ in range(8):
        tc.split_wait_probe(plan, x, out, side_by_side, tile)
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())  # nothing is written
    with pytest.raises(ops.KernelError, match="limit of a wait") as raised:
        ops.raise_on_device_error()
    assert f"code {5 << 8}" not in str(raised.value)  # the producer saw its copies land
    for form in [(tile, side_by_side), (16, True), (128, True)]:
        tc.gemm_split(plan, x, out, form)
        assert torch.equal(out, want)
    assert tc.take_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tile,side_by_side", [(64, False), (64, True), (128, True)])
def test_rows_beyond_the_room_for_pieces_run_in_parts(monkeypatch, tile, side_by_side):
    """The same bits, and no more room however many rows there are; a last part of few rows, room for less than a tile, and groups."""
    from mini_engine_b200.csrc import ops
    from mini_engine_b200.engine.workspace import Workspace

    tc = tensor_core()
    torch.manual_seed(11)
    x, w = torch.randn(1000, 1100, device="cuda"), torch.randn(300, 1100, device="cuda")
    plan, want = tc.SplitPlan(w), torch.empty(1000, 300, device="cuda")
    tc.gemm_split(plan, x, want, (tile, side_by_side))
    row = 3 * 2 * 1104
    for room in (row, 200 * row, 331 * row, 999 * row):
        monkeypatch.setattr(tc, "SPLIT_PIECES_BYTES", room)
        workspace, out = Workspace(16, "cuda"), torch.full((1000, 300), float("nan"), device="cuda")
        launches = ops.launch_count()
        tc.gemm_split(plan, x, out, (tile, side_by_side), workspace)
        assert ops.launch_count() - launches >= 4
        assert workspace.bytes_held() <= max(room, tile * row)
        assert torch.equal(out, want)
    monkeypatch.setattr(tc, "SPLIT_PIECES_BYTES", 2 * tile * row)
    groups = torch.tensor([1, -1, 0, 2, 2, 1, 0], dtype=torch.int32, device="cuda")
    grouped = tc.SplitPlan(w.clone(), group_rows=100)
    out = torch.full((7 * tile, 100), float("nan"), device="cuda")
    tc.gemm_split_grouped(grouped, x[: 7 * tile].contiguous(), out, groups, tile, 6, side_by_side)
    assert tc.take_error() == 0
    for b, group in enumerate(groups.tolist()):
        got = out[b * tile : (b + 1) * tile]
        if group < 0:
            assert bool(got.isnan().all())
            continue
        alone = torch.empty(tile, 100, device="cuda")
        tc.gemm_split(tc.SplitPlan(w[100 * group : 100 * group + 100].clone()), x[b * tile : (b + 1) * tile].clone(), alone)
        assert torch.equal(got, alone)
