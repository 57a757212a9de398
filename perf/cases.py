"""Timed cases of the engine: one step of a model through the step function, as a serving program drives it.

A case is a model (design, layer sizes, layers), a dtype, a page size and the entries of one step.  ``past`` and ``new`` list per
entry how many of its tokens the cache holds already and how many the step brings: ``past=2048, new=1`` is a decoding request,
``past=0, new=2048`` a whole prompt, ``past=512, new=512`` the second portion of a prompt.  A step of single tokens replays the
engine's decode graph, one short prompt alone the engine's prompt graph, every other step is run eagerly: the rule that the
engine's own loop follows.  The result is the logits behind every entry's last token.

Repeating a pass writes the same keys and values to the same places again; a design with states per request moves them on
by the same tokens.  Designs that route tokens to units (Molotar, Bizurax, Tobadra) are run in float32: in bfloat16 one token in
some fifty changes a unit when anything before the router is rounded in another way, and its logits then say nothing.

``exact`` restates every design over whole sequences in float64, without cache and batching.
"""

import math
import random

import torch

from mini_engine_b200 import EngineConfig, LLMEngine
from mini_engine_b200.cli.design_bench import SIZES, configs
from mini_engine_b200.config import Qwen3Config
from mini_engine_b200.config.registry import architecture_for
from mini_engine_b200.engine.batch import StepEntry
from mini_engine_b200.parts.model import DecoderModel
from mini_engine_b200.weights.loader import place_tensors

ROUTED = ("molotar", "bizurax", "tobadra")
QWEN3 = {  # width, feed-forward width, query heads, KV heads, vocabulary, tied head; heads of 128
    "0.6b": (1024, 3072, 16, 8, 151936, True),
    "1b": (2048, 6144, 16, 8, 32768, True),
    "8b": (4096, 12288, 32, 8, 151936, False),
    "32b": (5120, 25600, 64, 8, 151936, False),
}
FILL = 2048  # tokens of one step while the caches are filled


def listed():
    case = lambda name, design, size, layers, dtype, past, new, page=16: dict(  # noqa: E731
        name=name, design=design, size=size, layers=layers, dtype=dtype, page=page, past=past, new=new
    )
    return [
        # one conversation with a small model: launches and their latency
        case("qwen3 0.6b decode 1", "qwen3", "0.6b", 28, "bfloat16", "300", "1"),
        # the headline: eight conversations of 2,048 tokens, a quarter of the layers of the 8B sizes (all are alike)
        case("qwen3 8b decode 8", "qwen3", "8b", 9, "bfloat16", "2048" + ",2048" * 7, "1" + ",1" * 7),
        # the headline's other half: one prompt of 2,048 tokens
        case("qwen3 8b prompt 2048", "qwen3", "8b", 9, "bfloat16", "0", "2048"),
        # chunked prefill under load: portions of 512 tokens beside decoding requests of unlike lengths
        case("qwen3 32b mixed", "qwen3", "32b", 2, "bfloat16", "512,512,0,0" + ",4096,1777,255,3001" * 8, "512,512,512,437" + ",1" * 32),
        # the 32-bit path at full layer sizes: what a bfloat16 run is checked with
        case("qwen3 8b float32 256", "qwen3", "8b", 4, "float32", "0", "256"),
        # a long prompt for the design with mixed heads beside a linear attention
        case("pimezen 8b prompt 2048", "pimezen", "8b", 4, "bfloat16", "0", "2048"),
        # eight of its requests decoding at unlike lengths
        case("pimezen 1b decode 8", "pimezen", "1b", 4, "bfloat16", "2048,1999,1500,1024,777,300,65,16", "1" + ",1" * 7),
        # three short prompts at once, odd lengths; sorted units, gated recurrence, 32-bit
        case("molotar 1b float32 prompts", "molotar", "1b", 4, "float32", "0,0,0", "301,173,38"),
        # three prompts of very unlike lengths; latent attention, windows, distance bias
        case("bevadra 8b prompts", "bevadra", "8b", 4, "bfloat16", "0,0,0", "1337,700,11"),
        # eight requests decoding in 32-bit; several residual streams, retention, latent attention
        case("bizurax 1b float32 decode 8", "bizurax", "1b", 4, "float32", "512,512,500,411,256,255,100,17", "1" + ",1" * 7),
        # a prompt in 32-bit; lightning attention, delta rule, routed units beside a shared one
        case("tobadra 1b float32 prompt", "tobadra", "1b", 4, "float32", "0", "512"),
        # an odd prompt for the design with matrix states; loop, token shift, sigmoid attention in chunks
        case("vufadra 8b prompt 1777", "vufadra", "8b", 4, "bfloat16", "0", "1777"),
    ]


def spread(rng, low, high):
    """A whole number between low and high, evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng: random.Random):
    design = rng.choice(["qwen3", "qwen3", "pimezen", "molotar", "bevadra", "bizurax", "tobadra", "vufadra"])
    if design == "qwen3":
        size, layers = rng.choice([("0.6b", 28), ("1b", 4), ("8b", 4), ("32b", 2)])
    else:
        size, layers = rng.choice(["1b", "8b"]), 4
    dtype = "float32" if design in ROUTED or rng.random() < 0.2 else "bfloat16"
    if dtype == "float32":
        size, layers = "1b", 4
    most = 512 if dtype == "float32" else 2048
    past, new = [], []
    kind = rng.choice(["decode", "prompts", "prompts", "mixed"])
    if kind in ("prompts", "mixed"):
        room = spread(rng, 2, most if kind == "prompts" else most // 2)
        for i in range(rng.choice([1, 1, 2, 3])):
            count = room if i == 0 else spread(rng, 1, room)
            if sum(new) + count <= most:
                past.append(rng.choice([0, 0, spread(rng, 1, most - count)]) if count < most else 0)
                new.append(count)
    if kind in ("decode", "mixed"):
        for _ in range(spread(rng, 1, 16 if dtype == "float32" else 64)):
            context = spread(rng, 8, most)
            if sum(past) + context <= 16 * most:
                past.append(context)
                new.append(1)
    return dict(design=design, size=size, layers=layers, dtype=dtype, page=rng.choice([8, 16, 16, 32]),
                past=",".join(map(str, past)), new=",".join(map(str, new)))  # fmt: skip


def entries_of(case):
    return list(zip([int(n) for n in case["past"].split(",")], [int(n) for n in case["new"].split(",")]))


def config_of(case):
    if case["design"] != "qwen3":
        return configs(SIZES[case["size"]], case["design"])[case["design"]]
    width, ff, heads, kv_heads, vocab, tied = QWEN3[case["size"]]
    return Qwen3Config(
        vocab_size=vocab, hidden_size=width, intermediate_size=ff, num_hidden_layers=case["layers"], num_attention_heads=heads,
        num_key_value_heads=kv_heads, head_dim=128, rms_norm_eps=1e-6, rope_theta=1e6, max_position_embeddings=8192,
        tie_word_embeddings=tied,
    )  # fmt: skip


def weights_of(case, specs, seed):
    """Tensors by name, from the seed alone: matrices in the case's dtype, vectors in float32."""
    generator = torch.Generator("cuda").manual_seed(seed)
    made = {}
    for spec in specs:
        if spec.alias_of is not None or spec.optional:
            continue
        if spec.role == "table":
            made[spec.name] = torch.zeros(spec.shape, dtype=torch.int32, device="cuda")
            continue
        values = torch.randn(spec.shape, generator=generator, device="cuda")
        if spec.init == "ones_normal":
            values = 1.0 + 0.1 * values
        elif spec.init == "small_normal":
            values *= 0.1
        elif spec.init == "eye_normal":
            values = 0.1 * values + torch.eye(*spec.shape, device="cuda")
        elif spec.init == "positive":
            values = 0.05 + 0.1 * values.abs()
        elif spec.init != "wide_normal":
            values *= 0.02
        made[spec.name] = values.to(getattr(torch, case["dtype"])) if spec.role == "matrix" else values
    return made


def tokens_of(case, seed, vocab):
    """The tokens of every entry's request, past ones first."""
    generator = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (past + new,), generator=generator).tolist() for past, new in entries_of(case)]


@torch.inference_mode()
def prepare(case, seed):
    """An engine with loaded weights whose cache holds what the step's requests have behind them, and the step's entries."""
    config = config_of(case)
    model = DecoderModel(architecture_for(config.architecture).build_spec(config))
    specs = model.weight_specs()
    dtype = getattr(torch, case["dtype"])
    model.load(place_tensors(weights_of(case, specs, seed), specs, dtype, "cuda"))
    step, page = entries_of(case), case["page"]
    budget = max(sum(new for _, new in step), min(FILL, max(past for past, _ in step)), len(step))
    longest = max(past + new for past, new in step)
    engine = LLMEngine(model, EngineConfig(
        block_size=page, num_blocks=sum(-(-(past + new) // page) for past, new in step) + 1, max_num_seqs=len(step),
        max_num_batched_tokens=budget, max_model_len=-(-longest // page) * page, enable_prefix_caching=False, dtype=dtype))  # fmt: skip
    entries = []
    for (past, new), ids in zip(step, tokens_of(case, seed, config.vocab_size)):
        cache = engine.block_manager.new_request()
        if not engine.block_manager.try_allocate(cache, past + new):
            raise MemoryError("the pool is too small for the case")
        for begin in range(0, past, FILL):
            engine.runner.execute([StepEntry(cache, begin, ids[begin : min(past, begin + FILL)], ())])
        entries.append(StepEntry(cache, past, ids[past:], (new - 1,)))
    return engine, entries


@torch.inference_mode()
def run(state):
    """One step; float32 logits [entries, vocabulary]."""
    engine, entries = state
    if all(len(entry.token_ids) == 1 for entry in entries):
        return engine.decode_graphs.run(entries)
    logits = engine.prompt_graphs.run(entries[0]) if len(entries) == 1 and engine.prompt_graphs is not None else None
    return engine.runner.execute(entries) if logits is None else logits


# ------------------------------------------------------------------------------------------------ work


def layer_plans(case):
    """Per layer run: what its mixer keeps and reads, from the configuration's own keys."""
    config = config_of(case)
    if case["design"] == "qwen3":
        c = dict(heads=config.num_attention_heads, kv_heads=config.num_key_value_heads, dim=128, vdim=128)
        return [("attention", c)] * case["layers"]
    plans = []
    for layer in config.to_dict()["layers"]:
        plans.append((layer["type"], layer["mixer"]))
    return plans


def seen(past, new, mask):
    """Keys that the new tokens see, summed over them, and how many distinct ones of the past."""
    window = (mask or {}).get("size")
    if window is None:
        return new * past + new * (new + 1) // 2, past
    keep = (mask or {}).get("keep_first", 0)
    total = sum(min(p + 1, window + min(keep, max(0, p + 1 - window))) for p in range(past, past + new))
    return total, min(past, window + keep)


def work(case):
    """Every weight that the step needs once, the caches and states that it reads and writes, the logits; multiply-adds as two."""
    config = config_of(case)
    specs = DecoderModel(architecture_for(config.architecture).build_spec(config)).weight_specs()
    step, tokens = entries_of(case), sum(new for _, new in entries_of(case))
    size = 4 if case["dtype"] == "float32" else 2
    raw = config.to_dict()
    router = next((l["mlp"]["router"] for l in raw.get("layers", []) if l.get("mlp") and l["mlp"].get("router")), None)
    units = (router["experts"] + router.get("identity", 0)) if router else 1
    share = router["top"] / units if router else 1.0
    touched = 1.0 - (1.0 - share) ** tokens
    nbytes, flops, width = 0.0, 0.0, None
    for spec in specs:
        count = math.prod(spec.shape)
        if spec.role != "matrix" or spec.optional:
            continue
        name = spec.name
        if name in ("embed", "bigram", "model.embed_tokens.weight"):
            width = spec.shape[1]
            nbytes += tokens * width * size
            continue
        if name in ("lm_head.weight", "head"):
            continue
        if ".mlp.e" in name:
            nbytes, flops = nbytes + touched * count * size, flops + 2 * tokens * share * count
        else:
            nbytes, flops = nbytes + count * size, flops + 2 * tokens * count
    vocab = config.vocab_size
    nbytes += vocab * width * size + len(step) * vocab * 4
    flops += 2.0 * len(step) * vocab * width
    for kind, mixer in layer_plans(case):
        for part_kind, m in ((("attention", mixer["left"]), ("state", mixer["right"])) if kind == "parallel" else ((kind, mixer),)):
            for past, new in step:
                if part_kind in ("attention", "latent_attention"):
                    total, rows = seen(past, new, m.get("mask"))
                    if part_kind == "attention":
                        per_key, per_pair = m["kv_heads"] * (m["dim"] + m["vdim"]), 2 * m["heads"] * (m["dim"] + m["vdim"])
                    else:
                        per_key, per_pair = m["kv_rank"] + m["rot_dim"], 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
                    nbytes += (rows + new) * per_key * size
                    flops += total * per_pair
                elif part_kind == "rglru":
                    nbytes += 2 * m["width"] * 4
                    flops += new * m["width"] * 8
                else:
                    cells = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
                    nbytes += (2 if past else 1) * cells * 4
                    flops += new * cells * (8 if "delta" in part_kind else 5)
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """What the logits were seen to be off the float64 ones: 1e-6 to 2e-5 in float32 (four times that is stated), 0.003 to 0.042
    in bfloat16, where every activation is rounded between the kernels and a deep or looped model adds its layers' roundings up."""
    return {"rel": 8e-5} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.4}


# ------------------------------------------------------------------- the designs over whole sequences


class Weights:
    """Tensors by name, widened to float64 when they are asked for."""

    def __init__(self, tensors, prefix=""):
        self.tensors, self.prefix = tensors, prefix

    def __call__(self, name):
        return self.tensors[self.prefix + name].double()

    def under(self, prefix):
        return Weights(self.tensors, self.prefix + prefix)

    def has(self, name):
        return self.prefix + name in self.tensors


def linear(x, w, name):
    y = x @ w(name).T
    return y + w(name + ".b") if w.has(name + ".b") else y


def unit(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def rms(x, weight, eps):
    return unit(x, eps) * weight


def gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


silu = torch.nn.functional.silu


def places(x):
    return torch.arange(x.shape[0], device=x.device)


def turn(x, rot, pairs=False, back=False):
    """The first ``dims`` elements of every head of ``x [T, heads, d]`` turned by position times frequency."""
    dims, base, scaling = rot["dims"], rot["base"], rot.get("scaling") or {}
    half, gain = dims // 2, 1.0
    freq = [base ** (-2.0 * i / dims) for i in range(half)]
    if "high" in scaling:  # waves longer than `original` are stretched, those between blended
        for i, f in enumerate(freq):
            blend = (scaling["original"] * f / (2 * math.pi) - scaling["low"]) / (scaling["high"] - scaling["low"])
            blend = min(1.0, max(0.0, blend))
            freq[i] = (1 - blend) * f / scaling["factor"] + blend * f
    elif "fast" in scaling:  # a ramp over the elements between two numbers of turns, and a gain
        at = lambda t: dims * math.log(scaling["original"] / (2 * math.pi * t)) / (2 * math.log(base))  # noqa: E731
        low, high = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
        for i, f in enumerate(freq):
            ramp = min(1.0, max(0.0, (i - low) / max(high - low, 1e-3)))
            freq[i] = f / scaling["factor"] * ramp + f * (1 - ramp)
        gain = 0.1 * math.log(scaling["factor"]) + 1.0
    elif scaling:
        freq = [f / scaling["factor"] for f in freq]
    angle = places(x).double().view(-1, 1, 1) * torch.tensor(freq, dtype=torch.float64, device=x.device)
    cos, sin = angle.cos() * gain, angle.sin() * (-gain if back else gain)
    out = x.clone()
    first, second = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, half), slice(half, dims))
    u, v = x[..., first], x[..., second]
    out[..., first], out[..., second] = u * cos - v * sin, v * cos + u * sin
    return out


def visible(x, mask, chunks=False):
    i, j = places(x).view(-1, 1), places(x).view(1, -1)
    size = (mask or {}).get("size")
    if size is None:
        return j <= i
    if chunks:
        return (j <= i) & (i // size == j // size)
    return (j <= i) & ((i - j < size) | (j < mask.get("keep_first", 0)))


def weigh(scores, allowed, extra=None):
    """Softmax over the visible keys of ``[H, T, T]``; ``extra [H]`` joins the denominator alone."""
    scores = scores.masked_fill_(~allowed, -math.inf)
    if extra is None:
        return torch.softmax(scores, -1)
    extra = extra.view(-1, 1, 1).expand(-1, scores.shape[1], 1)
    return torch.softmax(torch.cat((scores, extra), -1), -1)[..., :-1]


def by_head(x, heads):
    return x.view(x.shape[0], heads, -1)


def attend(q, k, v, weights):
    """``weights(scores, heads)`` of groups of query heads, so that ``[H, T, T]`` stays small."""
    group = q.shape[1] // k.shape[1]
    out = []
    for g in range(k.shape[1]):
        heads = slice(g * group, (g + 1) * group)
        scores = torch.einsum("ihd,jd->hij", q[:, heads], k[:, g])
        out.append(torch.einsum("hij,jd->ihd", weights(scores, heads), v[:, g]))
    return torch.cat(out, 1)


def states(q, k, v, step):
    """``step(state, t)`` for every token: the next state ``[H, d, e]`` and the state that the query reads."""
    state, out = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=k.dtype, device=k.device), []
    for t in range(q.shape[0]):
        state, read = step(state, t)
        out.append((q[t].unsqueeze(1) @ read).squeeze(1))
    return torch.stack(out)


def shifted(x, taps):
    """Per channel the sum of the last tokens under ``taps [C, K]``."""
    count = taps.shape[1]
    x = torch.nn.functional.pad(x, (0, 0, count - 1, 0))
    return sum(x[j : x.shape[0] - count + 1 + j] * taps[:, j] for j in range(count))


def qwen3_attention(x, w, c, eps):
    q, k, v = (by_head(x @ w(n + "_proj.weight").T, h) for n, h in (("q", c["heads"]), ("k", c["kv_heads"]), ("v", c["kv_heads"])))
    rot = {"dims": c["dim"], "base": c["theta"]}
    q, k = turn(rms(q, w("q_norm.weight"), eps), rot), turn(rms(k, w("k_norm.weight"), eps), rot)
    o = attend(q, k, v, lambda s, h: weigh(s * c["dim"] ** -0.5, visible(x, None)))
    return o.flatten(1) @ w("o_proj.weight").T


def qwen3(config, w, ids, rows):
    c = dict(heads=config.num_attention_heads, kv_heads=config.num_key_value_heads, dim=config.head_dim, theta=config.rope_theta)
    eps, x = config.rms_norm_eps, w.tensors["model.embed_tokens.weight"][ids].double()
    for i in range(config.num_hidden_layers):
        l = w.under(f"model.layers.{i}.")
        x = x + qwen3_attention(rms(x, l("input_layernorm.weight"), eps), l.under("self_attn."), c, eps)
        h = rms(x, l("post_attention_layernorm.weight"), eps)
        gated = silu(h @ l("mlp.gate_proj.weight").T) * (h @ l("mlp.up_proj.weight").T)
        x = x + gated @ l("mlp.down_proj.weight").T
    head = "model.embed_tokens.weight" if config.tie_word_embeddings else "lm_head.weight"
    return rms(x[rows], w("model.norm.weight"), eps) @ w(head).T


def clamped_unit(x, w, limit):
    g, u = linear(x, w, "gate").clamp(max=limit), linear(x, w, "up").clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w("down").T


def pimezen(raw, w, ids, rows):
    eps, x = raw["norm"]["eps"], w.tensors["embed"][ids].double()
    for i, layer in enumerate(raw["layers"]):
        l, m, r = w.under(f"l{i}."), layer["mixer"]["left"], layer["mixer"]["right"]
        h = unit(x, eps) * (1 + l("norm1"))
        left, right = l.under("mix.left."), l.under("mix.right.")
        q = rms(by_head(linear(h, left, "q"), m["heads"]), left("q.norm"), eps)
        k = rms(by_head(linear(h, left, "k"), m["kv_heads"]), left("k.norm"), eps)
        v = by_head(linear(h, left, "v"), m["kv_heads"])
        apart = (places(x).view(-1, 1) - places(x).view(1, -1)).clamp(min=0).double()
        group, mixed = m["heads"] // m["kv_heads"], []
        probs = torch.cat([
            weigh((q[:, j] @ k[:, j // group].T * m["scale"] - left("r1")[j] * torch.log1p(left("r2")[j] * apart))[None], visible(x, m["mask"]))
            for j in range(m["heads"])])  # fmt: skip
        for j in range(m["heads"]):
            mixed.append(torch.einsum("g,gij->ij", left("talk")[j], probs) @ v[:, j // group])
        del probs
        y = layer["mixer"]["left_scale"] * (torch.cat(mixed, 1) @ left("o").T)
        q, k, v = (by_head(linear(h, right, n), r["heads"]) for n in "qkv")
        keep = torch.sigmoid(h @ right("a1").T @ right("a2").T + right("a2.b")).pow(1 / r["tau"]).view_as(k)

        def step(s, t):
            s = keep[t].unsqueeze(2) * s + k[t].unsqueeze(2) * v[t].unsqueeze(1)
            return s, s

        o = rms(states(q * r["dim"] ** -0.5, k, v, step), right("norm"), eps).flatten(1)
        y = y + layer["mixer"]["right_scale"] * ((o * silu(linear(h, right, "g"))) @ right("o").T)
        x = x + l("ls1") * y
        if layer["mlp"]:
            x = x + l("ls2") * clamped_unit(unit(x, eps) * (1 + l("norm2")), l.under("mlp."), layer["mlp"]["limit"])
    return unit(x[rows], eps) * (1 + w("final.norm")) @ w("embed").T


def pair_embedding(raw, w, ids):
    e = raw.get("embedding") or {}
    x = w.tensors["embed"][ids].double() * e.get("scale", 1.0)
    if e.get("bigram"):
        b = e["bigram"]
        row = torch.full_like(ids, b["buckets"])
        row[1:] = (ids[:-1] * b["mul_prev"] + ids[1:] * b["mul_cur"]) % b["buckets"]
        x = x + w.tensors["bigram"][row].double()
    return x


def channel_recurrence(h, w, m):
    blocks, gate = m["blocks"], {}
    y = gelu(linear(h, w, "y"))
    u = shifted(linear(h, w, "x"), w("conv")) + w("conv.b")
    for name in ("ra", "ri"):
        gate[name] = torch.sigmoid(torch.einsum("tbi,boi->tbo", by_head(u, blocks), w(name)) + w(name + ".b")).flatten(1)
    log_a = -8 * gate["ra"] * torch.nn.functional.softplus(w("lam"))
    a, drive = log_a.exp(), torch.sqrt(-torch.expm1(2 * log_a)) * gate["ri"] * u
    state, out = torch.zeros_like(a[0]), []
    for t in range(h.shape[0]):
        state = a[t] * state + drive[t]
        out.append(state)
    return (torch.stack(out) * y) @ w("o").T


def spread_units(h, chosen, weight, count, unit_of):
    out = torch.zeros_like(h)
    for e in range(count):
        row, place = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            out.index_add_(0, row, weight[row, place].unsqueeze(1) * unit_of(h[row], e))
    return out


def best_groups(worth, keep, per):
    kept = torch.zeros_like(worth, dtype=torch.bool).scatter_(1, worth.topk(keep, 1).indices, True)
    return kept.repeat_interleave(per, 1)


def molotar(raw, w, ids, rows):
    eps, alpha, x, kept = raw["norm"]["eps"], raw["postln_alpha"], pair_embedding(raw, w, ids), {}
    for i, layer in enumerate(raw["layers"]):
        l, m = w.under(f"l{i}."), layer["mixer"]
        p = l.under("mix.")
        if layer["type"] == "attention":
            q = by_head(rms(linear(x, p, "q"), p("q.norm"), eps), m["heads"])
            q = turn(q, m["rot"]) if m.get("rot") else q
            if m.get("kv_from") is None:
                k = by_head(rms(linear(x, p, "k"), p("k.norm"), eps), m["kv_heads"])
                kept[i] = (turn(k, m["rot"]) if m.get("rot") else k, by_head(linear(x, p, "v"), m["kv_heads"]))
            source = i if m.get("kv_from") is None else m["kv_from"]
            kept[i] = kept[source]
            silent, allowed = torch.zeros(m["heads"], dtype=x.dtype, device=x.device), visible(x, m.get("mask"))
            o = attend(q, *kept[i], lambda s, h: weigh(s * m["scale"], allowed, silent[h]))
            y = (o * torch.sigmoid(linear(x, p, "g")).unsqueeze(2)).flatten(1) @ p("o").T
        else:
            y = channel_recurrence(x, p, m)
        x = rms(alpha * x + y, l("norm1"), eps)
        if layer.get("mlp"):
            p, r = l.under("mlp."), layer["mlp"]["router"]
            score = torch.sigmoid(x @ p("router").T)
            if r.get("groups"):
                per = r["experts"] // r["groups"]["count"]
                worth = score.view(len(score), -1, per).topk(min(2, per), -1).values.sum(-1)
                allowed = best_groups(worth, r["groups"]["keep"], per)
            else:
                allowed = torch.ones_like(score, dtype=torch.bool)
            chosen = score.masked_fill(~allowed, -1).topk(r["top"], 1).indices
            weight = score.gather(1, chosen)
            weight = weight / (weight.sum(1, keepdim=True) + 1e-20) * r["scale"]
            limit = layer["mlp"]["expert"]["limit"]
            y = spread_units(x, chosen, weight, r["experts"], lambda h, e: clamped_unit(h, p.under(f"e{e}."), limit))
            x = rms(alpha * x + y, l("norm2"), eps)
    return rms(x[rows], w("final.norm"), eps) @ w("head").T


def layer_norm(x, w, name, eps):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], w(name), w(name + ".b"), eps)


def latent_attention(h, w, m, eps, pairs):
    q = rms(h @ w("dq").T, w("dq.norm"), eps) @ w("uq").T if w.has("dq") else h @ w("q").T
    q, down, rank = by_head(q, m["heads"]), h @ w("dkv").T, m["kv_rank"]
    c = rms(down[:, :rank], w("dkv.norm"), eps)
    q = torch.cat((q[..., : m["dim"]], turn(q[..., m["dim"] :], m["rot"], pairs)), -1)
    shared = turn(down[:, None, rank:], m["rot"], pairs).expand(-1, m["heads"], -1)
    k = torch.cat((by_head(c @ w("uk").T, m["heads"]), shared), -1)
    allowed = visible(h, m.get("mask"))
    o = attend(q, k, by_head(c @ w("uv").T, m["heads"]), lambda s, _: weigh(s * m["scale"], allowed))
    if w.has("g"):
        o = o * torch.sigmoid(h @ w("g").T).unsqueeze(2)
    return o.flatten(1) @ w("o").T


def bevadra(raw, w, ids, rows):
    eps, x, kept = raw["norm"]["eps"], w.tensors["embed"][ids].double(), {}
    for i, layer in enumerate(raw["layers"]):
        l, m = w.under(f"l{i}."), layer["mixer"]
        p, h = l.under("mix."), layer_norm(x, l, "norm1", eps)
        if layer["type"] == "attention":
            source = i if m.get("kv_from") is None else m["kv_from"]
            if source == i:
                kept[i] = tuple(by_head(linear(h, p, n), m["kv_heads"]) for n in "kv")
            slope = torch.tensor([2.0 ** (-8.0 * (j + 1) / m["heads"]) for j in range(m["heads"])], dtype=x.dtype, device=x.device)
            apart, allowed = (places(x).view(-1, 1) - places(x).view(1, -1)).double(), visible(x, m.get("mask"))
            o = attend(by_head(linear(h, p, "q"), m["heads"]), *kept[source],
                       lambda s, j: weigh(s * m["scale"] - slope[j].view(-1, 1, 1) * apart, allowed, p("sink")[j]))  # fmt: skip
            y = linear(o.flatten(1) * torch.sigmoid(h @ p("g").T), p, "o")
        else:
            y = latent_attention(h, p, m, eps, pairs=False)
        if layer.get("mlp"):
            f = l.under("mlp.")
            y = y + (gelu(h @ f("gate").T) * (h @ f("up").T)) @ f("down").T
        x = x + y
    logits = layer_norm(x[rows], w, "final.norm", eps) @ w("embed").T
    cap = raw.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def decaying(q, k, v, decay):
    a = torch.tensor(decay, dtype=k.dtype, device=k.device).view(-1, 1, 1)

    def step(s, t):
        s = a * s + k[t].unsqueeze(2) * v[t].unsqueeze(1)
        return s, s

    return states(q, k, v, step)


def swiglu(h, w):
    return (silu(h @ w("gate").T) * (h @ w("up").T)) @ w("down").T


def bizurax(raw, w, ids, rows):
    eps, mult = raw["norm"]["eps"], raw.get("residual_mult", 1.0)
    x = w.tensors["embed"][ids].double()
    s = x.unsqueeze(0).repeat(raw["streams"], 1, 1)
    for i, layer in enumerate(raw["layers"]):
        l, m = w.under(f"l{i}."), layer["mixer"]
        p = l.under("mix.")
        for n in (1, 2):
            if n == 2 and not layer.get("mlp"):
                continue
            c = l.under(f"hc{n}.")
            h = rms(torch.einsum("s,stw->tw", c("in"), s), l(f"norm{n}"), eps)
            if n == 2:
                p, mlp = l.under("mlp."), layer["mlp"]
                if mlp["kind"] == "dense":
                    y = torch.relu(h @ p("up").T).square() @ p("down").T
                else:
                    best = linear(h, p, "router").topk(mlp["router"]["top"], 1)
                    y = spread_units(h, best.indices, best.values.softmax(1), mlp["router"]["experts"], lambda z, e: swiglu(z, p.under(f"e{e}.")))
                    y = y + swiglu(h, p.under("shared.")) if mlp.get("shared") else y
            elif layer["type"] == "attention":
                q, k, v = (by_head(linear(h, p, a), b) for a, b in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
                cap = m["softcap"]
                o = attend(unit(turn(q, m["rot"]), eps), unit(turn(k, m["rot"]), eps), v,
                           lambda a, j: weigh(cap * torch.tanh(a * m["scale"] / cap), visible(h, None), p("sink")[j]))  # fmt: skip
                y = o.flatten(1) @ p("o").T
            elif layer["type"] == "latent_attention":
                y = latent_attention(h, p, m, eps, pairs=True)
            else:
                q, k, v = (by_head(h @ p(a).T, m["heads"]) for a in "qkv")
                o = unit(decaying(turn(q, m["rot"]), turn(k, m["rot"]) * m["dim"] ** -0.5, v, m["decay"]), eps)
                y = (o.flatten(1) * silu(h @ p("g").T)) @ p("o").T
            s = torch.einsum("sr,stw->rtw", c("mix"), s) + mult * c("out").view(-1, 1, 1) * y
    return rms(s.sum(0)[rows], w("final.norm"), eps) @ w("head").T


def channel_delta(h, w, m, eps):
    heads, group = m["heads"], m["heads"] // m["kv_heads"]
    q, k, v = (silu(shifted(h @ w(n).T, w(n + ".conv"))) for n in "qkv")
    length = lambda a: a * torch.rsqrt(a.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q, k = (length(by_head(a, m["kv_heads"])).repeat_interleave(group, 1) for a in (q, k))
    v, rate = by_head(v, heads), torch.sigmoid(h @ w("b").T)
    z = by_head(torch.nn.functional.softplus(h @ w("a1").T @ w("a2").T + w("dt_bias")), heads)
    keep = torch.exp(-w("A_log").exp().view(1, heads, 1) * z)

    def step(s, t):
        s = keep[t].unsqueeze(2) * s
        u = rate[t].unsqueeze(1) * (v[t] - (k[t].unsqueeze(1) @ s).squeeze(1))
        s = s + k[t].unsqueeze(2) * u.unsqueeze(1)
        return s, s

    o = rms(states(q * m["dim"] ** -0.5, k, v, step), w("norm"), eps).flatten(1)
    return (o * torch.sigmoid(h @ w("g1").T @ w("g2").T)) @ w("o").T


def tobadra_mixer(kind, h, w, m, eps):
    if kind == "channel_delta":
        return channel_delta(h, w, m, eps)
    if kind == "lightning":
        q, k, v = (by_head(silu(h @ w(n).T), m["heads"]) for n in "qkv")
        o = rms(decaying(q, k, v, m["decay"]).flatten(1), w("norm"), eps)
        return (o * torch.sigmoid(h @ w("g").T)) @ w("o").T
    q, k, v = (by_head(linear(h, w, a), b) for a, b in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
    whole, allowed = {"dims": m["vdim"], "base": m["rot"]["base"]}, visible(h, m["mask"])
    o = attend(turn(q, m["rot"]), turn(k, m["rot"]), turn(v, whole), lambda s, _: weigh(s * m["scale"], allowed))
    return linear(turn(o, whole, back=True).flatten(1), w, "o")


def tobadra_units(h, w, mlp):
    if mlp["kind"] == "dense":
        return gelu(h @ w("up").T) @ w("down").T
    r = mlp["router"]
    one = lambda z, p: torch.nn.functional.gelu(z @ p("up").T) @ p("down").T  # noqa: E731
    score = torch.softmax(h @ w("router").T, -1)
    choice, count = score + w("correction"), r["experts"] + r.get("identity", 0)
    if r.get("groups"):
        per = count // r["groups"]["count"]
        choice = choice.masked_fill(~best_groups(choice.view(len(h), -1, per).amax(-1), r["groups"]["keep"], per), -math.inf)
    chosen = choice.topk(r["top"], 1).indices
    weight = score.gather(1, chosen) * r.get("scale", 1.0)
    y = spread_units(h, chosen, weight, count, lambda z, e: one(z, w.under(f"e{e}.")) if e < r["experts"] else z)
    return y + torch.sigmoid(h @ w("shared.sg").T) * one(h, w.under("shared.")) if mlp.get("shared") else y


def tobadra(raw, w, ids, rows):
    eps = raw["norm"]["eps"]
    x = rms(w.tensors["embed"][ids].double(), w("embed.norm"), eps)
    for i, layer in enumerate(raw["layers"]):
        l = w.under(f"l{layer.get('weights_of', i) if layer.get('weights_of') is not None else i}.")
        h = rms(x, l("norm1"), eps)
        y = tobadra_mixer(layer["type"], h + shifted(h, l("canon1")), l.under("mix."), layer["mixer"], eps)
        x = x + rms(torch.sigmoid(linear(h, l, "rg1")) * y, l("norm1b"), eps)
        if layer.get("mlp"):
            h = rms(x, l("norm2"), eps)
            x = x + rms(torch.sigmoid(linear(h, l, "rg2")) * tobadra_units(h, l.under("mlp."), layer["mlp"]), l("norm2b"), eps)
    return rms(x[rows], w("final.norm"), eps) @ w("embed").T * raw.get("logit_scale", 1.0)


def saturating(x, w, name):
    return torch.tanh(w(name + ".alpha") * x) * w(name) + w(name + ".b")


def lean_back(h, share):
    return h + (torch.nn.functional.pad(h, (0, 0, 1, 0))[:-1] - h) * share


def general_delta(h, w, m, eps):
    r, k, v = (by_head(h @ w(n).T, m["heads"]) for n in "rkv")
    keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w("w1").T) @ w("w2").T + w("w0"))).view_as(k)
    u = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    away = torch.sigmoid(linear(h, w, "a")).view_as(k) * u

    def step(s, t):
        read = u[t].unsqueeze(1) @ s
        s = keep[t].unsqueeze(2) * s - away[t].unsqueeze(2) * read + k[t].unsqueeze(2) * v[t].unsqueeze(1)
        return s, s

    o = unit(states(r, k, v, step), eps).flatten(1) * w("norm") * torch.sigmoid(h @ w("g").T)
    return o @ w("o").T


def time_mixing(h, w, m, eps):
    mixed = {n: lean_back(h, w("mu." + n)) for n in "rkvgw"}
    r, k, v = (by_head(mixed[n] @ w(n).T, m["heads"]) for n in "rkv")
    keep = torch.exp(-torch.exp(torch.tanh(mixed["w"] @ w("w1").T) @ w("w2").T + w("w0"))).view_as(k)
    bonus = w("u").unsqueeze(2)

    def step(s, t):
        new = k[t].unsqueeze(2) * v[t].unsqueeze(1)
        return keep[t].unsqueeze(2) * s + new, s + bonus * new

    o = unit(states(r, k, v, step), eps).flatten(1)
    return (o * w("norm") * silu(mixed["g"] @ w("g").T)) @ w("o").T


def vufadra(raw, w, ids, rows):
    eps, first = raw["norm"]["eps"], pair_embedding(raw, w, ids)
    x, loop = first, raw.get("loop") or {"start": 0, "stop": 0, "times": 0}
    inner = list(range(loop["start"], loop["stop"]))
    order = [(i, None) for i in range(loop["start"])]
    order += [(i, t if i == loop["start"] else None) for t in range(loop["times"]) for i in inner]
    order += [(i, None) for i in range(loop["stop"], len(raw["layers"]))]
    for i, opens in order:
        layer, l = raw["layers"][i], w.under(f"l{i}.")
        p, m = l.under("mix."), layer["mixer"]
        if opens is not None:
            x = torch.cat((x, first), -1) @ w("loop.in").T + w("loop.step")[opens]
        h = lean_back(saturating(x, l, "norm1"), l("shift"))
        if layer["type"] == "general_delta":
            y = general_delta(h, p, m, eps)
        elif layer["type"] == "rglru":
            y = channel_recurrence(h, p, m)
        else:
            a, c = p.under("left."), m["left"]
            q, k, v = (by_head(h @ a(n).T, c["heads" if n == "q" else "kv_heads"]) for n in "qkv")
            q, k = turn(rms(q, a("q.norm"), eps), c["rot"]), turn(rms(k, a("k.norm"), eps), c["rot"])
            allowed = visible(h, c.get("mask"), chunks=True)
            o = attend(q, k, v, lambda s, j: torch.sigmoid(s * c["scale"] + a("pb")[j].view(-1, 1, 1)) * allowed)
            y = 0.5 * rms(o.flatten(1) @ a("o").T, p("left.out"), eps)
            y = y + 0.5 * rms(time_mixing(h, p.under("right."), m["right"], eps), p("right.out"), eps)
        if layer.get("mlp"):
            y = y + swiglu(saturating(x, l, "norm2"), l.under("mlp."))
        x = x + y
    return saturating(x[rows], w, "final.norm") @ w("head").T


@torch.inference_mode()
def exact(case, seed):
    """The step's logits in float64: every request as one whole sequence; None where that would take long."""
    config = config_of(case)
    specs = DecoderModel(architecture_for(config.architecture).build_spec(config)).weight_specs()
    every = [past + new for past, new in entries_of(case)]
    matrices = sum(math.prod(s.shape) for s in specs if s.role == "matrix" and s.name not in ("embed", "bigram", "model.embed_tokens.weight"))
    if 2.0 * sum(every) * matrices > 3e14 or sum(every) > 20000:
        return None
    w = Weights(weights_of(case, specs, seed))
    whole = qwen3 if case["design"] == "qwen3" else globals()[case["design"]]
    described = config if case["design"] == "qwen3" else config.to_dict()
    rows = []
    for ids in tokens_of(case, seed, config.vocab_size):
        rows.append(whole(described, w, torch.tensor(ids, device="cuda"), slice(len(ids) - 1, len(ids))))
    return torch.cat(rows)
