"""Whole passes through the engine that stand for what its users run.

A pass opens a set of requests, feeds their prompts in rounds of at most 2,048 tokens (requests whose prompt is through
decode one token each beside the portions of the others, as the scheduler does it), decodes a number of tokens and ends
the requests.  The tokens are given, as in trace replay, so that a pass means the same whatever rounding does to a
choice; every round goes through ``ModelRunner.step``, the one step function that generation, replay and the scheduler
share.  Outputs are float32 logits: at the wanted places of the prompts, and after each request's last token.

Models are four layers of the sizes that ``bench.py`` measures the designs at (Qwen3 and four others; widths 2,048 and
4,096, heads of 128), a vocabulary of 32,000, random weights from the seed.  Every weight is a bfloat16 value, so the
float64 computation of :func:`exact` starts from the very same model.
"""

import math
import zlib

import torch

VOCAB = 32000
LAYERS = 4
ROUND = 2048            # most tokens of one step
PAGE = 16
EPS = 1e-6
#: share of the residual stream that a normed branch adds: as in a deep trained model, a small one.  (It also keeps the
#: logits comparable where a token's expert choice is a tie that two correct implementations round apart.)
MIXER_SHARE, EXPERT_SHARE = 0.1, 0.02


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # one short conversation turn: the smallest calls, where latency and launches count
        dict(name="turn_small", model="qwen3", width=2048, dtype="bfloat16", requests=1, shortest=512, longest=512,
             new=32, places=1),
        # an offline batch of eight: prompts of 1,024 tokens, then decoding; what the benchmark measures
        dict(name="batch8", model="qwen3", width=4096, dtype="bfloat16", requests=8, shortest=1024, longest=1024,
             new=64, places=1),
        # a serving load of ragged requests: mixed rounds, then batch 64
        dict(name="serving64", model="qwen3", width=4096, dtype="bfloat16", requests=64, shortest=129, longest=1023,
             new=64, places=1),
        # the time to the first token of one prompt
        dict(name="prompt2048", model="qwen3", width=4096, dtype="bfloat16", requests=1, shortest=2048, longest=2048,
             new=0, places=1),
        # long documents in portions, ragged, and a few tokens after them
        dict(name="documents", model="qwen3", width=4096, dtype="bfloat16", requests=2, shortest=5003, longest=7907,
             new=8, places=1),
        # the float32 path, as used to check a model
        dict(name="check_float32", model="qwen3", width=2048, dtype="float32", requests=4, shortest=1, longest=130,
             new=10, places=1),
        # scoring of ragged texts with the delta rule and routed experts
        dict(name="delta_scoring", model="zifuzen", width=2048, dtype="bfloat16", requests=3, shortest=301,
             longest=1501, new=0, places=32),
        # a batch decoding through the delta rule's memories and routed experts
        dict(name="delta_batch32", model="zifuzen", width=4096, dtype="bfloat16", requests=32, shortest=63,
             longest=511, new=32, places=1),
        # the first token of a prompt through the gated and the constant-decay memories
        dict(name="memory_prompt", model="renadra", width=4096, dtype="bfloat16", requests=1, shortest=2048,
             longest=2048, new=0, places=1),
        # a batch of eight on the same kind of model
        dict(name="memory_batch8", model="renadra", width=2048, dtype="bfloat16", requests=8, shortest=257,
             longest=1024, new=32, places=1),
        # scoring with latent attention and routed experts
        dict(name="latent_scoring", model="ligirax", width=4096, dtype="bfloat16", requests=1, shortest=2048,
             longest=2048, new=0, places=64),
        # questions on two documents: latent attention over all keys beside capped attention in blocks
        dict(name="latent_documents", model="sukalorn", width=4096, dtype="bfloat16", requests=2, shortest=1001,
             longest=3003, new=16, places=1),
    ]


def draw(rng):
    """One more case of the same ranges; the tokens of a pass stay below those of the largest listed one."""
    def log_uniform(low, high):
        return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))

    model = rng.choice(("qwen3", "qwen3", "qwen3", "sukalorn", "zifuzen", "renadra", "ligirax"))
    routed = model in ("zifuzen", "ligirax")
    dtype = "float32" if model == "qwen3" and rng.random() < 0.15 else "bfloat16"
    most = 8 if dtype == "float32" else 64
    scoring = rng.random() < 0.5
    if scoring:
        requests, new, places = log_uniform(1, 4), 0, 64 if routed else rng.choice((1, 64))
        longest = log_uniform(257, 600 if dtype == "float32" else 6000 if model == "qwen3" else 3000)
    else:
        requests, new, places = log_uniform(16 if routed else 1, most), log_uniform(4, 64), 1
        longest = log_uniform(17, 300 if dtype == "float32" else 1023)
    shortest = max(1, longest - rng.randrange(longest))
    if requests == 1:
        shortest = longest
    return dict(model=model, width=2048 if dtype == "float32" else rng.choice((2048, 4096)), dtype=dtype,
                requests=requests, shortest=shortest, longest=longest, new=new, places=places)


def lengths(case):
    """The requests' prompt lengths, spread evenly between the shortest and the longest, long and short in turn."""
    n, low, high = case["requests"], case["shortest"], case["longest"]
    even = [low + (high - low) * i // max(1, n - 1) for i in range(n)] if n > 1 else [high]
    return [even[i // 2] if i % 2 == 0 else even[n - 1 - i // 2] for i in range(n)]


def rounds(case):
    """The steps of a pass: lists of (request, first token, last token + 1)."""
    prompt, new = lengths(case), case["new"]
    at, out = [0] * len(prompt), []
    while any(a < p + new for a, p in zip(at, prompt)):
        step = [(i, at[i], at[i] + 1) for i, p in enumerate(prompt) if p <= at[i] < p + new]
        room = ROUND - len(step)
        for i, p in enumerate(prompt):
            if at[i] < p and room > 0:
                take = min(p - at[i], room)
                step.append((i, at[i], at[i] + take))
                room -= take
        for i, _, stop in step:
            at[i] = stop
        out.append(step)
    return out


def wanted(case, length):
    """The places of a prompt whose logits are wanted: its last one, or ``places`` spread over it."""
    count = min(case["places"], length)
    return [(k + 1) * length // count - 1 for k in range(count)]


# ------------------------------------------------------------------------------------------------ the models

def sizes(case):
    width = case["width"]
    big = width >= 4096
    return dict(width=width, heads=width // 128, groups=width // 512, dim=128, ff=12288 if big else 8192,
                q_rank=1536 if big else 768, kv_rank=512, rot=64, window=1024, keep=64, experts=64 if big else 32,
                expert_ff=1024 if big else 768, shared_ff=2048 if big else 1024, identity=16 if big else 8)


def config(case):
    """The configuration, as config.json holds it."""
    z = sizes(case)
    d, heads, groups = z["dim"], z["heads"], z["groups"]
    if case["model"] == "qwen3":
        return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": LAYERS, "hidden_size": z["width"],
                "num_attention_heads": heads, "num_key_value_heads": groups, "head_dim": d,
                "intermediate_size": z["ff"], "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": EPS,
                "max_position_embeddings": 16384, "tie_word_embeddings": False}
    top = {"vocab": VOCAB, "width": z["width"], "norm": {"eps": EPS}}
    attention = {"heads": heads, "kv_heads": groups, "dim": d, "vdim": d, "scale": d ** -0.5}
    dense = {"kind": "dense", "ff": z["ff"]}
    latent = {"heads": heads, "dim": d, "rot_dim": z["rot"], "vdim": d, "kv_rank": z["kv_rank"],
              "scale": (d + z["rot"]) ** -0.5, "rot": {"base": 10000.0, "dims": z["rot"]}}
    yarn = {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    if case["model"] == "sukalorn":
        layers = [("attention", dict(attention, softcap=30.0, mask={"size": z["window"]}, v_mix=True), dense),
                  ("latent_attention", dict(latent, q_rank=z["q_rank"]), dense)] * 2
        top["architecture"] = "Sukalorn"
    elif case["model"] == "zifuzen":
        delta = {"heads": heads, "kv_heads": groups, "dim": d, "vdim": d, "conv": 4}
        moe = {"kind": "moe", "expert": {"ff": z["expert_ff"], "limit": 7.0}, "shared": {"ff": z["shared_ff"], "limit": 7.0},
               "router": {"experts": z["experts"], "top": 4, "scale": 2.5, "groups": {"count": 8, "keep": 4}}}
        layers = [("delta", delta, moe), ("attention", attention, dense), ("delta_2", delta, moe),
                  ("attention", dict(attention, kv_from=1), moe)]
        top.update(architecture="Zifuzen", max_positions=16384, embedding={"scale": math.sqrt(z["width"])},
                   logit_softcap=30.0)
    elif case["model"] == "renadra":
        rot = {"base": 1000000.0, "dims": d}
        memory = {"heads": heads, "dim": d, "vdim": d}
        seen = dict(attention, mask={"size": z["window"]}, rot=rot)
        left = dict(seen, softcap=30.0, mask={"size": z["window"], "keep_first": z["keep"]}, rot=dict(rot, scaling=yarn))
        right = dict(memory, decay=[1.0 - 2.0 ** -(2 + 8 * h / max(1, heads - 1)) for h in range(heads)])
        parallel = {"left": left, "right": right, "left_scale": 0.8, "right_scale": 1.1}
        layers = [("hgrn2", memory, dense), ("attention", seen, dense), ("parallel", parallel, dense),
                  ("hgrn2", memory, dense)]
        top.update(architecture="Renadra", embedding={"scale": 1.0, "bigram": {
            "buckets": 100003, "mul_prev": 1000003, "mul_cur": 31}})
    else:
        mixer = dict(latent, mask={"size": z["window"]}, rot=dict(latent["rot"], scaling=yarn))
        moe = {"kind": "moe", "expert": {"ff": z["expert_ff"], "limit": 7.0},
               "router": {"experts": z["experts"], "identity": z["identity"], "top": 6}}
        layers = [("latent_attention", dict(mixer, kv_from=1) if i == 2 else mixer, moe) for i in range(LAYERS)]
        top.update(architecture="Ligirax", residual_mult=0.5, logit_scale=z["width"] ** -0.5)
    top["layers"] = [{"type": kind, "mixer": mixer, "mlp": mlp} for kind, mixer, mlp in layers]
    return top


def tensor(case, seed, name, shape, device):
    """A weight by its name: float32, every value representable in bfloat16."""
    shape = tuple(shape)
    gen = torch.Generator(device=device).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
    model, last = case["model"], name.rsplit(".", 1)[-1]
    if last in ("A_log", "lower", "vmix", "conv", "dt_bias"):
        u = torch.rand(shape, generator=gen, device=device)
        if last == "A_log":           # decay rates of 1 to 16, as state-space models are initialised
            u = torch.log(1.0 + 15.0 * u)
        elif last == "dt_bias":       # steps of 0.001 to 0.1 behind the softplus
            u = torch.log(torch.expm1(torch.exp(math.log(1e-3) + u * math.log(100.0))))
        elif last == "conv":
            u = u - 0.5
        return u.bfloat16().float()
    n = torch.randn(shape, generator=gen, device=device)
    if last == "pb":                  # a sigmoid in a softmax's place starts from about minus the log of the keys
        n = n * 0.1 - 6.0
    elif last == "correction":        # small beside the scores it corrects
        n = n * (0.1 if model == "zifuzen" else 0.1 / shape[0])
    elif name == "embed" and model == "ligirax":
        pass                          # a stream of unit size from the start
    elif len(shape) == 1 and last != "b":
        share = 1.0
        if name.startswith("l") and model in ("zifuzen", "ligirax") and ".mix" not in name:
            inner = model == "ligirax" and not last.endswith("b")
            share = 1.0 if inner else MIXER_SHARE if last.startswith("norm1") else EXPERT_SHARE
            share = share if inner or model == "zifuzen" else 2.0 * share      # (times residual_mult)
        around_zero = model == "sukalorn" and not name.endswith("dq.norm") and not name.endswith("dkv.norm")
        n = n * 0.1 if around_zero else (1.0 + 0.1 * n) * share
    else:
        n = n * 0.02
    return n.bfloat16().float()


def token_ids(case, seed):
    gen = torch.Generator().manual_seed(seed * 7919 + 17)
    return [torch.randint(0, VOCAB, (n + case["new"],), generator=gen).tolist() for n in lengths(case)]


# ------------------------------------------------------------------------------------------------ a pass

def prepare(case, seed):
    from ampere_kv_engine_b200.config.engine_config import EngineConfig
    from ampere_kv_engine_b200.engine.engine import Engine, parse_dtype
    from ampere_kv_engine_b200.models.decoder import DecoderModel
    from ampere_kv_engine_b200.models.registry import config_from_dict
    from ampere_kv_engine_b200.weights.loader import cast_for

    arch, model_config = config_from_dict(config(case))
    dtype = parse_dtype(case["dtype"])
    model = DecoderModel(arch.build_spec(model_config), dtype=dtype, device="cuda")
    model.load_tensors({name: cast_for(spec, tensor(case, seed, name, spec.drawn_shape(), "cuda"), dtype)
                        for name, spec in model.param_specs().items() if not spec.optional})
    held = sum((n + case["new"] + PAGE) // PAGE + 1 for n in lengths(case)) * PAGE
    engine = Engine(model, EngineConfig(dtype=case["dtype"], page_size=PAGE, max_tokens=held + ROUND,
                                        max_seqs=case["requests"] + 1, max_batch_tokens=ROUND, max_context=16384))
    prompt = lengths(case)
    ids = token_ids(case, seed)
    steps = []
    for step in rounds(case):
        plan = []
        for i, start, stop in step:
            if stop <= prompt[i]:
                places = [p - start for p in wanted(case, prompt[i]) if start <= p < stop]
            else:
                places = [0]          # a decoding request chooses from the logits of every token
            plan.append((i, ids[i][start:stop], places))
        steps.append(plan)
    return {"engine": engine, "steps": steps, "requests": len(prompt), "prompt": prompt, "new": case["new"]}


def run(state):
    from ampere_kv_engine_b200.engine.batch import SeqStep

    runner, prompt, new = state["engine"].runner, state["prompt"], state["new"]
    held = [runner.open(i) for i in range(state["requests"])]
    fed = [0] * len(held)
    in_prompt, after = [], []
    for plan in state["steps"]:
        logits = runner.step([SeqStep(held[i], tokens, places) for i, tokens, places in plan])
        row = 0
        for i, tokens, places in plan:
            fed[i] += len(tokens)
            if fed[i] <= prompt[i]:
                if places:
                    in_prompt.append((i, fed[i], logits[row:row + len(places)].clone()))
            elif fed[i] == prompt[i] + new:
                after.append((i, fed[i], logits[row:row + 1].clone()))
            row += len(places)
    for seq in held:
        runner.close(seq)
    by_request = lambda kept: torch.cat([t for _, _, t in sorted(kept, key=lambda k: k[:2])])  # noqa: E731
    return {"prompt": by_request(in_prompt), **({"last": by_request(after)} if after else {})}


def work(case):
    """Matrices read once a step, keys and values (or memories) read and written once, logits written; the matrix
    products of every token and its attention or memory update."""
    z = sizes(case)
    w, d, heads, groups, ff = z["width"], z["dim"], z["heads"], z["groups"], z["ff"]
    element = 4 if case["dtype"] == "float32" else 2
    attn = w * d * (2 * heads + 2 * groups)
    gated, plain = 3 * w * ff, 2 * w * ff
    model = case["model"]
    # per layer: (dense matrix elements, expert matrix elements, experts, chosen, keys' width, flops per key, memory)
    if model == "qwen3":
        layers = [(attn + gated, 0, 0, 0, 2 * groups * d, 4 * heads * d, 0)] * 4
        reach = None
    elif model == "sukalorn":
        lat = w * z["q_rank"] + z["q_rank"] * heads * (d + z["rot"]) + w * (z["kv_rank"] + z["rot"]) + \
            2 * heads * d * z["kv_rank"] + w * heads * d
        layers = [(attn + plain, 0, 0, 0, 2 * groups * d, 4 * heads * d, 0),
                  (lat + plain, 0, 0, 0, z["kv_rank"] + z["rot"], 2 * heads * (2 * d + z["rot"]), 0)] * 2
        reach = None
    elif model == "zifuzen":
        expert, shared = 3 * w * z["expert_ff"], 3 * w * z["shared_ff"] + w * z["experts"]
        delta = w * d * (2 * groups + 3 * heads) + 2 * w * heads
        layers = [(delta + shared, expert, z["experts"], 4, 0, 0, heads * d * d),
                  (attn + gated, 0, 0, 0, 2 * groups * d, 4 * heads * d, 0),
                  (delta + shared, expert, z["experts"], 4, 0, 0, heads * d * d),
                  (2 * w * d * heads + shared, expert, z["experts"], 4, 2 * groups * d, 4 * heads * d, 0)]
        reach = None
    elif model == "renadra":
        memory = (4 * w * d * heads + gated, 0, 0, 0, 0, 0, heads * d * d)
        window = (attn + gated, 0, 0, 0, 2 * groups * d, 4 * heads * d, 0)
        both = (attn + 5 * w * d * heads - w * d * groups + gated, 0, 0, 0, 2 * groups * d, 4 * heads * d, heads * d * d)
        layers, reach = [memory, window, both, memory], z["window"]
    else:
        lat = w * heads * (d + z["rot"]) + w * (z["kv_rank"] + z["rot"]) + 2 * heads * d * z["kv_rank"] + w * heads * d
        layers = [(lat + w * (z["experts"] + z["identity"]), 3 * w * z["expert_ff"], z["experts"],
                   6.0 * z["experts"] / (z["experts"] + z["identity"]), z["kv_rank"] + z["rot"],
                   2 * heads * (2 * d + z["rot"]), 0)] * 4
        reach = z["window"]
    moved = flops = 0.0
    for step in rounds(case):
        tokens = sum(stop - start for _, start, stop in step)
        for dense, expert, experts, chosen, kept, per_key, memory in layers:
            used = experts * (1.0 - (1.0 - chosen / experts) ** tokens) if experts else 0.0
            moved += element * (dense + used * expert)
            flops += 2.0 * tokens * (dense + chosen * expert)
            for _, start, stop in step:
                far = min(stop, reach + stop - start) if reach else stop
                keys = sum(min(p + 1, reach) for p in range(start, stop)) if reach else \
                    (start + stop + 1) * (stop - start) / 2.0
                moved += element * kept * (far + stop - start) + 8 * memory
                flops += per_key * keys + 5.0 * memory * (stop - start)
        rows = sum(len([p for p in wanted(case, lengths(case)[i]) if start <= p < stop]) if stop <= lengths(case)[i] else 1
                   for i, start, stop in step)
        if rows:
            moved += element * w * VOCAB + 4.0 * rows * VOCAB
            flops += 2.0 * rows * w * VOCAB
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """About four times the distance to :func:`exact` that was measured: 4e-6 in float32; in bfloat16 0.007 to 0.015, and
    0.003 where a branch adds only its small share to an exact embedding."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4}
    if case["model"] in ("zifuzen", "ligirax"):
        return {"rel": 0.012, "max": 0.1}
    return {"rel": 0.03, "max": 0.2}


# ------------------------------------------------------------------------------------------------ in 64 bits

def rms(x):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS)


def silu(x):
    return x * torch.sigmoid(x)


def turn_table(count, dims, base, device, scaling=None):
    """cos and sin [count, dims / 2]; frequencies and angles are rounded to float32, as the designs state it."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=device)
    freq, factor = base ** (-2.0 * i / dims), 1.0
    if scaling is not None:
        where = lambda turns: dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        low, high = max(math.floor(where(scaling["fast"])), 0), min(math.ceil(where(scaling["slow"])), dims - 1)
        ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        freq = freq / scaling["factor"] * ramp + freq * (1.0 - ramp)
        factor = 0.1 * math.log(scaling["factor"]) + 1.0
    angle = (torch.arange(count, dtype=torch.float32, device=device)[:, None] * freq.float()).double()
    return angle.cos() * factor, angle.sin() * factor


def turn(x, table, pairs):
    """x [B, T, heads, 2n]: neighbouring pairs, or dim i with dim i + n, turned by the position's angles."""
    cos, sin = (t[None, :, None, :] for t in table)
    half = x.shape[-1] // 2
    u, v = (x[..., 0::2], x[..., 1::2]) if pairs else (x[..., :half], x[..., half:])
    a, b = u * cos - v * sin, v * cos + u * sin
    return torch.stack((a, b), -1).flatten(-2) if pairs else torch.cat((a, b), -1)


def attend(q, k, v, scale, see, weigh=None):
    """q [B, T, H, D], k [B, T, G, D], v [B, T, G, V]; ``see(i, j)`` says which keys a place sees, ``weigh(scores,
    head, mask, distance)`` makes weights of the scaled scores (softmax where it is left out)."""
    count, length, heads, per = q.shape[0], q.shape[1], q.shape[2], q.shape[2] // k.shape[2]
    at = torch.arange(length, device=q.device)
    out = q.new_empty(count, length, heads, v.shape[-1])
    for first in range(0, length, 2048):
        i = at[first:first + 2048, None]
        stop = int(i[-1]) + 1
        mask, distance = see(i, at[None, :stop]), (i - at[None, :stop]).double()
        for b in range(count):
            for h in range(heads):
                s = q[b, first:stop, h] @ k[b, :stop, h // per].T * scale
                if weigh is None:
                    s = torch.softmax(s.masked_fill(~mask, -math.inf), -1)
                else:
                    s = weigh(s, h, mask, distance)
                out[b, first:stop, h] = s @ v[b, :stop, h // per]
    return out


def causal(i, j):
    return j <= i


def window_of(size, keep=0):
    return lambda i, j: (j <= i) & ((i - j < size) | (j < keep))


def memory_of(q, k, v, stays):
    """S_t = diag(stays_t) S_(t-1) + k_t v_t^T, o_t = S_t^T q_t; all [B, T, H, .]."""
    state = q.new_zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3])
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        state = state * stays[:, t, :, :, None] + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = torch.einsum("bhdv,bhd->bhv", state, q[:, t])
    return out


def delta_of(q, k, v, beta, stays):
    """S *= stays; S += k (beta (v - S^T k))^T; o = S^T q; the heads of a group share q and k."""
    per = v.shape[2] // q.shape[2]
    state = q.new_zeros(q.shape[0], v.shape[2], q.shape[3], v.shape[3])
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        qt, kt = (a[:, t].repeat_interleave(per, 1) for a in (q, k))
        state = state * stays[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", state, kt))
        state = state + kt[..., None] * u[:, :, None, :]
        out[:, t] = torch.einsum("bhdv,bhd->bhv", state, qt)
    return out


def short_conv(x, taps):
    n = taps.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(n))


class Model:
    """The five designs on whole, padded sequences [B, T] (padding stands behind a sequence, where nothing sees it)."""

    def __init__(self, case, seed, device):
        self.case, self.seed, self.device, self.z, self.config = case, seed, device, sizes(case), config(case)

    def w(self, name, *shape):
        return tensor(self.case, self.seed, name, shape, self.device).double()

    def lin(self, x, name, out, bias=False):
        y = x @ self.w(name, out, x.shape[-1]).T
        return y + self.w(name + ".b", out) if bias else y

    def heads(self, x, name, count, dim, bias=False):
        return self.lin(x, name, count * dim, bias).unflatten(-1, (count, dim))

    def gain(self, x, name):
        return rms(x) * self.w(name, x.shape[-1])

    # --- feed-forwards, over rows [N, width]

    def rows(self, fn, x):
        flat = x.reshape(-1, x.shape[-1])
        return torch.cat([fn(part) for part in flat.split(16384)]).view_as(x)

    def clamped(self, x, name, ff):
        g = self.lin(x, name + ".gate", ff).clamp(max=7.0)
        u = self.lin(x, name + ".up", ff).clamp(-7.0, 7.0)
        return self.lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), name + ".down", x.shape[-1])

    def experts(self, x, name, mlp):
        """Rows [N, width] through the experts they choose."""
        r = mlp["router"]
        count = r["experts"] + r.get("identity", 0)
        z = self.lin(x, name + ".router", count)
        s = torch.softmax(z, -1) if self.case["model"] == "ligirax" else torch.sigmoid(z)
        choice = s + self.w(name + ".correction", count)
        if "groups" in r:
            grouped = choice.unflatten(-1, (r["groups"]["count"], -1))
            kept = grouped.topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
            allowed = torch.zeros(grouped.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, kept, True)
            choice = grouped.masked_fill(~allowed[..., None], -math.inf).flatten(1)
        chosen = choice.topk(r["top"], -1).indices
        share = s.gather(1, chosen)
        if self.case["model"] == "zifuzen":
            share = share / (share.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = torch.zeros_like(x)
        for e in range(count):
            t, place = (chosen == e).nonzero(as_tuple=True)
            if len(t):
                y = x[t] if e >= r["experts"] else self.clamped(x[t], f"{name}.e{e}", mlp["expert"]["ff"])
                out[t] += share[t, place][:, None] * y
        if "shared" in mlp:
            out = out + self.clamped(x, name + ".shared", mlp["shared"]["ff"])
        return out

    # --- mixers, x [B, T, width]

    def latent(self, x, name, m, kept):
        down = m["kv_rank"]
        if kept is None:
            c = self.lin(x, name + ".dkv", down + m["rot_dim"])
            table = turn_table(x.shape[1], m["rot_dim"], m["rot"]["base"], x.device, m["rot"].get("scaling"))
            kept = self.gain(c[..., :down], name + ".dkv.norm"), turn(c[..., None, down:], table, True), table
        c, r, table = kept
        per = m["dim"] + m["rot_dim"]
        source = self.gain(self.lin(x, name + ".dq", m["q_rank"]), name + ".dq.norm") if "q_rank" in m else x
        q = self.heads(source, name + (".uq" if "q_rank" in m else ".q"), m["heads"], per)
        q = torch.cat((q[..., :m["dim"]], turn(q[..., m["dim"]:], table, True)), -1)
        k = torch.cat((self.heads(c, name + ".uk", m["heads"], m["dim"]), r.expand(-1, -1, m["heads"], -1)), -1)
        o = attend(q, k, self.heads(c, name + ".uv", m["heads"], m["vdim"]), m["scale"],
                   window_of(m["mask"]["size"]) if "mask" in m else causal)
        if "q_rank" not in m:
            o = o * torch.sigmoid(self.lin(x, name + ".g", m["heads"]))[..., None]
        return self.lin(o.flatten(2), name + ".o", x.shape[-1]), kept

    def delta(self, x, name, m):
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (silu(short_conv(self.lin(x, f"{name}.{n}", h * D), self.w(f"{name}.{n}.conv", h * D, m["conv"])))
                   .unflatten(-1, (h, D)) for n, h in (("q", G), ("k", G), ("v", H)))
        q = q / torch.sqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5
        k = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
        step = torch.nn.functional.softplus(self.lin(x, name + ".a", H) + self.w(name + ".dt_bias", H))
        o = delta_of(q, k, v, torch.sigmoid(self.lin(x, name + ".b", H)),
                     torch.exp(-torch.exp(self.w(name + ".A_log", H)) * step))
        o = rms(o) * self.w(name + ".norm", D) * silu(self.heads(x, name + ".g", H, D))
        return self.lin(o.flatten(2), name + ".o", x.shape[-1])

    def rotated(self, x, m, pairs):
        table = turn_table(x.shape[1], m["rot"]["dims"], m["rot"]["base"], x.device, m["rot"].get("scaling"))
        return turn(x, table, pairs)

    def hgrn2(self, x, name, m):
        H, D = m["heads"], m["dim"]
        low = self.w(name + ".lower", H * D)
        f = low + (1.0 - low) * torch.sigmoid(x @ self.w(name + ".f", H * D, x.shape[-1]).T + self.w(name + ".f.b", H * D))
        f = f.unflatten(-1, (H, D))
        o = memory_of(silu(self.heads(x, name + ".q", H, D)), 1.0 - f, self.heads(x, name + ".v", H, D), f)
        return self.lin((rms(o) * self.w(name + ".norm", D)).flatten(2), name + ".o", x.shape[-1])

    def parallel(self, x, name, m):
        left, right = m["left"], m["right"]
        H, G, D = left["heads"], left["kv_heads"], left["dim"]
        q, k = self.heads(x, name + ".left.q", H, D, True), self.heads(x, name + ".left.k", G, D, True)
        bias, cap = self.w(name + ".left.pb", H), left["softcap"]
        o = attend(self.rotated(q, left, False), self.rotated(k, left, False), k, left["scale"],
                   window_of(left["mask"]["size"], left["mask"]["keep_first"]),
                   lambda s, h, mask, _: torch.sigmoid(cap * torch.tanh(s / cap) + bias[h]) * mask)
        a = self.lin(o.flatten(2), name + ".left.o", x.shape[-1])
        H = right["heads"]
        q, k, v = (silu(self.heads(x, f"{name}.right.{n}", H, D)) for n in "qkv")
        stays = torch.tensor(right["decay"], dtype=torch.float64, device=x.device)[None, None, :, None].expand_as(q)
        o = self.gain(memory_of(q, k, v, stays).flatten(2), name + ".right.norm")
        b = self.lin(o * torch.sigmoid(self.lin(x, name + ".right.g", H * D)), name + ".right.o", x.shape[-1])
        return m["left_scale"] * a + m["right_scale"] * b

    def grouped(self, x, name, m, model):
        """The plain attentions of three designs (and the capped one of Sukalorn)."""
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        bias = model == "renadra"
        q, k, v = (self.heads(x, f"{name}.{n}", h, D, bias) for n, h in (("q", H), ("k", G), ("v", G)))
        if model == "renadra":
            q, k, v = self.rotated(q, m, True), self.rotated(k, m, True), rms(v)
            o = attend(q, k, v, m["scale"], window_of(m["mask"]["size"]))
            return self.lin(o.flatten(2), name + ".o", x.shape[-1], True)
        own, size, cap = v, m["mask"]["size"], m["softcap"]
        if self.first is None:
            self.first = own
        else:
            blend = self.w(name + ".vmix")
            v = (1.0 - blend) * own + blend * self.first
        def weigh(s, h, mask, distance):
            s = cap * torch.tanh(s / cap) - 2.0 ** (-8.0 * (h + 1) / H) * distance
            return torch.softmax(s.masked_fill(~mask, -math.inf), -1)
        o = attend(rms(q), rms(k), v, m["scale"], lambda i, j: (j <= i) & (i // size == j // size), weigh)
        o = o * torch.sigmoid(self.lin(x, name + ".g", H))[..., None]
        return self.lin(o.flatten(2), name + ".o", x.shape[-1])

    def borrowing(self, x, name, m):
        """Zifuzen's attention, which may read an earlier layer's keys and values."""
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q = rms(self.heads(x, name + ".q", H, D)) * self.w(name + ".q.norm", D)
        if "kv_from" not in m:
            self.first = (rms(self.heads(x, name + ".k", G, D)) * self.w(name + ".k.norm", D),
                          self.heads(x, name + ".v", G, D))
        return self.lin(attend(q, *self.first, m["scale"], causal).flatten(2), name + ".o", x.shape[-1])

    # --- whole models: the stream [B, T, width] behind the final norm, and the head's matrix

    def qwen3(self, ids):
        z, c = self.z, self.config
        x = self.w("model.embed_tokens.weight", VOCAB, z["width"])[ids]
        table = turn_table(ids.shape[1], 128, c["rope_theta"], x.device)
        for i in range(LAYERS):
            p = f"model.layers.{i}."
            h = self.gain(x, p + "input_layernorm.weight")
            q, k, v = (self.heads(h, f"{p}self_attn.{n}_proj.weight", g, 128)
                       for n, g in (("q", z["heads"]), ("k", z["groups"]), ("v", z["groups"])))
            q, k = (turn(self.gain(a, f"{p}self_attn.{n}_norm.weight"), table, False) for n, a in (("q", q), ("k", k)))
            x = x + self.lin(attend(q, k, v, 128 ** -0.5, causal).flatten(2), p + "self_attn.o_proj.weight", z["width"])
            h = self.gain(x, p + "post_attention_layernorm.weight")
            x = x + self.rows(lambda r: self.lin(silu(self.lin(r, p + "mlp.gate_proj.weight", z["ff"])) *
                                                 self.lin(r, p + "mlp.up_proj.weight", z["ff"]),
                                                 p + "mlp.down_proj.weight", z["width"]), h)
        return self.gain(x, "model.norm.weight"), "lm_head.weight", lambda y: y

    def sukalorn(self, ids):
        one = lambda x, name: rms(x) * (1.0 + self.w(name, x.shape[-1]))  # noqa: E731
        x, self.first = one(self.w("embed", VOCAB, self.z["width"])[ids], "embed.norm"), None
        for i, layer in enumerate(self.config["layers"]):
            h, m = one(x, f"l{i}.norm1"), layer["mixer"]
            x = x + (self.grouped(h, f"l{i}.mix", m, "sukalorn") if layer["type"] == "attention"
                     else self.latent(h, f"l{i}.mix", m, None)[0])
            x = x + self.rows(lambda r: self.lin(torch.relu(self.lin(r, f"l{i}.mlp.up", self.z["ff"])).square(),
                                                 f"l{i}.mlp.down", r.shape[-1]), one(x, f"l{i}.norm2"))
        return one(x, "final.norm"), "head", lambda y: y

    def zifuzen(self, ids):
        centred = lambda x, name: (x - x.mean(-1, keepdim=True)) / torch.sqrt(  # noqa: E731
            x.var(-1, unbiased=False, keepdim=True) + EPS) * self.w(name, x.shape[-1])
        x = self.w("embed", VOCAB, self.z["width"])[ids] * self.config["embedding"]["scale"]
        x = x + self.w("pos", self.config["max_positions"], self.z["width"])[: ids.shape[1]]

        def dense(r, p):
            g = self.lin(r, p + ".gate", self.z["ff"]) + self.w(p + ".gate.b", self.z["ff"])
            u = self.lin(r, p + ".up", self.z["ff"]) + self.w(p + ".up.b", self.z["ff"])
            g = 0.5 * g * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (g + 0.044715 * g ** 3)))
            return self.lin(g * u, p + ".down", r.shape[-1]) + self.w(p + ".down.b", r.shape[-1])

        for i, layer in enumerate(self.config["layers"]):
            mix = self.borrowing if layer["type"] == "attention" else self.delta
            x = x + centred(mix(x, f"l{i}.mix", layer["mixer"]), f"l{i}.norm1")
            ff = dense if layer["mlp"]["kind"] == "dense" else lambda r, p: self.experts(r, p, layer["mlp"])
            x = x + centred(self.rows(lambda r: ff(r, f"l{i}.mlp"), x), f"l{i}.norm2")
        return centred(x, "final.norm"), "head", lambda y: 30.0 * torch.tanh(y / 30.0)

    def renadra(self, ids):
        b = self.config["embedding"]["bigram"]
        before = torch.cat((ids[:, :1], ids[:, :-1]), 1)
        pair = (before * b["mul_prev"] + ids * b["mul_cur"]) % b["buckets"]
        pair[:, 0] = b["buckets"]
        x = self.w("embed", VOCAB, self.z["width"])[ids] + self.w("bigram", b["buckets"] + 1, self.z["width"])[pair]
        for i, layer in enumerate(self.config["layers"]):
            h, m, name = self.gain(x, f"l{i}.norm1"), layer["mixer"], f"l{i}.mix"
            x = x + (self.grouped(h, name, m, "renadra") if layer["type"] == "attention"
                     else self.parallel(h, name, m) if layer["type"] == "parallel" else self.hgrn2(h, name, m))
            x = x + self.rows(lambda r: self.lin(silu(self.lin(r, f"l{i}.mlp.gate", self.z["ff"])) *
                                                 self.lin(r, f"l{i}.mlp.up", self.z["ff"]), f"l{i}.mlp.down", r.shape[-1]),
                              self.gain(x, f"l{i}.norm2"))
        return self.gain(x, "final.norm"), "head", lambda y: y

    def ligirax(self, ids):
        x, c = self.w("embed", VOCAB, self.z["width"])[ids], self.config
        kept = {}
        for i, layer in enumerate(c["layers"]):
            source = layer["mixer"].get("kv_from", i)
            y, kept[i] = self.latent(self.gain(x, f"l{i}.norm1"), f"l{i}.mix", layer["mixer"], kept.get(source))
            x = x + c["residual_mult"] * self.gain(y, f"l{i}.norm1b")
            y = self.rows(lambda r: self.experts(r, f"l{i}.mlp", layer["mlp"]), self.gain(x, f"l{i}.norm2"))
            x = x + c["residual_mult"] * self.gain(y, f"l{i}.norm2b")
        return self.gain(x, "final.norm"), "embed", lambda y: y * c["logit_scale"]


@torch.no_grad()
def exact(case, seed):
    """The logits of :func:`run` in float64, from the formulas of the designs on whole sequences."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    prompt, ids = lengths(case), token_ids(case, seed)
    longest = max(len(t) for t in ids)
    padded = torch.tensor([t + [0] * (longest - len(t)) for t in ids], device=device)
    model = Model(case, seed, device)
    x, head, last = getattr(model, case["model"])(padded)
    matrix = model.w(head, VOCAB, case["width"])
    out = {"prompt": torch.cat([x[i, wanted(case, n)] for i, n in enumerate(prompt)])}
    if case["new"]:
        out["last"] = torch.stack([x[i, n + case["new"] - 1] for i, n in enumerate(prompt)])
    return {name: last(rows @ matrix.T) for name, rows in out.items()}
