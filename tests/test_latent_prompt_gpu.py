"""Prompt attention through latents with keys and values written out: portions at the edges of the 128-token tiles and
key blocks, after earlier tokens, behind a window, of several sequences beside single tokens; widths that fill a chunk
partly; gates and sinks; pages in any order.  Against float64 attention over the written-out keys and values."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_the_plan_on_the_host():
    from ampere_kv_engine_b200.kernels import ops

    assert ops.latent_plan([1, 1], [5, 9], 0) is None
    plan = ops.latent_plan([1, 130, 2], [40, 200, 2], 0)
    assert plan.num_seqs == 2 and plan.rows == 256 + 128 and plan.num_tiles == 3 and plan.tokens == 132
    assert plan.numbers[:12] == [0, 0, 200, 130, 1, 1, 256, 0, 2, 2, 131, 2]
    assert plan.numbers[12:] == [0, 128, 0, 0, 1, 0]      # 200, 198 and 2 keys
    windowed = ops.latent_plan([130], [1000], 64)
    assert windowed.numbers[:6] == [0, 1000 - 130 - 63, 1000, 130, 0, 0] and windowed.rows == 256


@pytest.mark.parametrize("dim,rot,v_dim,rank,heads", [(128, 64, 128, 512, 4), (64, 32, 96, 64, 3), (40, 8, 16, 72, 2)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("q_lens,ctx_lens,extras", [([2], [2], False), ([128, 1, 129], [128, 300, 500], True),
                                                    ([257, 300], [257, 1025], True)])
def test_against_float64(dim, rot, v_dim, rank, heads, window, q_lens, ctx_lens, extras):
    from ampere_kv_engine_b200.kernels import ops

    g = torch.Generator(device="cuda").manual_seed(dim + window + sum(ctx_lens))
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    page, row = 16, rank + rot
    widest = max((c + page - 1) // page for c in ctx_lens)
    pages = len(q_lens) * widest + 3
    order = torch.randperm(pages, generator=g, device="cuda").int()
    table = order[:len(q_lens) * widest].view(len(q_lens), widest).contiguous()
    cache = torch.full((pages, 1, page, row), float("nan"), device="cuda").bfloat16()
    latents = [rand(c, row).bfloat16() for c in ctx_lens]
    for s, lat in enumerate(latents):
        for j in range(0, lat.shape[0], page):
            cache[table[s, j // page].item(), 0, : lat[j:j + page].shape[0]] = lat[j:j + page]
    tokens = sum(q_lens)
    q = rand(tokens, heads * (dim + rot) + 8).bfloat16()
    q_rows = torch.full((tokens, heads, row), float("nan"), device="cuda").bfloat16()
    q_rows[..., rank:] = rand(tokens, heads, rot).bfloat16()
    w_kv = (rand(heads * (dim + v_dim), rank) * rank ** -0.5).bfloat16()
    gate = torch.rand(tokens, heads, generator=g, device="cuda") if extras else None
    sink = rand(heads) if extras else None
    scale = (dim + rot) ** -0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    plan = ops.latent_plan(q_lens, ctx_lens, window).to("cuda")
    out = torch.full((tokens, heads * v_dim), 7.0, device="cuda").bfloat16()
    ops.latent_prompt_attention(q[:, :heads * (dim + rot)], q_rows.view(tokens, -1), cache, table, plan, w_kv, out,
                                heads=heads, dim=dim, rot_dim=rot, v_dim=v_dim, rank=rank, scale=scale, window=window,
                                gate=gate, sink=sink, status=status)
    assert int(status) == 0
    row0 = 0
    for n, c, lat in zip(q_lens, ctx_lens, latents):
        got = out[row0:row0 + n].view(n, heads, v_dim).double()
        if n == 1:
            assert bool((got == 7.0).all())          # single tokens are not the plan's
            row0 += 1
            continue
        kv = (lat[:, :rank].double() @ w_kv.double().T).bfloat16().double().view(c, heads, dim + v_dim)
        qh = torch.cat((q[row0:row0 + n, :heads * (dim + rot)].view(n, heads, dim + rot)[..., :dim],
                        q_rows[row0:row0 + n, :, rank:]), -1).double()
        kh = torch.cat((kv[..., :dim], lat[:, None, rank:].double().expand(c, heads, rot)), -1)
        s = torch.einsum("ihd,jhd->hij", qh, kh) * scale
        i, j = torch.arange(c - n, c, device="cuda")[:, None], torch.arange(c, device="cuda")[None]
        see = (j <= i) & ((i - j < window) if window else (j >= 0))
        s = s.masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink.double()[:, None, None].expand(heads, n, 1)), -1)
        p = torch.softmax(s, -1)[..., :c]
        want = torch.einsum("hij,jhd->ihd", p, kv[..., dim:])
        spread = torch.einsum("hij,jhd->ihd", p, kv[..., dim:].abs())
        if gate is not None:
            want, spread = want * gate[row0:row0 + n, :, None], spread * gate[row0:row0 + n, :, None]
        # a probability and the result are rounded to bfloat16 (2^-9 each); keys and values may round the other way than
        # here where the product's sum order differs (2^-8 of a value, and of a score: up to 2^-8 times its size)
        size = torch.einsum("ihd,jhd->hij", qh.abs(), kh.abs()).amax() * scale * 2.0 ** -8 * 0.02
        error = (got - want).abs()
        assert bool((error <= 2.0 ** -7 * spread + 2.0 ** -8 * want.abs() + size * spread + 1e-6).all()), error.max()
        row0 += n


def test_a_missing_page_is_reported():
    from ampere_kv_engine_b200.kernels import ops

    cache = torch.zeros(4, 1, 16, 72, device="cuda").bfloat16()
    table = torch.tensor([[0, 9]], dtype=torch.int32, device="cuda")
    plan = ops.latent_plan([20], [20], 0).to("cuda")
    out = torch.zeros(20, 64, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.latent_prompt_attention(torch.zeros(20, 72, device="cuda").bfloat16(), torch.zeros(20, 72, device="cuda").bfloat16(),
                                cache, table, plan, torch.zeros(128, 64, device="cuda").bfloat16(), out, heads=1, dim=64,
                                rot_dim=8, v_dim=64, rank=64, scale=1.0, status=status)
    assert int(status) == 1
