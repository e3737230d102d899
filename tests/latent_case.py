"""A ragged prompt batch over paged latents, with float64 attention over the written-out keys and values: shared by the
tests of ``ops.latent_prompt_attention``."""

import math

import torch


class LatentCase:
    def __init__(self, q_lens, ctx_lens, *, heads=4, dim=64, rot=32, v_dim=64, rank=64, window=0, gated=False, sink=None,
                 seed=0):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
        self.q_lens, self.ctx_lens, self.window, self.sink = q_lens, ctx_lens, window, sink
        self.heads, self.dim, self.rot, self.v_dim, self.rank, self.page = heads, dim, rot, v_dim, rank, 16
        self.scale = (dim + rot) ** -0.5
        widest = max((c + self.page - 1) // self.page for c in ctx_lens)
        order = torch.randperm(len(q_lens) * widest + 3, generator=g, device="cuda").int()
        self.table = order[:len(q_lens) * widest].view(len(q_lens), widest).contiguous()
        self.latents = [rand(c, rank + rot).bfloat16() for c in ctx_lens]
        tokens = sum(q_lens)
        self.q = rand(tokens, heads, dim + rot).bfloat16()
        self.q_rows = torch.full((tokens, heads, rank + rot), float("nan"), device="cuda").bfloat16()
        self.q_rows[..., rank:] = rand(tokens, heads, rot).bfloat16()
        self.w_kv = (rand(heads * (dim + v_dim), rank) * rank ** -0.5).bfloat16()
        self.gate = torch.rand(tokens, heads, generator=g, device="cuda") if gated else None
        self.pages = order.numel()

    def run(self, ops, fill=7.0):
        """The kernels' output [tokens, heads, v_dim] (rows that are not the plan's keep ``fill``)."""
        cache = torch.full((self.pages, 1, self.page, self.rank + self.rot), float("nan"), device="cuda").bfloat16()
        for s, lat in enumerate(self.latents):
            for j in range(0, lat.shape[0], self.page):
                part = lat[j:j + self.page]
                cache[self.table[s, j // self.page].item(), 0, :part.shape[0]] = part
        tokens = self.q.shape[0]
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        plan = ops.latent_plan(self.q_lens, self.ctx_lens, self.window).to("cuda")
        out = torch.full((tokens, self.heads * self.v_dim), fill, device="cuda").bfloat16()
        ops.latent_prompt_attention(self.q.view(tokens, -1), self.q_rows.view(tokens, -1), cache, self.table, plan,
                                    self.w_kv, out, heads=self.heads, dim=self.dim, rot_dim=self.rot, v_dim=self.v_dim,
                                    rank=self.rank, scale=self.scale, window=self.window, gate=self.gate,
                                    sink=self.sink, status=status)
        assert int(status) == 0
        return out.view(tokens, self.heads, self.v_dim).double()

    def plain(self, s):
        """float64 (result, bound) of sequence s's rows.  The bound: a probability and the result are rounded to bfloat16
        (2^-9 each); keys and values may round the other way than here where the product's sum order differs (2^-8 of a
        value, and of a score: up to 2^-8 times its size, of which a sum of many takes a small part)."""
        n, c, lat = self.q_lens[s], self.ctx_lens[s], self.latents[s]
        row0 = sum(self.q_lens[:s])
        kv = (lat[:, :self.rank].double() @ self.w_kv.double().T).bfloat16().double()
        kv = kv.view(c, self.heads, self.dim + self.v_dim)
        qh = torch.cat((self.q[row0:row0 + n, :, :self.dim], self.q_rows[row0:row0 + n, :, self.rank:]), -1).double()
        kh = torch.cat((kv[..., :self.dim], lat[:, None, self.rank:].double().expand(c, self.heads, self.rot)), -1)
        score = torch.einsum("ihd,jhd->hij", qh, kh) * self.scale
        i, j = torch.arange(c - n, c, device="cuda")[:, None], torch.arange(c, device="cuda")[None]
        see = (j <= i) & ((i - j < self.window) if self.window else (j >= 0))
        score = score.masked_fill(~see, -math.inf)
        if self.sink is not None:
            score = torch.cat((score, self.sink.double()[:, None, None].expand(self.heads, n, 1)), -1)
        p, v = torch.softmax(score, -1)[..., :c], kv[..., self.dim:]
        # a key that a row does not see gives it nothing, whatever its value is
        v = v.masked_fill(~v.isfinite(), 0.0)
        want, spread = torch.einsum("hij,jhd->ihd", p, v), torch.einsum("hij,jhd->ihd", p, v.abs())
        if self.gate is not None:
            gate = self.gate[row0:row0 + n, :, None]
            want, spread = want * gate, spread * gate
        finite = lambda x: x.masked_fill(~x.isfinite(), 0.0).abs()  # noqa: E731
        size = torch.einsum("ihd,jhd->hij", finite(qh), finite(kh)).amax() * self.scale * 2.0 ** -8 * 0.02
        return want, 2.0 ** -7 * spread + 2.0 ** -8 * want.abs() + size * spread + 1e-6
