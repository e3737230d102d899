"""What the latent prompt kernel and the experts' tcgen05 products do when a wait runs out: with a bound of no tries every
wait gives up at once, copies are under way by then; the kernels report it, let the copies land, free their tensor memory
(more CTAs than the GPU holds follow one another, each with all of it) and leave, and the next launch is right."""

import pytest
import torch

from latent_case import LatentCase

pytestmark = pytest.mark.gpu

WAIT_TIMEOUT = 5


def test_latent_prompt_attention(monkeypatch):
    from ampere_kv_engine_b200.kernels import ops

    case = LatentCase([600, 130], [900, 130], heads=40)
    want = case.run(ops)
    attention, codes = ops.ext().latent_prompt_attention, []

    class Impatient:
        def __getattr__(self, name):
            return getattr(ops_ext, name)

        def latent_prompt_attention(self, *args):
            attention(*args, wait_limit=0)
            codes.append(int(args[-1]))
            args[-1].zero_()

    ops_ext = ops.ext()
    monkeypatch.setattr(ops, "ext", lambda: Impatient())
    assert bool((case.run(ops) == 7.0).all())        # nothing is written
    monkeypatch.undo()
    assert codes == [WAIT_TIMEOUT]
    assert torch.equal(case.run(ops), want)


@pytest.mark.parametrize("form", ["gated", "up", "down"])
def test_expert_products(form):
    from ampere_kv_engine_b200.kernels import ops

    g = torch.Generator(device="cuda").manual_seed(0)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    tokens, experts, k, n = 300, 8, 256, 2048
    chosen = rand(tokens, experts).topk(2, dim=-1).indices.int()
    order, offsets = ops.moe_sort(chosen, experts)
    x, w = rand(tokens, k).bfloat16(), rand(experts, 2 * n if form == "gated" else n, k).bfloat16()
    act, weights = rand(2 * tokens, k).bfloat16(), torch.rand(tokens, 2, generator=g, device="cuda")
    tc = ops.MOE_FORMS["tc"]

    def run(limit):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        out = torch.zeros(2 * tokens, n, device="cuda", dtype=torch.float32 if form == "down" else torch.bfloat16)
        if form == "gated":
            ops.ext().moe_gate_up(x, w, order, offsets, out, 2, 7.0, 1.702, tc, 1.0, status=status, wait_limit=limit)
        elif form == "up":
            ops.ext().moe_up(x, w, order, offsets, out, 2, 2, tc, status=status, wait_limit=limit)
        else:
            ops.ext().moe_down(act, w, order, offsets, weights, out, tc, status=status, wait_limit=limit)
        return out, int(status)

    want, code = run(-1)
    assert code == 0
    out, code = run(0)
    assert code == WAIT_TIMEOUT and not bool(out.any())
    again, code = run(-1)
    assert code == 0 and torch.equal(again, want)
