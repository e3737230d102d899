"""Which form the first product of experts without a gate takes: the few-rows form up to eight tokens and 384 blocks of 32
features, the tcgen05 tiles beyond either; both against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,top,features,few", [(1, 4, 96, True), (8, 1, 40, True), (9, 1, 40, False),
                                                     (8, 16, 96, True), (8, 16, 97, False), (1, 12, 1024, True),
                                                     (1, 12, 1056, False), (5, 30, 32, False)])
@pytest.mark.parametrize("same", [False, True])
def test_the_form_of_a_few_tokens(tokens, top, features, few, same):
    from ampere_kv_engine_b200.kernels import ops

    experts, k = 32, 136
    g = torch.Generator(device="cuda").manual_seed(tokens * features)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    chosen = rand(1 if same else tokens, experts).topk(top, dim=-1).indices.int().expand(tokens, top).contiguous()
    x, w = rand(tokens, k).bfloat16(), (rand(experts, features, k) * k ** -0.5).bfloat16()
    order, offsets = ops.moe_sort(chosen, experts)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.moe_up(x, w, order, offsets, top=top, activation="silu", status=status)
    forced = ops.moe_up(x, w, order, offsets, top=top, activation="silu", kernel="few" if few else "tc", status=status)
    assert int(status) == 0 and torch.equal(got, forced)
    pair = order.long()
    a, we = x[pair // top].double(), w[chosen.view(-1)[pair].long()].double()
    z = torch.einsum("rk,rnk->rn", a, we)
    size = torch.einsum("rk,rnk->rn", a.abs(), we.abs())
    want = z * torch.sigmoid(z)
    # k products added up in float32, |silu'| <= 1.1, an exponential and a division, one rounding to bfloat16
    bound = 1.1 * k * 2.0 ** -23 * size + (2.0 ** -21 + 2.0 ** -8) * want.abs() + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())
