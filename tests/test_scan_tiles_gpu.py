"""Prompt scans in register tiles at the ends of their chunks of 16 tokens and of their dims, against the same tokens one by
one (the form that decoding takes, which adds up a column's sums in another order)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = (1, 15, 16, 17, 32, 33)
DIMS = [(4, 4), (64, 32), (68, 36), (128, 20), (132, 64), (256, 4)]


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _both(run, width):
    """run(rows, state, cu, slots) over all sequences at once, and sequence by sequence a token at a time; a padded
    sequence's slot and the slots of nobody must stay as they were."""
    cu = [0]
    for n in LENS:
        cu.append(cu[-1] + n)
    slots = [3, 0, 6, 1, 5, 2]
    whole, single = torch.zeros(8, width, device="cuda"), torch.zeros(8, width, device="cuda")
    whole[[4, 7]] = 2.5
    got = run(slice(0, cu[-1]), whole, cu + [cu[-1]], slots + [-1])
    assert bool((whole[[4, 7]] == 2.5).all())
    want = torch.empty_like(got)
    for s, slot in enumerate(slots):
        for t in range(cu[s], cu[s + 1]):
            want[t:t + 1] = run(slice(t, t + 1), single, [0, 1], [slot])
    # sums of up to 256 products in another order, each within 256 x 2^-24 of the sums' size, over at most 33 tokens of a
    # recurrence that does not grow
    bound = dict(atol=33 * 256 * 2.0 ** -24 * float(want.abs().max()), rtol=0.0)
    torch.testing.assert_close(got, want, **bound)
    torch.testing.assert_close(whole[slots], single[slots], atol=33 * 256 * 2.0 ** -24 * float(single.abs().max()), rtol=0.0)


@pytest.mark.parametrize("mode", ["gated_write", "constant_decay", "plain_decay", "token_decay"])
@pytest.mark.parametrize("dim,vdim", DIMS)
def test_linear_scan(mode, dim, vdim):
    from ampere_kv_engine_b200.kernels import ops

    heads, g = 4, torch.Generator(device="cuda").manual_seed(dim)
    x = torch.randn(sum(LENS), heads * (2 * dim + vdim) + heads, generator=g, device="cuda")
    x[:, -heads:] = torch.sigmoid(x[:, -heads:])
    extra = {"gated_write": {"lower": torch.rand(heads * dim, generator=g, device="cuda")}, "token_decay": {"decay_off": x.shape[1] - heads}
             }.get(mode, {"decay": torch.rand(heads, generator=g, device="cuda")})

    def run(rows, state, cu, slots):
        return ops.linear_scan(x[rows].contiguous(), state, _i32(cu), _i32(slots), num_heads=heads, head_dim=dim, v_dim=vdim, mode=mode,
                               q_off=0, k_off=heads * dim, v_off=2 * heads * dim, **extra)

    _both(run, ops.linear_scan_state_floats(heads, dim, vdim))


@pytest.mark.parametrize("dim,vdim", DIMS)
def test_delta_scan(dim, vdim):
    from ampere_kv_engine_b200.kernels import ops

    heads, g = 4, torch.Generator(device="cuda").manual_seed(dim)
    n, channels = sum(LENS), heads * (2 * dim + vdim)
    qkv = torch.randn(n, channels, generator=g, device="cuda")
    for lo in (0, heads * dim):
        part = qkv[:, lo:lo + heads * dim].view(n, heads, dim)
        part /= part.norm(dim=-1, keepdim=True)
    coef = torch.sigmoid(torch.randn(n, 2 * heads, generator=g, device="cuda"))
    x = torch.ones(n, channels + heads * vdim + 2 * heads, device="cuda")
    sizes = dict(num_heads=heads, num_kv_heads=heads, head_dim=dim, v_dim=vdim, taps=1)

    def run(rows, state, cu, slots):
        return ops.delta_scan(qkv[rows].contiguous(), coef[rows].contiguous(), x[rows].contiguous(), torch.ones(vdim, device="cuda"), state,
                              _i32(cu), _i32(slots), norm_eps=1.0, **sizes)

    _both(run, ops.delta_state_floats(heads, heads, dim, vdim, 1)[1])
