"""A sequence whose state slot or rows do not exist is reported by the scans and not walked: its rows (those that are rows
of the batch) come out as zeros, no state changes for it, and the other sequences are what they are without it.  Prompt
forms in register tiles, the other prompt forms (odd widths) and the decode forms."""

import pytest
import torch

pytestmark = pytest.mark.gpu

BAD_SLOT, BAD_ROW = 2, 4
SLOTS = 5
#: (rows of the sequences, state slots, the rows that must be zeros, status)
STEPS = [([0, 9, 12, 30], [1, SLOTS, 3], slice(9, 12), BAD_SLOT),
         ([0, 9, 12, 30], [1, 2 ** 30, 3], slice(9, 12), BAD_SLOT),
         ([0, 9, 12, 40], [1, 0, 3], slice(12, 30), BAD_ROW),
         ([-4, 9, 12, 30], [1, 0, 3], slice(0, 9), BAD_ROW),
         ([0, 1, 2, 3], [1, SLOTS, 3], slice(1, 2), BAD_SLOT),
         ([0, 1, 2, 9], [1, 0, 3], slice(2, 3), BAD_ROW)]


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _check(run, width, cu, slots, zeros, code):
    """run(tokens, state, cu, slots, status): the step against the same one in which the bad sequence is padding."""
    tokens = 3 if max(slots) < 100 and cu[1] == 1 else 30
    g = torch.Generator(device="cuda").manual_seed(1)
    start = torch.randn(SLOTS, width, generator=g, device="cuda")
    state, status = start.clone(), _i32([0])
    got = run(tokens, state, cu, slots, status)
    assert int(status) == code
    assert bool((got[zeros] == 0).all())
    bad = [i for i in range(3) if slots[i] >= SLOTS or cu[i] < 0 or cu[i + 1] > tokens][0]
    clean = [-1 if i == bad else s for i, s in enumerate(slots)]
    want_state, fine = start.clone(), _i32([0])
    rows = [min(max(c, 0), tokens) for c in cu]
    want = run(tokens, want_state, rows, clean, fine)
    assert int(fine) == 0 and torch.equal(state, want_state)
    others = torch.ones(tokens, dtype=torch.bool, device="cuda")
    others[zeros] = False
    assert torch.equal(got[others], want[others])


@pytest.mark.parametrize("mode", ["gated_write", "constant_decay", "plain_decay", "token_decay"])
@pytest.mark.parametrize("dim,vdim", [(64, 36), (20, 33), (160, 64)])
@pytest.mark.parametrize("step", range(len(STEPS)))
def test_linear_scan(mode, dim, vdim, step):
    from ampere_kv_engine_b200.kernels import ops

    heads, g = 2, torch.Generator(device="cuda").manual_seed(dim)
    x = torch.randn(30, heads * (2 * dim + vdim) + heads, generator=g, device="cuda")
    x[:, -heads:] = torch.sigmoid(x[:, -heads:])
    extra = {"gated_write": {"lower": torch.rand(heads * dim, generator=g, device="cuda")},
             "token_decay": {"decay_off": x.shape[1] - heads}}.get(mode, {"decay": torch.rand(heads, generator=g, device="cuda")})

    def run(tokens, state, cu, slots, status):
        return ops.linear_scan(x[:tokens].contiguous(), state, _i32(cu), _i32(slots), num_heads=heads, head_dim=dim, v_dim=vdim,
                               mode=mode, q_off=0, k_off=heads * dim, v_off=2 * heads * dim, status=status, **extra)

    _check(run, ops.linear_scan_state_floats(heads, dim, vdim), *STEPS[step])


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("dim,vdim", [(64, 36), (20, 33), (160, 64)])
@pytest.mark.parametrize("step", range(len(STEPS)))
def test_delta_scan(channel, dim, vdim, step):
    from ampere_kv_engine_b200.kernels import ops

    heads, taps, g = 4, 4, torch.Generator(device="cuda").manual_seed(dim)
    channels = heads * (2 * dim + vdim)
    qkv = torch.randn(30, channels, generator=g, device="cuda") * dim ** -0.5
    coef = torch.sigmoid(torch.randn(30, heads * (1 + (dim if channel else 1)), generator=g, device="cuda"))
    x = torch.randn(30, channels + heads * vdim + 2 * heads, generator=g, device="cuda")
    gates = torch.ones(30, heads * vdim, device="cuda")

    def run(tokens, state, cu, slots, status):
        return ops.delta_scan(qkv[:tokens].contiguous(), coef[:tokens].contiguous(), x[:tokens].contiguous(),
                              torch.ones(vdim, device="cuda"), state, _i32(cu), _i32(slots), num_heads=heads,
                              num_kv_heads=heads, head_dim=dim, v_dim=vdim, taps=taps, norm_eps=1.0,
                              gates=gates[:tokens].contiguous(), channel_decay=channel, status=status)

    _check(run, ops.delta_state_floats(heads, heads, dim, vdim, taps)[1], *STEPS[step])
