"""The scans against their recurrences in float64, from memories that hold something, in every form a step can select by its
size: a long sequence among short ones, many short sequences, one short sequence, single tokens; decays per head, per token
and per channel; heads that share q and k; the four-column preparation with a gate's bias in both storage types."""

import pytest
import torch

pytestmark = pytest.mark.gpu

#: what bounds a float32 result here: a sum of up to 256 products errs by some 2^-20 of its size, and the decays (below
#: 0.95) keep at most about 20 tokens' errors in the memory
REL = 20 * 2.0 ** -20

#: lengths of a step's sequences: a chain beyond 256 tokens; many blocks of one to four tokens; one portion that few blocks
#: walk; single tokens
STEPS = {"long": [1, 15, 16, 17, 300], "many": [1 + i % 4 for i in range(150)], "few": [33], "single": [1] * 9}


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _rand(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def _step(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    slots = torch.randperm(len(lens) + 2, generator=torch.Generator().manual_seed(len(lens)))[:len(lens)].tolist()
    return cu, slots


def _close(got, want, what):
    error = (got.double() - want).abs().max()
    assert float(error) <= REL * float(want.abs().max()), (what, float(error), float(want.abs().max()))


@pytest.mark.parametrize("step", list(STEPS))
@pytest.mark.parametrize("dim,vdim", [(64, 64), (36, 20), (128, 96), (100, 32), (256, 64), (132, 36), (30, 20)])
@pytest.mark.parametrize("mode,dtype", [("gated_write", torch.bfloat16), ("gated_write", torch.float32), ("constant_decay", torch.bfloat16),
                                        ("plain_decay", torch.float32), ("token_decay", torch.float32)])
def test_linear_scan(mode, dtype, dim, vdim, step):
    from ampere_kv_engine_b200.kernels import ops

    lens, heads = STEPS[step], 4
    group = 2 if mode == "token_decay" else 1
    cu, slots = _step(lens)
    n, qk = cu[-1], heads // group * dim
    x = _rand(n, 2 * qk + heads * vdim + 8, seed=dim).to(dtype)
    extra = {}
    if mode == "gated_write":
        extra = {"lower": 0.9 * torch.sigmoid(_rand(qk, seed=1)), "gate_bias": _rand(qk, seed=2) - 1.0}
    elif mode == "token_decay":
        x[:, -heads:] = 0.95 * torch.sigmoid(x[:, -heads:])
        extra = {"decay_off": x.shape[1] - heads, "qk_group": group}
    else:
        extra = {"decay": torch.linspace(0.3, 0.95, heads, device="cuda")}
    state = _rand(len(lens) + 2, ops.linear_scan_state_floats(heads, dim, vdim), seed=3)
    start, status = state.clone(), _i32([0])
    got = ops.linear_scan(x, state, _i32(cu), _i32(slots), num_heads=heads, head_dim=dim, v_dim=vdim, mode=mode, q_off=0, k_off=qk,
                          v_off=2 * qk, status=status, **extra).view(n, heads, vdim)
    assert int(status) == 0
    z = x.double()
    silu = torch.nn.functional.silu
    q, k = (z[:, i * qk:(i + 1) * qk].view(n, heads // group, dim).repeat_interleave(group, 1) for i in (0, 1))
    v = z[:, 2 * qk:2 * qk + heads * vdim].view(n, heads, vdim)
    if mode == "gated_write":
        low = extra["lower"].double().view(heads, dim)
        a = low + (1.0 - low) * torch.sigmoid(k + extra["gate_bias"].double().view(heads, dim))
        q, k = silu(q), 1.0 - a
    else:
        a = z[:, -heads:] if mode == "token_decay" else extra["decay"].double().expand(n, heads)
        a = a[:, :, None].expand(n, heads, dim)
        if mode == "constant_decay":
            q, k, v = silu(q), silu(k), silu(v)
    want = torch.empty(n, heads, vdim, dtype=torch.float64, device="cuda")
    for s, slot in enumerate(slots):
        S = ops.linear_scan_memory(start[slot], heads, dim, vdim).double()
        for t in range(cu[s], cu[s + 1]):
            S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hdv,hd->hv", S, q[t])
        _close(ops.linear_scan_memory(state[slot], heads, dim, vdim), S, ("memory", s))
    _close(got, want, "output")
    rest = [i for i in range(len(lens) + 2) if i not in slots]
    assert torch.equal(state[rest], start[rest])


def _delta_memory(ops, row, heads, dim, vdim):
    per_lane, lanes = ops.delta_shape(dim, vdim)
    row = row[:heads * vdim * lanes * per_lane].view(heads, per_lane // 4, vdim, lanes, 4)
    return row.permute(0, 3, 1, 4, 2).reshape(heads, lanes * per_lane, vdim)


@pytest.mark.parametrize("step", list(STEPS))
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (36, 20), (128, 96), (100, 32), (256, 64), (132, 36), (30, 20)])
def test_delta_scan(dim, vdim, channel, step):
    from ampere_kv_engine_b200.kernels import ops

    lens, heads, kv_heads, taps, eps = STEPS[step], 4, 2, 3, 1e-2
    cu, slots = _step(lens)
    n, channels = cu[-1], 2 * kv_heads * dim + heads * vdim
    qkv = _rand(n, channels, seed=dim)
    for lo in (0, kv_heads * dim):
        part = qkv[:, lo:lo + kv_heads * dim].view(n, kv_heads, dim)
        part /= part.norm(dim=-1, keepdim=True)
    coef = 0.95 * torch.sigmoid(_rand(n, heads * (1 + (dim if channel else 1)), seed=1))
    x, gates = _rand(n, channels + heads * vdim + 2 * heads, seed=2), _rand(n, heads * vdim, seed=3)
    memory, floats = ops.delta_state_floats(heads, kv_heads, dim, vdim, taps)
    state = _rand(len(lens) + 2, floats, seed=4)
    # rows beyond the width are zeros in a state
    per_lane, lanes = ops.delta_shape(dim, vdim)
    for row in state:
        view = row[:memory].view(heads, per_lane // 4, vdim, lanes, 4)
        index = torch.arange(lanes * per_lane, device="cuda").view(lanes, per_lane // 4, 4).permute(1, 0, 2)[:, None]
        view.masked_fill_((index >= dim).expand(per_lane // 4, vdim, lanes, 4), 0.0)
    start, status, weight = state.clone(), _i32([0]), 1.0 + 0.1 * _rand(vdim, seed=5)
    got = ops.delta_scan(qkv, coef, x, weight, state, _i32(cu), _i32(slots), num_heads=heads, num_kv_heads=kv_heads, head_dim=dim,
                         v_dim=vdim, taps=taps, norm_eps=eps, gates=gates, channel_decay=channel, status=status).view(n, heads, vdim)
    assert int(status) == 0
    z = qkv.double()
    q, k = (z[:, i * kv_heads * dim:(i + 1) * kv_heads * dim].view(n, kv_heads, dim).repeat_interleave(heads // kv_heads, 1) for i in (0, 1))
    v, beta = z[:, 2 * kv_heads * dim:].view(n, heads, vdim), coef[:, :heads].double()
    decay = coef[:, heads:].double().view(n, heads, -1).expand(n, heads, dim)
    raw = torch.empty(n, heads, vdim, dtype=torch.float64, device="cuda")
    for s, slot in enumerate(slots):
        S = _delta_memory(ops, start[slot], heads, dim, vdim)[:, :dim].double()
        for t in range(cu[s], cu[s + 1]):
            S = S * decay[t][:, :, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            raw[t] = torch.einsum("hdv,hd->hv", S, q[t])
        _close(_delta_memory(ops, state[slot], heads, dim, vdim)[:, :dim], S, ("memory", s))
        kept = torch.cat((start[slot, memory:memory + (taps - 1) * channels].view(taps - 1, channels), x[cu[s]:cu[s + 1], :channels]))
        assert torch.equal(state[slot, memory:memory + (taps - 1) * channels].view(taps - 1, channels), kept[-(taps - 1):])
    g = gates.double().view(n, heads, vdim)
    want = raw / torch.sqrt(raw.square().mean(-1, keepdim=True) + eps) * weight.double() * torch.nn.functional.silu(g)
    _close(got, want, "output")
    rest = [i for i in range(len(lens) + 2) if i not in slots]
    assert torch.equal(state[rest], start[rest])
