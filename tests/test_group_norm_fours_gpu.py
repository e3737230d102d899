"""The output norm of whole groups of four columns: the group sizes at which its kernel changes form."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("group,groups", [(128, 3), (256, 2), (512, 5), (1024, 2), (2048, 1), (4096, 2), (8192, 1)])
def test_norm_of_whole_fours(dtype, group, groups):
    from ampere_kv_engine_b200.kernels import ops

    n, width = 5, group * groups
    g = torch.Generator(device="cuda").manual_seed(group)
    o = torch.randn(n, width, generator=g, device="cuda") * 3.0
    x = torch.randn(n, width + 12, generator=g, device="cuda").to(dtype)
    skip, coef = torch.randn(n, width + 4, generator=g, device="cuda"), torch.randn(width // 32, generator=g, device="cuda")
    od, zd = o.double(), x[:, 8:8 + width].double()
    shape = (n, groups, group)
    for weight in (None, torch.rand(group, generator=g, device="cuda") + 0.5, torch.rand(width, generator=g, device="cuda")):
        wd = 1.0 if weight is None else weight.double().repeat(width // weight.numel())
        for gate, first, skipped in ((None, False, False), ("sigmoid", False, False), ("silu", False, True), ("silu", True, True)):
            v, z = od, None
            if skipped:
                v = v + coef.double().repeat_interleave(32) * skip[:, 4:].double()
            if gate:
                z = torch.sigmoid(zd) * (zd if gate == "silu" else 1.0)
                v = v * z if first else v
            want = (v.view(shape) / torch.sqrt(v.view(shape).square().mean(-1, keepdim=True) + 1e-6)).view(n, width) * wd * 0.7
            if gate and not first:
                want = want * z
            got = ops.group_norm_gate(o, weight, group=group, eps=1e-6, out_dtype=dtype, factor=0.7, x=x if gate else None,
                                      gate_off=8, gate=gate or "sigmoid", gate_first=first, skip=skip if skipped else None,
                                      skip_off=4, skip_coef=coef if skipped else None, skip_head=32)
            # a few float32 roundings (2^-24 each) of the value and of the root mean square, the skip's own cancellation,
            # and one rounding to the result's dtype
            size = want.abs() + (wd * 0.7 * (od.abs() + (skip[:, 4:].double().abs() * coef.double().abs().repeat_interleave(32))) if skipped else 0)
            assert bool(((got.double() - want).abs() <= 2.0 ** -19 * size + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0) + 1e-6).all())
