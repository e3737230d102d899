"""A sink of minus infinity, or of the lowest bfloat16 (whose score in log2 units overflows to it), is a sink that takes
nothing: in every kernel that knows sinks, beside heads with finite ones."""

import pytest
import torch

from latent_case import LatentCase
from test_gosizen_kernels_gpu import SINK_CASES, TOL, _attend, _attend_plain
from paged_case import PagedCase

pytestmark = pytest.mark.gpu


def _sinks(heads):
    lowest = torch.finfo(torch.bfloat16).min
    return torch.tensor([(-float("inf"), 0.7, lowest, -2.0)[h % 4] for h in range(heads)], device="cuda")


@pytest.mark.parametrize("dtype,nh,nkv,d,page", SINK_CASES)
@pytest.mark.parametrize("window", [0, 33])
def test_a_sink_that_takes_nothing(dtype, nh, nkv, d, page, window):
    from ampere_kv_engine_b200.kernels import ops

    sink = _sinks(nh)
    for q_lens, ctx, splits in (([1, 1, 1], [200, 3, 41], (1, 4)), ([70, 2, 33], [170, 2, 73], (1,))):
        case = PagedCase(dtype, nh, nkv, d, page, q_lens, ctx, seed=d, q_tile=32)
        want = _attend_plain(case, sink, d ** -0.5, window)
        for n in splits:
            for kernel in ("auto", "general"):
                if n > 1 and kernel == "auto" and d == 20:
                    continue
                got = _attend(ops, case, sink, d ** -0.5, window, splits=n, kernel=kernel)
                torch.testing.assert_close(got, want, **TOL[dtype])


@pytest.mark.parametrize("row,v_dim", [(80, 64), (52, 33)])
def test_a_sink_that_takes_nothing_over_shared_rows(row, v_dim):
    from ampere_kv_engine_b200.kernels import ops

    sink, dtype = _sinks(20), torch.bfloat16
    for q_lens, ctx, splits in (([1, 1], [300, 7], (1, 3)), ([40, 5], [90, 5], (1, 2))):
        case = PagedCase(dtype, 20, 1, row, 16, q_lens, ctx, seed=row, q_tile=32)
        want = _attend_plain(case, sink, row ** -0.5, shared=True, v_dim=v_dim)
        for n in splits:
            got = _attend(ops, case, sink, row ** -0.5, splits=n, shared=True, v_dim=v_dim)
            torch.testing.assert_close(got, want, **TOL[dtype])


@pytest.mark.parametrize("window", [0, 100])
def test_a_sink_that_takes_nothing_over_latents(window):
    from ampere_kv_engine_b200.kernels import ops

    case = LatentCase([2, 130], [2, 200], heads=4, window=window, sink=_sinks(4), seed=window)
    got = case.run(ops)
    for s, rows in ((0, slice(0, 2)), (1, slice(2, 132))):
        want, bound = case.plain(s)
        assert bool(((got[rows] - want).abs() <= bound).all())
