"""A latent that is not finite reaches the queries that see it and no other, though they share a tile with them."""

import pytest
import torch

from latent_case import LatentCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("window,key", [(0, 60), (0, 199), (0, 130), (40, 75), (40, 90)])
@pytest.mark.parametrize("column", [0, 37])
def test_a_latent_that_is_not_finite(value, window, key, column):
    from ampere_kv_engine_b200.kernels import ops

    case = LatentCase([120, 100], [200, 130], window=window, seed=key)      # positions 80 to 199, 30 to 129
    case.latents[0][key, column] = value
    got = case.run(ops)
    pos = torch.arange(80, 200, device="cuda")
    sees = (pos >= key) & ((pos - key < window) if window else (pos >= 0))
    want, bound = case.plain(0)
    first = got[:120]
    assert not bool(first[sees].isfinite().all(-1).any())
    assert bool(((first - want).abs() <= bound)[~sees].all())
    want, bound = case.plain(1)
    assert bool(((got[120:] - want).abs() <= bound).all())


@pytest.mark.parametrize("window,sink,sharpness", [(1, -4.0, 1.0), (2, -4.0, 1.0), (1, -12.0, 1.0), (0, None, 12.0)])
def test_a_row_that_one_key_dominates(window, sink, sharpness):
    """Such a row is nearly that key's value: a weight's rounding must not stay in it, only the result's.  (With a sink the
    walk refers its weights to the sink's score while no key stands far above it, so the largest is no power of two.)"""
    from ampere_kv_engine_b200.kernels import ops

    heads = 6
    case = LatentCase([300], [900], heads=heads, window=window, seed=5,
                      sink=None if sink is None else torch.full((heads,), sink, device="cuda"))
    case.scale *= sharpness
    got, (want, _) = case.run(ops), case.plain(0)
    # rounding the exact result alone; what the sink's share leaves of a weight's rounding, and further keys', fits into a
    # quarter of it (a weight's whole rounding would make it 1.4 times as much)
    rounding = (want.bfloat16().double() - want).norm()
    assert float((got - want).norm()) <= 1.25 * float(rounding)
