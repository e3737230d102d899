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
