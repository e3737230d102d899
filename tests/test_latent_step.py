"""Which portions of a step have their keys and values written out (no GPU needed): each by its own length and reach, in
groups of bounded size; the others' tiles."""

import pytest

from ampere_kv_engine_b200.kernels import ops

SIZES = dict(window=0, portion=16, row_bytes=1000, q_tile=8, group_bytes=1 << 30, most_bytes=1 << 30)


def _taken(step):
    return [] if step is None else [plan.numbers[6 * i + 5] for plan in step.plans for i in range(plan.num_seqs)]


@pytest.mark.parametrize("n,context,taken", [(1, 500, False), (2, 2, False), (15, 15, False), (15, 4096, False), (16, 16, True),
                                             (16, 128, True), (16, 2064, True), (45, 45, True), (46, 130, True)])
@pytest.mark.parametrize("window", [0, 100])
def test_a_portion_is_judged_by_itself(n, context, taken, window):
    sizes = dict(SIZES, window=window)
    alone = _taken(ops.latent_step([n], [context], **sizes)) == [0]
    # beside a long prompt, short ones and single tokens
    among = 2 in _taken(ops.latent_step([2000, 1, n, 3], [2000, 700, context, 3], **sizes))
    assert alone == among == taken


def test_a_portion_that_needs_too_much_stays():
    sizes = dict(SIZES, most_bytes=256_000)
    assert _taken(ops.latent_step([20, 20, 20], [257, 256, 20], **sizes)) == [1, 2]
    assert ops.latent_step([20], [257], **sizes) is None
    # behind a window the gathered keys count, not the context
    assert _taken(ops.latent_step([20], [5000], **dict(sizes, window=100))) == [0]


def test_groups_and_what_stays():
    step = ops.latent_step([20, 1, 130, 19, 3, 40, 1], [20, 9, 400, 300, 8, 100, 2], **dict(SIZES, group_bytes=640_000))
    # 128, 512, 384 and 128 gathered rows
    assert [[p.numbers[6 * i + 5] for i in range(p.num_seqs)] for p in step.plans] == [[0, 2], [3, 5]]
    assert [p.rows for p in step.plans] == [640, 512]
    assert [p.numbers[4] for p in step.plans] == [0, 151]         # first batch rows
    # the three-token portion is one tile of the latent space; the last row that stays is the last single token's
    assert step.num_tiles == 1 and step.numbers[-3:] == [4, 170, 3] and step.rows == 214
    assert sum(len(p.numbers) for p in step.plans) + 3 == len(step.numbers)
    step = ops.latent_step([17, 15], [17, 15], **SIZES)
    assert step.numbers[-6:] == [1, 1, 17, 25, 8, 7] and step.rows == 32
    assert ops.latent_step([50, 60], [50, 60], **SIZES).rows == 0
