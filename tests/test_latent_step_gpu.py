"""A step whose portions go both ways through latents, beside single tokens: every sequence once, by its own length,
whatever order they come in."""

import pytest
import torch

import ligirax_util
import sukalorn_util

pytestmark = pytest.mark.gpu


def _run(monkeypatch, portion, held, new, group_bytes=None):
    """(logits of every entry's last token, portions written out, prompt tiles in the latent space) of a mixed step."""
    from ampere_kv_engine_b200.config.engine_config import EngineConfig
    from ampere_kv_engine_b200.engine.batch import SeqStep
    from ampere_kv_engine_b200.engine.engine import Engine
    from ampere_kv_engine_b200.kernels import ops
    from ampere_kv_engine_b200.parts import latent_attention

    runner = Engine.from_pretrained(sukalorn_util.model_folder("S3"),
                                    config=EngineConfig(dtype="bfloat16", num_pages=200)).runner
    tokens = torch.randint(0, 320, (2000,), generator=torch.Generator().manual_seed(1)).tolist()
    seqs = [runner.open(f"r{i}") for i in range(len(new))]
    for i, n in enumerate(held):
        if n:
            runner.step([SeqStep(seqs[i], tokens[7 * i:7 * i + n], [])])
    monkeypatch.setattr(latent_attention, "LATENT_PORTION", portion)
    if group_bytes is not None:
        monkeypatch.setattr(ops, "LATENT_GROUP_BYTES", group_bytes)
    written, stayed = [], []
    attention, scored = ops.latent_prompt_attention, ops.scored_attention

    def record_written(q, q_rows, cache, table, plan, *args, **kw):
        written.extend(int(plan.plan[6 * i + 5]) for i in range(plan.num_seqs))
        return attention(q, q_rows, cache, table, plan, *args, **kw)

    def record_stayed(q, k, v, table, cu, ctx, tile_seq, tile_q0, tile_nq, **kw):
        if k is v and kw["q_tile"] > 1:
            stayed.extend(zip(tile_seq.tolist(), tile_nq.tolist()))
        return scored(q, k, v, table, cu, ctx, tile_seq, tile_q0, tile_nq, **kw)

    monkeypatch.setattr(ops, "latent_prompt_attention", record_written)
    monkeypatch.setattr(ops, "scored_attention", record_stayed)
    logits = runner.step([SeqStep(seqs[i], tokens[1000 + 11 * i:1000 + 11 * i + n], [n - 1]) for i, n in enumerate(new)])
    runner.raise_on_status()
    monkeypatch.undo()
    return logits.double(), written, stayed


@pytest.mark.parametrize("held,new", [([0, 50, 0, 200, 7, 130], [16, 1, 3, 40, 1, 15]), ([130, 0], [17, 150]),
                                      ([300, 9, 20], [1, 1, 20])])
def test_a_step_that_goes_both_ways(monkeypatch, held, new):
    got, written, stayed = _run(monkeypatch, 16, held, new)
    assert written == [i for i, n in enumerate(new) if n >= 16]
    assert sorted(stayed) == [(i, n) for i, n in enumerate(new) if 1 < n < 16]
    want, written, _ = _run(monkeypatch, 10 ** 9, held, new)
    assert written == []
    # two ways through one of four layers, all in bfloat16: roundings of 2^-9 in another place, against the logits' size
    assert float((got - want).norm() / want.norm()) < 2.0 ** -6


def test_groups_one_after_the_other(monkeypatch):
    held, new = [0, 50, 0, 100, 7], [100, 1, 30, 20, 40]
    want, whole, _ = _run(monkeypatch, 16, held, new)
    # a row of keys and values of this layer takes 20 * (48 + 40) * 2 bytes: two portions of 128 rows a group
    got, grouped, _ = _run(monkeypatch, 16, held, new, group_bytes=256 * 20 * 88 * 2)
    assert whole == grouped == [0, 2, 3, 4]
    assert float((got - want).norm() / want.norm()) < 2.0 ** -6


def test_a_step_travels_in_one_copy(monkeypatch):
    """The plans of two layers that differ in their windows go with the step's index data, and are counted."""
    from ampere_kv_engine_b200.config.engine_config import EngineConfig
    from ampere_kv_engine_b200.engine.batch import SeqStep
    from ampere_kv_engine_b200.engine.engine import Engine

    runner = Engine.from_pretrained(ligirax_util.model_folder("L3"), config=EngineConfig(dtype="bfloat16", num_pages=100)).runner
    seqs = [runner.open(f"r{i}") for i in range(2)]
    pins, sizes = torch.Tensor.pin_memory, []

    def pin(tensor, *args, **kw):
        sizes.append(tensor.numel() * tensor.element_size())
        return pins(tensor, *args, **kw)

    monkeypatch.setattr(torch.Tensor, "pin_memory", pin)
    runner.step([SeqStep(seqs[0], list(range(40)), [39]), SeqStep(seqs[1], list(range(5)), [4])])
    runner.raise_on_status()
    assert len(sizes) == 1 and runner.last_h2d_bytes == sizes[0]


def test_a_step_without_room_for_keys_and_values(monkeypatch):
    """An engine whose weights and cache leave no room for a portion's written-out keys and values works on in the latent
    space, and asks for less from then on."""
    from ampere_kv_engine_b200.config.engine_config import EngineConfig
    from ampere_kv_engine_b200.engine.batch import SeqStep
    from ampere_kv_engine_b200.engine.engine import Engine
    from ampere_kv_engine_b200.parts import latent_attention

    runner = Engine.from_pretrained(sukalorn_util.model_folder("S3"),
                                    config=EngineConfig(dtype="bfloat16", num_pages=2200)).runner
    tokens = torch.randint(0, 320, (16400,), generator=torch.Generator().manual_seed(1)).tolist()
    seqs = [runner.open("a"), runner.open("b")]
    monkeypatch.setattr(latent_attention, "LATENT_PORTION", 10 ** 9)
    for lo in range(0, 16384, 2048):
        for seq in seqs:
            runner.step([SeqStep(seq, tokens[lo:lo + 2048], [])])
    want = runner.step([SeqStep(seqs[0], tokens[16384:], [15])])
    monkeypatch.undo()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # a portion of 16 tokens has small activations, but 58 MB of keys and values of its 16,400 latents
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (24 << 20)) / total)
    taken = []
    try:
        # what the process has reserved earlier and not given back must not hold them either
        with pytest.raises(torch.OutOfMemoryError):
            while True:
                taken.append(torch.empty(32 << 20, dtype=torch.uint8, device="cuda"))
        got = runner.step([SeqStep(seqs[1], tokens[16384:], [15])])
        torch.cuda.synchronize()
    finally:
        taken.clear()
        torch.cuda.set_per_process_memory_fraction(1.0)
    runner.raise_on_status()
    torch.testing.assert_close(got, want, atol=0, rtol=0)
    mixer = next(p for p in runner.model._parts() if isinstance(p, latent_attention.LatentAttention))
    assert mixer.most_bytes == 16512 * 20 * 88 * 2 // 2
