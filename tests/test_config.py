"""Configuration and registry (no GPU)."""
import json

import pytest

from lgml_b200.config import (ConfigError, LlamaConfig, ModelConfig, architectures, config_from_dict, load_config,
                              lookup_architecture, register_architecture)
from tests import helpers as H


def test_llama_defaults_follow_the_reference():
    d = {"architectures": ["LlamaForCausalLM"], "vocab_size": 100, "hidden_size": 96, "intermediate_size": 50,
         "num_hidden_layers": 1, "num_attention_heads": 6, "rms_norm_eps": 1e-5, "max_position_embeddings": 64}
    c = config_from_dict(d)
    assert c.num_key_value_heads == 6            # defaults to the heads
    assert c.head_dim == 16                      # hidden // heads
    assert c.rope_theta == 10000.0
    assert c.rope_scaling is None and not c.tie_word_embeddings and not c.attention_bias and not c.mlp_bias


@pytest.mark.parametrize("which", ["A", "B", "C"])
def test_round_trip(which):
    cfg, _ = H.TINY[which]
    c = config_from_dict(cfg)
    again = config_from_dict(json.loads(json.dumps(c.to_dict())))
    assert again == c
    assert c.head_dim == cfg["head_dim"] and c.vocab_size == cfg["vocab_size"]


def test_head_width_may_differ_from_hidden():
    c = config_from_dict(H.TINY_B)
    assert c.num_attention_heads * c.head_dim == 192 != c.hidden_size


def test_rope_parameters_style():
    d = dict(H.TINY_B)
    rs = d.pop("rope_scaling")
    theta = d.pop("rope_theta")
    d["rope_parameters"] = dict(rs, rope_theta=theta)
    assert config_from_dict(d) == config_from_dict(H.TINY_B)
    d["rope_parameters"] = {"rope_type": "default", "rope_theta": 1234.0}
    c = config_from_dict(d)
    assert c.rope_theta == 1234.0 and c.rope_scaling is None


@pytest.mark.parametrize("key", ["vocab_size", "hidden_size", "intermediate_size", "num_hidden_layers", "num_attention_heads",
                                 "rms_norm_eps", "max_position_embeddings"])
def test_missing_key_is_named(key):
    d = dict(H.TINY_A)
    del d[key]
    with pytest.raises(ConfigError, match=key):
        config_from_dict(d)


@pytest.mark.parametrize("change,match", [
    ({"num_key_value_heads": 3}, "multiple"),
    ({"head_dim": 15}, "even"),
    ({"hidden_act": "gelu"}, "hidden_act"),
    ({"rope_scaling": {"rope_type": "yarn", "factor": 2.0}}, "rope_type"),
    ({"rope_scaling": {"rope_type": "llama3", "factor": 8.0}}, "low_freq_factor"),
    ({"rms_norm_eps": 0.0}, "rms_norm_eps"),
    ({"vocab_size": 0}, "vocab_size"),
])
def test_bad_values_are_refused(change, match):
    with pytest.raises(ConfigError, match=match):
        config_from_dict({**H.TINY_A, **change})


def test_unknown_architecture_is_named():
    with pytest.raises(ConfigError, match="MambaForCausalLM"):
        config_from_dict({**H.TINY_A, "architectures": ["MambaForCausalLM"]})
    with pytest.raises(ConfigError, match="architectures"):
        config_from_dict({k: v for k, v in H.TINY_A.items() if k != "architectures"})
    assert "LlamaForCausalLM" in architectures()


def test_load_config_errors(tmp_path):
    with pytest.raises(ConfigError, match="config.json"):
        load_config(tmp_path)
    (tmp_path / "config.json").write_text("{not json")
    with pytest.raises(ConfigError, match="JSON"):
        load_config(tmp_path)
    (tmp_path / "config.json").write_text(json.dumps(H.TINY_B))
    assert isinstance(load_config(tmp_path), LlamaConfig)


def test_eos_forms():
    assert config_from_dict({**H.TINY_A, "eos_token_id": 7}).eos_token_ids == [7]
    assert config_from_dict({**H.TINY_A, "eos_token_id": [7, 9]}).eos_token_ids == [7, 9]


def test_registry_takes_a_new_architecture():
    class Toy(ModelConfig):
        @classmethod
        def from_dict(cls, d):
            return cls(architecture="ToyForTest")

        def validate(self):
            pass

    register_architecture("ToyForTest", Toy, lambda cfg: "model")
    cls, builder = lookup_architecture("ToyForTest")
    assert cls is Toy and builder(None) == "model"
    assert config_from_dict({"architectures": ["ToyForTest"]}).architecture == "ToyForTest"


def test_k_ranges_of_a_small_product_are_never_empty():
    """The number of K ranges a product is cut into: every range gets at least one block (9 ranges
    of 8 blocks would leave the ninth of 64 blocks empty).  A block is 64 elements up to 64 tokens
    and a stage of 128 from 65 tokens on, where the product runs on pairs of CTAs; many tokens
    and many tiles leave K whole."""
    from lgml_b200.ops import tcgen05_splits

    for M in (1, 8, 16, 17, 64, 65, 128, 200, 256, 300, 2048):
        for N in (1024, 3072, 4096, 5120, 6144, 9216, 14336, 28672, 128256):
            for K in (64, 512, 3072, 4096, 5120, 8192, 13824, 14336):
                s = tcgen05_splits(M, N, K)
                blocks = -(-K // (64 if M <= 64 else 128))
                per = -(-blocks // s)
                assert 1 <= s <= (16 if M <= 64 else 8) and (s - 1) * per < blocks, (M, N, K, s)
                if M > 64 and s > 1:
                    assert per >= 4                         # no range shorter than four stages
                if M >= 2048 and N >= 3072:
                    assert s == 1


def test_key_ranges_of_the_decode_attention_stay_within_their_bounds():
    """The rule that cuts a token's keys into ranges: at least one range, never more than the
    merge kernel takes, no range shorter than four pages, never more CTAs than fill the SMs twice
    (once for one or two short requests), and one range from 37 requests on 8 KV heads up."""
    from lgml_b200.ops import decode_splits, sm_count

    for n in (1, 2, 3, 4, 8, 16, 37, 64, 256):
        for kv, group in ((8, 4), (40, 1), (1, 12), (5, 9)):
            for ctx in (1, 64, 65, 1024, 4096, 16384, 32768, 131072, 1 << 20):
                s = decode_splits(n, kv, group, ctx)
                pages = -(-ctx // 64)
                ctas = n * kv * ((group + 7) // 8)
                assert 1 <= s <= 512
                assert s == 1 or -(-pages // s) >= 4 or s * 4 <= pages + 3, (n, kv, group, ctx, s)
                assert s == 1 or s * ctas <= 2 * sm_count(), (n, kv, group, ctx, s)
    assert decode_splits(37, 8, 4, 4096) == 1 and decode_splits(1, 8, 4, 4096) == 16 and decode_splits(2, 8, 4, 4096) == 9


def test_ranges_of_contexts_that_fill_their_last_round_badly():
    """More than one range for many CTAs only where all measured contexts gain: heads with keys of their own, even contexts over 1,024
    tokens, a last round of the chip that is nearly empty.  Everything else is ``decode_splits``."""
    from lgml_b200.engine.runner import context_reach
    from lgml_b200.ops import decode_ranges, decode_splits, sm_count

    R = 2 * sm_count()                                              # CTAs of head size 128 that the chip holds at once
    for ctas, want in ((R, 1), (R + 1, 3), (int(1.3 * R), 3), (int(1.32 * R), 1), (2 * R, 1), (2 * R + 1, 3), (int(2.2 * R), 3), (int(2.3 * R), 1),
                       (3 * R + 1, 1), (8 * R + 1, 1)):
        assert decode_ranges(1, ctas, 1, 128, 1025, 2048) == want
        assert decode_ranges(1, 2 * ctas, 1, 64, 3000, 4096) == want
        for group, dim, shortest, longest in ((1, 128, 1024, 2048), (1, 128, 70, 1024), (1, 128, 2047, 4096), (1, 128, 1, 4096), (1, 96, 4096, 4096),
                                              (4, 128, 4096, 4096), (1, 256, 4096, 4096), (1, 128, 512, 512)):
            assert decode_ranges(1, ctas, group, dim, shortest, longest) == decode_splits(1, ctas, group, longest) == 1
    for n, g, group in ((1, 8, 4), (4, 8, 1), (8, 32, 1), (2, 5, 9)):
        assert decode_ranges(n, g, group, 128, 3000, 3000) == decode_splits(n, g, group, 3000)
    # a captured step is told only what its graph is for: the same answer at both ends of what it replays
    for lengths, reach, even in (([1], 1024, False), ([513, 1024], 1024, True), ([512, 1024], 1024, False), ([1025], 2048, True),
                                 ([1025, 2048], 2048, True), ([1024, 1025], 2048, False), ([3585] * 16, 4096, True), ([3585, 20], 4096, False)):
        assert context_reach(lengths) == (reach, even)
        if even:
            answers = {decode_ranges(16, 40, 1, 128, reach // 2 + 1, reach), decode_ranges(16, 40, 1, 128, max(lengths), max(lengths))}
            assert len(answers) == 1


def test_chunks_and_scratch_of_tokens_taken_by_themselves():
    """float32 attention: a window is given the chunks it can touch wherever it starts, not its context's, and the scratch has a bound
    whatever the batch and the context."""
    from lgml_b200 import ops

    for window in (1, 2, 100, 127, 128, 129, 256, 257, 4096):
        touched = max((start + window - 1) // 128 - start // 128 + 1 for start in range(256))
        assert ops.attention_f32_chunks(1, 8, 8, 64, 1 << 20, window)[0] == (0 if touched == 1 else touched)
    assert ops.attention_f32_chunks(1, 8, 8, 64, 300, 1000)[0] == 3 and ops.attention_f32_chunks(1, 8, 8, 64, 128, 0) == (0, 0)
    assert ops.attention_f32_chunks(64, 8, 8, 64, 1024, 0) == (0, 0) and ops.attention_f32_chunks(64, 8, 8, 64, 1025, 0)[0] == 9
    for n, heads, kv, dim, ctx in ((32, 32, 8, 128, 32768), (2048, 40, 40, 128, 131072), (8, 64, 1, 16, 4096)):
        chunks, tokens = ops.attention_f32_chunks(n, heads, kv, dim, ctx, 0)
        floats = tokens * heads * chunks * (dim + 2)
        assert chunks == -(-ctx // 128) and 1 <= tokens <= n and (4 * floats <= ops.ATTENTION_F32_SCRATCH or tokens == 1)


def test_requests_taken_token_by_token_and_as_tiles():
    """float32 attention: which requests of a step go token by token (those whose tokens are less work than their tiles, and the shortest as
    long as all of them take less than one tile), and the two lists of a step that holds both kinds."""
    from types import SimpleNamespace

    import numpy as np
    import torch

    from lgml_b200 import ops
    from lgml_b200.engine.batch import StepBatch

    short = lambda lens, *shape: ops.attention_f32_short(lens, *shape)
    assert short([9], 16, 4, 128) == 9 and short([96], 16, 4, 128) == 96 and short([300], 16, 4, 128) < 300
    assert short([9] * 16, 40, 40, 128) == 9 and short([12] * 16, 40, 40, 128) == 9 and short([1] * 500 + [40], 40, 40, 128) == 9 and short([1, 1, 30], 8, 8, 64) == 30
    for shape in ((8, 8, 64), (40, 40, 128), (64, 1, 128), (24, 8, 128)):
        assert short([1] * 4096, *shape) >= 1 and short([2048], *shape) < 64

    lens, pos0 = [1, 70, 2, 1, 9], [40, 0, 7, 500, 3]
    reqs = [SimpleNamespace(id=i, slot=i, n_tokens=p, tables=[]) for i, p in enumerate(pos0)]
    manager = SimpleNamespace(groups=[])
    batch = StepBatch(manager, reqs, [[0] * n for n in lens], [[] for _ in lens], torch.device("cpu"))
    tiles, few, longest = batch.tiles_and_short(16, lambda got: 2 if got == lens else None, "a")
    assert few.tolist() == [0, 71, 72, 73] and longest == 501
    rows = sorted((t, n, s) for s, t, n, _ in tiles.tolist())
    assert rows == [(1, 16, 1), (17, 16, 1), (33, 16, 1), (49, 16, 1), (65, 6, 1), (74, 9, 4)]
    assert batch.tiles_and_short(16, None, "a")[0] is tiles                     # made once
    assert batch.tiles_and_short(16, lambda _: 70, "b") == (None, None, 501)
    tiles, few, longest = batch.tiles_and_short(16, lambda _: 0, "c")
    assert few is None and longest == 0 and np.array_equal(tiles.numpy(), batch.attention_tiles(16).numpy())


def test_layouts_that_the_host_sizes_are_the_kernels_own():
    """Scratch is sized by what the libraries say of themselves: a record holds at least a block's vectors, triangles and steps."""
    from lgml_b200 import ops

    n = ops.delta_block_tokens()
    for dim in (4, 12, 64, 128):
        assert ops.delta_block_record(dim) >= (3 * n + 1) * dim + 2 * n * n + n and ops.delta_block_record(dim) % 4 == 0
    assert ops.attention_f32_chunk() % 64 == 0


def test_end_tokens_of_generation_config_join_those_of_config(tmp_path):
    import json

    from lgml_b200.config import ConfigError, load_config
    from tests import helpers as H

    d = dict(H.TINY_B, eos_token_id=7)
    (tmp_path / "config.json").write_text(json.dumps(d))
    assert load_config(tmp_path).eos_token_ids == [7]
    (tmp_path / "generation_config.json").write_text(json.dumps({"eos_token_id": [9, 7, 11], "temperature": 0.6}))
    assert load_config(tmp_path).eos_token_ids == [7, 9, 11]
    (tmp_path / "generation_config.json").write_text(json.dumps({"eos_token_id": 3}))
    assert load_config(tmp_path).eos_token_ids == [7, 3]
    (tmp_path / "generation_config.json").write_text(json.dumps({"eos_token_id": "x"}))
    with pytest.raises(ConfigError, match="eos_token_id"):
        load_config(tmp_path)


@pytest.mark.parametrize("lens,pos0", [([1], [5]), ([64], [0]), ([65, 1, 300, 2, 300], [0, 900, 12, 63, 40]), ([28, 27, 29], [7, 7, 7])])
def test_tiles_and_pieces_of_a_step(lens, pos0):
    """Against the rule in Python, asked for one by one and sent with the step's description; from 16-byte boundaries there."""
    from types import SimpleNamespace

    import torch

    from lgml_b200.engine.batch import StepBatch

    reqs = [SimpleNamespace(id=i, slot=i, n_tokens=p, tables=[]) for i, p in enumerate(pos0)]
    ids = [[7 * s + j for j in range(n)] for s, n in enumerate(lens)]
    lists = {}
    starts = [sum(lens[:s]) for s in range(len(lens))]
    for round_ in range(2):
        pinned = torch.full((4096,), -7, dtype=torch.int32)
        b = StepBatch(SimpleNamespace(groups=[]), reqs, ids, [[n - 1] for n in lens], torch.device("cpu"), pinned, lists=lists)
        assert len(b._tiles) == (0 if round_ == 0 else len(lists))
        assert b.token_ids.tolist() == sum(ids, []) and b.seq_start.tolist() == starts + [sum(lens)] and b.logit_rows.tolist() == [a + n - 1 for a, n in zip(starts, lens)]
        assert b.positions.tolist() == [p + j for p, n in zip(pos0, lens) for j in range(n)] and b.seq_of_token.tolist() == [s for s, n in enumerate(lens) for _ in range(n)]
        for tile, longer in ((16, 0), (64, 0), (16, 27)):
            want = [(s, a + t, min(tile, n - t), p + min(t + tile, n)) for s, (a, n, p) in enumerate(zip(starts, lens, pos0)) if n > longer for t in range(0, n, tile)]
            got = b.attention_tiles(tile, longer)
            assert got.tolist() == [[s, a, n, 0] for s, a, n, _ in sorted(want, key=lambda r: -r[3])]
            assert round_ == 0 or (got.data_ptr() - b._dev.data_ptr()) % 16 == 0
        for ctas in (1, 8, 1000):           # half a tile while each has an SM to itself
            size = 32 if sum(-(-n // 32) for n in lens) * ctas <= 148 else 64
            assert b.twin_tiles(64, ctas).tolist() == b.attention_tiles(size).tolist()
        pieces, first = b.scan_pieces(16)
        want = [[[a + t, a + min(t + 16, n)] for t in range(0, n, 16)] for a, n in zip(starts, lens)]
        assert pieces.tolist() == sum(want, []) and first.tolist() == [sum(map(len, want[:s])) for s in range(len(lens) + 1)]
        got = b.scan_chunks(32, 27)
        long = [s for s, n in enumerate(lens) if n > 27]
        assert (got is None) == (not long)
        if long:
            want = [[[starts[s] + t, starts[s] + min(t + 32, lens[s])] for t in range(0, lens[s], 32)] for s in long]
            assert got.rows.tolist() == sum(want, []) and got.requests.tolist() == long and got.short == (len(long) < len(lens))
            assert got.first.tolist() == [sum(map(len, want[:s])) for s in range(len(long) + 1)] and (got.longer_than, got.chunk_tokens) == (27, 32)
