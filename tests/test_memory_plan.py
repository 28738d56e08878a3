"""The memory plan: bytes of weights, cache and workspace from a configuration alone, and the
refusal before anything is allocated."""
import pytest
import torch

import camelid_b200
from camelid_b200 import MemoryBudgetError, benchmark, memory_plan
from conftest import TINY_A, TINY_B


def test_plan_counts_what_the_survey_counts():
    """Llama 3.2 1B: 973.1 M linear + 262.7 M embedding (tied) + 67.6 k norm parameters; the
    cache keeps 2 * 16 layers * 8 kv heads * 64 = 16,384 elements a position."""
    cfg = benchmark.config_for(2)
    p = memory_plan(cfg, "bfloat16", max_tokens=8 * 4096, max_slots=8)
    assert p.weights == (973_078_528 + 262_668_288 + 33 * 2048) * 2
    assert p.cache == 8 * 4096 * 16_384 * 2
    assert p.total == p.weights + p.cache + p.workspace and 0 < p.workspace < 1 << 30
    f = memory_plan(cfg, "float32", max_tokens=8 * 4096, max_slots=8)
    assert f.weights == 2 * p.weights and f.cache == 2 * p.cache
    untied = memory_plan({**cfg, "tie_word_embeddings": False}, "bfloat16")
    assert untied.weights - p.weights == 262_668_288 * 2 and untied.cache == 0
    # tokens are rounded up to pages of 64
    assert memory_plan(TINY_A, "float32", max_tokens=65).cache == memory_plan(TINY_A, "float32", max_tokens=128).cache


def test_8b_in_float32_is_refused_on_a_32_gb_device_with_the_numbers():
    cfg = benchmark.config_for(4)
    plan = memory_plan(cfg, "float32", max_tokens=8 * 8192, max_slots=8)
    assert 32.0e9 < plan.weights < 32.3e9                      # 8.03 G parameters in 4 bytes
    with pytest.raises(MemoryBudgetError) as e:
        plan.check(32 * 2 ** 30, "Llama 3.1 8B in float32")
    assert e.value.needed == plan.total and e.value.available == 32 * 2 ** 30
    assert f"{plan.weights:,}" in str(e.value) and f"{plan.cache:,}" in str(e.value)
    plan.check(64 * 2 ** 30)
    assert isinstance(e.value, camelid_b200.CacheError) and isinstance(e.value, camelid_b200.CamelidError)


def test_load_refuses_before_it_reads_a_tensor():
    """``load_tensors`` checks names, shapes and then the bytes: a source whose tensors would
    not fit is refused without one tensor having been asked for."""
    from camelid_b200 import DecoderModel
    model = DecoderModel.from_config(TINY_B, dtype=torch.float32, device="cpu")
    specs = model.tensor_specs()

    class Source:
        asked = []

        def names(self):
            return list(specs)

        def shape(self, name):
            return list(specs[name].shape)

        def dtype(self, name):
            return torch.bfloat16

        def tensor(self, name):
            self.asked.append(name)
            raise AssertionError("no tensor may be read")
    src = Source()
    need = model.memory_plan().weights
    with pytest.raises(MemoryBudgetError) as e:
        model.load_tensors(src, available_bytes=need - 1)
    assert src.asked == [] and not model.loaded and e.value.needed == need


def test_chunked_portions_and_their_scratch():
    """Tiles of the portions that run by chunks and of no other; the bound on their number holds for every mix; the plan
    counts what single tokens and ragged portions beside a prompt take."""
    import random
    from camelid_b200.config.plan import PartSpec
    from camelid_b200.csrc import ops
    from camelid_b200.engine.context import StepContext
    from camelid_b200.parts import build_part
    rng = random.Random(5)
    for _ in range(300):
        news = [int(2 ** rng.uniform(0, 9)) for _ in range(rng.randint(1, 40))]
        if max(news) == 1:
            continue
        size, least = key = rng.choice(((64, 128), (64, 64), (64, 32), (32, 128)))
        layout, host, _, _ = StepContext.host_arrays(range(len(news)), [0] * len(news), [[0] * n for n in news], [[] for _ in news], [], [64, key])
        for r, floor in ((64, 1), (key, least)):
            want = [(s, q) for s, n in enumerate(news) for q in range(0, n, r if floor == 1 else size) if n >= floor]
            assert list(zip(layout.view(host, f"tile_seq{r}"), layout.view(host, f"tile_q0{r}"))) == want and layout.n_tiles[r] == len(want)
        assert len(want) <= ops.chunks_at_most(sum(news), len(news), size, least)
    common = {"hidden_size": 64, "num_heads": 16, "key_dim": 128, "value_dim": 128, "state_size": 128, "conv_taps": 4, "gate_cap": 15.0}
    square = 64 * 64
    floats = {"retention": 16 * (square + 4 * 64 + 128 * 128), "matrix_memory": 16 * (square + 4 * 64 + 129 * 128),
              "state_space": square + 16 * (3 * 64 + 128 * 128), "gated_delta": 16 * ops.gated_chunk_floats(128, 128)}
    for kind, per_chunk in floats.items():
        part = build_part("mixer", PartSpec(kind, {**common, "decay": [0.9] * 16 if kind == "retention" else None}))
        size, least = part.query_tile_sizes()[0]
        for news in ([128] + [1] * 63, [2048] + [1] * 200, [least] * 40, [least + 1] * 30, [2047]):
            assert part.workspace(sum(news), len(news)) >= 4 * per_chunk * sum(-(-n // size) for n in news if n >= least)


def test_shares_of_single_tokens_over_a_latent():
    """Every multiprocessor gets at most two blocks, a row at most 64 shares; the plan counts what the shares take."""
    import random
    from camelid_b200.config.plan import PartSpec
    from camelid_b200.csrc import ops
    from camelid_b200.parts import build_part
    from camelid_b200.parts.latent_attention import pages_a_block
    rng = random.Random(6)
    for _ in range(500):
        pages, rows, heads = int(2 ** rng.uniform(0, 10)), int(2 ** rng.uniform(0, 9)), rng.choice((1, 16, 64, 65, 128))
        part = build_part("mixer", PartSpec("latent_attention", {"hidden_size": 64, "num_heads": heads, "head_dim": 32, "value_dim": 32, "rank": 96, "rot_dim": 0}))
        windowed = rng.random() < 0.5
        per = pages_a_block(pages, rows * part.row_blocks, ops.SMS, windowed)
        assert 0 <= per < max(pages, 1)
        if per:
            shares = -(-pages // per)
            assert 1 < shares <= 64 and rows * part.row_blocks * shares <= 2 * ops.SMS
            assert part.workspace(rows, rows) >= 4 * shares * rows * heads * (96 + 2)
        else:
            assert pages < 4 or rows * part.row_blocks * 2 > ops.SMS
    assert pages_a_block(32, 1, 148) == 1 and pages_a_block(128, 1, 148) == 2 and pages_a_block(8, 128, 148) == 0
    assert [pages_a_block(p, 2, 148, True) for p in (4, 9, 17)] == [2, 3, 3] and pages_a_block(9, 128, 148, True) == 6
