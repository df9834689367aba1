"""Prompt steps whose layers are launched from native code (engine/prompt_layers.py) against the same steps launched part
by part: the same kernels with the same arguments, so the same bits and as many launches."""

import numpy as np
import pytest

import tiny_configs as C
from gpu_utils import engine_for, make_model, random_tokens
from test_parts_gpu import engine_from_spec, spec_with

pytestmark = pytest.mark.gpu


def engine(d, cfg, window, **kw):
    if not window:
        return engine_for(d, "bfloat16", kv_cache_tokens=1536, **kw)
    return engine_from_spec(d, cfg, spec_with(cfg, window=window), "bfloat16", kv_cache_tokens=1536, **kw)


@pytest.mark.parametrize("name,window", [("tiny_a", 0), ("tiny_b", 0), ("tiny_c", 0), ("tiny_a", 40)])
def test_the_same_bits_as_part_by_part(name, window, tmp_path, monkeypatch):
    from redline_b200.engine.prompt_layers import PromptLayers
    from redline_b200.ops import kernels
    cfg = C.ALL[name]
    d, _ = make_model(tmp_path, cfg, seed=90)
    vocab = cfg["vocab_size"]
    seqs = {i: random_tokens(vocab, 420, 30 + i) for i in range(3)}
    # (request, tokens) of every step: the sizes on both sides of the products' borders (17, 64, 65, 127, 128 rows),
    # alone, beside single tokens, and on a cached past
    steps = [[(0, 17)], [(0, 1), (1, 63)], [(0, 1), (1, 64)], [(0, 2), (1, 1), (2, 61)], [(0, 100), (1, 26), (2, 1)],
             [(0, 1), (1, 127)], [(0, 130), (2, 70)], [(0, 16)], [(1, 1), (2, 20)]]
    outs, launches = {}, {}
    for mode in ("1", "0"):
        monkeypatch.setenv("REDLINE_PROMPT_LAYERS", mode)
        eng = engine(d, cfg, window)
        at, outs[mode], launches[mode] = {0: 0, 1: 0, 2: 0}, [], []
        for step in steps:
            entries = []
            for i, n in step:
                entries.append((i, seqs[i][at[i]:at[i] + n], [n - 1]))
                at[i] += n
            before = kernels.LAUNCHES
            outs[mode].append(eng.step_tokens(entries).cpu().numpy())
            launches[mode].append(kernels.LAUNCHES - before)
        plan = eng.runner.model._prompt_layers
        assert isinstance(plan, PromptLayers) if mode == "1" else plan is False
        eng.runner.check_status()
    assert launches["1"] == launches["0"]
    for a, b in zip(outs["1"], outs["0"]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("window", [0, 40])
def test_full_portions_as_a_graph(window, tmp_path, monkeypatch):
    """Full portions of a prompt are captured once and replayed for the next ones; the rest of the prompt runs eagerly."""
    from redline_b200.engine.prompt_layers import PromptLayers
    cfg = C.ALL["tiny_a"]
    d, _ = make_model(tmp_path, cfg, seed=92)
    tokens = random_tokens(cfg["vocab_size"], 128 * 3 + 70, 33)
    outs = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("REDLINE_PROMPT_LAYERS", mode)
        eng = engine(d, cfg, window, cuda_graphs=True, max_num_batched_tokens=128)
        outs[mode] = [eng.step_tokens([("a", tokens[i:i + 128], [min(128, len(tokens) - i) - 1])], graphs=True).cpu().numpy()
                      for i in range(0, len(tokens), 128)]
        assert eng.runner.num_graph_steps == 3 and eng.runner.num_eager_steps == 1 and len(eng.runner._graphs) == 1
        plan = eng.runner.model._prompt_layers
        assert isinstance(plan, PromptLayers) if mode == "1" else plan is False
        eng.runner.check_status()
    for a, b in zip(outs["1"], outs["0"]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("what", ["weights", "moved", "part", "caches", "builder", "forward", "_attend"])
def test_a_model_changed_between_steps(what, tmp_path, monkeypatch):
    """The plan is of the model as it is at the step: after the change, the same bits as part by part."""
    import torch
    from redline_b200.cache.storage import CacheStorage
    from redline_b200.engine.batch import BatchBuilder
    from redline_b200.engine.prompt_layers import PromptLayers
    from redline_b200.weights.safetensors_io import CheckpointReader
    cfg = C.ALL["tiny_a"]
    d, _ = make_model(tmp_path / "a", cfg, seed=90)
    d2, _ = make_model(tmp_path / "b", cfg, seed=91)
    tokens = [random_tokens(cfg["vocab_size"], 200, 60 + i) for i in range(2)]
    outs, calls, kept = {}, {"1": 0, "0": 0}, []
    for mode in ("1", "0"):
        monkeypatch.setenv("REDLINE_PROMPT_LAYERS", mode)
        eng = engine_for(d, "bfloat16", kv_cache_tokens=1536)
        run, model = eng.runner, eng.runner.model
        eng.step_tokens([("a", tokens[0], [199])])
        first = model._prompt_layers
        if what == "weights":
            model.load_weights(CheckpointReader(d2))
        elif what == "moved":
            w = model.blocks[1].ffn.w_down
            kept.append(w.detach())
            w.data = -w.data
        elif what == "part":
            model.blocks[0], model.blocks[1] = model.blocks[1], model.blocks[0]
        elif what == "caches":
            run.storage = CacheStorage(run.groups, [run.storage.of_owner(0, True).k.shape[0]], run.cfg.block_size, run.dtype, run.device)
            run._caches = [run.storage.of_owner(i, True) for i in range(cfg["num_hidden_layers"])]
        elif what == "builder":
            b, c = run.builder, run.cfg
            run.builder = BatchBuilder(run.cache, c.max_num_batched_tokens, c.max_num_seqs, run.max_rows, c.max_seq_len, run.device,
                                       b.tile_rows, b.partition)
            assert run.builder.status.data_ptr() != b.status.data_ptr()
        else:
            part = model.blocks[1] if what == "forward" else model.blocks[1].mixer
            inner = getattr(part, what)

            def wrapped(*args, mode=mode, inner=inner):
                calls[mode] += 1
                return inner(*args)
            setattr(part, what, wrapped)
        # a prompt in two portions of both kinds, then a token that reads what they left in the cache
        outs[mode] = [eng.step_tokens([("b", part, [len(part) - 1])]).cpu().numpy()
                      for part in (tokens[1][:150], tokens[1][150:199], tokens[1][199:])]
        run.check_status()
        assert isinstance(first, PromptLayers) if mode == "1" else first is False
        if what == "builder" and mode == "1":            # (the word in which the step's kernels report belongs to the builder)
            assert model._prompt_layers is not first
        torch.cuda.synchronize()
    for a, b in zip(outs["1"], outs["0"]):
        assert np.array_equal(a, b)
    assert calls["1"] == calls["0"] == (3 if what in ("forward", "_attend") else 0)


def test_no_workspace_for_single_tokens_before_there_are_some(tmp_path):
    """The partial results of decode attention, which grow with sequences and their length, are not asked for by prompts."""
    import torch
    cfg = C.ALL["tiny_a"]
    d, _ = make_model(tmp_path, cfg, seed=93)
    eng = engine(d, cfg, 0)
    held = eng.runner.rt.workspace._bufs
    for steps in ([("a", [5] * 150, [149])], [("a", [6] * 40, [39]), ("b", [7] * 20, [19])]):
        eng.step_tokens(steps)
        assert ("attn.part_o", torch.float32) not in held and ("attn.part_ml", torch.float32) not in held
    eng.step_tokens([("a", [8], [0]), ("b", [9] * 30, [29])])
    assert ("attn.part_o", torch.float32) in held and ("attn.part_ml", torch.float32) in held
    eng.runner.check_status()
