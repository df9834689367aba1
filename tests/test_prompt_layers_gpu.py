"""Prompt steps whose layers are launched from native code (engine/prompt_layers.py) against the same steps launched part
by part: the same kernels with the same arguments, so the same bits and as many launches."""

import numpy as np
import pytest

import tiny_configs as C
from gpu_utils import engine_for, make_model, random_tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny_a", "tiny_b"])
def test_the_same_bits_as_part_by_part(name, tmp_path, monkeypatch):
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
        eng = engine_for(d, "bfloat16", kv_cache_tokens=1536)
        at, outs[mode], launches[mode] = {0: 0, 1: 0, 2: 0}, [], []
        for step in steps:
            entries = []
            for i, n in step:
                entries.append((i, seqs[i][at[i]:at[i] + n], [n - 1]))
                at[i] += n
            before = kernels.LAUNCHES
            outs[mode].append(eng.step_tokens(entries).cpu().numpy())
            launches[mode].append(kernels.LAUNCHES - before)
        assert (eng.runner.model._prompt_layers is False) == (mode == "0")
        eng.runner.check_status()
    assert launches["1"] == launches["0"]
    for a, b in zip(outs["1"], outs["0"]):
        assert np.array_equal(a, b)
