"""Entries of the Python host whose use of the arenas or kernels depends on sizes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import graft

pkg = graft.load_package()
g = pkg.gpt_lm
from test_gpu_gpt_lm import small_cfg  # noqa: E402

pytestmark = pytest.mark.gpu


def test_generation_with_a_data_slot_for_the_prompts_only():
    """1.5 KB of prompt words fit the slot, with 5 KB of generated ids they do not."""
    cfg = small_cfg(dropout_p=0.0, mlp_hidden=256)
    hp = g.init_params(cfg, seed=12, residual_scaled=False)
    prompts = np.random.default_rng(1).integers(0, cfg.vocab_size, size=(32, 4)).astype(np.int32)
    out = []
    for data_bytes in (2048, 1 << 20):
        with pkg.runtime.Context(params_bytes=64 << 20, state_bytes=64 << 20, scratch_bytes=256 << 20, data_bytes=data_bytes) as c:
            model = g.GptLm(c, cfg, hp)
            model.training = False
            out.append(g.greedy_generate_native(model, prompts, new_tokens=40, capacity=48))
    assert np.array_equal(*out)
