"""Entries of the Python host whose use of the arenas or kernels depends on sizes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import graft

pkg = graft.load_package()
abi, g = pkg.abi, pkg.gpt_lm
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


def compare_decode_forms(monkeypatch, cfg, batch, prompt, new):
    """Ids and caches of one launch for all steps against one launch per operation. Every sum is formed alike: a difference in the last bit of
    a cache is enough to turn a greedy choice between two nearly equal logits, as those of an untrained model are."""
    hp = g.init_params(cfg, seed=12, residual_scaled=False)
    prompts = np.random.default_rng(batch).integers(0, cfg.vocab_size, size=(batch, prompt)).astype(np.int32)
    forms = []
    with pkg.runtime.Context(params_bytes=256 << 20, state_bytes=1 << 30, scratch_bytes=2 << 30) as c:
        model = g.GptLm(c, cfg, hp)
        model.training = False
        for one_launch in ("1", "0"):
            monkeypatch.setenv("GDB200_DECODE_MEGA", one_launch)
            mark, timing = c.state.top, {}
            ids = g.greedy_generate_native(model, prompts, new, prompt + new, timing=timing)
            forms.append([ids] + [t.read() for t in model.k_cache + model.v_cache])
            c.state.top = mark
            assert (timing["decode_launches"] <= 2) == (one_launch == "1")
    assert all(np.array_equal(a, b) for a, b in zip(*forms))


def other_model(dtype, d_model, mlp_hidden, vocab, layers, window):
    cfg = g.GptConfig.baseline()
    cfg.dropout_p, cfg.sdpa_window, cfg.n_layers, cfg.vocab_size, cfg.dtype = 0.0, window, layers, vocab, dtype
    cfg.d_model, cfg.n_heads, cfg.mlp_hidden, cfg.context_length = d_model, d_model // 64, mlp_hidden, 4096
    return cfg


# the benchmark model, seven clusters of 16 CTAs: one sequence to a cluster, clusters that are not full, the first batch of two to a
# cluster, of three, of five and of nine (two column tiles instead of one) and the ones before, another number of heads to an
# attention unit at 20, 34 and 64, a window, the largest batch
@pytest.mark.parametrize("dtype", [abi.F16, abi.BF16])
@pytest.mark.parametrize("batch,prompt,new,window", [(1, 16, 32, 0), (13, 77, 45, 64), (16, 40, 24, 0), (17, 40, 24, 0), (32, 30, 24, 0), (33, 100, 40, 0), (64, 200, 48, 0),
                                                     (7, 20, 6, 0), (8, 20, 6, 0), (14, 20, 6, 0), (15, 20, 6, 0), (28, 40, 6, 9), (29, 40, 6, 0), (56, 20, 6, 0), (57, 20, 6, 0)])
def test_decode_agrees_bit_for_bit(monkeypatch, dtype, batch, prompt, new, window):
    cfg = g.GptConfig.baseline()
    cfg.dropout_p, cfg.sdpa_window, cfg.dtype = 0.0, window, dtype
    compare_decode_forms(monkeypatch, cfg, batch, prompt, new)


# twice the layers: one sequence, an odd count, a window, a tied head
@pytest.mark.parametrize("dtype", [abi.F16, abi.BF16])
@pytest.mark.parametrize("batch,prompt,new,window,tied", [(1, 5, 20, 0, False), (7, 70, 20, 48, True), (33, 20, 12, 0, False), (64, 60, 16, 0, False)])
def test_decode_of_a_larger_model_agrees_bit_for_bit(monkeypatch, dtype, batch, prompt, new, window, tied):
    cfg = g.GptConfig.baseline()
    cfg.dropout_p, cfg.sdpa_window, cfg.dtype, cfg.n_layers, cfg.tied_lm_head = 0.0, window, dtype, 6, tied
    compare_decode_forms(monkeypatch, cfg, batch, prompt, new)


# clusters of four and eight CTAs; more than 16 units of a phase to a CTA (rounds), a CTA with one unit more than another, k ranges of 16 and
# 32, one 128-wide tile of the down projection; positions behind the cos / sin table (512); more than eight tiles of keys to
# a warp, and several units to a CTA
@pytest.mark.parametrize("dtype", [abi.F16, abi.BF16])
@pytest.mark.parametrize("d_model,mlp_hidden,vocab,layers,batch,prompt,new,window", [
    (128, 128, 4096, 2, 5, 6, 12, 0), (128, 2560, 272, 1, 64, 4, 9, 3), (256, 640, 272, 2, 20, 30, 20, 0), (256, 768, 4112, 1, 3, 17, 8, 5),
    (512, 1536, 2048, 1, 3, 490, 40, 0), (512, 512, 16, 1, 59, 250, 12, 200),
    (512, 512, 272, 1, 2, 3000, 9, 0), (512, 512, 272, 2, 58, 900, 5, 0), (256, 256, 272, 1, 61, 700, 5, 0), (128, 128, 272, 1, 35, 600, 5, 0)])
def test_decode_of_other_shapes_agrees_bit_for_bit(monkeypatch, dtype, d_model, mlp_hidden, vocab, layers, batch, prompt, new, window):
    cfg = other_model(dtype, d_model, mlp_hidden, vocab, layers, window)
    compare_decode_forms(monkeypatch, cfg, batch, prompt, new)


# gate rows in one pass and in several: the last hidden width of one pass and the first of several for ten, nine, eight and two sequences to a
# cluster, chunks of 512, 256 and 128, a short last pass; more places between two warps of the down projection than the ring has barriers
@pytest.mark.parametrize("dtype", [abi.F16, abi.BF16])
@pytest.mark.parametrize("d_model,mlp_hidden,batch", [
    (512, 4096, 64), (512, 4224, 64), (512, 8192, 64), (512, 8960, 64), (512, 4736, 63), (512, 4864, 63), (512, 4736, 56), (512, 4864, 56), (512, 4992, 56),
    (512, 8192, 49), (512, 8448, 45), (512, 16384, 30), (512, 16896, 1), (256, 9600, 64), (256, 9728, 64), (128, 26112, 64), (128, 26240, 64)])
def test_decode_with_gate_rows_in_passes_agrees_bit_for_bit(monkeypatch, dtype, d_model, mlp_hidden, batch):
    compare_decode_forms(monkeypatch, other_model(dtype, d_model, mlp_hidden, 272, 2, 0), batch, 5, 6)
