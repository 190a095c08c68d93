"""Parameter gradients of the native step driver against those of the op capsules, where the driver's schedule changes: with and without
the one-pass cross entropy, with and without the second stream, tied and untied head, small workspaces."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, graft
from gpu_util import BF16, F16

pkg = graft.load_package()
g = pkg.gpt_lm
from test_gpu_gpt_lm import small_cfg  # noqa: E402

pytestmark = pytest.mark.gpu


def step_gradients(kind, cfg, hp, batch, scratch=1 << 30, used=None):
    """Loss and gradients of one step in a context of its own."""
    with pkg.runtime.Context(params_bytes=64 << 20, state_bytes=256 << 20, scratch_bytes=scratch) as c:
        trainer = kind(g.GptLm(c, cfg, hp), g.TrainConfig.baseline())
        loss = float(trainer.train_batch(batch).read()[()])
        if used is not None:
            used.append(c.scratch.high_water)
        if kind is g.NativeTrainer:
            return loss, g.native_step_gradients(trainer)
        c.flush()
        return loss, {n: p.grad.read_f32() for n, p in trainer.model.params.items()}


def problem(n_seqs=5, max_len=64, **kw):
    cfg = small_cfg(**kw)
    return cfg, g.init_params(cfg, seed=4), g.synthetic_batch(cfg, n_seqs=n_seqs, min_len=4, max_len=max_len, seed=8, pad_to=64)


def agree(got, want, dtype, only=None):
    """The two hosts issue the same contractions; statistics that one forms in another order move single results by a rounding of the storage
    type (2^-11, 2^-8), which some ten operations per layer pass on: at most eight and five times that over a whole tensor. (Logits taken
    for their gradients put a tensor off by its own size and more.)"""
    assert abs(got[0] - want[0]) <= 1e-5 * want[0]
    for name in only or want[1]:
        off = np.linalg.norm(got[1][name] - want[1][name]) / max(np.linalg.norm(want[1][name]), 1e-20)
        assert off <= (4e-3 if dtype == F16 else 2e-2), (name, off)


def check(dtype=F16, **kw):
    p = problem(dtype=dtype, **kw)
    native = step_gradients(g.NativeTrainer, *p)
    agree(native, step_gradients(g.Trainer, *p), dtype)
    again = step_gradients(g.NativeTrainer, *p)
    head = [n for n in native[1] if n.startswith("lm_head")]
    assert native[0] == again[0] and head and all(np.array_equal(native[1][n], again[1][n]) for n in head)


# 324, 1001: no multiple of eight, the one-pass kernel declines; 328, 2040: it takes them
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("vocab,tied,dropout", [(324, False, 0.1), (324, True, 0.1), (324, False, 0.0), (1001, False, 0.1), (328, True, 0.1), (2040, False, 0.1),
                                                (328, False, 0.0)])
def test_gradients_match_the_op_capsules(vocab, tied, dropout, dtype):
    check(dtype, vocab_size=vocab, tied_lm_head=tied, dropout_p=dropout)


def test_gradients_with_one_chunk_of_more_classes_than_the_one_pass_kernel_takes(monkeypatch):
    monkeypatch.setenv("GD_LM_CE_CHUNK_SIZE", "32776")
    check(vocab_size=32776)


@pytest.mark.parametrize("tied", [False, True])
def test_gradients_without_the_one_pass_kernel(tied):
    """GDB200_LMCE_FUSED is read once per process."""
    code = f"import sys; sys.path.insert(0, 'tests'); import test_gpu_native_gradients as t; t.check(vocab_size=328, tied_lm_head={tied})"
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, GDB200_LMCE_FUSED="0"), check=True, timeout=300)


def test_gradients_with_scratch_too_small_for_the_second_stream():
    """The driver asks for more room than the step with two streams then uses: given just that, it keeps to one stream."""
    p = problem(vocab_size=328)
    used = []
    wide = step_gradients(g.NativeTrainer, *p, used=used)
    narrow = step_gradients(g.NativeTrainer, *p, scratch=used[0], used=used)
    assert used[1] < used[0]      # scratch is reused from block to block
    agree(narrow, wide, F16)


@pytest.mark.parametrize("mib,n_seqs", [(1, 64), (1, 192), (2, 64)])
def test_gradients_with_a_small_workspace(monkeypatch, mib, n_seqs):
    """Two streams share the workspace by halves. 64 sequences (2 k tokens of 16 heads): 0.26 MiB of attention statistics fit a half of either
    workspace; 192: 0.81 MiB fit one MiB but not its half, and the step keeps to one stream. Column sums and partial sums get
    half a MiB (256 MiB by default): other slices, FP32 rounding only."""
    p = problem(vocab_size=2040, d_model=1024, n_heads=16, mlp_hidden=512, n_seqs=n_seqs)
    want = step_gradients(g.NativeTrainer, *p, scratch=3 << 30)
    monkeypatch.setenv("GD_CUDA_WORKSPACE_MB", str(mib))
    agree(step_gradients(g.NativeTrainer, *p, scratch=3 << 30), want, F16)


def test_profiled_step_keeps_to_one_stream():
    """A pair of events around a contraction must not hold the work of another stream. With one stream scratch is reused from block to block."""
    cfg, hp, batch = problem(vocab_size=328)
    with pkg.runtime.Context(params_bytes=64 << 20, state_bytes=256 << 20, scratch_bytes=1 << 30) as c:
        trainer, used = g.NativeTrainer(g.GptLm(c, cfg, hp), g.TrainConfig.baseline()), []
        for enabled in (0, 1, 0):
            c.lib.gdb200_gemm_profile_enable(c.backend, enabled)
            trainer.train_batch(batch)
            used.append(c.scratch.top)
        c.flush()
    assert used[1] < used[0] == used[2]
