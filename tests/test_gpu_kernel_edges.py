"""Kernels at the sizes where their splits change: edges of tiles, remainders, the smallest and largest of a dispatch's range."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from conftest import graft
from gpu_util import BF16, F16, F32, I32, close, dev, host, rnd_np, storage_name

pkg = graft.load_package()
abi, ops, g, optim = pkg.abi, pkg.ops, pkg.gpt_lm, pkg.optim
from oracle import ops as O  # noqa: E402
from test_gpu_gpt_lm import small_cfg  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = pkg.runtime.Context(params_bytes=64 << 20, state_bytes=64 << 20, scratch_bytes=1 << 30)
    yield c
    c.destroy()


# one 64-key step, one 128-row item, one row more, an odd number of steps, sequences that begin inside a tile, rows behind the last one
@pytest.mark.parametrize("dtype,dh", [(F16, 64), (BF16, 64), (F16, 128), (BF16, 128)])
@pytest.mark.parametrize("lengths,window,behind", [([128], 0, 0), ([129], 0, 0), ([64, 64, 1], 0, 0), ([1, 191, 65, 3], 0, 5), ([320], 65, 0), ([127, 200], 1, 130),
                                                   ([400], 192, 0)])
def test_attention_tile_edges(ctx, dtype, dh, lengths, window, behind):
    r, sd, h = np.random.default_rng(3), storage_name(dtype), 2
    cu = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    nv = int(cu[-1])
    q, k, v, go = (rnd_np(r.standard_normal((nv + behind, h, dh)).astype(np.float32), dtype) for _ in range(4))
    q *= np.linspace(0.1, 4.0, nv + behind, dtype=np.float32)[:, None, None]          # row maxima that grow along the keys
    q = rnd_np(q, dtype)
    ctx.begin_step()
    qt, kt, vt, cut = dev(ctx, q, dtype), dev(ctx, k, dtype), dev(ctx, v, dtype), dev(ctx, cu, I32)
    qt.requires_grad = kt.requires_grad = vt.requires_grad = True
    out = ops.gd_sdpa_varlen(ctx, qt, kt, vt, cut, causal=True, sliding_window=window, max_seqlen=max(lengths))
    out.grad = dev(ctx, go, dtype)
    ctx.run_backward()
    t = [torch.from_numpy(a[:nv]) for a in (go, q, k, v)]
    got = host(out)
    close(got[:nv], O.sdpa_varlen_forward(t[1], t[2], t[3], cu, 0.0, True, window, 0, sd)[0], dtype, scale=2, what="forward")
    grads = [host(x.grad) for x in (qt, kt, vt)]
    for name, a, b in zip(("dq", "dk", "dv"), grads, O.sdpa_varlen_backward(*t, cu, 0.0, True, window, 0, sd)):
        close(a[:nv], b, dtype, scale=12, what=name)
    assert all(np.all(a[nv:] == 0) for a in [got] + grads)
    ctx.end_step()


# fewer ids than table rows (rows named by the ids), as many, more (whole table); ids outside it; a width of one vector
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("vocab,n,dim", [(97, 1, 8), (97, 96, 64), (97, 97, 64), (40, 333, 520)])
def test_embedding_backward_by_row_and_whole(ctx, dtype, vocab, n, dim):
    r = np.random.default_rng(5)
    ids = r.integers(0, vocab, size=n).astype(np.int32)
    if n > 8:
        ids[[2, 7]] = [-1, vocab]
    grad = rnd_np(r.standard_normal((n, dim)).astype(np.float32), dtype)
    ctx.begin_step()
    table = dev(ctx, np.zeros((vocab, dim), np.float32), dtype)
    table.requires_grad = True
    out = ops.gd_embedding(ctx, table, dev(ctx, ids, I32))
    out.grad = dev(ctx, grad, dtype)
    ctx.run_backward()
    close(host(table.grad), O.embedding_backward(torch.from_numpy(grad), torch.from_numpy(ids), vocab, storage_name(dtype)), dtype, scale=4)
    ctx.end_step()


# partial sums: one, a remainder before and behind the 16-byte loads, more than one round of the block
@pytest.mark.parametrize("blocks,skew", [(1, 0), (3, 1), (4, 3), (9, 2), (4099, 0), (9000, 1)])
def test_gradient_norm_over_many_partials(ctx, blocks, skew):
    count = blocks * optim.NORM_BLOCK - 5
    x = np.random.default_rng(blocks).standard_normal(count).astype(np.float16)
    ctx.begin_step()
    t, part, inv = dev(ctx, x, F16), ctx.zeros(ctx.scratch, F32, (blocks + 8,)), dev(ctx, np.array([0.5, 0.0, 0.0, 0.0], np.float32), F32)
    d = abi.GradNormDesc()
    d.grad_buffer, d.grad_offset, d.count, d.grad_dtype = t.buffer, t.offset, count, F16
    d.partial_buffer, d.partial_offset, d.partial_count = part.buffer, part.offset + 4 * skew, blocks
    d.grad_scale_buffer, d.grad_scale_offset = inv.buffer, inv.offset
    d.found_inf_buffer, d.found_inf_offset, d.has_found_inf = inv.buffer, inv.offset + 4, 1
    ctx.check(ctx.lib.gd_backend_grad_clip_scale(ctx.backend, C.byref(d), 1, inv.buffer, inv.offset + 8, 1.0, 1e-6), "grad_clip_scale")
    ctx.flush()
    got = inv.read()
    want = 0.5 * np.linalg.norm(x.astype(np.float64))
    assert got[1] == 0.0 and abs(got[3] - want) <= 1e-5 * want
    ctx.end_step()


# several chunks of classes formed at once: the last block of 256 threads, the first of 1024, odd remainders of a chunk, the largest
@pytest.mark.parametrize("vocab,dtype", [(4096, F16), (8192, BF16), (8200, F16), (32768, F16)])
def test_native_step_with_a_chunked_vocabulary(vocab, dtype):
    cfg = small_cfg(vocab_size=vocab, dtype=dtype)
    hp = g.init_params(cfg, seed=4)
    batch = g.synthetic_batch(cfg, n_seqs=5, min_len=4, max_len=64, seed=8, pad_to=64)
    res = []
    for kind in (g.Trainer, g.NativeTrainer):
        with pkg.runtime.Context(params_bytes=64 << 20, state_bytes=256 << 20, scratch_bytes=1 << 30) as c:
            trainer = kind(g.GptLm(c, cfg, hp), g.TrainConfig.baseline())
            loss = float(trainer.train_batch(batch).read()[()])
            if kind is g.NativeTrainer:
                grads = g.native_step_gradients(trainer)
            else:
                c.flush()
                grads = {n: p.grad.read_f32() for n, p in trainer.model.params.items()}
            res.append((loss, grads))
    assert abs(res[0][0] - res[1][0]) <= 1e-5 * res[0][0]
    for name, want in res[0][1].items():
        off = np.linalg.norm(res[1][1][name] - want) / max(np.linalg.norm(want), 1e-20)
        assert off <= (4e-3 if dtype == F16 else 2e-2), (name, off)


# one sequence, the most that one tile of rows takes, one more; a head that ends inside a unit of 16 classes (one launch per operation)
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("batch,vocab,window,prompt", [(1, 512, 0, 1), (2, 520, 0, 5), (16, 512, 24, 30), (17, 512, 0, 7)])
def test_greedy_generation_batch_edges(dtype, batch, vocab, window, prompt):
    cfg = small_cfg(dropout_p=0.0, mlp_hidden=256, vocab_size=vocab, sdpa_window=window, dtype=dtype)
    hp = g.init_params(cfg, seed=12, residual_scaled=False)
    prompts = np.random.default_rng(batch).integers(0, vocab, size=(batch, prompt)).astype(np.int32)
    with pkg.runtime.Context(params_bytes=64 << 20, state_bytes=256 << 20, scratch_bytes=1 << 30) as c:
        model = g.GptLm(c, cfg, hp)
        model.training = False
        want = g.greedy_generate(model, prompts, new_tokens=11, capacity=48)
        caches = [host(t) for t in model.k_cache + model.v_cache]
        got = g.greedy_generate_native(model, prompts, new_tokens=11, capacity=48)
        for a, b in zip(caches, model.k_cache + model.v_cache):
            close(host(b), a, dtype, scale=2)
    assert np.array_equal(got, want)


# enough tiles for one k-slice (both results written directly), with ragged edges in all three extents; one tile fewer than that takes slices
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("m,n,k", [(2560, 1024, 200), (2568, 1032, 72), (4096, 776, 1096), (1024, 1024, 2048), (1536, 512, 1501),
                                   (3000, 1000, 33), (136, 72, 65)])
def test_weight_gradient_with_column_sums(ctx, dtype, m, n, k):
    r, sd = np.random.default_rng(m + k), storage_name(dtype)
    a, b = (rnd_np(r.standard_normal(s).astype(np.float32), dtype) for s in ((k, m), (k, n)))
    ctx.begin_step()
    y, s = ctx.scratch_empty(dtype, (m, n)), ctx.scratch_empty(dtype, (m,))
    am, bm, ym, sv = dev(ctx, a, dtype).mv(k, m), dev(ctx, b, dtype).mv(k, n), y.mv(m, n), s.vv()
    ctx.check(ctx.lib.gdb200_matmul_tn_colsum(ctx.backend, C.byref(am), C.byref(bm), C.byref(ym), C.byref(sv)), "tn_colsum")
    ctx.flush()
    scale = np.sqrt(k) / 8
    close(host(y), O.rnd(torch.from_numpy(a).t() @ torch.from_numpy(b), sd), dtype, scale=scale, what="dW")
    close(host(s), O.rnd(torch.from_numpy(a).sum(dim=0), sd), dtype, scale=scale, what="db")
    ctx.end_step()


# a last wave of tiles in halves: the only wave, behind whole waves, with a half that lies behind the last column, ragged k and rows
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("m,n,k", [(2560, 512, 264), (2600, 392, 72), (19200, 264, 128), (9728, 512, 520)])
def test_contractions_with_half_tiles_in_the_last_wave(ctx, dtype, m, n, k):
    r, sd, lib = np.random.default_rng(m + n), storage_name(dtype), ctx.lib
    a, b = (rnd_np(r.standard_normal(s).astype(np.float32), dtype) for s in ((m, k), (k, n)))
    want = O.rnd(torch.from_numpy(a) @ torch.from_numpy(b), sd)
    ctx.begin_step()
    for fn, x, w in ((lib.gd_backend_matmul, a, b), (lib.gd_backend_matmul_nt, a, b.T.copy()), (lib.gd_backend_matmul_tn, a.T.copy(), b)):
        y = ctx.scratch_empty(dtype, (m, n))
        xm, wm, ym = dev(ctx, x, dtype).mv(*x.shape), dev(ctx, w, dtype).mv(*w.shape), y.mv(m, n)
        ctx.check(fn(ctx.backend, C.byref(xm), C.byref(wm), C.byref(ym)), "matmul")
        ctx.flush()
        close(host(y), want, dtype, scale=np.sqrt(k) / 8)
    ctx.end_step()


# few rows with contractions that are no multiple of the staged kernel's chunk, or of eight; a last tile of one row
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("m,n,k", [(1, 176, 312), (33, 3000, 1000), (64, 128, 136), (65, 264, 72), (129, 1000, 128)])
def test_contractions_of_few_rows(ctx, dtype, m, n, k):
    r, sd, lib = np.random.default_rng(m + n), storage_name(dtype), ctx.lib
    a, w, b = (rnd_np(r.standard_normal(s).astype(np.float32), dtype) for s in ((m, k), (n, k), (n,)))
    ta, tw = torch.from_numpy(a), torch.from_numpy(w)
    ctx.begin_step()
    y, dx, wt = ctx.scratch_empty(dtype, (m, n)), ctx.scratch_empty(dtype, (m, n)), dev(ctx, w.T.copy(), dtype)
    am, wm, ym, xm, tm, bv = dev(ctx, a, dtype).mv(m, k), dev(ctx, w, dtype).mv(n, k), y.mv(m, n), dx.mv(m, n), wt.mv(k, n), dev(ctx, b, dtype).vv()
    ctx.check(lib.gdb200_matmul_nt_bias(ctx.backend, C.byref(am), C.byref(wm), C.byref(bv), C.byref(ym)), "nt_bias")
    ctx.check(lib.gd_backend_matmul(ctx.backend, C.byref(am), C.byref(tm), C.byref(xm)), "matmul")
    ctx.flush()
    product = O.rnd(ta @ tw.t(), sd)
    close(host(dx), product, dtype, scale=np.sqrt(k) / 8)
    close(host(y), O.rnd(product + torch.from_numpy(b), sd), dtype, scale=np.sqrt(k) / 8)
    ctx.end_step()
