"""GPU: a device-side give-up reaches the host as GD_ERR_INTERNAL at flush, names its code, is cleared, and leaves the
backend usable. The failure is made without a fault: a code stored in the backend's error word in stream order, and a
one-warp kernel whose bounded wait on a barrier nobody arrives at runs out (a few thousand polls) and returns; a CTA of the
decode kernel that falls silent, so that the exchanges of its cluster run out."""
import ctypes as C
import time

import numpy as np
import pytest

from gpu_util import F16, I32, abi, dev, host, pkg

pytestmark = pytest.mark.gpu


def still_usable(ctx):
    ctx.begin_step()
    x = np.arange(64, dtype=np.float32).reshape(8, 8)
    t = dev(ctx, x, F16)
    out = ctx.scratch_empty(F16, (8, 8))
    ctx.check(ctx.lib.gd_backend_scale(ctx.backend, out.buffer, out.offset, t.buffer, t.offset, 64, F16, 2.0), "scale")
    got = host(out)
    ctx.end_step()
    return np.array_equal(got, 2 * x)


@pytest.mark.parametrize("how", ["injected", "bounded_wait"])
def test_device_give_up_surfaces_at_flush_once_and_the_backend_stays_usable(how):
    with pkg.runtime.Context(params_bytes=16 << 20, state_bytes=16 << 20, scratch_bytes=64 << 20) as ctx:
        lib, be = ctx.lib, ctx.backend
        assert lib.gd_backend_flush(be) == abi.GD_OK
        if how == "injected":
            assert lib.gdb200_inject_device_error(be, 777) == abi.GD_OK
            code = 777
        else:
            assert lib.gdb200_selftest_bounded_wait(be, 4096) == abi.GD_OK
            code = 399
        assert lib.gd_backend_flush(be) == abi.GD_ERR_INTERNAL
        assert f"code {code}".encode() in lib.gdb200_last_error(be)
        assert lib.gd_backend_flush(be) == abi.GD_OK          # reported once, then cleared
        assert still_usable(ctx)
        assert lib.gdb200_inject_device_error(be, 0) == abi.GD_ERR_INVALID_ARGUMENT
        assert lib.gdb200_selftest_bounded_wait(be, 0) == abi.GD_ERR_INVALID_ARGUMENT


class DecodeRun:
    """Prefilled state of a small model whose decode steps can be run again from where the prefill left them."""

    def __init__(self, ctx, d_model, mlp_hidden, batch, new, prompt=9):
        g = pkg.gpt_lm
        cfg = g.GptConfig.baseline()
        cfg.dropout_p, cfg.n_layers, cfg.vocab_size, cfg.d_model, cfg.n_heads, cfg.mlp_hidden = 0.0, 2, 272, d_model, d_model // 64, mlp_hidden
        self.ctx, self.new, self.batch = ctx, new, batch
        self.model = g.GptLm(ctx, cfg, g.init_params(cfg, seed=4))
        self.model.alloc_kv_cache(batch, prompt + new)
        n = batch * prompt
        self.at = np.cumsum([0, n, n, batch + 1, batch, batch, batch, batch, new * batch, 1])
        words = np.zeros(int(self.at[-1]), dtype=np.int32)
        words[:n] = np.random.default_rng(2).integers(0, cfg.vocab_size, size=n)
        words[n:2 * n].reshape(batch, prompt)[:] = np.arange(prompt)
        words[self.at[2]:self.at[3]] = np.arange(batch + 1) * prompt
        words[self.at[4]:self.at[5]] = np.arange(1, batch + 1) * prompt - 1
        words[self.at[6]:self.at[7]] = prompt - 1
        ctx.begin_step()
        self.io = ctx.from_numpy(ctx.state, I32, words)
        off = [self.io.offset + 4 * int(i) for i in self.at]
        self.state = abi.GptDecodeState()
        self.state.cache_buffer, self.state.io_buffer = ctx.state.buffer, self.io.buffer
        for i in range(cfg.n_layers):
            self.state.k_cache_offset[i], self.state.v_cache_offset[i] = self.model.k_cache[i].offset, self.model.v_cache[i].offset
        self.state.tokens_offset, self.state.positions_offset, self.state.out_tokens_offset, self.state.step_counter_offset = off[5:9]
        self.state.batch, self.state.capacity, self.state.max_steps = batch, prompt + new, new
        self.spec = g.model_spec(self.model)
        prompts = abi.GptBatch(self.io.buffer, off[0], 0, off[1], off[2], n, batch + 1)
        ctx.check(ctx.lib.gdb200_gpt_prefill(ctx.backend, C.byref(self.spec), C.byref(prompts), off[3], off[4], C.byref(self.state), None), "prefill")
        ctx.end_step()
        ctx.flush()

    def words(self):
        """tokens, positions, out_tokens [new, batch], step counter"""
        w = self.io.read()
        return [w[self.at[5]:self.at[6]], w[self.at[6]:self.at[7]], w[self.at[7]:self.at[8]].reshape(self.new, self.batch), w[self.at[8]]]

    def decode(self):
        self.ctx.begin_step()
        st = self.ctx.lib.gdb200_gpt_decode_steps(self.ctx.backend, C.byref(self.spec), C.byref(self.state), self.new - 1, 1, None)
        self.ctx.end_step()
        assert st == abi.GD_OK
        return self.ctx.lib.gd_backend_flush(self.ctx.backend)


# clusters of 16 and of four CTAs; CTAs without an attention unit (one sequence); up to eight gate units to a CTA (hidden 1024) and more;
# the CTA that records the ids; the first step and later ones; gate rows in passes (hidden 8192)
@pytest.mark.parametrize("d_model,mlp_hidden,batch,cta,step", [(512, 1024, 1, 15, 0), (512, 1024, 1, 0, 3), (512, 1536, 20, 7, 2), (512, 1536, 64, 3, 1),
                                                               (256, 512, 7, 2, 4), (128, 256, 64, 1, 2), (512, 8192, 64, 9, 2)])
def test_decode_that_gives_up_leaves_ids_and_positions_where_they_were(d_model, mlp_hidden, batch, cta, step):
    with pkg.runtime.Context(params_bytes=256 << 20, state_bytes=256 << 20, scratch_bytes=1 << 30) as ctx:
        run = DecodeRun(ctx, d_model, mlp_hidden, batch, new=8)
        before = run.words()
        assert ctx.lib.gdb200_selftest_decode_give_up(ctx.backend, cta, step, 50) == abi.GD_OK
        assert run.decode() == abi.GD_ERR_INTERNAL and b"code 398" in ctx.lib.gdb200_last_error(ctx.backend)
        failed = run.words()
        assert np.array_equal(failed[0], before[0]) and np.array_equal(failed[1], before[1]) and failed[3] == before[3] == 1
        assert run.decode() == abi.GD_OK          # once only, and from the state of before
        tokens, positions, ids, count = run.words()
        done = step if cta != 0 else max(step - 1, 0)      # (CTA 0 records the ids of a step at the start of the next one)
        assert np.array_equal(failed[2][:1 + done], ids[:1 + done]) and not failed[2][1 + done:].any()
        assert np.array_equal(tokens, ids[-1]) and np.array_equal(positions, before[1] + 7) and count == 8
        assert still_usable(ctx)
        want = pkg.gpt_lm.greedy_generate_native(run.model, run.io.read()[:batch * 9].reshape(batch, 9), 8, 17, use_graph=False)
        assert np.array_equal(ids.T, want)


def test_decode_gives_up_within_seconds():
    with pkg.runtime.Context(params_bytes=256 << 20, state_bytes=256 << 20, scratch_bytes=1 << 30) as ctx:
        run = DecodeRun(ctx, 512, 1024, 3, new=4)
        assert ctx.lib.gdb200_selftest_decode_give_up(ctx.backend, 5, 1, 0) == abi.GD_OK
        start = time.monotonic()
        assert run.decode() == abi.GD_ERR_INTERNAL and b"code 398" in ctx.lib.gdb200_last_error(ctx.backend)
        assert 1.5 < time.monotonic() - start < 10.0        # two seconds, once: no CTA waits a second time
        assert run.decode() == abi.GD_OK
