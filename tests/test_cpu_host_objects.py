"""CPU: descriptors that the Python host lays out once or copies follow the objects they describe."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from conftest import graft

pkg = graft.load_package()
abi, g, optim, runtime = pkg.abi, pkg.gpt_lm, pkg.optim, pkg.runtime


def host_context():
    """A context's arenas without device memory behind them."""
    def arena(address):
        a = runtime.Arena.__new__(runtime.Arena)
        a.buffer, a.capacity, a.top, a.high_water, a._views = address, 1 << 30, 0, 0, {}
        return a
    ctx = SimpleNamespace(backend=None, params=arena(0x1000), state=arena(0x2000), scratch=arena(0x3000))
    ctx.empty = lambda arena, dtype, shape, name="": runtime.Context.empty(ctx, arena, dtype, shape, name)
    return ctx


def test_model_description_follows_the_parameters():
    model = g.GptLm.__new__(g.GptLm)
    model.cfg, model.ctx = g.GptConfig.baseline(), host_context()
    model.params = {n: model.ctx.empty(model.ctx.params, abi.F16, shape, n) for n, shape, _ in g.param_specs(model.cfg)}
    names, first = list(model.params), g.model_spec(model)
    assert list(first.param_offset[:len(names)]) == [model.params[n].offset for n in names]
    # one weight loaded into a new place: what is described next is that place, and what was handed out before stays as it was
    moved = "blocks.1.up_gate.weight"
    old = model.params[moved]
    model.params[moved] = model.ctx.empty(model.ctx.params, abi.F16, old.shape, moved)
    second = g.model_spec(model)
    assert second.param_offset[names.index(moved)] == model.params[moved].offset != old.offset
    assert first.param_offset[names.index(moved)] == old.offset
    second.scratch_bytes = 1
    assert g.model_spec(model).scratch_bytes == model.ctx.scratch.capacity


@pytest.mark.parametrize("offset,shape", [(np.int64(512), (np.int64(3), np.int32(4))), (512, [3, 4]), (np.uint32(512), np.array([3, 4])), (512, (3.0, 4))])
def test_tensor_of_any_whole_numbers(offset, shape):
    ctx = host_context()
    t = runtime.Tensor(ctx, ctx.params, offset, abi.F16, shape)
    assert t.shape == (3, 4) and all(type(v) is int for v in (t.offset, t.count, t.nbytes) + t.shape)
    v = t.tv()
    assert (v.offset, v.count, v.rank, list(v.shape[:2]), list(v.strides[:2])) == (512, 12, 2, [3, 4], [4, 1])
    assert ctx.empty(ctx.params, abi.F16, shape).shape == (3, 4)


def test_optimizer_descriptors_follow_replaced_state():
    ctx, seen = host_context(), []
    ctx.check = lambda st, what: None
    ctx.lib = SimpleNamespace(gd_backend_grad_clip_scale=lambda *a: seen.append([("clip", a[4])]),
                              gd_backend_adamw_batch=lambda be, d, n: seen[-1].extend((x.grad_scale_offset, x.beta1_power_offset, x.param_step_offset, x.m_offset)
                                                                                      for x in d[:n]))
    place = lambda count, dtype=abi.F32: ctx.empty(ctx.state, dtype, (count,))
    opt = optim.AdamW.__new__(optim.AdamW)
    opt.ctx, opt.config, opt.n = ctx, optim.AdamwConfig(1e-3, 0.9, 0.95, 1e-8, 0.0, True), 2
    opt.slots = [optim.ParamSlot(ctx.empty(ctx.params, abi.F16, (8,)), 0.0, 1.0, place(8), place(8), place(8)) for _ in range(2)]
    opt.state_f32, opt.state_i32, opt.partials, opt.grad_clip_scale = place(10), place(3, abi.I32), place(2), place(2)
    opt._norm_descs, opt._adamw_descs, opt._laid_out = (abi.GradNormDesc * 2)(), (abi.AdamwDesc * 2)(), [None] * 2
    scaler = SimpleNamespace(begin_step=lambda: None, finish_step=lambda: None, scale_state=place(2), flag_state=place(3, abi.I32))

    def step():
        for s in opt.slots:
            s.param.grad = ctx.empty(ctx.scratch, abi.F16, (8,))
        opt.step_amp_clip_lr(scaler, 1e-3, 1.0)
        return seen[-1][1:]

    want = lambda: [(opt.grad_clip_scale.offset, opt._f32_off(0, i), opt.state_i32.offset + 4 * i, opt.slots[i].m.offset) for i in range(2)]
    assert step() == want() == step()
    for replace in (lambda: setattr(opt, "state_f32", place(10)), lambda: setattr(opt, "state_i32", place(3, abi.I32)),
                    lambda: setattr(opt, "grad_clip_scale", place(2)), lambda: setattr(opt.slots[1], "m", place(8))):
        replace()
        assert step() == want()


def test_data_slot_takes_what_it_was_asked_for_beside_a_running_step():
    """Batches copied beside the running step alternate between two places; what a step adds to its batch has the asked-for size in both."""
    def no_device(be, size, out):
        out._obj.value = 0x9000
        return abi.GD_OK
    copies = []
    lib = SimpleNamespace(gd_backend_buffer_create=no_device, gdb200_upload_beside=lambda be, buf, n, offs, src, sizes: copies.append((offs[0], offs[n - 1] + sizes[n - 1])) or 0)
    ctx = runtime.Context.__new__(runtime.Context)
    ctx.lib, ctx.backend, ctx.run_ahead, ctx.tape, ctx.in_step = lib, 1, 1, [], False
    ctx.check, ctx.wait_steps = (lambda st, what: None), (lambda n: None)
    lib.gd_backend_scope_begin = lambda be: 0
    ctx.scratch = host_context().scratch
    ctx._make_data_slot(10000)
    batch = [np.zeros(n, dtype=np.int32) for n in (1100, 1100, 60)]
    for step in range(4):
        ctx.begin_step()
        ts = ctx.upload_beside(batch)
        assert ts is not None and copies[-1] == (ts[0].offset, ts[-1].offset + ts[-1].nbytes)
        assert step == 0 or copies[-1][0] >= copies[-2][1] or copies[-2][0] >= copies[-1][1]
        ctx.empty(ctx.data, abi.I32, (130,))    # 9992 bytes in use with it
        ctx.in_step = False
