"""CPU: descriptors that the Python host lays out once or copies follow the objects they describe."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from conftest import graft

pkg = graft.load_package()
abi, g, runtime = pkg.abi, pkg.gpt_lm, pkg.runtime


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
