"""The work that users of this backend have it do, as cases that can be timed and compared.

Four kinds, each through the entry points a program calls:

* `train`: one optimizer step of a gpt_lm model, `NativeTrainer.train_batch` (host "native") or the op capsules with the tape,
  `Trainer.train_batch` (host "tape", the call sequence of the reference's own host). The batch comes from page-locked memory, the
  loss goes to page-locked memory, both in stream order with one step of run-ahead, as a training loop runs it.
* `generate`: greedy KV-cache generation, `greedy_generate_native` (packed prefill, all decode steps, ids back on the host).
* `sdpa`: qkv_split_rope + packed causal attention, forward and backward, through the op capsules.
* `linear`: forward and backward of one linear layer through the C ABI (Y = X W^T + b, dX, dW + db).

All states of a process share one `Context` (one backend, one stream, one scratch arena), as a program has one; the weights,
optimizer state and caches of a state live in arenas of its own.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

import __graft_entry__ as graft

pkg = graft.load_package()
g, abi, ops, runtime = pkg.gpt_lm, pkg.abi, pkg.ops, pkg.runtime

DTYPES = {"f16": abi.F16, "bf16": abi.BF16}
TORCH = {abi.F16: torch.float16, abi.BF16: torch.bfloat16, abi.F32: torch.float32, abi.I32: torch.int32}
SCRATCH_BYTES = 24 << 30


# ------------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest training call: the two-layer model of the smoke test, six short sequences; launches and host work are all of it
        dict(name="train tiny f16", kind="train", host="native", model="tiny", dtype="f16", seqs=6, min_len=8, max_len=64),
        # the reference's default model (tied head, window 256, dropout 0.05) on a small batch, as on one rank of many
        dict(name="train default 8 f16", kind="train", host="native", model="default", dtype="f16", seqs=8, min_len=64, max_len=512),
        # the benchmark configuration: 64 sequences, untied biased head
        dict(name="train bench 64 f16", kind="train", host="native", model="bench", dtype="f16", seqs=64, min_len=64, max_len=512),
        # a large batch of the benchmark model in bfloat16
        dict(name="train bench 200 bf16", kind="train", host="native", model="bench", dtype="bf16", seqs=200, min_len=64, max_len=512),
        # two layers of the scaled configuration (d2048, 16 heads of 128, vocabulary 32768 in chunks): the largest step
        dict(name="train wide 8 bf16", kind="train", host="native", model="wide", dtype="bf16", seqs=8, min_len=256, max_len=2048),
        # the reference's own call sequence (op capsules and tape, no fused driver) on its default model
        dict(name="train tape 64 f16", kind="train", host="tape", model="default", dtype="f16", seqs=64, min_len=64, max_len=512),
        # a single short prompt answered, as in interactive use: latency of every step
        dict(name="generate 1x16+32 f16", kind="generate", dtype="f16", window=0, batch=1, prompt=16, new=32),
        # an odd batch with a sliding window in bfloat16
        dict(name="generate 13x77+45 bf16", kind="generate", dtype="bf16", window=256, batch=13, prompt=77, new=45),
        # the benchmark's generation: 64 prompts of 256 tokens, 256 new ones each
        dict(name="generate 64x256+256 f16", kind="generate", dtype="f16", window=0, batch=64, prompt=256, new=256),
        # packed attention of the benchmark: 32768 tokens in sequences of 16 to 512
        dict(name="sdpa 8x64 f16 32768", kind="sdpa", dtype="f16", heads=8, head_dim=64, window=0, tokens=32768, min_len=16, max_len=512),
        # attention of the scaled configuration's heads: long ragged sequences, a sliding window, bfloat16
        dict(name="sdpa 16x128 bf16 8191", kind="sdpa", dtype="bf16", heads=16, head_dim=128, window=1024, tokens=8191, min_len=256, max_len=2048),
        # one projection of the model by itself: forward and backward, a few tens of microseconds
        dict(name="linear 4096x512x1536 f16", kind="linear", dtype="f16", m=4096, k=512, n=1536),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["train", "train", "generate", "sdpa", "linear"])
    dtype = rng.choice(["f16", "bf16"])
    if kind == "train":
        model = rng.choice(["tiny", "default", "default", "bench", "bench", "wide"])
        ctx = {"tiny": 64, "default": 512, "bench": 512, "wide": 2048}[model]
        most = {"tiny": 64, "default": 200, "bench": 200, "wide": 8}[model]
        return dict(kind=kind, host="tape" if model != "wide" and rng.random() < 0.2 else "native", model=model, dtype="bf16" if model == "wide" else dtype,
                    seqs=_log_uniform(rng, 2, most), min_len=rng.randint(4, ctx // 8), max_len=rng.randint(ctx // 2, ctx))
    if kind == "generate":
        prompt = _log_uniform(rng, 4, 256)
        return dict(kind=kind, dtype=dtype, window=rng.choice([0, 256]), batch=_log_uniform(rng, 1, 64), prompt=prompt, new=_log_uniform(rng, 4, 256))
    if kind == "sdpa":
        heads, head_dim = rng.choice([(8, 64), (8, 64), (2, 64), (16, 128)])
        tokens = _log_uniform(rng, 256, 32768)
        longest = rng.choice([64, 512, 2048])
        return dict(kind=kind, dtype=dtype, heads=heads, head_dim=head_dim, window=rng.choice([0, 0, 256]), tokens=tokens,
                    min_len=rng.randint(1, 16), max_len=min(longest, tokens))
    # layer widths are multiples of eight (rows of 16 bytes), the number of rows is any
    return dict(kind=kind, dtype=dtype, m=_log_uniform(rng, 1, 32768), k=8 * _log_uniform(rng, 16, 256), n=8 * _log_uniform(rng, 16, 512))


# ------------------------------------------------------------------------------------------------------------- models
def _config(case):
    dt = DTYPES[case["dtype"]]
    if case["kind"] == "generate":
        cfg = g.GptConfig.baseline()
        cfg.dropout_p, cfg.sdpa_window = 0.0, case["window"]
    elif case["model"] == "tiny":
        cfg = g.GptConfig(vocab_size=256, context_length=64, d_model=128, n_layers=2, n_heads=2, head_dim=64, mlp_hidden=256, tied_lm_head=False,
                          dropout_p=0.1, sdpa_window=0)
    elif case["model"] == "default":
        cfg = g.GptConfig.reference_default()
    elif case["model"] == "bench":
        cfg = g.GptConfig.baseline()
    else:
        cfg = g.GptConfig.scaled()
        cfg.n_layers = 2
    cfg.dtype = dt
    return cfg


def _n_matmul(cfg):
    d, f = cfg.d_model, cfg.mlp_hidden
    return cfg.n_layers * (4 * d * d + 3 * d * f) + cfg.vocab_size * d


def _n_params(cfg):
    return sum(math.prod(shape) for _, shape, _ in g.param_specs(cfg))


def _pairs(n, window):
    """Allowed (query, key) pairs of a causal sequence of n tokens."""
    return n * (n + 1) / 2 if window <= 0 or n <= window else window * (window + 1) / 2 + (n - window) * window


def _mean_pairs(lo, hi, window):
    """Mean pairs per token when lengths are uniform in [lo, hi]."""
    lens = np.unique(np.linspace(lo, hi, 33).astype(np.int64))
    return sum(_pairs(int(n), window) for n in lens) / float(lens.sum())


def work(case):
    kind = case["kind"]
    if kind == "train":
        cfg = _config(case)
        tokens = case["seqs"] * (case["min_len"] + case["max_len"]) / 2
        flops = 6.0 * _n_matmul(cfg) * tokens
        flops += 14.0 * cfg.d_model * cfg.n_layers * tokens * _mean_pairs(case["min_len"], case["max_len"], cfg.sdpa_window)
        # parameters read and written, gradients written, masters and both moments read and written; the batch and the loss
        return {"bytes": (2 + 2 + 2 + 24.0) * _n_params(cfg) + 12.0 * tokens, "flops": flops}
    if kind == "generate":
        cfg = _config(case)
        b, p, n = case["batch"], case["prompt"], case["new"]
        d, layers = cfg.d_model, cfg.n_layers
        body = _n_matmul(cfg) - cfg.vocab_size * d
        live = [min(p + t + 1, cfg.sdpa_window or 1 << 30) for t in range(n - 1)]
        flops = 2.0 * body * b * (p + n - 1) + 2.0 * cfg.vocab_size * d * b * n + 4.0 * d * layers * b * (_pairs(p, cfg.sdpa_window) + sum(live))
        # every decode step reads the weights and the live keys and values; the prompt's and the new rows are written to the caches
        return {"bytes": 2.0 * _n_matmul(cfg) * n + 4.0 * d * layers * b * (sum(live) + p + n - 1), "flops": flops}
    if kind == "sdpa":
        el = float(case["tokens"]) * case["heads"] * case["head_dim"]
        pairs = case["tokens"] * _mean_pairs(case["min_len"], case["max_len"], case["window"])
        # the fused projection and the output's gradient read, the output and the projection's gradient written
        return {"bytes": 2.0 * (3 + 1 + 1 + 3) * el, "flops": 14.0 * case["heads"] * case["head_dim"] * pairs}
    m, k, n = case["m"], case["k"], case["n"]
    return {"bytes": 2.0 * (2 * m * k + 2 * n * k + 2 * m * n + 2 * n), "flops": 6.0 * m * n * k}


def tolerance(case):
    """16-bit storage with FP32 sums. A training step passes every value through some ten roundings per layer in each direction; single
    gradient elements that nearly cancel are off by much more than the tensor is."""
    f16 = case["dtype"] == "f16"
    if case["kind"] == "train":
        return {"rel": 5e-3, "max": 0.3} if f16 else {"rel": 2e-2, "max": 0.6}
    if case["kind"] == "generate":
        return {"rel": 4e-3, "max": 0.1} if f16 else {"rel": 1.5e-2, "max": 0.3}
    return {"rel": 2e-3, "max": 0.05} if f16 else {"rel": 1e-2, "max": 0.3}


# ----------------------------------------------------------------------------------------------------------- program
_ctx = None


def _context():
    """The process's context. Its own parameter and state arenas stay almost empty: every state brings its own."""
    global _ctx
    if _ctx is None:
        _ctx = runtime.Context(params_bytes=1 << 20, state_bytes=1 << 20, scratch_bytes=SCRATCH_BYTES, data_bytes=64 << 20)
    return _ctx


class _Arenas:
    """The two arenas of a state, given back when neither the state nor a view of their memory is left."""

    def __init__(self, params_bytes, state_bytes):
        self.params, self.state = runtime.Arena(_context(), "params", params_bytes), runtime.Arena(_context(), "state", state_bytes)

    def __del__(self):
        for name in ("params", "state"):
            if hasattr(self, name):
                getattr(self, name).destroy()


class _Span:
    """A range of the backend's memory for torch."""

    def __init__(self, owner, pointer, nbytes):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (nbytes // 2,), "typestr": "<i2", "data": (int(pointer), False), "version": 3}


class _State:
    """What a program has in hand before the call."""

    def __init__(self, case, params_bytes, state_bytes):
        self.case, self.ctx = case, _context()
        self.arenas = _Arenas(params_bytes, state_bytes)
        self.where, self.views = None, None
        self.enter()
        for arena in (self.arenas.params, self.arenas.state):
            self.view(arena.buffer, 0, arena.capacity // 4, abi.F32).zero_()
        torch.cuda.synchronize()   # torch's stream and the backend's are not ordered

    def enter(self):
        self.ctx.params, self.ctx.state = self.arenas.params, self.arenas.state

    def view(self, buffer, offset, count, dtype, shape=None):
        pointer = self.ctx.lib.gdb200_buffer_device_ptr(buffer, offset)
        out = torch.as_tensor(_Span(self.arenas, pointer, count * abi.DTYPE_SIZE[dtype]), device="cuda").view(TORCH[dtype])
        return out if shape is None else out.view(shape)

    def of(self, t):
        return self.view(t.buffer, t.offset, t.count, t.dtype, t.shape)

    def outputs(self, tensors, more=()):
        """Torch's views of the outputs; made anew only when these lie elsewhere than in the pass before."""
        where = [t.offset for t in tensors]
        if where != self.where:
            self.where, self.views = where, [self.of(t) for t in tensors] + [self.view(*m) for m in more]
        return self.views


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _normal(gen, shape, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * std


def _tensor(state, arena, dtype, shape, values=None):
    t = state.ctx.empty(arena, dtype, shape)
    if values is not None:
        state.of(t).copy_(values)
    return t


def _model(state, cfg, seed, trained):
    """A model whose weights are drawn on the GPU: initial weights, or weights with a trained model's peaked predictions (each token has
    a likely successor), so that greedy ids do not hang on the last bit of two nearly equal logits."""
    storage = np.uint16 if cfg.dtype == abi.BF16 else np.float16
    model = g.GptLm(state.ctx, cfg, {name: np.zeros(shape, dtype=storage) for name, shape, _ in g.param_specs(cfg)})
    gen = _generator(seed)
    for name, shape, kind in g.param_specs(cfg):
        if kind == "ones":
            w = torch.ones(shape, device="cuda") + (_normal(gen, shape, 0.1) if trained else 0.0)
        elif kind == "zeros":
            w = _normal(gen, shape, 0.02) if trained else torch.zeros(shape, device="cuda")
        else:
            w = _normal(gen, shape, 0.02 / math.sqrt(2.0 * cfg.n_layers) if kind == "residual" else 0.02)
        if trained and name == "token_embedding":
            w = embedding = w * 10.0
        if trained and name == "lm_head.weight":
            w[torch.randperm(shape[0], generator=gen, device="cuda")] = embedding * 0.1
        state.of(model.params[name]).copy_(w)
    torch.cuda.synchronize()
    return model


# ------------------------------------------------------------------------------------------------------------- train
def _prepare_train(case, seed):
    cfg = _config(case)
    n = _n_params(cfg)
    state = _State(case, 2 * n + (1 << 20), 12 * n + n // 64 + (2 << 20))
    ctx = state.ctx
    model = _model(state, cfg, seed, trained=False)
    config = g.TrainConfig() if case["model"] == "default" else g.TrainConfig.baseline()
    state.trainer = (g.NativeTrainer if case["host"] == "native" else g.Trainer)(model, config)
    batch = g.synthetic_batch(cfg, case["seqs"], case["min_len"], case["max_len"], seed=int(seed) & 0x7FFFFFFF, pad_to=cfg.context_length)
    for field in ("input_ids", "targets", "positions", "cu_seqlens"):
        setattr(batch, field, ctx.pinned_copy(getattr(batch, field)))
    state.batch, state.loss = batch, [ctx.pinned_copy(np.zeros(1, dtype=np.float32)) for _ in range(2)]
    # what a step updates: the parameters, then masters and both moments (ranges of their arenas that hold nothing else)
    opt, arenas = state.trainer.optimizer, state.arenas
    first = opt.slots[0].master.offset
    state.updated = [(arenas.params.buffer, 0, arenas.params.top // 2, cfg.dtype),
                     (arenas.state.buffer, first, (opt.state_f32.offset - first) // 4, abi.F32)]
    return state


def _run_train(state):
    ctx, trainer = state.ctx, state.trainer
    state.enter()
    ctx.run_ahead = 1
    loss = trainer.train_batch(state.batch, loss_out=state.loss[trainer.global_step & 1])
    slots = trainer.optimizer.slots
    if state.case["host"] == "native":
        offsets = (C.c_size_t * len(slots))()
        ctx.lib.gdb200_gpt_train_step_grad_offsets(ctx.backend, offsets, len(slots))
        grads = [runtime.Tensor(ctx, ctx.scratch, off, s.param.dtype, s.param.shape) for off, s in zip(offsets, slots)]
    else:
        grads = [s.param.grad for s in slots]
    return state.outputs([loss] + grads, state.updated)


# ---------------------------------------------------------------------------------------------------------- generate
def _prepare_generate(case, seed):
    cfg = _config(case)
    capacity = case["prompt"] + case["new"]
    cache = 2 * cfg.n_layers * case["batch"] * capacity * cfg.d_model * 2
    state = _State(case, 2 * _n_params(cfg) + (1 << 20), cache + (2 << 20))
    state.capacity = capacity
    state.model = _model(state, cfg, seed, trained=True)
    state.model.training = False
    state.prompts = np.random.default_rng(int(seed)).integers(0, cfg.vocab_size, size=(case["batch"], case["prompt"])).astype(np.int32)
    return state


def _run_generate(state):
    ctx, model = state.ctx, state.model
    state.enter()
    ctx.run_ahead = 0
    mark = ctx.state.top
    ids = g.greedy_generate_native(model, state.prompts, state.case["new"], state.capacity)
    ctx.state.top = mark   # the caches of this call may be overwritten by the next one
    return [ids] + state.outputs(model.k_cache + model.v_cache)


# -------------------------------------------------------------------------------------------------------- operations
def _lengths(case, seed):
    """Sequence lengths uniform in [min_len, max_len] that add up to the tokens."""
    rng, lens = np.random.default_rng(int(seed)), []
    while sum(lens) < case["tokens"]:
        lens.append(int(rng.integers(case["min_len"], case["max_len"] + 1)))
    lens[-1] -= sum(lens) - case["tokens"]
    return lens


def _prepare_sdpa(case, seed):
    t, h, d = case["tokens"], case["heads"], case["head_dim"]
    state = _State(case, 8 * t * h * d + (1 << 20), 8 * t + (1 << 20))
    dt, gen, lens = DTYPES[case["dtype"]], _generator(seed), _lengths(case, seed)
    state.qkv = _tensor(state, state.arenas.params, dt, (t, 3 * h * d), _normal(gen, (t, 3 * h * d)))
    state.go = _tensor(state, state.arenas.params, dt, (t, h, d), _normal(gen, (t, h, d)))
    state.cu = _tensor(state, state.arenas.state, abi.I32, (len(lens) + 1,), torch.tensor([0] + list(np.cumsum(lens))))
    state.pos = _tensor(state, state.arenas.state, abi.I32, (t,), torch.from_numpy(np.concatenate([np.arange(n) for n in lens])))
    state.qkv.requires_grad = True
    torch.cuda.synchronize()
    return state


def _run_sdpa(state):
    case, ctx = state.case, state.ctx
    state.enter()
    ctx.run_ahead = 1
    ctx.begin_step()
    state.qkv.grad = None
    q, k, v = ops.gd_qkv_split_rope(ctx, state.qkv, state.pos, case["heads"], case["head_dim"])
    out = ops.gd_sdpa_varlen(ctx, q, k, v, state.cu, causal=True, sliding_window=case["window"], max_seqlen=case["max_len"])
    out.grad = state.go
    ctx.run_backward()
    ctx.end_step()
    return state.outputs([out, state.qkv.grad])


def _prepare_linear(case, seed):
    m, k, n = case["m"], case["k"], case["n"]
    state = _State(case, 4 * (m * k + n * k + m * n + n) + (1 << 20), 1 << 20)
    arena, dt, gen = state.arenas.params, DTYPES[case["dtype"]], _generator(seed)
    x, dy = (_tensor(state, arena, dt, s, _normal(gen, s)) for s in ((m, k), (m, n)))
    w, b = _tensor(state, arena, dt, (n, k), _normal(gen, (n, k), 0.02)), _tensor(state, arena, dt, (n,), _normal(gen, (n,), 0.02))
    y, dx, dw, db = state.results = [_tensor(state, arena, dt, s) for s in ((m, n), (m, k), (n, k), (n,))]
    state.args = [C.byref(v) for v in (x.mv(m, k), w.mv(n, k), b.vv(), y.mv(m, n), dy.mv(m, n), dx.mv(m, k), dw.mv(n, k), db.vv())]
    torch.cuda.synchronize()
    return state


def _run_linear(state):
    x, w, b, y, dy, dx, dw, db = state.args
    ctx, lib = state.ctx, state.ctx.lib
    ctx.check(lib.gdb200_matmul_nt_bias(ctx.backend, x, w, b, y), "y")
    ctx.check(lib.gd_backend_matmul(ctx.backend, dy, w, dx), "dx")
    ctx.check(lib.gdb200_matmul_tn_colsum(ctx.backend, dy, x, dw, db), "dw + db")
    return state.outputs(state.results)


_KINDS = {"train": (_prepare_train, _run_train), "generate": (_prepare_generate, _run_generate), "sdpa": (_prepare_sdpa, _run_sdpa),
          "linear": (_prepare_linear, _run_linear)}


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return _KINDS[state.case["kind"]][1](state)
