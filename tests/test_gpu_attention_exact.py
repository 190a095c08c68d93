"""Attention on the tensor path: what the order of sums, the choice of the row maximum and the rows behind the last sequence may not change."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import graft
from gpu_util import BF16, F16, I32, close, dev, host, rnd_np

pkg = graft.load_package()
ops = pkg.ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = pkg.runtime.Context(params_bytes=64 << 20, state_bytes=64 << 20, scratch_bytes=2 << 30)
    yield c
    c.destroy()


@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("dh", [64, 128])
def test_largest_probability_is_not_rounded(ctx, dtype, dh):
    """Probabilities are rounded to 16 bits relative to the row's maximum, so the largest one is exactly 1. Every 64 keys bring a record, 3.3
    above the one before in powers of two; columns of V that only the record names then come out as V / sum with the output's rounding alone
    (half a unit in the last place; 1e-5 for the FP32 sum and exponentials). Relative to an older maximum they carry a second rounding."""
    n, blocks, width = 384, 6, dh // 8
    a, v = np.zeros(n, np.float32), np.zeros((n, 1, dh), np.float32)
    records = np.arange(1, blocks) * 64 + 3
    a[records] = np.arange(1, blocks) * 3.3 / np.log2(np.e) * np.sqrt(dh) / 4.0
    rng = np.random.default_rng(dh)
    for t, r in enumerate(records, 1):
        v[r, 0, t * width:(t + 1) * width] = rng.uniform(1.0, 2.0, width)
    q, k = np.zeros((2, n, 1, dh), np.float32)
    q[:, 0, 0], k[:, 0, 0] = 4.0, a
    k, v = rnd_np(k, dtype), rnd_np(v, dtype)
    ctx.begin_step()
    out = ops.gd_sdpa_varlen(ctx, dev(ctx, q, dtype), dev(ctx, k, dtype), dev(ctx, v, dtype), dev(ctx, np.array([0, n], np.int32), I32), causal=True,
                             sliding_window=0, max_seqlen=n)
    got = host(out).astype(np.float64)
    ctx.end_step()
    s = 4.0 * k[:, 0, 0].astype(np.float64) / np.sqrt(dh)
    half_unit = 2.0 ** (-11 if dtype == F16 else -8)   # of a value just above a power of two, relative
    for t, r in enumerate(records, 1):
        cols = slice(t * width, (t + 1) * width)
        for row in range(r, (t + 1) * 64):
            want = v[r, 0, cols].astype(np.float64) / np.exp(s[:row + 1] - s[r]).sum()
            # spacing of the storage type at each value
            spacing = 2.0 ** np.floor(np.log2(want)) * 2.0 * half_unit
            assert np.all(np.abs(got[row, 0, cols] - want) <= 0.5 * spacing + 1e-5 * want), (t, row)


# behind the last sequence: inside its last tile, a whole tile and more; one key step only; a last row that begins a tile; grouped heads
@pytest.mark.parametrize("dtype,dh", [(F16, 64), (BF16, 64), (F16, 128), (BF16, 128)])
@pytest.mark.parametrize("lengths,behind,hq,hkv,window", [([150, 43], 7, 2, 2, 0), ([130, 63], 200, 4, 2, 40), ([64, 65], 63, 2, 1, 0), ([20], 120, 2, 2, 0),
                                                          ([300, 1], 19, 2, 2, 128)])
def test_rows_behind_the_last_sequence_are_not_read(ctx, dtype, dh, lengths, behind, hq, hkv, window):
    """They may hold anything (scratch memory is not cleared): with NaN and infinities there every result is that of zeros there, bit for bit
    (head_dim 64: but for dQ, whose contributions are added in no fixed order there)."""
    rng, nv = np.random.default_rng(7), sum(lengths)
    cu = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    shapes = [(nv + behind, h, dh) for h in (hq, hkv, hkv, hq)]
    clean = [rnd_np(rng.standard_normal(s).astype(np.float32), dtype) for s in shapes]
    results = []
    for fill in (0.0, np.nan, np.inf):
        arrays = [a.copy() for a in clean]
        for a in arrays:
            a[nv:] = fill
        ctx.begin_step()
        q, k, v, go = (dev(ctx, a, dtype) for a in arrays)
        q.requires_grad = k.requires_grad = v.requires_grad = True
        out = ops.gd_sdpa_varlen(ctx, q, k, v, dev(ctx, cu, I32), causal=True, sliding_window=window, max_seqlen=max(lengths))
        out.grad = go
        ctx.run_backward()
        results.append([host(t) for t in (out, k.grad, v.grad, q.grad)])
        ctx.end_step()
    for got in results[1:]:
        for name, a, b in zip(("out", "dk", "dv", "dq"), got, results[0]):
            if name == "dq" and dh == 64:
                close(a, b, dtype, what=name)
            else:
                assert np.array_equal(a, b), name


# many key tiles to a query tile, with and without a window that ends inside a tile; sequences that share tiles; grouped heads
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("lengths,hq,hkv,window", [([2048, 1999], 16, 16, 0), ([700, 1500, 900, 37], 8, 8, 1000), ([130, 260, 390] * 6, 16, 4, 200), ([64] * 40, 16, 16, 0)])
def test_backward_of_128_dimensions_repeats_bit_for_bit(ctx, dtype, lengths, hq, hkv, window):
    """Every sum has one order, whichever CTA forms it."""
    rng, n = np.random.default_rng(11), sum(lengths)
    arrays = [rnd_np(rng.standard_normal((n, h, 128)).astype(np.float32), dtype) for h in (hq, hkv, hkv, hq)]
    cu, first = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32), None
    for _ in range(5):
        ctx.begin_step()
        q, k, v, go = (dev(ctx, a, dtype) for a in arrays)
        q.requires_grad = k.requires_grad = v.requires_grad = True
        out = ops.gd_sdpa_varlen(ctx, q, k, v, dev(ctx, cu, I32), causal=True, sliding_window=window, max_seqlen=max(lengths))
        out.grad = go
        ctx.run_backward()
        grads = [t.grad.read() for t in (q, k, v)]
        ctx.end_step()
        first = first or grads
        assert all(np.array_equal(a, b) for a, b in zip(grads, first))


# Scores, probabilities and weighted sums are FP32 sums of 16-bit factors (products of the tensor cores for one new token at head_dim 64): their
# error is at most 64 x 2^-22 x sum |q k| x scale, some 1e-4 of a probability, and a third of that in the 2-norm of a result over
# dozens of keys. Beside the result's own rounding (2e-4 for 11 bits) that is 2 %; probabilities in 16 bits would be 5e-4 each. (Three, five
# and seven key ranges of a query are among the shapes, with some but not all of them to a warp.)
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("b,tq,hq,hkv,dh,tmax,window", [(1, 1, 8, 8, 64, 48, 0), (13, 1, 8, 8, 64, 122, 50), (64, 1, 8, 8, 64, 512, 0), (30, 1, 4, 4, 64, 900, 0), (64, 1, 2, 2, 64, 300, 0),
                                                        (100, 1, 12, 4, 64, 200, 0), (100, 1, 8, 8, 64, 160, 0), (200, 1, 3, 3, 64, 400, 90), (5, 1, 8, 8, 128, 200, 0), (9, 3, 8, 2, 64, 150, 0), (100, 2, 16, 16, 64, 70, 0)])
def test_decode_attention_has_the_rounding_of_its_result(ctx, dtype, b, tq, hq, hkv, dh, tmax, window):
    rng = np.random.default_rng(b * tmax)
    q, k, v = (rnd_np((rng.standard_normal(shape) * f).astype(np.float32), dtype) for shape, f in (((b, tq, hq, dh), 1.5), ((b, tmax, hkv, dh), 1.0), ((b, tmax, hkv, dh), 1.0)))
    pos = rng.integers(0, tmax - tq + 1, size=b).astype(np.int32)
    ctx.begin_step()
    got = host(ops.gd_sdpa_decode_positions(ctx, dev(ctx, q, dtype), dev(ctx, k, dtype), dev(ctx, v, dtype), dev(ctx, pos, I32), sliding_window=window)).astype(np.float64)
    ctx.end_step()
    want = np.zeros((b, tq, hq, dh))
    for i in range(b):
        for t in range(tq):
            hi = pos[i] + t + 1
            lo = max(0, hi - window) if window > 0 else 0
            for h in range(hq):
                kk, vv = (c[i, lo:hi, h // (hq // hkv)].astype(np.float64) for c in (k, v))
                s = kk @ q[i, t, h].astype(np.float64) / np.sqrt(dh)
                p = np.exp(s - s.max())
                want[i, t, h] = p @ vv / p.sum()
    rounding = np.linalg.norm(rnd_np(want.astype(np.float32), dtype) - want)
    assert np.linalg.norm(got.reshape(want.shape) - want) <= 1.02 * rounding
