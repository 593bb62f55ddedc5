"""The batched tcgen05 path (three or more sequences) against the fp64 oracle: edges of its 32-row tiles,
128- and 256-row groups, 4 / 8 / 16 / 32-sequence forms, row groups cut over several CTAs, several passes."""
import numpy as np
import pytest

from lutmac_b200 import _lib, api, synth
from lutmac_b200.blocks import BINARY, INT2, INT3, INT4, INT5, INT6, INT8, TERNARY, blocks_per_row
from lutmac_b200.model import Model
from oracle.oracle import OracleModel
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# (M, K, batch): one row; one row over a tile and a group; ragged K; every accumulator form; split row groups; two passes
SHAPES = [(1, 256, 3), (33, 300, 4), (129, 700, 5), (257, 4, 9), (300, 2300, 16), (64, 2560, 17), (512, 1024, 31), (40, 512, 33)]
# fixed-point activations (2^-31 of a block's largest) and fp32 sums over at most 10 blocks: a few 2^-24
TOL = 1e-6


@pytest.mark.parametrize("kind", (TERNARY, BINARY, INT2, INT3, INT4, INT5, INT6, INT8))
def test_batched_linear_vs_fp64(ctx, oracle, kind):
    rng = np.random.default_rng(900 + kind)
    for M, K, batch in SHAPES:
        t = synth.tensor(rng, kind, M, K)
        kp = blocks_per_row(K) * 256
        x = np.stack([synth.activations(rng, kp) for _ in range(batch)])
        w, dx, dy = ctx.upload(t), ctx.to_device(x), ctx.malloc(batch * M * 4)
        for _ in range(2):  # twice: the arrival counters must be back at zero
            dy.zero()
            ctx.linear(w, dx, dy, batch=batch, flags=0, x_len=kp, x_stride=kp)
            y = dy.download(np.float32).reshape(batch, M)
            for q in {0, 1, batch // 2, batch - 1}:
                want = oracle.gemv_f64(kind, t.blocks, x[q], M, K)
                err = np.linalg.norm(y[q] - want)
                assert err < TOL * np.linalg.norm(np.abs(want) + 1e-3 * np.linalg.norm(x[q])), (M, K, batch, q, err)
        w.free()


@pytest.mark.parametrize("M", (64, 128, 512))
@pytest.mark.parametrize("kind", (TERNARY, INT4, INT8))
def test_batched_error_of_few_rows_and_a_long_row(ctx, oracle, kind, M):
    """112 blocks per row in 56 parts, twice what the planner takes: the fp32 error against 64 bits is that of the same
    sequences one at a time, whose sums are short slices (both are sums of M x 8 independent errors, whose norms agree
    within a few percent when the orders are equally good; one serial chain of 56 parts is 1.3 to 1.5 times off)."""
    rng = np.random.default_rng(40 + kind)
    K, batch = 28672, 8
    t = synth.tensor(rng, kind, M, K)
    x = np.stack([synth.activations(rng, K) for _ in range(batch)])
    w, dx, dy = ctx.upload(t), ctx.to_device(x), ctx.malloc(batch * M * 4)
    one = np.empty((batch, M), np.float32)
    for q in range(batch):
        dq = ctx.to_device(x[q])
        ctx.linear(w, dq, dy, flags=0)
        one[q] = dy.download(np.float32, M)
    _lib.check(_lib.lib().lmb_debug_batched_plan(ctx.h, 8, 56 * -(-M // (128 if kind == INT8 else 256))))
    try:
        ctx.linear(w, dx, dy, batch=batch, flags=0)
    finally:
        _lib.check(_lib.lib().lmb_debug_batched_plan(ctx.h, 0, 0))
    y = dy.download(np.float32).reshape(batch, M)
    want = np.stack([oracle.gemv_f64(kind, t.blocks, x[q], M, K) for q in range(batch)])
    assert np.linalg.norm(y - want) < 1.15 * np.linalg.norm(one - want)
    w.free()


def test_batched_sums_are_deterministic_and_match_single_sequences(ctx):
    """A row group cut over many CTAs gives the same bits every time, and a sequence's result does not
    depend on what the other sequences hold (infinities and NaN among them)."""
    rng = np.random.default_rng(31)
    t = synth.int4_tensor(rng, 512, 8192)
    x = np.stack([synth.activations(rng, 8192) for _ in range(6)])
    first = api.lut_linear(t, None, x, None, 6, ctx=ctx).reshape(6, -1).copy()
    assert np.array_equal(first, api.lut_linear(t, None, x, None, 6, ctx=ctx).reshape(6, -1))
    x[1, 5], x[3, 7] = np.inf, np.nan
    again = api.lut_linear(t, None, x, None, 6, ctx=ctx).reshape(6, -1)
    for q in (0, 2, 4, 5):
        assert np.array_equal(first[q], again[q])
    for q in (0, 2):
        one = api.lut_linear(t, None, x[q], None, 1, ctx=ctx)
        assert rel_l2(again[q], one) < TOL


def test_batched_expired_wait_is_reported(ctx):
    """A barrier that expects one arrival too many: the waits run out, the kernel leaves, the next host call says so."""
    L = _lib.lib()
    rng = np.random.default_rng(5)
    t = synth.int4_tensor(rng, 512, 2048)
    x = np.stack([synth.activations(rng, 2048) for _ in range(4)])
    want = api.lut_linear(t, None, x, None, 4, ctx=ctx).copy()
    try:
        _lib.check(L.lmb_debug_batched_waits(ctx.h, 1, 2000))
        with pytest.raises(_lib.LutmacError):
            api.lut_linear(t, None, x, None, 4, ctx=ctx)
    finally:
        _lib.check(L.lmb_debug_batched_waits(ctx.h, 0, 0))
    assert np.array_equal(api.lut_linear(t, None, x, None, 4, ctx=ctx), want)


def test_batched_limit_does_not_count_the_kernels_before(ctx):
    """A launch that waits a long time (and gives up), and behind it one with a limit a fraction of that: the second
    is let in early, but its waits begin when the first has ended, so its result is there."""
    L = _lib.lib()
    rng = np.random.default_rng(6)
    t = synth.int4_tensor(rng, 256, 256)
    x = np.stack([synth.activations(rng, 256) for _ in range(4)])
    w, dx, dy, dy2 = ctx.upload(t), ctx.to_device(x), ctx.malloc(4 * 256 * 4), ctx.malloc(4 * 256 * 4)
    try:
        _lib.check(L.lmb_debug_batched_plan(ctx.h, 4, 1))
        ctx.linear(w, dx, dy2, batch=4)
        want = dy2.download(np.float32)
        dy2.zero()
        _lib.check(L.lmb_debug_batched_waits(ctx.h, 1, 100000))
        ctx.linear(w, dx, dy, batch=4)
        _lib.check(L.lmb_debug_batched_waits(ctx.h, 0, 2000))
        ctx.linear(w, dx, dy2, batch=4)
        with pytest.raises(_lib.LutmacError) as e:
            ctx.sync()  # the first launch's
        assert e.value.status == _lib.ERR_TIMEOUT
    finally:
        _lib.check(L.lmb_debug_batched_waits(ctx.h, 0, 0))
        _lib.check(L.lmb_debug_batched_plan(ctx.h, 0, 0))
    assert np.array_equal(dy2.download(np.float32), want)
    w.free()


@pytest.mark.parametrize("head_dim,n_heads,n_kv", [(64, 8, 2), (64, 6, 1), (128, 4, 2)])
def test_batched_attention_positions(ctx, oracle, head_dim, n_heads, n_kv):
    """The streaming attention form: chunk edges (32 and 64 positions), sequences at different positions, an empty
    cache, splits without positions; every sequence against the oracle's own decode."""
    shape = dict(synth.tiny_model_shape(), head_dim=head_dim, n_heads=n_heads, n_kv_heads=n_kv, n_layers=1)
    spec = synth.model_spec(shape, INT4, seed=3, max_seq=160)
    m = Model(spec, ctx, max_batch=3)
    refs = [OracleModel(oracle, spec) for _ in range(3)]
    rng = np.random.default_rng(8)
    for p in range(131):
        toks, pos = rng.integers(0, spec.cfg["vocab"], size=3), [p, p // 2, p // 5]
        got = m.forward(toks.astype(np.int32), pos)
        for q in range(3):
            want = refs[q].forward(int(toks[q]), pos[q])
            if p in (0, 1, 31, 32, 33, 63, 64, 65, 66, 127, 128, 130):
                assert rel_l2(got[q], want) < 1e-5, (p, q)
    m.close()


def _models_with_context(ctx, oracle, head_dim, n_heads, n_kv, positions, seed):
    """A one-layer model and one oracle per sequence, all holding the same random cache."""
    shape = dict(synth.tiny_model_shape(), head_dim=head_dim, n_heads=n_heads, n_kv_heads=n_kv, n_layers=1)
    spec = synth.model_spec(shape, INT4, seed=seed, max_seq=max(positions) + 8)
    m = Model(spec, ctx, max_batch=len(positions))
    refs = [OracleModel(oracle, spec) for _ in positions]
    rng = np.random.default_rng(seed)
    for q, ref in enumerate(refs):
        ref.kv[...] = rng.standard_normal(ref.kv.shape).astype(np.float32)
        m.kv_import(ref.kv, q)
    return spec, m, refs, rng


@pytest.mark.parametrize("head_dim,pos", [(64, 385), (128, 193)])
def test_step_after_an_expired_attention_wait(ctx, oracle, head_dim, pos, monkeypatch):
    """Two splits, of which the first has one chunk more than the ring has stages and the second has not: with
    a refill barrier that never completes the first leaves without arriving, the second arrives.  The step
    reports it, and the following steps (other tokens) are right."""
    monkeypatch.setenv("LMB_MODEL_GRAPH", "0")
    L = _lib.lib()
    spec, m, refs, rng = _models_with_context(ctx, oracle, head_dim, 4, 2, [pos, pos], 17)
    toks = rng.integers(0, spec.cfg["vocab"], size=(4, 2)).astype(np.int32)
    try:
        _lib.check(L.lmb_debug_attn_stream(ctx.h, 2, 1, 2000))
        with pytest.raises(_lib.LutmacError) as e:
            m.forward(toks[0], [pos, pos])
        assert e.value.status == _lib.ERR_TIMEOUT
        _lib.check(L.lmb_debug_attn_stream(ctx.h, 2, 0, 0))
        for s in range(1, 4):
            got = m.forward(toks[s], [pos + s - 1] * 2)
            for q in range(2):
                assert rel_l2(got[q], refs[q].forward(int(toks[s][q]), pos + s - 1)) < 1e-5, (s, q)
    finally:
        _lib.check(L.lmb_debug_attn_stream(ctx.h, 0, 0, 0))
    m.close()


@pytest.mark.parametrize("splits", (1, 3))
@pytest.mark.parametrize("head_dim,n_heads,n_kv", [(64, 8, 2), (64, 6, 1), (128, 4, 2)])
def test_batched_attention_refills_its_ring(ctx, oracle, head_dim, n_heads, n_kv, splits, monkeypatch):
    """Four to six chunks per split through the ring of three stages, in each of the three forms: refills, phase
    flips and a ragged tail behind full chunks, over a random cache."""
    monkeypatch.setenv("LMB_MODEL_GRAPH", "0")
    L = _lib.lib()
    chunk = splits * (32 if head_dim == 128 else 64)
    start = [5 * chunk - 1, 4 * chunk - 2, 3 * chunk + 7]
    spec, m, refs, rng = _models_with_context(ctx, oracle, head_dim, n_heads, n_kv, start, 23)
    try:
        _lib.check(L.lmb_debug_attn_stream(ctx.h, splits, 0, 0))
        for s in range(4):
            toks, pos = rng.integers(0, spec.cfg["vocab"], size=3).astype(np.int32), [p + s for p in start]
            got = m.forward(toks, pos)
            for q in range(3):
                assert rel_l2(got[q], refs[q].forward(int(toks[q]), pos[q])) < 1e-5, (s, q)
    finally:
        _lib.check(L.lmb_debug_attn_stream(ctx.h, 0, 0, 0))
    m.close()


# (sequences, sequences per pass, CTAs per pass): every accumulator form with all units of the launch in one CTA (20 to
# 60 units, ranges over several row groups, every stage reused, sums folded every 8 blocks), ranges that end inside a
# row group, several passes, and as many CTAs as there are units
PLANS = [(3, 4, 1), (8, 8, 3), (16, 16, 1), (17, 32, 2), (32, 32, 1), (32, 8, 2), (9, 16, 1000), (31, 32, 7)]


@pytest.mark.parametrize("kind", (TERNARY, BINARY, INT2, INT3, INT4, INT5, INT6, INT8))
def test_batched_long_ranges_vs_fp64(ctx, oracle, kind):
    """Odd strides (rows that are not 16-byte aligned), a bias, and every plan of PLANS."""
    L = _lib.lib()
    rng = np.random.default_rng(70 + kind)
    M, K = 300, 5000
    t = synth.tensor(rng, kind, M, K)
    w, stride = ctx.upload(t), K + 3
    bias = rng.standard_normal(M).astype(np.float32)
    db = ctx.to_device(bias)
    for batch, seqs, ctas in PLANS:
        x = np.stack([synth.activations(rng, stride) for _ in range(batch)])
        dx, dy = ctx.to_device(x), ctx.malloc(batch * M * 4)
        _lib.check(L.lmb_debug_batched_plan(ctx.h, seqs, ctas))
        try:
            for _ in range(2):  # twice: the arrival counters must be back at zero
                dy.zero()
                ctx.linear(w, dx, dy, batch=batch, bias=db, flags=0, x_len=K, x_stride=stride)
                y = dy.download(np.float32).reshape(batch, M)
        finally:
            _lib.check(L.lmb_debug_batched_plan(ctx.h, 0, 0))
        for q in sorted({0, 1, batch // 2, batch - 1}):
            padded = np.zeros(blocks_per_row(K) * 256, np.float32)
            padded[:K] = x[q, :K]
            want = oracle.gemv_f64(kind, t.blocks, padded, M, K) + bias
            err = np.linalg.norm(y[q] - want)
            assert err < TOL * np.linalg.norm(np.abs(want) + 1e-3 * np.linalg.norm(padded)), (batch, seqs, ctas, q, err)
    w.free()
