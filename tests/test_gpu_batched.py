"""The batched tcgen05 path (three or more sequences) against the fp64 oracle: edges of its 32-row tiles,
128- and 256-row groups, 4 / 8 / 16 / 32-sequence forms, row groups cut over several CTAs, several passes."""
import numpy as np
import pytest

from lutmac_b200 import _lib, api, synth
from lutmac_b200.blocks import BINARY, INT2, INT3, INT4, INT5, INT6, INT8, TERNARY, blocks_per_row
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
