"""ameva_flash_attn over prompts (the tensor-core kernel: 128 rows of positions x grouped heads per CTA, key tiles of 64,
masked tiles left out) against fp64 attention. Inputs are sized so that the fp16 rounding of queries and probabilities is
the only error that matters: |q|, |k| ~ 1 and D = 128 give scores of a few units, whose fp16 query rounding (2^-12 relative
per term) moves a probability by less than 1e-3 of itself; the outputs are averages of values of order 1."""
import struct

import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu
pkg = load_pkg()
rt = pkg.runtime
TOL = 2e-3      # (measured: 3e-4)


def fbits(v):
    return struct.unpack("<I", struct.pack("<f", float(v)))[0]


@pytest.fixture(scope="module")
def ctx():
    c = rt.init()
    yield c
    c.destroy()


def causal(n_q, n_kv, pitch):
    m = np.full((n_q, pitch), -np.inf, np.float16)
    for i in range(n_q):
        m[i, :n_kv - n_q + i + 1] = 0
    return m


def attention(q, k, v, mask, scale, softcap=0.0):
    """q [n_q][H][D], k / v [n_kv][Hkv][D], mask [n_q][n_kv] or [Hm][n_q][n_kv] or None, all fp64 sums -> [n_q][H][D]."""
    n_q, H, D = q.shape
    rep = H // k.shape[1]
    out = np.zeros((n_q, H, D))
    for h in range(H):
        s = q[:, h].astype(np.float64) @ k[:, h // rep].astype(np.float64).T * scale
        if softcap:
            s = softcap * np.tanh(s / softcap)
        if mask is not None:
            m = mask if mask.ndim == 2 else mask[h % mask.shape[0]]
            s = s + m.astype(np.float64)
        p = np.exp(s - s.max(axis=1, keepdims=True))
        out[:, h] = (p @ v[:, h // rep].astype(np.float64)) / p.sum(axis=1, keepdims=True)
    return out


def run(ctx, q, k, v, mask, scale, softcap=0.0, scratch=1 << 22, o_off=0, m_off=0, kv_pitch=None):
    n_q, H, D = q.shape
    n_kv, Hkv, _ = k.shape
    s1 = kv_pitch or Hkv * D
    kk, vv = (np.zeros((n_kv, s1), np.float16) for _ in range(2))
    kk[:, :Hkv * D], vv[:, :Hkv * D] = k.reshape(n_kv, -1), v.reshape(n_kv, -1)
    has = mask is not None
    m = np.zeros(8, np.float16) if not has else np.concatenate([np.zeros(m_off, np.float16), mask.ravel()])
    ne2 = 1 if not has or mask.ndim == 2 else mask.shape[0]
    pitch = mask.shape[-1] if has else 0
    push = [D, D, n_kv, n_q, H, Hkv, 0x11, int(has), 0, H * D, D, 0, s1, D, 0, s1, D, m_off, pitch, pitch * n_q, ne2, o_off,
            fbits(scale), fbits(softcap), 0, 0, 0, 0, 0, 0, 0]
    bufs = [ctx.buffer(data=np.ascontiguousarray(q.astype(np.float32))), ctx.buffer(data=kk), ctx.buffer(data=vv), ctx.buffer(data=m),
            ctx.buffer((n_q * H * D + o_off) * 4), ctx.buffer(scratch)]
    batch = ctx.batch(4)
    batch.dispatch(ctx.kernel("ameva_flash_attn"), bufs, push, (1, 1, 1))
    ev = batch.submit()
    ev.wait()
    ev.destroy()
    batch.destroy()
    out = bufs[4].read(np.float32)[o_off:].reshape(n_q, H, D)
    for b in bufs:
        b.destroy()
    return out


def inputs(n_q, n_kv, H, Hkv, D, seed=0):
    rng = np.random.default_rng(seed + n_q * 7 + n_kv)
    return (rng.standard_normal((n_q, H, D)).astype(np.float32), rng.standard_normal((n_kv, Hkv, D)).astype(np.float16),
            rng.standard_normal((n_kv, Hkv, D)).astype(np.float16))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("n_q,n_kv,H,Hkv", [(17, 17, 1, 1), (33, 64, 8, 2), (43, 65, 3, 1), (128, 128, 2, 2), (129, 300, 4, 4),
                                            (64, 1000, 8, 1), (50, 63, 7, 1), (300, 700, 6, 2)])
def test_causal_prompts(ctx, D, n_q, n_kv, H, Hkv):
    """Ragged tiles of rows and keys, G = 1, 3, 4, 7, 8; with and without room for key splits."""
    q, k, v = inputs(n_q, n_kv, H, Hkv, D)
    pitch = (n_kv + 63) // 64 * 64
    mask = causal(n_q, n_kv, pitch)
    want = attention(q, k, v, mask[:, :n_kv], D ** -0.5)
    for scratch in (64, 1 << 24):
        assert np.max(np.abs(run(ctx, q, k, v, mask, D ** -0.5, scratch=scratch) - want)) < TOL


@pytest.mark.parametrize("n_q,n_kv", [(40, 200), (64, 64)])
def test_forms_of_mask_scale_and_layout(ctx, n_q, n_kv):
    H, Hkv, D = 4, 2, 128
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 3)
    rng = np.random.default_rng(n_q)
    bias = rng.standard_normal((n_q, n_kv)).astype(np.float16)                     # a mask that is a bias
    per_head = np.where(rng.random((H, n_q, n_kv)) < 0.5, -np.inf, 0).astype(np.float16)
    per_head[:, :, 0] = 0
    for name, mask, scale, cap, kw in [("none", None, 0.09, 0.0, {}), ("bias", bias, 0.09, 0.0, {}), ("heads", per_head, 0.09, 0.0, {}),
                                       ("odd", bias[:, :n_kv], 0.09, 0.0, {"m_off": 3}), ("cap", bias, 0.5, 5.0, {}),
                                       ("negative", None, -0.05, 0.0, {}), ("zero", None, 0.0, 0.0, {}),
                                       ("output offset", None, 0.09, 0.0, {"o_off": 3, "scratch": 64}),
                                       ("pitch", bias, 0.09, 0.0, {"kv_pitch": Hkv * D + 8})]:
        got = run(ctx, q, k, v, mask, scale, cap, **kw)
        want = attention(q, k, v, mask, scale, cap)
        assert np.max(np.abs(got - want)) < TOL, name


def test_growing_scores_rescale_the_accumulator(ctx):
    """Keys sorted so that every tile raises the maximum, some by more than the rescale step and some by less."""
    n_q, n_kv, D = 64, 1024, 128
    q, k, v = inputs(n_q, n_kv, 2, 2, D, 9)
    q[:] = np.abs(q)
    k = (np.abs(k.astype(np.float32)) * np.linspace(0, 1, n_kv)[:, None, None]).astype(np.float16)
    for scale in (0.02, 0.2, 1.0):
        want = attention(q.astype(np.float16), k, v, None, scale)
        got = run(ctx, q.astype(np.float16).astype(np.float32), k, v, None, scale)
        assert np.max(np.abs(got - want)) < TOL


def test_masked_rows_and_lowest_values(ctx):
    """A key cache with an unused, wholly masked tail of infinities; rows whose every key is masked give NaN and no other row
    does; a mask of the type's lowest finite value leaves the row's own softmax."""
    n_q, n_kv, D = 64, 512, 128
    q, k, v = inputs(n_q, n_kv, 2, 2, D, 5)
    k[320:], v[320:] = np.inf, np.nan        # whole tiles nobody may read
    mask = np.zeros((n_q, n_kv), np.float16)
    mask[:, 320:] = -np.inf
    mask[7, :] = -np.inf
    mask[9, :320] = -65504
    got = run(ctx, q, k, v, mask, D ** -0.5)
    want = attention(q, k[:320], v[:320], mask[:, :320], D ** -0.5)
    assert np.isnan(got[7]).all()
    keep = [i for i in range(n_q) if i not in (7, 9)]
    assert np.max(np.abs(got[keep] - want[keep])) < TOL
    # scores next to -65504 are spaced 2^-8 apart in fp32: probabilities within 2^-8
    assert np.max(np.abs(got[9] - want[9])) < 2e-2


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("last,m_off", [(288, 0), (272, 0), (304, 3), (16, 0)])
def test_unused_cache_behind_the_last_key_of_a_tile(ctx, D, last, m_off):
    """The keys in use end inside a tile of 64; behind them the cache holds NaN and infinities that no row sees (the mask read
    in pieces of eight and one by one)."""
    n_q, n_kv = 64, 512
    q, k, v = inputs(n_q, n_kv, 2, 2, D, 5)
    k[last:], v[last:] = np.inf, np.nan
    mask = np.zeros((n_q, n_kv), np.float16)
    mask[:, last:] = -np.inf
    got = run(ctx, q, k, v, mask, D ** -0.5, m_off=m_off)
    want = attention(q, k[:last], v[:last], None, D ** -0.5)
    assert np.max(np.abs(got - want)) < TOL


def seen(q, k, v, mask, scale):
    """As attention(), each row over the keys it sees only: what is masked is no term of the sum."""
    out = np.zeros(q.shape)
    rep = q.shape[1] // k.shape[1]
    with np.errstate(invalid="ignore"):
        for h in range(q.shape[1]):
            for i in range(q.shape[0]):
                at = mask[i] != -np.inf
                s = k[at, h // rep].astype(np.float64) @ q[i, h].astype(np.float16).astype(np.float64) * scale
                p = np.exp(s - s.max())
                out[i, h] = (p[:, None] * v[at, h // rep].astype(np.float64)).sum(0) / p.sum()
    return out


@pytest.mark.parametrize("D,H,Hkv", [(64, 4, 4), (128, 4, 2), (128, 8, 1)])
@pytest.mark.parametrize("scratch", [64, 1 << 24])
def test_values_that_are_not_finite_reach_the_rows_that_see_them(ctx, D, H, Hkv, scratch):
    """V rows of infinities, of either sign, and of NaN: a position in front of them (causal mask) gives what it would give
    without them, one behind them +inf, -inf or NaN in the same columns as the sum over its keys."""
    n_q, n_kv = 150, 700
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 31)
    mask = causal(n_q, n_kv, 704)
    v[600, :, 1::3] = np.inf
    v[655, :, 2::5] = -np.inf
    v[690, 0, ::7] = np.nan
    v[697:, :, :] = np.nan
    mask[:, 697:] = -np.inf
    want = seen(q, k, v, mask[:, :n_kv], D ** -0.5)
    got = run(ctx, q, k, v, mask, D ** -0.5, scratch=scratch)
    finite = np.isfinite(want)
    assert finite.any() and np.isposinf(want).any() and np.isneginf(want).any() and np.isnan(want).any()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    assert np.max(np.abs(got[finite] - want[finite])) < TOL


def test_more_keys_than_one_window(ctx):
    """More key tiles than one scan of the mask covers (512), in one split."""
    n_q, n_kv, D = 17, 512 * 64 + 200, 64
    q, k, v = inputs(n_q, n_kv, 1, 1, D, 6)
    mask = causal(n_q, n_kv, n_kv)
    mask[:, 1000:20000] = -np.inf
    got = run(ctx, q, k, v, mask, D ** -0.5, scratch=64)
    assert np.max(np.abs(got - attention(q, k, v, mask, D ** -0.5))) < TOL


@pytest.mark.parametrize("D,H,Hkv", [(64, 14, 2), (64, 8, 1), (128, 32, 32), (128, 20, 5), (128, 8, 1), (256, 8, 1), (256, 6, 2)])
@pytest.mark.parametrize("n_kv", [1, 15, 16, 17, 95, 96, 97, 193, 256, 257, 400, 5000])
def test_one_position_over_few_and_many_blocks(ctx, D, H, Hkv, n_kv):
    """Blocks of 16 keys per warp, one to many per CTA, one to many CTAs per KV head (merged by the last one)."""
    q, k, v = inputs(1, n_kv, H, Hkv, D, 11)
    rng = np.random.default_rng(n_kv)
    mask = np.where(rng.random((1, (n_kv + 63) // 64 * 64)) < 0.3, -np.inf, rng.standard_normal((1, (n_kv + 63) // 64 * 64))).astype(np.float16)
    mask[0, n_kv // 2] = 0
    want = attention(q, k, v, mask[:, :n_kv], D ** -0.5)
    for _ in range(2):      # (the second launch finds the arrival counters as the first left them)
        assert np.max(np.abs(run(ctx, q, k, v, mask, D ** -0.5) - want)) < TOL
    assert np.max(np.abs(run(ctx, q, k, v, mask, D ** -0.5, scratch=64) - want)) < TOL


@pytest.mark.parametrize("D,H,Hkv,n_q,n_kv", [(128, 8, 8, 1, 1536), (128, 8, 8, 1, 1537), (64, 8, 2, 1, 1536), (64, 8, 2, 1, 1537),
                                              (128, 32, 32, 1, 3551), (128, 8, 1, 1, 20000), (64, 32, 8, 1, 14301), (256, 8, 1, 1, 2500),
                                              (256, 4, 2, 3, 700)])
def test_one_position_on_both_sides_of_the_rules(ctx, D, H, Hkv, n_q, n_kv):
    """The longest context with fine splits and the first with the wider CTAs and coarse ones; long ones; D = 256."""
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 13)
    mask = causal(n_q, n_kv, (n_kv + 63) // 64 * 64)
    want = attention(q, k, v, mask[:, :n_kv], D ** -0.5)
    for scratch in (1 << 24, n_q * H * (D + 4) * 4 * 3 + 64):
        assert np.max(np.abs(run(ctx, q, k, v, mask, D ** -0.5, scratch=scratch) - want)) < TOL


def test_prompt_attention_among_kernels_with_tensor_memory(ctx):
    """Attention and tensor-core products in turn in one batch: each holds tensor memory, and each may be scheduled while the
    one before it still runs. Same bytes as one by one."""
    qmm = pkg.qmm
    from helpers import Q8_0, make_acts, make_weights
    n_q, H, Hkv, D = 256, 32, 8, 128
    q, k, v = inputs(n_q, n_q, H, Hkv, D, 21)
    mask = causal(n_q, n_q, 256)
    N, K = 384, 256
    blocks, scale = make_weights(Q8_0, N, K, 3)
    w = qmm.QuantWeight.from_ggml(ctx, Q8_0, blocks, N, K, scale)
    mm = qmm.MulMat(ctx, w, n_q)
    push = [D, D, n_q, n_q, H, Hkv, 0x11, 1, 0, H * D, D, 0, Hkv * D, D, 0, Hkv * D, D, 0, 256, 256 * n_q, 1, 0, fbits(D ** -0.5), 0, 0, 0,
            0, 0, 0, 0, 0]
    bufs = [ctx.buffer(data=np.ascontiguousarray(a)) for a in (q, k, v, mask)] + [ctx.buffer(n_q * H * D * 4), ctx.buffer(1 << 22)]
    x, y = ctx.buffer(data=make_acts(n_q, K, 4)), ctx.buffer(n_q * N * 4)

    def go(rounds):
        batch = ctx.batch(64)
        for _ in range(rounds):
            batch.dispatch(ctx.kernel("ameva_flash_attn"), bufs, push, (1, 1, 1))
            mm.record(batch, x, y, n_q)
            batch.dispatch(ctx.kernel("ameva_flash_attn"), bufs, push, (1, 1, 1))
            mm.record(batch, x, y, n_q, quantize=False)
        ev = batch.submit()
        ev.wait()
        ev.destroy()
        batch.destroy()
        return bufs[4].read(np.uint8), y.read(np.uint8)

    one, many = go(1), go(8)
    assert np.array_equal(one[0], many[0]) and np.array_equal(one[1], many[1])
    want = attention(q, k, v, mask[:, :n_q], D ** -0.5)
    assert np.max(np.abs(one[0].view(np.float32).reshape(n_q, H, D) - want)) < TOL
    mm.destroy()
    w.destroy()
    for b in bufs + [x, y]:
        b.destroy()


@pytest.mark.parametrize("n_q,n_kv,H,Hkv,D", [(60, 1041, 32, 8, 128), (60, 1043, 32, 8, 128), (129, 1000, 14, 2, 64), (300, 1000, 14, 2, 64),
                                              (75, 1250, 32, 32, 128), (150, 1250, 32, 32, 128), (130, 4100, 8, 8, 64), (420, 1800, 8, 8, 64)])
def test_prompts_on_both_sides_of_the_work_rule(ctx, n_q, n_kv, H, Hkv, D):
    """Little work (64 rows per CTA) and more (128 rows, tensor memory), grouped heads and not; the same tolerance."""
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 41)
    mask = causal(n_q, n_kv, (n_kv + 63) // 64 * 64)
    want = attention(q, k, v, mask[:, :n_kv], D ** -0.5)
    for scratch in (64, 1 << 24):
        assert np.max(np.abs(run(ctx, q, k, v, mask, D ** -0.5, scratch=scratch) - want)) < TOL


# ---- the 128-row kernel: the same edges with enough heads that the work rule picks it -------------------------------------
@pytest.mark.parametrize("n_q,n_kv,H,Hkv,D", [(50, 1100, 48, 16, 128), (43, 3001, 28, 4, 128), (129, 700, 24, 3, 128), (65, 2000, 32, 16, 64),
                                              (300, 2600, 8, 8, 128), (17, 8200, 64, 64, 64)])
def test_ragged_tiles_of_the_large_kernel(ctx, n_q, n_kv, H, Hkv, D):
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 51)
    mask = causal(n_q, n_kv, (n_kv + 63) // 64 * 64)
    want = attention(q, k, v, mask[:, :n_kv], D ** -0.5)
    for scratch in (64, 1 << 26):
        assert np.max(np.abs(run(ctx, q, k, v, mask, D ** -0.5, scratch=scratch) - want)) < TOL


def test_forms_of_the_large_kernel(ctx):
    n_q, n_kv, H, Hkv, D = 64, 520, 64, 32, 128
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 53)
    rng = np.random.default_rng(53)
    bias = rng.standard_normal((n_q, n_kv)).astype(np.float16)
    per_head = np.where(rng.random((H, n_q, n_kv)) < 0.5, -np.inf, 0).astype(np.float16)
    per_head[:, :, 0] = 0
    for name, mask, scale, cap, kw in [("none", None, 0.09, 0.0, {}), ("bias", bias, 0.09, 0.0, {}), ("heads", per_head, 0.09, 0.0, {}),
                                       ("odd", bias, 0.09, 0.0, {"m_off": 3}), ("cap", bias, 0.5, 5.0, {}), ("negative", None, -0.05, 0.0, {}),
                                       ("zero", None, 0.0, 0.0, {}), ("output offset", None, 0.09, 0.0, {"o_off": 3, "scratch": 64}),
                                       ("pitch", bias, 0.09, 0.0, {"kv_pitch": Hkv * D + 8})]:
        assert np.max(np.abs(run(ctx, q, k, v, mask, scale, cap, **kw) - attention(q, k, v, mask, scale, cap))) < TOL, name


def test_growing_scores_in_the_large_kernel(ctx):
    n_q, n_kv, D = 64, 1024, 128
    q, k, v = inputs(n_q, n_kv, 32, 16, D, 9)
    q = np.abs(q).astype(np.float16)
    k = (np.abs(k.astype(np.float32)) * np.linspace(0, 1, n_kv)[:, None, None]).astype(np.float16)
    for scale in (0.02, 0.2, 1.0):
        assert np.max(np.abs(run(ctx, q.astype(np.float32), k, v, None, scale) - attention(q, k, v, None, scale))) < TOL


@pytest.mark.parametrize("D,H,Hkv", [(64, 128, 64), (128, 64, 32)])
@pytest.mark.parametrize("last,m_off", [(320, 0), (288, 0), (272, 0), (304, 3), (16, 0)])
def test_unused_cache_in_the_large_kernel(ctx, D, H, Hkv, last, m_off):
    n_q, n_kv = 64, 512
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 5)
    k[last:], v[last:] = np.inf, np.nan
    mask = np.zeros((n_q, n_kv), np.float16)
    mask[:, last:] = -np.inf
    mask[7, :] = -np.inf
    got = run(ctx, q, k, v, mask, D ** -0.5, m_off=m_off)
    want = attention(q, k[:last], v[:last], None, D ** -0.5)
    keep = [i for i in range(n_q) if i != 7]
    assert np.isnan(got[7]).all() and np.max(np.abs(got[keep] - want[keep])) < TOL


@pytest.mark.parametrize("D,H,Hkv", [(64, 48, 6), (128, 24, 12)])
@pytest.mark.parametrize("scratch", [64, 1 << 26])
def test_values_that_are_not_finite_in_the_large_kernel(ctx, D, H, Hkv, scratch):
    n_q, n_kv = 150, 700
    q, k, v = inputs(n_q, n_kv, H, Hkv, D, 31)
    mask = causal(n_q, n_kv, 704)
    v[600, :, 1::3] = np.inf
    v[655, :, 2::5] = -np.inf
    v[690, 0, ::7] = np.nan
    v[697:, :, :] = np.nan
    mask[:, 697:] = -np.inf
    want = seen(q, k, v, mask[:, :n_kv], D ** -0.5)
    got = run(ctx, q, k, v, mask, D ** -0.5, scratch=scratch)
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    assert np.max(np.abs(got[finite] - want[finite])) < TOL


def test_more_keys_than_one_window_of_the_large_kernel(ctx):
    n_q, n_kv, D = 17, 512 * 64 + 200, 64
    q, k, v = inputs(n_q, n_kv, 8, 1, D, 6)
    mask = causal(n_q, n_kv, n_kv)
    mask[:, 1000:20000] = -np.inf
    got = run(ctx, q, k, v, mask, D ** -0.5, scratch=64)
    assert np.max(np.abs(got - attention(q, k, v, mask, D ** -0.5))) < TOL
