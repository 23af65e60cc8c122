"""Order of the dispatches of a batch as the host sees it: products request their weights before the launches in front of them
have completed, except where one of those may write the weights."""
import numpy as np
import pytest

from conftest import load_pkg
from helpers import I2_S, Q4_0, Q4_K, Q6_K, Q8_0, make_acts, make_weights

pytestmark = pytest.mark.gpu
pkg = load_pkg()
rt, qmm = pkg.runtime, pkg.qmm
ONE = (1, 1, 1)


@pytest.fixture(scope="module")
def ctx():
    c = rt.init()
    yield c
    c.destroy()


def copy(ctx, batch, src, dst, nbytes):
    n = nbytes // 4
    batch.dispatch(ctx.kernel("ameva_cpy"), [src, dst], [n, 1, 1, 1, 0, 1, n, n, n, n, 1, 1, 0, 1, n, n, n, 0, 0], ONE)


@pytest.mark.parametrize("t,M,N,K", [(Q4_0, 1, 4096, 4096), (Q8_0, 3, 1000, 4096), (Q4_K, 1, 4096, 4096), (Q4_K, 8, 2048, 4096),
                                     (Q6_K, 1, 4096, 4096), (Q6_K, 5, 515, 2048), (I2_S, 1, 4096, 2560), (I2_S, 64, 1024, 2560),
                                     (Q8_0, 64, 2048, 2048), (Q4_K, 300, 1024, 2048)])
@pytest.mark.parametrize("flush", [False, True])
def test_weights_written_by_the_dispatch_in_front(ctx, t, M, N, K, flush):
    """The weight buffer filled from two others in turn, a product behind each copy: the bytes of products with weights that
    were there all along."""
    ws = []
    for seed in (1, 2, 3):
        ws.append(qmm.QuantWeight.from_ggml(ctx, t, make_weights(t, N, K, seed)[0], N, K, 0.0625))   # (the scale is I2_S's)
    x, out = ctx.buffer(data=make_acts(M, K, 9)), [ctx.buffer(M * N * 4) for _ in range(2)]
    nbytes = ws[0].buf.size_bytes // 4 * 4
    want = []
    for w in ws[:2]:
        mm = qmm.MulMat(ctx, w, M)
        mm.run(x, out[0], M)
        want.append(out[0].read(np.uint8))
        mm.destroy()
    mm = qmm.MulMat(ctx, ws[2], M)

    def record():
        batch = ctx.batch(16)
        for w, o in zip(ws, out):
            copy(ctx, batch, w.buf, ws[2].buf, nbytes)
            if flush:
                batch.flush()
            mm.record(batch, x, o, M)
        return batch

    batch = record()
    if flush:
        ev = batch.submit()
        ev.wait()
        ev.destroy()
        for o, y in zip(out, want):
            assert np.array_equal(o.read(np.uint8), y)
        assert batch.launches()[1] >= 3        # the first of each flush and the second product at least
    else:
        batch.instantiate()
        assert batch.launches()[1] == 2        # both products
        for _ in range(6):
            ev = batch.replay()
            ev.wait()
            ev.destroy()
            for o, y in zip(out, want):
                assert np.array_equal(o.read(np.uint8), y)
    batch.destroy()
    for o in [mm, x] + out + ws:
        o.destroy()


def test_products_that_only_share_memory_with_reads_start_early(ctx):
    """A table that rows are taken from and that is also a weight (tied embeddings), a weight used twice, and a group with
    unused slots bound to its output: nothing writes the weights, nothing has to wait."""
    N, K = 512, 1024
    blocks, _ = make_weights(Q4_K, N, K, 4)
    w = qmm.QuantWeight.from_ggml(ctx, Q4_K, blocks, N, K)
    mm, g = qmm.MulMat(ctx, w, 1), qmm.MulMatGroup(ctx, [w, w], fused_quantize=False)
    x, o, o2 = ctx.buffer(data=make_acts(1, K, 5)), ctx.buffer(N * 4), ctx.buffer(N * 4)
    idx, status = ctx.buffer(data=np.array([3], np.int32)), ctx.buffer(data=np.array([0, -1], np.int32))
    q_row, s_row = K // 256 * qmm.Q_BYTES[Q4_K], K // 256 * qmm.S_BYTES[Q4_K]
    batch = ctx.batch(16)
    batch.dispatch(ctx.kernel("ameva_get_rows_q4_k_rp"), [w.buf, idx, status, x],
                   [K, 1, 1, 1, 0, 0, 0, 0, 0, 1, 0, 0, 0, K, 0, 0, N, 3, 0, N, 0, w.s_off, q_row, 0, s_row], ONE)
    mm.record(batch, x, o, 1)
    mm.record(batch, x, o2, 1)
    g.record(batch, x, [o, o2])
    batch.instantiate()
    assert batch.launches()[1] == 0
    batch.destroy()
    for b in (mm, g, x, o, o2, idx, status, w):
        b.destroy()
