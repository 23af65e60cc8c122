"""The f32 row ops that sit between two quantized mul_mats (ADD, MUL, split SWIGLU, RMS norm with and without the weight
multiply), through the C ABI against numpy statements of ggml's CPU arithmetic (silu(x) = x / (1 + exp(-x)); rms_norm:
y = x / sqrt(mean(x^2) + eps), the mean accumulated in double by ggml)."""
import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu
pkg = load_pkg()
rt = pkg.runtime


@pytest.fixture(scope="module")
def ctx():
    c = rt.init()
    yield c
    c.destroy()


def _run(ctx, name, bufs, push):
    batch = ctx.batch(4)
    batch.dispatch(ctx.kernel(name), bufs, push, (1, 1, 1))
    ev = batch.submit()
    ev.wait()
    ev.destroy()
    batch.destroy()


@pytest.mark.parametrize("rows,cols,b_rows", [(1, 4096, 1), (7, 130, 1), (7, 130, 7), (512, 11008, 1), (3, 1, 3)])
@pytest.mark.parametrize("op", ["add", "mul"])
def test_binary_rows(ctx, rows, cols, b_rows, op):
    rng = np.random.default_rng(rows + cols)
    a = rng.standard_normal((rows, cols)).astype(np.float32)
    b = rng.standard_normal((b_rows, cols)).astype(np.float32)
    ab, bb, db = ctx.buffer(data=a), ctx.buffer(data=b), ctx.buffer(a.nbytes)
    _run(ctx, f"ameva_{op}_f32", [ab, bb, db], [rows, cols, b_rows])
    want = a + b if op == "add" else a * b
    assert np.array_equal(db.read(np.float32).reshape(rows, cols), want)
    _run(ctx, f"ameva_{op}_f32", [ab, bb, ab], [rows, cols, b_rows])     # in place
    assert np.array_equal(ab.read(np.float32).reshape(rows, cols), want)
    for v in (ab, bb, db):
        v.destroy()


def test_swiglu(ctx):
    rng = np.random.default_rng(1)
    g = (rng.standard_normal(11008) * 3).astype(np.float32)
    g[:4] = [0.0, -30.0, 30.0, -100.0]
    u = rng.standard_normal(11008).astype(np.float32)
    gb, ub, db = ctx.buffer(data=g), ctx.buffer(data=u), ctx.buffer(g.nbytes)
    _run(ctx, "ameva_swiglu_f32", [gb, ub, db], [g.size])
    want = (g.astype(np.float64) / (1.0 + np.exp(-g.astype(np.float64)))) * u
    got = db.read(np.float32)
    assert np.isfinite(got).all()
    assert np.max(np.abs(got - want)) <= 2e-6 * np.max(np.abs(want))
    for v in (gb, ub, db):
        v.destroy()


@pytest.mark.parametrize("rows,cols", [(1, 4096), (5, 2560), (512, 4096), (3, 100), (2, 28672)])
@pytest.mark.parametrize("with_weight", [0, 1])
def test_rms_norm(ctx, rows, cols, with_weight):
    rng = np.random.default_rng(rows * 7 + cols)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    x[0] *= 1e-3
    w = (1 + 0.1 * rng.standard_normal(cols)).astype(np.float32)
    eps = np.float32(1e-5)
    xb, wb, db = ctx.buffer(data=x), ctx.buffer(data=w), ctx.buffer(x.nbytes)
    _run(ctx, "ameva_rms_norm_f32", [xb, wb, db], [rows, cols, int(eps.view(np.uint32)), with_weight])
    x64 = x.astype(np.float64)
    scale = 1.0 / np.sqrt(np.mean(x64 * x64, axis=1, keepdims=True) + float(eps))
    want = (x64 * scale).astype(np.float32)
    if with_weight:
        want = want * w
    got = db.read(np.float32).reshape(rows, cols)
    assert np.max(np.abs(got - want) / np.max(np.abs(want), axis=1, keepdims=True)) <= 3e-6
    for v in (xb, wb, db):
        v.destroy()


def test_argument_checks(ctx):
    a = ctx.buffer(64 * 4)
    for name, bufs, push in (("ameva_add_f32", [a, a, a], [4, 16, 3]), ("ameva_add_f32", [a, a, a], [8, 16, 1]),
                             ("ameva_swiglu_f32", [a, a, a], [0]), ("ameva_rms_norm_f32", [a, a, a], [8, 16, 0, 0]),
                             ("ameva_rms_norm_f32", [a, a, a], [1, 16, 0, 2])):
        batch = ctx.batch(4)
        with pytest.raises(rt.AmevaComputeError):
            batch.dispatch(ctx.kernel(name), bufs, push, (1, 1, 1))
            batch.submit().wait()
        batch.destroy()
    a.destroy()


@pytest.mark.parametrize("n", [1, 2049, 65535, 65536, 65537, 67583, 67584, 67587, 200003])
def test_swiglu_and_add_at_the_edges_of_the_vector_forms(ctx, n):
    """From 65536 elements: pieces of four, two per thread, 2048 elements per CTA; below, one element per thread."""
    rng = np.random.default_rng(n)
    g, u = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    g64 = g.astype(np.float64)
    want = g64 / (1.0 + np.exp(-g64)) * u
    gb, ub, db = ctx.buffer(data=g), ctx.buffer(data=u), ctx.buffer(4 * n)
    _run(ctx, "ameva_swiglu_f32", [gb, ub, db], [n])
    # expf (2 ulp), one division and two multiplications: well below 1e-6 of the value
    assert np.all(np.abs(db.read(np.float32) - want) <= 1e-6 * np.abs(want) + 1e-30)
    _run(ctx, "ameva_add_f32", [gb, ub, db], [n, 1, n])
    assert np.array_equal(db.read(np.float32), g + u)
    for b in (gb, ub, db):
        b.destroy()


@pytest.mark.parametrize("cols", [4, 1020, 1024, 1028, 4100, 8192, 8196])
def test_rms_norm_at_the_edges_of_the_register_form(ctx, cols):
    rng = np.random.default_rng(cols)
    x = rng.standard_normal((3, cols)).astype(np.float32)
    w = (1 + 0.1 * rng.standard_normal(cols)).astype(np.float32)
    eps = np.float32(1e-5)
    xb, wb = ctx.buffer(data=x), ctx.buffer(data=w)
    _run(ctx, "ameva_rms_norm_f32", [xb, wb, xb], [3, cols, int(eps.view(np.uint32)), 1])      # in place
    x64 = x.astype(np.float64)
    want = x64 / np.sqrt(np.mean(x64 * x64, axis=1, keepdims=True) + float(eps)) * w
    # the fp32 sum of squares (8192 terms by a tree: well below 1e-6) and four roundings
    assert np.all(np.abs(xb.read(np.float32).reshape(3, cols) - want) <= 1.5e-6 * np.abs(want) + 1e-30)
    xb.destroy()
    wb.destroy()


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 3, (1 << 20) + 2047, (1 << 20) + 2050])
def test_swiglu_on_both_sides_of_its_vector_form(ctx, n):
    rng = np.random.default_rng(n)
    g, u = (rng.standard_normal(n).astype(np.float32) * 3 for _ in range(2))
    gb, ub, db = ctx.buffer(data=g), ctx.buffer(data=u), ctx.buffer(n * 4 + 64)
    db.write(np.zeros(n + 16, np.float32))
    _run(ctx, "ameva_swiglu_f32", [gb, ub, db], [n])
    got = db.read(np.float32)
    g64 = g.astype(np.float64)
    assert np.allclose(got[:n], g64 / (1 + np.exp(-g64)) * u, rtol=2e-6, atol=1e-7)
    assert not got[n:].any()
    for b in (gb, ub, db):
        b.destroy()
