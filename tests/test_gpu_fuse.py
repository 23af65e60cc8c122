"""Dispatches that leave the host in one launch (csrc/fuse.cu) against the same dispatches submitted one by one: every buffer
ends with the same bytes, whether the operands allow a fused form or (aliased, overlapping, strided) do not."""
import struct

import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu
pkg = load_pkg()
rt, qmm = pkg.runtime, pkg.qmm


def fbits(v):
    return struct.unpack("<I", struct.pack("<f", float(v)))[0]


@pytest.fixture(scope="module")
def ctx():
    c = rt.init()
    yield c
    c.destroy()


def check(ctx, bufs, ops):
    """bufs: name -> initial array; ops: (kernel, [name or (name, byte offset[, bytes])], push, grid)."""
    held = {n: ctx.buffer(data=a) for n, a in bufs.items()}

    def bind(x):
        return held[x] if isinstance(x, str) else (held[x[0]],) + tuple(x[1:])

    def run(groups, replay=False):
        for n, a in bufs.items():
            held[n].write(a)
        for g in groups:
            batch = ctx.batch(len(g) + 1)
            for name, binds, push, grid in g:
                batch.dispatch(ctx.kernel(name), [bind(b) for b in binds], push, grid)
            if replay:
                batch.instantiate()
                ev = batch.replay()
            else:
                ev = batch.submit()
            ev.wait()
            ev.destroy()
            batch.destroy()
        return {n: held[n].read(np.uint8) for n in bufs}

    alone = run([[op] for op in ops])
    for got in (run([ops]), run([ops], replay=True)):
        for n in bufs:
            assert np.array_equal(alone[n], got[n]), n
    for b in held.values():
        b.destroy()
    return alone


ONE = (1, 1, 1)


def i2_s(prefix, src, M, N, K, rng, bufs, out, y=None):
    """The quantize and the product of one I2_S weight."""
    bufs[prefix + "w"] = rng.integers(0, 256, N * K // 4).astype(np.uint8)
    for name, size in (("y", M * K * 4), ("q", M * K), ("act", M * 8), ("qeo", 64)):
        bufs[prefix + name] = np.zeros(size, np.uint8)
    bufs[out] = np.zeros(M * N, np.float32)
    return [("bitnet_norm_q8", [src, src, src, y or prefix + "y", prefix + "q", prefix + "act", prefix + "qeo"], [K, 0, 0, 0], (M, 1, 1)),
            ("bitnet_gemv_i2_s_l32w1", [prefix + "w", prefix + "q", out, prefix + "act"], [K, N, fbits(0.02), 0, M, N], ONE)]


@pytest.mark.parametrize("M,K,ns", [(1, 128, (1, 2)), (1, 2560, (2560, 640, 641)), (3, 1152, (33, 7, 64, 9)), (8, 8192, (5, 6)),
                                    (1, 8320, (40, 41)), (2, 256, (17, 18, 19, 20, 21))])
def test_bitnet_products_of_one_row(ctx, M, K, ns):
    rng = np.random.default_rng(K + M)
    bufs = {"x": rng.standard_normal(M * K).astype(np.float32), "w": rng.standard_normal(K).astype(np.float32),
            "h": np.zeros(M * K, np.float32)}
    ops = [("ameva_rms_norm_f32", ["x", "w", "h"], [M, K, fbits(1e-5), 1], ONE)]
    for j, N in enumerate(ns):
        ops += i2_s(f"p{j}", "h", M, N, K, rng, bufs, f"o{j}")
    out = check(ctx, bufs, ops)
    assert any(out["o0"])
    # no weight row; the norm in place; a quantize that writes its own source (that one and what follows stay apart)
    check(ctx, bufs, [("ameva_rms_norm_f32", ["x", "w", "x"], [M, K, fbits(1e-5), 0], ONE)] +
          [(k, ["x" if b == "h" else b for b in binds], p, g) for k, binds, p, g in ops[1:]])
    bufs2 = dict(bufs)
    check(ctx, bufs2, ops[:1] + i2_s("p0", "h", M, ns[0], K, rng, bufs2, "o0", y="h") + ops[3:])


@pytest.mark.parametrize("M,N", [(1, 77), (1, 2560), (4, 130)])
@pytest.mark.parametrize("form", ["ab", "ba", "in place", "onto the activations"])
def test_bitnet_gate_and_residual(ctx, M, N, form):
    K = 384
    rng = np.random.default_rng(N)
    bufs = {n: rng.standard_normal(M * K).astype(np.float32) for n in ("gate", "up", "act")}
    bufs["res"], bufs["sum"] = rng.standard_normal(M * N).astype(np.float32), np.zeros(max(M * N, M * K), np.float32)
    ops = [("ameva_swiglu_f32", ["gate", "up", "act"], [M * K], ONE)] + i2_s("d", "act", M, N, K, rng, bufs, "tmp")
    a, b, o = {"ab": ("tmp", "res", "sum"), "ba": ("res", "tmp", "sum"), "in place": ("tmp", "res", "res"),
               "onto the activations": ("tmp", "res", "sum")}[form]
    if form == "onto the activations":   # the sum overwrites what the product reads: not in one launch
        ops = [(k, ["sum" if x == "dq" else x for x in binds], p, g) for k, binds, p, g in ops]
    ops.append(("ameva_add_f32", [a, b, o], [M, N, M], ONE))
    check(ctx, bufs, ops)
    check(ctx, bufs, [(ops[0][0], ["gate", "up", "gate"], ops[0][2], ONE)] +     # the gate in place
          [(k, ["gate" if x == "act" else x for x in binds], p, g) for k, binds, p, g in ops[1:]])


def rope(a, d, D, heads, M, pos="pos", neox=1, d_off=0):
    w = heads * D
    return ("ameva_rope", [a, pos, pos, d], [D, heads, M, 1, 0, D, w, w * M, d_off, D, w, w * M, 0, 0, D, neox, 0, fbits(0.9), fbits(1.0),
                                            fbits(0.0), fbits(1.0), 0, 0], ONE)


def store(src, cache, width, M, rows, f16=1, a_off=0, node=3):
    return ("ameva_set_rows", [src, "idx", "status", cache],
            [width, M, 1, 1, a_off, width, width * M, width * M, 0, 2, 2 * M, 2 * M, 1, 1, 1, rows, 0, width, width * rows, width * rows,
             f16, node], ONE)


@pytest.mark.parametrize("M", [1, 5, 160])
@pytest.mark.parametrize("D,heads,kv,f16", [(128, 32, 8, 1), (64, 14, 2, 1), (64, 3, 1, 0), (6, 5, 3, 1)])
def test_ropes_and_cache_writes(ctx, M, D, heads, kv, f16):
    rng = np.random.default_rng(M + D)
    rows = 300
    bufs = {n: rng.standard_normal(M * w * D).astype(np.float32) for n, w in (("q", heads), ("k", kv), ("v", kv), ("qr", heads), ("kr", kv))}
    bufs["pos"] = rng.integers(0, 4096, M).astype(np.int32)
    idx = rng.permutation(rows)[:M].astype(np.int64)
    if M > 1:
        idx[1] = rows + 7          # reported, not written
    bufs["idx"], bufs["status"] = idx, np.array([0, 0xFFFFFFFF], np.uint32)
    bufs["kc"], bufs["vc"] = (rng.standard_normal(rows * kv * D).astype(np.float16 if f16 else np.float32) for _ in range(2))
    q, k = rope("q", "qr", D, heads, M), rope("k", "kr", D, kv, M)
    ks, vs = store("kr", "kc", kv * D, M, rows, f16), store("v", "vc", kv * D, M, rows, f16, node=9)
    out = check(ctx, bufs, [q, k, ks, vs])
    assert list(out["status"].view(np.uint32)) == ([2, 3] if M > 1 else [0, 0xFFFFFFFF])
    for ops in ([q, k, vs, ks], [k, ks, q, vs], [q, k], [ks, vs], [k, vs, q, ks, rope("q", "kr2", D, heads, M)],
                [rope("q", "q", D, heads, M, neox=0), rope("k", "k", D, kv, M, neox=0), store("k", "kc", kv * D, M, rows, f16), vs],
                [q, rope("qr", "q", D, heads, M), k, ks],          # the second reads what the first writes
                [k, store("kr", "kc", kv * D, M, rows, f16), store("kr", "vc", kv * D, M, rows, f16)],   # one result stored twice
                [k, rope("k", "k", D, kv, M), vs]):                # writes what the first reads
        b = dict(bufs, kr2=np.zeros(M * heads * D, np.float32))
        check(ctx, b, ops)


QUANT = {("a8", 0): "ameva_quant_a8", ("a8", 1): "ameva_quant_a8_f16", ("a8b", 0): "ameva_quant_a8b", ("a8b", 1): "ameva_quant_a8b_f16"}


def quant(scheme, f16, src, dst, M, K, bufs, stride=None, mode=0):
    ab = M * (K // 256) * 48 if scheme == "a8b" else M * (K // 32) * 4
    for name, size in ((dst + "q", M * K), (dst + "d", ab), (dst + "h", M * K * 2), (dst + "e", M * 4)):
        bufs[name] = np.zeros(size, np.uint8)
    return (QUANT[scheme, f16], [src, dst + "q", dst + "d"] + ([dst + "h", dst + "e"] if f16 else []), [M, K, stride or K, mode], ONE)


@pytest.mark.parametrize("scheme", ["a8", "a8b"])
@pytest.mark.parametrize("M,K,f16", [(1, 256, 0), (1, 4864, 0), (8, 1024, 0), (1, 11008, 0), (9, 256, 1), (40, 2304, 1), (12, 14336, 1)])
def test_quantizes_of_the_same_rows(ctx, scheme, M, K, f16):
    rng = np.random.default_rng(K + M)
    bufs = {n: (rng.standard_normal(M * K) * 2).astype(np.float32) for n in ("x", "gate", "up")}
    bufs.update(y=np.zeros(M * K, np.float32), w=rng.standard_normal(K).astype(np.float32))
    qs = [quant(scheme, f16, "y", f"m{j}", M, K, bufs) for j in range(5)]
    other = quant("a8b" if scheme == "a8" and K % 256 == 0 else "a8", f16, "y", "o", M, K, bufs)
    gate = ("ameva_swiglu_f32", ["gate", "up", "y"], [M * K], ONE)
    norm = (f"ameva_rms_norm_quant_{scheme}", ["x", "w", "y", "nq", "nd", "nh", "ne"], [M, K, K, 0, fbits(1e-5), 1, f16], (M, 1, 1))
    for a, b in zip("qdhe", "qdhe"):
        bufs["n" + a] = np.zeros_like(bufs["m0" + b])
    out = check(ctx, bufs, [gate] + qs[:1])
    assert any(out["m0q"])
    for ops in ([gate] + qs, [gate, other] + qs, [norm] + qs, [norm, other, qs[0]], [gate, quant(scheme, f16, "y", "m0", M, K, bufs, mode=1), qs[1]],
                [(gate[0], ["gate", "up", "gate"], gate[2], ONE)] + [(q[0], ["gate"] + q[1][1:], q[2], ONE) for q in qs[:2]],
                [norm, (qs[0][0], ["y"] + norm[1][3:3 + len(qs[0][1]) - 1], qs[0][2], ONE), qs[1]]):     # the same destination twice
        check(ctx, bufs, ops)


@pytest.mark.parametrize("name,unit,rec,act", [("ameva_mmvqb_q6_K", 256, 18, 48), ("ameva_mmvqb_q5_K", 256, 16, 48), ("ameva_mmvqb_iq4_xs", 256, 8, 48),
                                               ("ameva_mmvq_q4_1", 32, 4, 4), ("ameva_mmvqb_q3_K", 256, 14, 48), ("ameva_mmvqb_q2_K", 256, 20, 48)])
@pytest.mark.parametrize("M,N,K", [(1, 9, 256), (1, 130, 4352), (3, 17, 2048), (8, 8, 768)])
def test_byte_decoded_products_with_the_add_behind_them(ctx, name, unit, rec, act, M, N, K):
    rng = np.random.default_rng(N + K)
    u = K // unit
    S = rng.integers(0, 64, (N, u, rec)).astype(np.uint8)
    A = rng.integers(0, 16, (M, u, act)).astype(np.uint8)
    bufs = {"q": rng.integers(0, 16, N * K).astype(np.uint8), "s": S, "aq": rng.integers(0, 256, M * K).astype(np.uint8), "ad": A,
            "o": np.zeros(M * N, np.float32), "e": rng.standard_normal(M * N).astype(np.float32), "r": np.zeros(M * N, np.float32)}
    gemv = (name, ["q", "s", "aq", "ad", "o"], [M, N, K, N], ONE)
    for a, b, out in (("o", "e", "r"), ("e", "o", "r"), ("o", "e", "e"), ("o", "e", "o"), ("o", "o", "r")):
        check(ctx, bufs, [gemv, ("ameva_add_f32", [a, b, out], [M, N, M], ONE)])
    check(ctx, bufs, [gemv, ("ameva_add_f32", ["o", "e", "r"], [M, N, 1], ONE)])      # one row of e over all


@pytest.mark.parametrize("bad", ["gemv", "gemm", "mmv", "mmtc", "quant"])
def test_nothing_behind_a_refused_dispatch_has_run(ctx, bad):
    """A dispatch with arguments its launcher refuses, between two quantizes of the same rows that would otherwise leave in one
    launch: the batch fails there, what is in front has run and what is behind has not."""
    M, K, N = 1, 512, 64
    rng = np.random.default_rng(1)
    bufs = {"x": rng.standard_normal(M * K).astype(np.float32)}
    ops = [i2_s(f"p{j}", "x", M, N, K, rng, bufs, f"o{j}")[0] for j in (0, 1)]
    for n, size in (("w", N * K), ("s", N * K), ("aq", M * K), ("ad", M * K), ("ah", 2 * M * K), ("ae", 4 * M), ("o", 4 * M * N)):
        bufs[n] = np.zeros(size, np.uint8)
    wrong = {"gemv": ("bitnet_gemv_i2_s_l32w1", ["w", "aq", "o", "ad"], [K - 64, N, fbits(0.02), 0, M, N]),       # K % 128
             "gemm": ("bitnet_gemm_i2_s", ["w", "aq", "o", "ad"], [M, 16 * N, K, 16 * N, fbits(0.02)]),            # outputs too small
             "mmv": ("ameva_mmvq_q8_0", ["w", "s", "aq", "ad", "o"], [M, N, K - 1, N]),
             "mmtc": ("ameva_mmtc_q8_0", ["w", "s", "ah", "o", "ae"], [M, N, K, N - 1, 0]),                        # rows closer than N
             "quant": ("ameva_quant_a8", ["o", "aq", "ad"], [M, K, K, 7])}[bad] + (ONE,)
    held = {n: ctx.buffer(data=a) for n, a in bufs.items()}
    batch = ctx.batch(4)
    for name, binds, push, grid in [ops[0], wrong, ops[1]]:
        batch.dispatch(ctx.kernel(name), [held[b] for b in binds], push, grid)
    with pytest.raises(rt.AmevaComputeError):
        batch.submit()
    batch.destroy()
    ctx.synchronize()
    assert any(held["p0q"].read(np.uint8)) and not any(held["p1q"].read(np.uint8)) and not any(held["p1y"].read(np.uint8))
    for b in held.values():
        b.destroy()


def launches(ctx, bufs, ops):
    """How many launches the dispatches leave in when they are one batch."""
    held = {n: ctx.buffer(data=a) for n, a in bufs.items()}
    batch = ctx.batch(len(ops))
    for name, binds, push, grid in ops:
        batch.dispatch(ctx.kernel(name), [held[b] for b in binds], push, grid)
    ev = batch.submit()
    ev.wait()
    n = batch.launches()[0]
    ev.destroy()
    batch.destroy()
    for b in held.values():
        b.destroy()
    return n


def test_number_of_launches(ctx):
    """The forms above leave in fewer launches, aliased operands in as many as before."""
    rng = np.random.default_rng(7)
    K = 512

    def base(M):
        return {n: rng.standard_normal(M * K).astype(np.float32) for n in ("x", "w", "h", "gate", "up", "act")}

    # I2_S: norm, three quantizes and three products (one or two rows: two launches; three rows: the products alone)
    for M, want in ((1, 2), (2, 2), (3, 4)):
        bufs = base(M)
        ops = [("ameva_rms_norm_f32", ["x", "w", "h"], [M, K, fbits(1e-5), 1], ONE)]
        for j, N in enumerate((64, 33, 128)):
            ops += i2_s(f"p{j}", "h", M, N, K, rng, bufs, f"o{j}")
        assert launches(ctx, bufs, ops) == want
    # the quantize writes the rows that it reads: it stays apart from the norm, and so does what follows
    bufs = base(1)
    ops = [("ameva_rms_norm_f32", ["x", "w", "h"], [1, K, fbits(1e-5), 1], ONE)] + i2_s("p0", "h", 1, 64, K, rng, bufs, "o0", y="h")
    assert launches(ctx, bufs, ops) == 3
    # gate, quantize, product and residual: two; with the sum written over the quantized row: three
    bufs = dict(base(1), res=np.zeros(64, np.float32), sum=np.zeros(K, np.float32))
    ops = [("ameva_swiglu_f32", ["gate", "up", "act"], [K], ONE)] + i2_s("d", "act", 1, 64, K, rng, bufs, "tmp")
    add = ("ameva_add_f32", ["tmp", "res", "sum"], [1, 64, 1], ONE)
    assert launches(ctx, bufs, ops + [add]) == 2
    assert launches(ctx, bufs, [(k, ["sum" if b == "dq" else b for b in binds], p, g) for k, binds, p, g in ops] + [add]) == 3
    # ropes and cache writes: one; a rope of the rotated rows: not
    D, kv, heads, M, rows = 64, 2, 14, 3, 40
    bufs = {n: rng.standard_normal(M * c * D).astype(np.float32) for n, c in (("q", heads), ("k", kv), ("v", kv), ("qr", heads), ("kr", kv))}
    bufs.update(pos=np.arange(M, dtype=np.int32), idx=np.arange(M, dtype=np.int64), status=np.array([0, 0xFFFFFFFF], np.uint32))
    bufs.update({c: np.zeros(rows * kv * D, np.float16) for c in ("kc", "vc")})
    q, k = rope("q", "qr", D, heads, M), rope("k", "kr", D, kv, M)
    ks, vs = store("kr", "kc", kv * D, M, rows), store("v", "vc", kv * D, M, rows)
    assert launches(ctx, bufs, [q, k, ks, vs]) == 1
    assert launches(ctx, bufs, [q, rope("qr", "q", D, heads, M), k, ks]) == 2
    # quantizes of the same rows: up to four together, with the gate in front; of other arguments: apart
    for scheme, f16 in (("a8", 0), ("a8", 1), ("a8b", 0), ("a8b", 1)):
        bufs = base(9)
        qs = [quant(scheme, f16, "act", f"m{j}", 9, K, bufs) for j in range(4)]
        gate = ("ameva_swiglu_f32", ["gate", "up", "act"], [9 * K], ONE)
        assert launches(ctx, bufs, qs) == 1 and launches(ctx, bufs, [gate] + qs) == 1
        assert launches(ctx, bufs, [qs[0], quant(scheme, f16, "act", "m1", 9, K, bufs, mode=1)]) == 2
    # a product of a byte-decoded type and the ADD behind it: one; in place of the product: two
    N = 96
    bufs = {"q": np.zeros(N * K, np.uint8), "s": np.zeros(N * (K // 256) * 18, np.uint8), "aq": np.zeros(K, np.uint8),
            "ad": np.zeros(K // 256 * 48, np.uint8), "o": np.zeros(N, np.float32), "e": np.zeros(N, np.float32), "r": np.zeros(N, np.float32)}
    gemv = ("ameva_mmvqb_q6_K", ["q", "s", "aq", "ad", "o"], [1, N, K, N], ONE)
    assert launches(ctx, bufs, [gemv, ("ameva_add_f32", ["o", "e", "r"], [1, N, 1], ONE)]) == 1
    assert launches(ctx, bufs, [gemv, ("ameva_add_f32", ["o", "e", "o"], [1, N, 1], ONE)]) == 2
