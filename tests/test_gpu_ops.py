"""GPU parity tests of the individual kernels, through the C ABI, against the CPU oracle."""
import numpy as np
import pytest

from caten_b200 import _lib as L
from caten_b200 import synthetic as S
from caten_b200._lib import B200Error

pytestmark = pytest.mark.gpu

TYPES = {"f32": 0, "f16": 1, "q4_0": 2, "q8_0": 8}


def make_weight(rng, rows, cols, wtype, std=0.05):
    """Returns (uploadable, ggml_type, raw bytes for the oracle)."""
    if wtype == "f32":
        a = (rng.standard_normal((rows, cols), dtype=np.float32) * np.float32(std))
        return a, 0, a.view(np.uint8).reshape(-1)
    if wtype == "f16":
        a = (rng.standard_normal((rows, cols), dtype=np.float32) * np.float32(std)).astype(np.float16)
        return a, 1, a.view(np.uint8).reshape(-1)
    p = S._rand_packed(rng, rows, cols, wtype, std)
    return p, p.ggml_type, p.data


def acc_check(got, ref32, ref64, slack=4.0, floor=1e-6):
    """`got` must be about as close to the float64 result as the strict-fp32 oracle is."""
    scale = max(1.0, float(np.abs(ref64).max()))
    e_ref = float(np.abs(ref32 - ref64).max())
    e_got = float(np.abs(got - ref64).max())
    assert e_got <= slack * e_ref + floor * scale, (e_got, e_ref)


@pytest.mark.parametrize("wtype", ["q4_0", "q8_0", "f16", "f32"])
def test_dequant_bit_exact(rt, oracle, wtype):
    rng = np.random.Generator(np.random.PCG64(1))
    up, t, raw = make_weight(rng, 37, 160, wtype)
    w = rt.upload_weight(up)
    got = w.dequantize()
    want = oracle.dequant(t, raw, 37 * 160).reshape(37, 160)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    w.close()


def test_dequant_golden_fixture(rt, golden):
    g = golden["gguf_dequant"]
    for name, t, bb in (("q4_0", 2, 18), ("q8_0", 8, 34)):
        w = rt.upload_weight(S.Packed(t, 6, 96, g[f"rand_{name}_raw"]))
        np.testing.assert_array_equal(w.dequantize().view(np.uint32), g[f"rand_{name}"].view(np.uint32))
        w.close()
    w = rt.upload_weight(S.Packed(2, 6, 32, g["edge_q4_0_raw"]))  # zero / subnormal / negative / max scales
    np.testing.assert_array_equal(w.dequantize().view(np.uint32), g["edge_q4_0"].view(np.uint32))
    w.close()
    w = rt.upload_weight(S.Packed(8, 1, 64, g["arange_q8_0_raw"]))  # the reference's own 64-element fixture
    np.testing.assert_array_equal(w.dequantize().reshape(-1), g["arange_q8_0"])
    w.close()


def test_weight_upload_rejects_bad_input(rt):
    with pytest.raises(B200Error) as e:
        rt.upload_weight(S.Packed(12, 4, 64, np.zeros(1000, np.uint8)))
    assert e.value.code == L.EUNSUPPORTED
    with pytest.raises(B200Error):
        rt.upload_weight(S.Packed(2, 4, 48, np.zeros(1000, np.uint8)))  # cols not a multiple of 32


@pytest.mark.parametrize("rows,d", [(1, 128), (7, 768), (33, 1600), (5, 2048)])
def test_layernorm(rt, oracle, rows, d):
    rng = np.random.Generator(np.random.PCG64(rows + d))
    x = rng.standard_normal((rows, d), dtype=np.float32) * 3 + 1
    g = rng.standard_normal(d, dtype=np.float32)
    b = rng.standard_normal(d, dtype=np.float32)
    y = rt.layernorm(rt.transfer_from_array(x), rt.transfer_from_array(g), rt.transfer_from_array(b)).numpy()
    np.testing.assert_allclose(y, oracle.layernorm(x, g, b, mode=0), atol=1e-5, rtol=1e-5)
    acc_check(y, oracle.layernorm(x, g, b, mode=0), oracle.layernorm(x, g, b, mode=2), slack=6.0)


def test_layernorm_golden(rt, golden):
    g = golden["torch_ops"]
    y = rt.layernorm(rt.transfer_from_array(g["ln_x"]), rt.transfer_from_array(g["ln_g"]), rt.transfer_from_array(g["ln_b"])).numpy()
    np.testing.assert_allclose(y, g["ln_y"], atol=1e-5, rtol=1e-2)  # the reference's tolerance


def test_layernorm_unsupported_width(rt):
    x = rt.open_buffer((2, 4100))
    with pytest.raises(B200Error) as e:
        rt.layernorm(x, x, x)
    assert e.value.code == L.EUNSUPPORTED


@pytest.mark.parametrize("dtype", [np.float32, np.int64])
def test_embed(rt, oracle, dtype):
    rng = np.random.Generator(np.random.PCG64(3))
    V, T, d = 301, 24, 192
    wte = rng.standard_normal((V, d), dtype=np.float32)
    wpe = rng.standard_normal((T, d), dtype=np.float32)
    ids = rng.integers(0, V, size=(3, 7))
    ids[1, 2] = V + 5      # outside the vocabulary: zero token row
    ids[2, 0] = -3
    got = rt.embed(rt.transfer_from_array(ids, dtype), rt.transfer_from_array(wte), rt.transfer_from_array(wpe), 5).numpy()
    want = oracle.embedding(ids.astype(np.float32), 5, wte, wpe)
    np.testing.assert_array_equal(got, want)
    if dtype == np.float32:
        frac = ids.astype(np.float32)
        frac[0, 0] += 0.5  # a non-integer id matches no row either
        got = rt.embed(rt.transfer_from_array(frac), rt.transfer_from_array(wte), rt.transfer_from_array(wpe), 5).numpy()
        np.testing.assert_array_equal(got, oracle.embedding(frac, 5, wte, wpe))


def test_argmax(rt, oracle):
    rng = np.random.Generator(np.random.PCG64(4))
    x = rng.standard_normal((5, 50257), dtype=np.float32)
    x[0, [100, 40000]] = 9.0          # tie: lowest index wins
    x[1, :] = 0.25                    # all equal
    x[2, 50256] = 11.0                # last element
    x[3, 0] = 12.0
    got = rt.argmax(rt.transfer_from_array(x)).numpy()
    np.testing.assert_array_equal(got, oracle.argmax(x))
    assert got[0] == 100 and got[1] == 0 and got[2] == 50256 and got[3] == 0


def _argmax_of_256_walkers(row):
    """One walker per index residue mod 256 that keeps its first value and then greater ones, and a tree over the walkers."""
    V = row.size
    c = []
    for r in range(256):
        v, i = -np.inf, V
        for k in range(r, V, 256):
            if i == V or row[k] > v: v, i = row[k], k
        c.append((v, i))
    o = 128
    while o:
        for t in range(o):
            (mv, mi), (ov, oi) = c[t], c[t + o]
            if oi < V and (mi == V or ov > mv or (ov == mv and oi < mi)): c[t] = c[t + o]
        o >>= 1
    return c[0][1]


@pytest.mark.parametrize("rows,V", [(1, 1), (2, 255), (1, 512), (1, 513), (3, 2048), (5, 16385), (74, 8193), (149, 4100), (150, 12287), (149, 12289)])
def test_argmax_however_a_row_is_cut(rt, rows, V):
    """One block that walks a row; one, two and four CTAs per row, one to four parts in them; ties, minus infinity only, and NaNs, which stand where no comparison admits them."""
    rng = np.random.Generator(np.random.PCG64(V))
    x = rng.integers(-40, 40, (rows, V)).astype(np.float32)
    x[0] = -np.inf
    x[-1, rng.integers(0, V, 5)] = np.nan
    x[-1, 0] = np.nan
    got = rt.argmax(rt.transfer_from_array(x)).numpy()
    at = sorted({0, 1 % rows, rows // 2, rows - 1})
    np.testing.assert_array_equal(got[at], [_argmax_of_256_walkers(x[r]) for r in at])
    finite = np.isfinite(x).all(1)
    np.testing.assert_array_equal(got[finite], x[finite].argmax(1))


GEMV_SHAPES = [(96, 128), (200, 768), (1000, 1600), (130, 3072), (77, 6400)]


@pytest.mark.parametrize("wtype", ["q4_0", "q8_0", "f32", "f16"])
@pytest.mark.parametrize("N,K", GEMV_SHAPES)
def test_gemv(rt, oracle, wtype, N, K):
    rng = np.random.Generator(np.random.PCG64(N * 7 + K))
    up, t, raw = make_weight(rng, N, K, wtype)
    Wf = oracle.dequant(t, raw, N * K).reshape(N, K)
    x = rng.standard_normal((1, K), dtype=np.float32) * 2
    bias = rng.standard_normal(N, dtype=np.float32)
    res = rng.standard_normal((1, N), dtype=np.float32)
    w = rt.upload_weight(up)
    dx, db, dr = rt.transfer_from_array(x), rt.transfer_from_array(bias), rt.transfer_from_array(res)
    for act in (L.ACT_NONE, L.ACT_GELU):
        got = rt.linear(w, dx, db, dr, act).numpy()
        r32 = oracle.linear(x, Wf, bias, res, act, mode=0)
        r64 = oracle.linear(x, Wf, bias, res, act, mode=2)
        np.testing.assert_allclose(got, r32, atol=1e-4, rtol=1e-4)
        acc_check(got, r32, r64)
    got = rt.linear(w, dx).numpy()  # no bias, no residual
    np.testing.assert_allclose(got, oracle.linear(x, Wf, mode=0), atol=1e-4, rtol=1e-4)
    w.close()


@pytest.mark.parametrize("wtype", ["q4_0", "q4_1", "q5_0", "q5_1", "q8_0"])
@pytest.mark.parametrize("N,K", [(9, 32), (50, 224), (2000, 4128), (1900, 8192), (591, 8224), (592, 8224), (700, 10240), (593, 11008), (100, 16384)])
def test_gemv_packed_formats_and_launch_shapes(rt, wtype, N, K):
    """A handful of 32-wide blocks per row and up to the most there may be, rows that fit the resident CTAs and rows that do not, one
    to four rows of x.  A product passes through at most 38 roundings: two chains of 16 in its block and their sum, 16 blocks of a
    lane, 5 across lanes."""
    rng = np.random.Generator(np.random.PCG64(N + K))
    up, _, _ = make_weight(rng, N, K, wtype)
    w = rt.upload_weight(up)
    W = w.dequantize().astype(np.float64)
    x, bias, res = rng.standard_normal((4, K), dtype=np.float32), rng.standard_normal(N, dtype=np.float32), rng.standard_normal((4, N), dtype=np.float32)
    bound = 42 * 2.0 ** -24 * (np.abs(x.astype(np.float64)) @ np.abs(W).T + np.abs(bias) + np.abs(res))
    # (minima enter as m times the sum of a block's x, and codes without their offset: products are larger than their sum)
    slack = 4.0 if wtype in ("q4_1", "q5_1") else 1.0
    want = res + (x.astype(np.float64) @ W.T + bias)
    db = rt.transfer_from_array(bias)
    for M in (1, 2, 3, 4):
        got = rt.linear(w, rt.transfer_from_array(x[:M]), db, rt.transfer_from_array(res[:M])).numpy()
        assert (np.abs(got - want[:M]) <= slack * bound[:M]).all()
    w.close()


def test_gemv_up_to_four_rows(rt, oracle):
    rng = np.random.Generator(np.random.PCG64(8))
    up, t, raw = make_weight(rng, 300, 1024, "q4_0")
    Wf = oracle.dequant(t, raw, 300 * 1024).reshape(300, 1024)
    x = rng.standard_normal((4, 1024), dtype=np.float32)
    res = rng.standard_normal((4, 300), dtype=np.float32)
    w = rt.upload_weight(up)
    got = rt.linear(w, rt.transfer_from_array(x), None, rt.transfer_from_array(res)).numpy()
    np.testing.assert_allclose(got, oracle.linear(x, Wf, None, res, mode=0), atol=1e-4, rtol=1e-4)
    w.close()


@pytest.mark.parametrize("wtype", ["q4_0", "q8_0", "f32", "f16"])
@pytest.mark.parametrize("M,N,K", [(2, 77, 3072), (3, 1301, 768), (4, 6402, 64), (4, 5000, 1600), (1, 9001, 1600)])
def test_gemv_rows_share_the_weights(rt, oracle, wtype, M, N, K):
    """One to four rows of x; a CTA's rows once, several loads deep and walked, the last ones partial."""
    rng = np.random.Generator(np.random.PCG64(M * N + K))
    up, t, raw = make_weight(rng, N, K, wtype)
    Wf = oracle.dequant(t, raw, N * K).reshape(N, K)
    x, bias, res = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal(N, dtype=np.float32), rng.standard_normal((M, N), dtype=np.float32)
    w = rt.upload_weight(up)
    got = rt.linear(w, rt.transfer_from_array(x), rt.transfer_from_array(bias), rt.transfer_from_array(res), L.ACT_GELU).numpy()
    np.testing.assert_allclose(got, oracle.linear(x, Wf, bias, res, L.ACT_GELU, mode=0), atol=1e-4, rtol=1e-4)
    w.close()


def test_gemv_large_activations_and_zero_scale(rt, oracle):
    """The Q4_0 path pre-scales x by powers of two: large and tiny activations must survive."""
    rng = np.random.Generator(np.random.PCG64(9))
    up, t, raw = make_weight(rng, 64, 256, "q4_0")
    Wf = oracle.dequant(t, raw, 64 * 256).reshape(64, 256)
    w = rt.upload_weight(up)
    for mag in (1e-12, 1e-3, 1e6, 1e12):
        x = rng.standard_normal((1, 256), dtype=np.float32) * np.float32(mag)
        got = rt.linear(w, rt.transfer_from_array(x)).numpy()
        ref = oracle.linear(x, Wf, mode=2)
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    w.close()


SIMT_CASES = [("f32", 5, 96, 64), ("q4_0", 70, 200, 256), ("q8_0", 33, 130, 128), ("f16", 9, 64, 96)]


@pytest.mark.parametrize("wtype,M,N,K", SIMT_CASES)
def test_gemm_fp32_is_bit_exact(rt, oracle, wtype, M, N, K):
    """PREC_FP32 accumulates k in ascending order with a rounded multiply and a rounded add:
    the same arithmetic as the reference's rendered C loop, hence identical bits."""
    rng = np.random.Generator(np.random.PCG64(M + N + K))
    up, t, raw = make_weight(rng, N, K, wtype)
    Wf = oracle.dequant(t, raw, N * K).reshape(N, K)
    x = rng.standard_normal((M, K), dtype=np.float32)
    bias = rng.standard_normal(N, dtype=np.float32)
    res = rng.standard_normal((M, N), dtype=np.float32)
    w = rt.upload_weight(up)
    dx, db, dr = rt.transfer_from_array(x), rt.transfer_from_array(bias), rt.transfer_from_array(res)
    got = rt.linear(w, dx, db, dr, L.ACT_RELU, L.PREC_FP32).numpy()
    want = oracle.linear(x, Wf, bias, res, 2, mode=0)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    got = rt.linear(w, dx, db, None, L.ACT_GELU, L.PREC_FP32).numpy()
    np.testing.assert_allclose(got, oracle.linear(x, Wf, bias, None, 1, mode=0), atol=2e-6, rtol=2e-6)
    w.close()


TC_CASES = [("q4_0", 256, 1600, 6400), ("q4_0", 32, 1600, 1600), ("q4_0", 8, 128, 64), ("q4_0", 5, 200, 128), ("q4_0", 64, 4800, 1600), ("q8_0", 33, 130, 192),
            ("f32", 130, 256, 128), ("f16", 17, 128, 64), ("q4_0", 300, 384, 256), ("q8_0", 256, 256, 768)]


@pytest.mark.parametrize("wtype,M,N,K", TC_CASES)
@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
def test_gemm_tensor_core(rt, oracle, wtype, M, N, K, prec):
    rng = np.random.Generator(np.random.PCG64(M * 3 + N + K))
    up, t, raw = make_weight(rng, N, K, wtype)
    Wf = oracle.dequant(t, raw, N * K).reshape(N, K)
    x = rng.standard_normal((M, K), dtype=np.float32)
    bias = rng.standard_normal(N, dtype=np.float32) * 0.1
    res = rng.standard_normal((M, N), dtype=np.float32) * 0.1
    w = rt.upload_weight(up)
    dx, db, dr = rt.transfer_from_array(x), rt.transfer_from_array(bias), rt.transfer_from_array(res)
    oracle.set_threads(8)
    ref_lin = oracle.linear(x, Wf, mode=0)
    ref = oracle.linear(x, Wf, bias, res, 1, mode=0)
    oracle.set_threads(1)
    got_lin = rt.linear(w, dx, None, None, L.ACT_NONE, L.PRECISIONS[prec]).numpy()
    got = rt.linear(w, dx, db, dr, L.ACT_GELU, L.PRECISIONS[prec]).numpy()
    rt.sync()
    tol = 2e-2 if prec == "bf16" else 1e-4   # relative to the largest output
    assert np.abs(got_lin - ref_lin).max() <= tol * np.abs(ref_lin).max()
    assert np.abs(got - ref).max() <= tol * max(1.0, np.abs(ref).max())
    w.close()


# thousands of rows: the weights are expanded to bf16 once and both operands reach the tensor cores through TMA
# (persistent kernel, two accumulators).  Ragged rows and features, every weight format, both precisions.
MANY_ROW_CASES = [("q4_0", 2048, 2560, 1600), ("q4_0", 2000, 2500, 768), ("q8_0", 1100, 4800, 128), ("q5_1", 1500, 3200, 256),
                  ("f32", 1024, 4864, 192), ("f16", 4100, 1200, 64),
                  ("q4_0", 1665, 260, 1088), ("q4_0", 1537, 2560, 5184)]   # (long rows: the converting GEMM)


@pytest.mark.parametrize("wtype,M,N,K", MANY_ROW_CASES)
@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
def test_gemm_tensor_core_many_rows(rt, oracle, wtype, M, N, K, prec):
    rng = np.random.Generator(np.random.PCG64(M + 7 * N + K))
    up, t, raw = make_weight(rng, N, K, wtype)
    Wf = oracle.dequant(t, raw, N * K).reshape(N, K)
    x = rng.standard_normal((M, K), dtype=np.float32)
    bias = rng.standard_normal(N, dtype=np.float32) * 0.1
    res = rng.standard_normal((M, N), dtype=np.float32) * 0.1
    w = rt.upload_weight(up)
    dx, db, dr = rt.transfer_from_array(x), rt.transfer_from_array(bias), rt.transfer_from_array(res)
    ref_lin = (x.astype(np.float64) @ Wf.T.astype(np.float64))
    got_lin = rt.linear(w, dx, None, None, L.ACT_NONE, L.PRECISIONS[prec]).numpy()
    got = rt.linear(w, dx, db, dr, L.ACT_GELU, L.PRECISIONS[prec]).numpy()
    rt.sync()
    tol = 2e-2 if prec == "bf16" else 1e-4   # relative to the largest output
    assert np.abs(got_lin - ref_lin).max() <= tol * np.abs(ref_lin).max()
    # bias, GELU (as the reference composes it) and residual on a sample of rows through the oracle
    rows = np.unique(np.concatenate([np.arange(0, 8), np.arange(M - 8, M), rng.integers(0, M, 48)]))
    ref = oracle.linear(x[rows], Wf, bias, res[rows], 1, mode=0)
    assert np.abs(got[rows] - ref).max() <= tol * max(1.0, np.abs(ref).max())
    # and everywhere against the kernel's own un-fused result
    z = got_lin + bias
    full = res + 0.5 * z * (1.0 + np.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))
    assert np.abs(got - full).max() <= 1e-4 * max(1.0, np.abs(full).max())
    w.close()


def test_gemm_many_rows_matches_the_tile_per_cta_kernel(oracle, monkeypatch):
    """CATEN_B200_DENSE_GEMM=0 sends many-row linears through the decode GEMM (weights dequantised inside the
    kernel): the two kernels must agree to split-bf16 accuracy, and relu(matmul) likewise."""
    from caten_b200.runtime import B200Runtime
    rng = np.random.Generator(np.random.PCG64(91))
    up, _, _ = make_weight(rng, 2560, 1600, "q4_0")
    x = rng.standard_normal((2048, 1600), dtype=np.float32)
    a, b = S.synth_relu_gemm(seed=1, M=4096, K=768, N=3072)
    outs = []
    for flag in ("1", "0"):
        monkeypatch.setenv("CATEN_B200_DENSE_GEMM", flag)
        with B200Runtime(0) as r2:
            w = r2.upload_weight(up)
            y = r2.linear(w, r2.transfer_from_array(x), None, None, L.ACT_NONE, L.PREC_BF16X3).numpy()
            c = r2.relu_matmul(r2.transfer_from_array(a), r2.transfer_from_array(b), L.PREC_BF16X3).numpy()
            r2.sync()
            outs.append((y, c))
            w.close()
    assert np.abs(outs[0][0] - outs[1][0]).max() <= 1e-4 * np.abs(outs[1][0]).max()
    assert np.abs(outs[0][1] - outs[1][1]).max() <= 1e-4 * np.abs(outs[1][1]).max()
    ref = np.maximum(a[:64].astype(np.float64) @ b.astype(np.float64), 0.0)
    np.testing.assert_allclose(outs[0][1][:64], ref, atol=1e-5, rtol=1e-5)   # test-gemm.lisp:3-22


@pytest.mark.parametrize("wtype", ["q8_0", "f16", "bf16"])
@pytest.mark.parametrize("prec,tol", [(L.PREC_BF16X3, 1e-4), (L.PREC_BF16, 4e-2)])
@pytest.mark.parametrize("M,N,K", [(2400, 2052, 2048), (2561, 4100, 1088), (1793, 260, 64), (1537, 508, 320), (1700, 2052, 192), (2049, 2300, 640)])
def test_gemm_pairs_of_ctas(rt, monkeypatch, wtype, prec, tol, M, N, K):
    """Tiles of 256 features by two CTAs, the second one partly or wholly past the last feature, rows that end within a half, one
    stage of k and more than the ring holds; every instance of the kernel, whatever the expected time, and the same linear with
    one CTA per tile.  Sums of K products of unit variance over sqrt(K): rounding errors of a few 2^-16, or of 2^-9 with both
    operands in bf16."""
    import re
    import torch
    from torch.profiler import ProfilerActivity, profile
    from caten_b200.runtime import B200Runtime
    rng = np.random.Generator(np.random.PCG64(M + N))
    if wtype == "bf16":
        raw = (rng.standard_normal((N, K), dtype=np.float32) * K ** -0.5).view(np.uint32) >> 16
        up = S.Packed(L.BF16, N, K, np.ascontiguousarray(raw.astype(np.uint16)).view(np.uint8).reshape(-1))
    else:
        up, _, _ = make_weight(rng, N, K, wtype, std=K ** -0.5)
    x, bias, res = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal(N, dtype=np.float32), rng.standard_normal((M, N), dtype=np.float32)
    for mode in ("2", "0"):
        monkeypatch.setenv("CATEN_B200_DENSE_PAIR", mode)
        with B200Runtime(0) as r:
            w = r.upload_weight(up)
            dx, db, dr = r.transfer_from_array(x), r.transfer_from_array(bias), r.transfer_from_array(res)
            want = res + (x.astype(np.float64) @ w.dequantize().astype(np.float64).T + bias)
            r.sync()
            with profile(activities=[ProfilerActivity.CUDA]) as p:
                got = r.linear(w, dx, db, dr, precision=prec).numpy()
                torch.cuda.synchronize()
            assert np.abs(got - want).max() < tol
            kernels = [m.groups() for m in (re.search(r"gemm_dense_kernel<(\d), (\w+), (\w+), (\w+)>", e.name) for e in p.events()) if m]
            split, lo = ("3", "false" if wtype == "bf16" else "true") if prec == L.PREC_BF16X3 else ("1", "false")
            assert kernels == [(split, "false", lo, "true" if mode == "2" else "false")]
            w.close()


def test_gemm_tensor_core_split_k_is_deterministic(rt):
    """Few output tiles and a long inner dimension: several CTAs share a tile (split-K) and the
    last one to finish adds the partial tiles in a fixed order, so repeated runs give equal bits."""
    rng = np.random.Generator(np.random.PCG64(33))
    up, _, _ = make_weight(rng, 256, 6400, "q4_0")
    w = rt.upload_weight(up)
    dx = rt.transfer_from_array(rng.standard_normal((64, 6400), dtype=np.float32))
    first = rt.linear(w, dx, None, None, L.ACT_NONE, L.PREC_BF16X3).numpy()
    for _ in range(5):
        again = rt.linear(w, dx, None, None, L.ACT_NONE, L.PREC_BF16X3).numpy()
        np.testing.assert_array_equal(first.view(np.uint32), again.view(np.uint32))
    w.close()


def test_gemm_tensor_core_in_place_residual(rt, oracle):
    rng = np.random.Generator(np.random.PCG64(21))
    up, t, raw = make_weight(rng, 128, 128, "q4_0")
    Wf = oracle.dequant(t, raw, 128 * 128).reshape(128, 128)
    x = rng.standard_normal((40, 128), dtype=np.float32)
    h = rng.standard_normal((40, 128), dtype=np.float32)
    w = rt.upload_weight(up)
    dh = rt.transfer_from_array(h)
    rt.linear(w, rt.transfer_from_array(x), None, dh, L.ACT_NONE, L.PREC_BF16X3, out=dh)
    ref = oracle.linear(x, Wf, None, h, mode=0)
    assert np.abs(dh.numpy() - ref).max() <= 1e-4 * np.abs(ref).max()
    w.close()


@pytest.mark.parametrize("prec,tol", [("fp32", 0.0), ("bf16x3", 1e-5), ("bf16", 2e-2)])
def test_relu_matmul(rt, oracle, prec, tol):
    a, b = S.synth_relu_gemm(seed=1, M=200, K=768, N=384)
    oracle.set_threads(8)
    ref = oracle.relu_matmul(a, b, mode=0)
    oracle.set_threads(1)
    got = rt.relu_matmul(rt.transfer_from_array(a), rt.transfer_from_array(b), L.PRECISIONS[prec]).numpy()
    assert (got >= 0).all()
    if prec == "fp32":
        np.testing.assert_array_equal(got.view(np.uint32), ref.view(np.uint32))
    elif prec == "bf16x3":
        np.testing.assert_allclose(got, ref, atol=1e-5, rtol=1e-5)  # test-gemm.lisp:3-22
    else:
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("prec", ["bf16x3", "bf16"])
@pytest.mark.parametrize("M,K,N", [(1537, 64, 68), (1600, 192, 132), (2100, 128, 64), (1536, 320, 1000)])
def test_relu_matmul_of_many_rows(rt, prec, M, K, N):
    """Both operands converted in one launch: partial tiles of b, rows of a that end inside a block of threads.  Products of split
    bf16 are within 2^-15 of sum |a b|, of plain bf16 within 2^-7."""
    rng = np.random.Generator(np.random.PCG64(M + K + N))
    a, b = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((K, N), dtype=np.float32)
    got = rt.relu_matmul(rt.transfer_from_array(a), rt.transfer_from_array(b), L.PRECISIONS[prec]).numpy()
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    assert (np.abs(got - np.maximum(a64 @ b64, 0)) <= 2.0 ** (-15 if prec == "bf16x3" else -7) * (np.abs(a64) @ np.abs(b64))).all()


def test_relu_matmul_golden(rt, golden):
    g = golden["torch_ops"]
    a = np.zeros((37, 64), np.float32); a[:] = g["mm_a"]
    got = rt.relu_matmul(rt.transfer_from_array(a), rt.transfer_from_array(g["mm_b"]), L.PREC_FP32).numpy()
    np.testing.assert_allclose(got, g["relu_mm_c"], atol=1e-5, rtol=1e-5)


def _to_gpu_cache(c):  # oracle [B,T,H,hd] -> device [B,H,T,hd]
    return np.ascontiguousarray(c.transpose(0, 2, 1, 3))


@pytest.mark.parametrize("B,H,T", [(1, 1, 16), (3, 2, 40), (2, 12, 300)])
def test_attention_decode_steps(rt, oracle, B, H, T):
    rng = np.random.Generator(np.random.PCG64(B + H + T))
    d = H * 64
    kc = np.zeros((B, T, H, 64), np.float32)
    vc = np.zeros_like(kc)
    dk, dv = rt.open_buffer((B, H, T, 64)), rt.open_buffer((B, H, T, 64))
    n0 = T - 6
    if n0 > 0:  # pre-existing context
        kc[:, :n0] = rng.standard_normal((B, n0, H, 64), dtype=np.float32)
        vc[:, :n0] = rng.standard_normal((B, n0, H, 64), dtype=np.float32)
        dk.close(); dv.close()
        dk, dv = rt.transfer_from_array(_to_gpu_cache(kc)), rt.transfer_from_array(_to_gpu_cache(vc))
    for n in range(max(n0, 0), T):
        qkv = rng.standard_normal((B, 3 * d), dtype=np.float32)
        want = oracle.attention(qkv, kc, vc, B, 1, n, H, mode=0)
        got = rt.attention(rt.transfer_from_array(qkv), dk, dv, B, 1, n).numpy()
        np.testing.assert_allclose(got, want, atol=1e-5, rtol=1e-5)
    np.testing.assert_array_equal(dk.numpy(), _to_gpu_cache(kc))
    np.testing.assert_array_equal(dv.numpy(), _to_gpu_cache(vc))


@pytest.mark.parametrize("B,H,T", [(1, 2, 1030), (1, 25, 515), (2, 3, 259), (5, 30, 130), (4, 74, 103), (3, 99, 103), (1, 4, 99), (2, 60, 1000)])
def test_attention_decode_shared_histories(rt, oracle, B, H, T):
    """One to eight CTAs per history, around the lengths and the numbers of heads and sequences where their number and the kernel change;
    histories of one round of a half-warp's rows and of several."""
    test_attention_decode_steps(rt, oracle, B, H, T)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_attention_decode_from_any_float(rt, oracle, offset):
    """qkv may start between two 16-byte boundaries, also where few heads and sequences would be read in such pieces."""
    B, H, T = 2, 3, 140
    rng = np.random.Generator(np.random.PCG64(offset))
    kc, vc = (rng.standard_normal((B, T, H, 64), dtype=np.float32) for _ in range(2))
    dk, dv = rt.transfer_from_array(_to_gpu_cache(kc)), rt.transfer_from_array(_to_gpu_cache(vc))
    for n in (0, 17, T - 1):
        qkv = rng.standard_normal((B, 3 * H * 64), dtype=np.float32)
        want = oracle.attention(qkv, kc, vc, B, 1, n, H, mode=0)
        moved = rt.transfer_from_array(np.concatenate([np.zeros(offset, np.float32), qkv.ravel()])).view(offset, qkv.shape)
        np.testing.assert_allclose(rt.attention(moved, dk, dv, B, 1, n).numpy(), want, atol=1e-5, rtol=1e-5)
    np.testing.assert_array_equal(dk.numpy(), _to_gpu_cache(kc))


def test_attention_refuses_addresses_that_its_kernels_cannot_read(rt):
    """Refused on the host, before anything is launched."""
    B, H, T = 1, 2, 20
    cache = [rt.open_buffer((B * H * T * 64 + 4,), np.float32) for _ in range(2)]
    qkv = rt.open_buffer((2 * 3 * H * 64 + 4,), np.float32)
    shape = (B, H, T, 64)
    for s, q, k, v in ((1, 0, 1, 0), (1, 0, 0, 2), (2, 0, 3, 0), (2, 1, 0, 0)):
        with pytest.raises(B200Error) as e:
            rt.attention(qkv.view(q, (B * s, 3 * H * 64)), cache[0].view(k, shape), cache[1].view(v, shape), B, s, 0)
        assert e.value.code == L.EINVAL
    for b in (*cache, qkv):
        b.close()


@pytest.mark.parametrize("B,H,n,at", [(1, 4, 5, 5), (1, 4, 5, 2), (1, 4, 20, 3), (1, 4, 140, 130), (1, 4, 140, 5), (2, 30, 140, 77), (5, 30, 139, 130), (5, 70, 20, 3)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_attention_decode_of_scores_that_are_no_numbers(rt, B, H, n, at, value):
    """One key with a NaN or an infinity: a NaN score makes its head's output NaN wherever it lies (a half-warp's only row, a part of
    a cluster's, among others), a score of -inf counts nothing, one of +inf gives NaN; the other heads do not notice."""
    T = n + 3
    rng = np.random.Generator(np.random.PCG64(n + at))
    kc, vc = (rng.standard_normal((B, H, T, 64), dtype=np.float32) for _ in range(2))
    qkv = np.abs(rng.standard_normal((B, 3, H, 64), dtype=np.float32))
    b, h = B - 1, H // 2
    if at == n:
        qkv[b, 1, h, 7] = value
    else:
        kc[b, h, at, 7] = value
    got = rt.attention(rt.transfer_from_array(qkv.reshape(B, -1)), rt.transfer_from_array(kc), rt.transfer_from_array(vc), B, 1, n).numpy().reshape(B, H, 64)
    kc[:, :, n], vc[:, :, n] = qkv[:, 1], qkv[:, 2]
    with np.errstate(invalid="ignore"):
        s = np.einsum("bhd,bhtd->bht", qkv[:, 0].astype(np.float64), kc[:, :, :n + 1].astype(np.float64)) * 0.125
        p = np.exp(s - s.max(-1, keepdims=True))
        want = np.einsum("bht,bhtd->bhd", p / p.sum(-1, keepdims=True), vc[:, :, :n + 1].astype(np.float64))
    assert np.isnan(want[b, h]).all() == (value != -np.inf)
    np.testing.assert_allclose(got, want, atol=1e-5, rtol=1e-5)


def test_attention_prefill_tensor_cores_in_groups(rt):
    """Histories so long that the operand tiles of one sequence fill the memory they are given."""
    torch = pytest.importorskip("torch")
    B, H, s, n = 2, 20, 65, 16300
    g = torch.Generator().manual_seed(5)
    k, v = (torch.randn(B, H, n + s, 64, generator=g) for _ in range(2))
    q = torch.randn(B, H, s, 64, generator=g)
    rows = torch.cat([a.transpose(1, 2).reshape(B * s, H * 64) for a in (q, k[:, :, n:], v[:, :, n:])], 1)
    want = torch.nn.functional.scaled_dot_product_attention(q, k, v, attn_mask=torch.ones(s, n + s, dtype=torch.bool).tril(n))
    kc, vc = (rt.transfer_from_array(torch.cat([a[:, :, :n], torch.zeros(B, H, s, 64)], 2).numpy()) for a in (k, v))
    got = rt.attention(rt.transfer_from_array(rows.numpy()), kc, vc, B, s, n, precision=L.PREC_BF16X3).numpy()
    np.testing.assert_allclose(got, want.transpose(1, 2).reshape(B * s, H * 64).numpy(), atol=2e-5, rtol=2e-5)
    np.testing.assert_array_equal(kc.numpy(), k.numpy())


@pytest.mark.parametrize("B,H,T,s,n", [(2, 2, 64, 5, 0), (1, 3, 200, 64, 0), (2, 1, 200, 70, 9), (1, 2, 300, 130, 40), (1, 1, 8, 2, 6)])
def test_attention_prefill(rt, oracle, B, H, T, s, n):
    rng = np.random.Generator(np.random.PCG64(B + H + T + s + n))
    d = H * 64
    kc = np.zeros((B, T, H, 64), np.float32)
    vc = np.zeros_like(kc)
    kc[:, :n] = rng.standard_normal((B, n, H, 64), dtype=np.float32)
    vc[:, :n] = rng.standard_normal((B, n, H, 64), dtype=np.float32)
    dk, dv = rt.transfer_from_array(_to_gpu_cache(kc)), rt.transfer_from_array(_to_gpu_cache(vc))
    qkv = rng.standard_normal((B * s, 3 * d), dtype=np.float32)
    want = oracle.attention(qkv, kc, vc, B, s, n, H, mode=0)
    got = rt.attention(rt.transfer_from_array(qkv), dk, dv, B, s, n).numpy()
    np.testing.assert_allclose(got, want, atol=1e-5, rtol=1e-5)
    np.testing.assert_array_equal(dk.numpy(), _to_gpu_cache(kc))
    np.testing.assert_array_equal(dv.numpy(), _to_gpu_cache(vc))


@pytest.mark.parametrize("B,H,T,s,n", [(2, 2, 64, 5, 0), (1, 3, 200, 64, 0), (2, 1, 200, 70, 9), (1, 2, 300, 130, 40),
                                       (1, 1, 8, 2, 6), (2, 2, 600, 300, 0), (1, 2, 700, 257, 391), (1, 1, 1024, 128, 896),
                                       (3, 1, 520, 129, 127)])
def test_attention_prefill_tensor_cores(rt, oracle, B, H, T, s, n):
    """q.K^T and P.V as split-bf16 tensor-core products: within 2^-16-class error of the fp32
    statement, the cache append still exact; tiles of 128 queries x 128 keys, so the cases cover
    partial tiles, several tiles, and a history that starts inside a key step."""
    rng = np.random.Generator(np.random.PCG64(B + H + T + s + n))
    d = H * 64
    kc = np.zeros((B, T, H, 64), np.float32)
    vc = np.zeros_like(kc)
    kc[:, :n] = rng.standard_normal((B, n, H, 64), dtype=np.float32)
    vc[:, :n] = rng.standard_normal((B, n, H, 64), dtype=np.float32)
    # stale rows past the end of the context must not leak in (they are masked, and 0 * NaN would show)
    kg, vg = _to_gpu_cache(kc), _to_gpu_cache(vc)
    kg[:, :, n + s:] = np.nan
    vg[:, :, n + s:] = np.nan
    dk, dv = rt.transfer_from_array(kg), rt.transfer_from_array(vg)
    qkv = rng.standard_normal((B * s, 3 * d), dtype=np.float32)
    want = oracle.attention(qkv, kc, vc, B, s, n, H, mode=0)
    for prec in (L.PREC_BF16X3, L.PREC_BF16):
        got = rt.attention(rt.transfer_from_array(qkv), dk, dv, B, s, n, precision=prec).numpy()
        np.testing.assert_allclose(got, want, atol=2e-5, rtol=2e-5)
    np.testing.assert_array_equal(dk.numpy()[:, :, :n + s], _to_gpu_cache(kc)[:, :, :n + s])
    np.testing.assert_array_equal(dv.numpy()[:, :, :n + s], _to_gpu_cache(vc)[:, :, :n + s])


@pytest.mark.parametrize("B,H,T,s,n", [(1, 1, 128, 128, 0), (1, 2, 130, 63, 1), (2, 50, 300, 2, 130), (4, 25, 330, 65, 191), (4, 25, 400, 128, 200), (2, 48, 200, 64, 64),
                                       (1, 2, 160, 129, 0), (2, 25, 400, 130, 64), (2, 25, 512, 256, 200), (10, 40, 700, 255, 400)])
def test_attention_of_few_tokens_without_a_pass_of_tiles(rt, B, H, T, s, n):
    """One and two query tiles whose CTAs split the keys themselves: steps that begin inside, at and behind a block of 64 keys."""
    torch = pytest.importorskip("torch")
    g = torch.Generator().manual_seed(s + n)
    k, v = (torch.randn(B, H, n + s, 64, generator=g) for _ in range(2))
    q = torch.randn(B, H, s, 64, generator=g)
    rows = torch.cat([a.transpose(1, 2).reshape(B * s, H * 64) for a in (q, k[:, :, n:], v[:, :, n:])], 1)
    want = torch.nn.functional.scaled_dot_product_attention(q, k, v, attn_mask=torch.ones(s, n + s, dtype=torch.bool).tril(n))
    end = torch.full((B, H, T - n, 64), float("nan"))   # (what is past the context must not leak in, and stays)
    kc, vc = (rt.transfer_from_array(torch.cat([a[:, :, :n], end], 2).numpy()) for a in (k, v))
    got = rt.attention(rt.transfer_from_array(rows.numpy()), kc, vc, B, s, n, precision=L.PREC_BF16X3).numpy()
    np.testing.assert_allclose(got, want.transpose(1, 2).reshape(B * s, H * 64).numpy(), atol=2e-5, rtol=2e-5)
    for cache, a in ((kc, k), (vc, v)):
        np.testing.assert_array_equal(cache.numpy()[:, :, :n + s], a.numpy())
        assert np.isnan(cache.numpy()[:, :, n + s:]).all()


@pytest.mark.parametrize("B,H,T,s,n,grow", [(2, 2, 600, 300, 0, 1.0), (1, 2, 700, 257, 391, 1.02), (1, 1, 512, 512, 0, 1.01)])
def test_attention_prefill_tensor_cores_moving_maximum(rt, oracle, B, H, T, s, n, grow):
    """Large scores whose maximum keeps rising along the keys (key j scaled by grow^j on top of
    3x inputs): the kernel's reference maximum has to move, and O and the row sums have to be
    rescaled, many times per row."""
    rng = np.random.Generator(np.random.PCG64(7 + s + n))
    d = H * 64
    t = n + s
    ramp = (grow ** np.arange(t, dtype=np.float64)).astype(np.float32)
    ramp = ramp / ramp.max() * 3.0                         # the largest keys are 3x
    kc = np.zeros((B, T, H, 64), np.float32)
    vc = np.zeros_like(kc)
    kc[:, :n] = rng.standard_normal((B, n, H, 64), dtype=np.float32) * ramp[None, :n, None, None]
    vc[:, :n] = rng.standard_normal((B, n, H, 64), dtype=np.float32)
    dk, dv = rt.transfer_from_array(_to_gpu_cache(kc)), rt.transfer_from_array(_to_gpu_cache(vc))
    qkv = rng.standard_normal((B * s, 3 * d), dtype=np.float32)
    qkv[:, :d] *= 3.0
    qkv[:, d:2 * d] = (qkv[:, d:2 * d].reshape(B, s, d) * ramp[None, n:, None]).reshape(B * s, d)
    want = oracle.attention(qkv, kc, vc, B, s, n, H, mode=0)
    got = rt.attention(rt.transfer_from_array(qkv), dk, dv, B, s, n, precision=L.PREC_BF16X3).numpy()
    # scores reach the hundreds here, so the split-bf16 products carry an absolute error of a few 1e-4 in the
    # exponent; the outputs are convex combinations of unit-normal V rows
    np.testing.assert_allclose(got, want, atol=2e-3, rtol=0)


def test_attention_golden_sdpa(rt, golden):
    g = golden["torch_ops"]
    q, k, v = g["sdpa_q"], g["sdpa_k"], g["sdpa_v"]  # [4,4,8,64]
    B, H, T, hd = q.shape
    qkv = np.concatenate([x.transpose(0, 2, 1, 3).reshape(B * T, H * hd) for x in (q, k, v)], axis=1)
    dk, dv = rt.open_buffer((B, H, T, hd)), rt.open_buffer((B, H, T, hd))
    got = rt.attention(rt.transfer_from_array(qkv), dk, dv, B, T, 0).numpy()
    np.testing.assert_allclose(got.reshape(B, T, H, hd).transpose(0, 2, 1, 3), g["sdpa_causal_o"], atol=1e-5, rtol=1e-5)
    got = rt.attention(rt.transfer_from_array(qkv), dk, dv, B, T, 0, precision=L.PREC_BF16X3).numpy()
    np.testing.assert_allclose(got.reshape(B, T, H, hd).transpose(0, 2, 1, 3), g["sdpa_causal_o"], atol=2e-5, rtol=2e-5)


def test_attention_rejects_positions_outside_cache(rt):
    dk, dv = rt.open_buffer((1, 1, 8, 64)), rt.open_buffer((1, 1, 8, 64))
    qkv = rt.open_buffer((4, 192))
    with pytest.raises(B200Error) as e:
        rt.attention(qkv, dk, dv, 1, 4, 6)
    assert e.value.code == L.EINVAL


def test_open_buffer_is_zero_filled_and_roundtrips(rt):
    b = rt.open_buffer((1000,))
    assert not b.numpy().any()
    a = np.arange(1000, dtype=np.float32)
    c = rt.copy_buffer_value(rt.transfer_from_array(a))
    np.testing.assert_array_equal(c.numpy(), a)
    e = rt.open_buffer((0,))
    assert e.numpy().size == 0


def test_work_can_be_queued_on_a_stream_of_the_caller(oracle):
    """caten_b200_set_stream: the context queues its kernels on a stream the host owns (here a torch stream), then
    returns to its own."""
    torch = pytest.importorskip("torch")
    from caten_b200.runtime import B200Runtime
    rng = np.random.Generator(np.random.PCG64(9))
    up, t, raw = make_weight(rng, 384, 256, "q4_0")
    Wf = oracle.dequant(t, raw, 384 * 256).reshape(384, 256)
    x = rng.standard_normal((3, 256), dtype=np.float32)
    ref = oracle.linear(x, Wf, mode=0)
    with B200Runtime(0) as r2:
        own = r2.stream
        w = r2.upload_weight(up)
        dx = r2.transfer_from_array(x)
        host_stream = torch.cuda.Stream()
        L.check(r2.ctx, r2.lib.caten_b200_set_stream(r2.ctx, host_stream.cuda_stream))
        assert r2.stream == host_stream.cuda_stream
        y1 = r2.linear(w, dx).numpy()
        L.check(r2.ctx, r2.lib.caten_b200_set_stream(r2.ctx, None))
        assert r2.stream == own
        y2 = r2.linear(w, dx).numpy()
        w.close()
    np.testing.assert_array_equal(y1.view(np.uint32), y2.view(np.uint32))
    np.testing.assert_allclose(y1, ref, atol=1e-5, rtol=1e-5)


def test_large_copies_through_the_pinned_bounce_buffers(rt, oracle):
    """Copies of 4 MiB and more from pageable host memory are cut into 16 MiB pieces that alternate between two
    pinned buffers: sizes around the piece boundaries, and a packed weight larger than one piece."""
    rng = np.random.Generator(np.random.PCG64(5))
    for n in ((4 << 20) // 4, (16 << 20) // 4 + 3, (40 << 20) // 4 + 1):
        a = rng.integers(0, 2 ** 31, n, dtype=np.int64).astype(np.float32)
        buf = rt.transfer_from_array(a)
        np.testing.assert_array_equal(buf.numpy().view(np.uint32), a.view(np.uint32))
        buf.close()
    p = S._rand_packed(rng, 4100, 4096, "q8_0")      # 17.8 MB of blocks
    w = rt.upload_weight(p)
    want = oracle.dequant(p.ggml_type, p.data, p.rows * p.cols).reshape(p.rows, p.cols)
    np.testing.assert_array_equal(w.dequantize().view(np.uint32), want.view(np.uint32))
    w.close()


@pytest.mark.parametrize("act", [L.ACT_GELU, L.ACT_NONE])
@pytest.mark.parametrize("M,N,K,offset", [(5, 128, 512, 0), (40, 260, 768, 0), (40, 257, 768, 0), (40, 260, 768, 1), (200, 388, 1024, 0), (300, 132, 512, 2), (1601, 260, 192, 0)])
def test_tensor_core_epilogues_in_fours_and_one_by_one(rt, act, M, N, K, offset):
    """Bias, activation and residual behind every way a sum can end: by a cluster, by the second kernel and in the tile's own
    CTA, with features in aligned fours or not (a width that is no multiple of four, a residual that starts between), large and
    small arguments of GELU.  Split-bf16 products are within 2^-16 of sum |x w|; the activation's slope is at most 1.13."""
    rng = np.random.Generator(np.random.PCG64(M + N + K + offset))
    W = rng.standard_normal((N, K), dtype=np.float32) * np.float32(K ** -0.5)
    x = rng.standard_normal((M, K), dtype=np.float32) * rng.choice(np.float32([0.05, 1.0, 6.0]), (M, 1))
    bias, res = rng.standard_normal(N, dtype=np.float32), rng.standard_normal((M, N), dtype=np.float32)
    w = rt.upload_weight(W)
    dres = rt.transfer_from_array(np.concatenate([np.zeros(offset, np.float32), res.ravel()])).view(offset, (M, N))
    got = rt.linear(w, rt.transfer_from_array(x), rt.transfer_from_array(bias), dres, act, L.PREC_BF16X3).numpy()
    z = x.astype(np.float64) @ W.T.astype(np.float64) + bias
    with np.errstate(over="ignore"):
        want = z / (1 + np.exp(-2 * np.sqrt(2 / np.pi) * (z + 0.044715 * z ** 3))) if act == L.ACT_GELU else z
    bound = 2.0 ** -15 * (np.abs(x).astype(np.float64) @ np.abs(W.T).astype(np.float64)) + 1e-6 * (np.abs(z) + np.abs(res))
    assert (np.abs(got - (want + res)) <= bound).all()
    w.close()


@pytest.mark.parametrize("M,N,K,dtype", [(1, 2304, 768, np.float32), (3, 2304, 768, np.float32), (2, 3840, 1280, np.float32), (1, 1024, 4096, np.float16), (4, 6400, 1600, np.float16)])
def test_dense_gemv_adds_short_chains(rt, M, N, K, dtype):
    """A lane adds its share of a row four products at a time, so that the error against 64 bits (2-norm) stays below what two warps a row
    had (9.3e-8 at 768, 1.27e-7 at 4096 columns; product by product 1.1e-7 and 1.59e-7).  Measured 8.9e-8 to 1.1e-7."""
    rng = np.random.Generator(np.random.PCG64(M + N + K))
    W, x = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(K ** -0.5)).astype(dtype), rng.standard_normal((M, K), dtype=np.float32)
    w = rt.upload_weight(W)
    got, want = rt.linear(w, rt.transfer_from_array(x)).numpy(), x.astype(np.float64) @ W.astype(np.float64).T
    w.close()
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= {768: 1.0e-7, 1280: 1.0e-7, 1600: 1.1e-7, 4096: 1.2e-7}[K], err


@pytest.mark.parametrize("M,precision", [(1, L.PREC_FP32), (5, L.PREC_FP32), (5, L.PREC_BF16X3), (200, L.PREC_BF16X3), (1700, L.PREC_BF16X3)])
def test_activations_over_their_whole_range(rt, M, precision):
    """Weights of zero, so that the activation's argument is the bias.  silu: exp within two ulps, one rounding of the sum and at most one
    ulp of the quotient, down to where exp(-z) overflows; GELU, one form in every kernel and precision: the exponent has
    a few roundings of its own size."""
    z = np.concatenate([np.linspace(-104, 104, 4177), -10.0 ** np.linspace(-30, 30, 301), 10.0 ** np.linspace(-30, 30, 301),
                        [0.0, -0.0, np.inf, -np.inf, np.nan, -83.3, -84.0, -86.0, -87.5, -88.6, -9.5, -9.9, -10.1]]).astype(np.float32)
    z = z[np.abs(z + 88.72) > 0.05]
    z = np.concatenate([z, np.zeros(-len(z) % 4, np.float32)])
    N = len(z)
    x = rt.transfer_from_array(np.ones((M, 64), np.float32))
    w, ww = rt.upload_weight(np.zeros((N, 64), np.float32)), rt.upload_weight(np.zeros((2 * N, 64), np.float32))
    gelu = rt.linear(w, x, rt.transfer_from_array(z), act=L.ACT_GELU, precision=precision).numpy()
    silu = rt.linear(ww, x, rt.transfer_from_array(np.stack([z, np.ones_like(z)], 1).ravel()), act=L.ACT_SILU_GLU, precision=precision, out=rt.open_buffer((M, N), np.float32)).numpy()
    with np.errstate(all="ignore"):
        z64 = z.astype(np.float64)
        e = np.exp(-z64)
        want = z64 / (1 + np.where(e > np.finfo(np.float32).max, np.inf, e))
        a = 2 * np.sqrt(2 / np.pi) * (z64 + 0.044715 * z64 ** 3)
        wg = z64 / (1 + np.where(-a > 127.99 * np.log(2), np.inf, np.exp(-a)))
        bound = (2.0 ** -20 + 2.0 ** -21 * np.minimum(np.abs(a), 200)) * np.abs(wg) + 2.0 ** -100
        for row in (0, M - 1):
            np.testing.assert_array_equal(np.isnan(silu[row]), np.isnan(want))
            np.testing.assert_array_equal(np.isnan(gelu[row]), np.isnan(wg))
            ok = (silu[row] == want) | np.isnan(want) | (np.abs(silu[row] - want) <= 2.0 ** -21 * np.abs(want))
            assert ok.all(), (z[~ok][:5], silu[row][~ok][:5], want[~ok][:5])
            ok = (gelu[row] == wg) | np.isnan(wg) | (np.abs(gelu[row] - wg) <= bound)
            assert ok.all(), (z[~ok][:5], gelu[row][~ok][:5], wg[~ok][:5])
    w.close(); ww.close()


def test_gemm_split_k_cluster_reduction_matches_global_reduction(oracle, monkeypatch):
    """CATEN_B200_SPLITK_CLUSTER=1 reduces split-K partial tiles inside a thread-block cluster
    (distributed shared memory) instead of a second kernel: same splits order, same epilogue."""
    from caten_b200.runtime import B200Runtime
    rng = np.random.Generator(np.random.PCG64(77))
    up, t, raw = make_weight(rng, 1600, 1600, "q4_0")
    x = rng.standard_normal((40, 1600), dtype=np.float32)
    bias = rng.standard_normal(1600, dtype=np.float32) * 0.1
    res = rng.standard_normal((40, 1600), dtype=np.float32) * 0.1
    outs = []
    for flag in ("0", "1"):
        monkeypatch.setenv("CATEN_B200_SPLITK_CLUSTER", flag)
        with B200Runtime(0) as r2:
            w = r2.upload_weight(up)
            y = r2.linear(w, r2.transfer_from_array(x), r2.transfer_from_array(bias), r2.transfer_from_array(res), L.ACT_GELU,
                          L.PREC_BF16X3).numpy()
            r2.sync()
            outs.append(y)
            w.close()
    Wf = oracle.dequant(t, raw, 1600 * 1600).reshape(1600, 1600)
    oracle.set_threads(8)
    ref = oracle.linear(x, Wf, bias, res, 1, mode=0)
    oracle.set_threads(1)
    for y in outs:
        assert np.abs(y - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    assert np.abs(outs[0] - outs[1]).max() <= 1e-5


@pytest.mark.parametrize("prec", [L.PREC_FP32, L.PREC_BF16X3])
def test_attention_block_golden(rt, golden, prec):
    """The attention block of source/test-suite/test-llm.lisp:257-301 (c_attn -> heads -> softmax
    attention -> c_proj vs `attn_impl_torch`, atol 1e-4 / rtol 1e-4) at head dim 64 with the causal
    mask of external/llm/layers.lisp:86, through the three C-ABI calls the block lowers to."""
    g = golden["attn_block"]
    x, H = g["hd64_x"], int(g["hd64_heads"])
    B, T, d = x.shape
    wa, wp = rt.upload_weight(g["hd64_wa"]), rt.upload_weight(g["hd64_wp"])
    ba, bp = rt.transfer_from_array(g["hd64_ba"]), rt.transfer_from_array(g["hd64_bp"])
    qkv = rt.linear(wa, rt.transfer_from_array(x.reshape(B * T, d)), ba, precision=prec)
    dk, dv = rt.open_buffer((B, H, T, 64)), rt.open_buffer((B, H, T, 64))
    o = rt.attention(qkv, dk, dv, B, T, 0, precision=prec)
    y = rt.linear(wp, o, bp, precision=prec).numpy()
    np.testing.assert_allclose(y.reshape(B, T, d), g["hd64_y"], atol=1e-4, rtol=1e-4)
    wa.close(); wp.close()


def test_kv_cache_protocol(rt):
    """source/test-suite/test-dynamic-shape.lisp:189-222: a prompt of 10 rows at start_pos 0, then one
    row per call; after every call cache rows [0, start_pos + seq_len) are exactly the rows fed so
    far, in order, and the rest of the cache is still zero."""
    rng = np.random.Generator(np.random.PCG64(4))
    B, T, H = 1, 128, 4
    d = H * 64
    dk, dv = rt.open_buffer((B, H, T, 64)), rt.open_buffer((B, H, T, 64))
    fed_k, fed_v, start = [], [], 0
    for nth in range(10):
        s = 10 if nth == 0 else 1
        qkv = rng.random((B * s, 3 * d), dtype=np.float32)
        rt.attention(rt.transfer_from_array(qkv), dk, dv, B, s, start).close()
        fed_k.append(qkv[:, d:2 * d]); fed_v.append(qkv[:, 2 * d:])
        start += s
        k, v = dk.numpy(), dv.numpy()   # [B, H, T, 64]
        np.testing.assert_array_equal(k[0, :, :start].transpose(1, 0, 2).reshape(start, d), np.concatenate(fed_k))
        np.testing.assert_array_equal(v[0, :, :start].transpose(1, 0, 2).reshape(start, d), np.concatenate(fed_v))
        assert not k[0, :, start:].any() and not v[0, :, start:].any()


@pytest.mark.parametrize("rows,d", [(30, 40), (9, 1600), (3, 4096)])
def test_rmsnorm(rt, oracle, golden, rows, d):
    """`!rms-norm` (source/nn/normalization.lisp:70-85): the oracle within 1e-5, the torchtune function of
    source/test-suite/test-normalization.lisp:57-63 at its tolerance, with and without a weight."""
    g = golden["llama_ops"]
    rng = np.random.Generator(np.random.PCG64(rows + d))
    x = g["rms_ref_x"] if (rows, d) == (30, 40) else g["rms_wide_x"] if (rows, d) == (9, 1600) else rng.standard_normal((rows, d), dtype=np.float32) * 2
    w = (rng.random(d, dtype=np.float32) + 0.5)
    dx = rt.transfer_from_array(x)
    got = rt.rmsnorm(dx).numpy()
    np.testing.assert_allclose(got, oracle.rmsnorm(x), atol=1e-5, rtol=1e-5)
    acc_check(got, oracle.rmsnorm(x), oracle.rmsnorm(x, mode=2))
    if (rows, d) == (30, 40):
        np.testing.assert_allclose(got, g["rms_ref_y"], atol=1e-3, rtol=1e-6)
    np.testing.assert_allclose(rt.rmsnorm(dx, rt.transfer_from_array(w)).numpy(), oracle.rmsnorm(x, w), atol=1e-5, rtol=1e-5)
    with pytest.raises(B200Error):
        rt.rmsnorm(rt.open_buffer((2, 10)))    # d % 4 != 0


@pytest.mark.parametrize("tag", ["ref", "hd64"])
def test_rope(rt, oracle, golden, tag):
    """`!rope` (source/nn/positional-encoding.lisp:3-56): bit-exact against the oracle (the same fp32 formula,
    transcendentals through double), the torchtune function of source/test-suite/test-rope.lisp:60-66 at its
    tolerance, and a continued sequence (pos0 > 0) equal to the tail of the full one."""
    g = golden["llama_ops"]
    x = g[f"rope_{tag}_x"]
    got = rt.rope(rt.transfer_from_array(x)).numpy()
    np.testing.assert_allclose(got, oracle.rope(x), atol=1e-6, rtol=1e-6)
    np.testing.assert_allclose(got, g[f"rope_{tag}_y"], atol=1e-5, rtol=5e-4)
    tail = rt.rope(rt.transfer_from_array(x[:, 4:]), pos0=4).numpy()
    np.testing.assert_array_equal(tail, got[:, 4:])
    odd = np.random.Generator(np.random.PCG64(1)).random((2, 5, 3, 7), dtype=np.float32)
    np.testing.assert_allclose(rt.rope(rt.transfer_from_array(odd)).numpy(), oracle.rope(odd), atol=1e-6, rtol=1e-6)
