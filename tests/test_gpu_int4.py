"""GPU parity of the int4-grouped scheme (row f4) through the C ABI against the CPU oracle: unpacked
nibbles and dequantized weights bit-exact, f32-accumulated outputs within 1e-3 and 16-bit outputs
within 1e-2 on the reference probes' metric |x - ref| / max(1, |ref|); routes counted like the int8
path (m <= 16: fused-dequant GEMV; larger m: explicit dequant + dense matmul)."""
import numpy as np
import pytest

import cases
from launches import launches
from oracle import oracle as orc
from torchlette_b200 import backend as tb

pytestmark = pytest.mark.gpu


def _weight(be, n, k, g, seed):
    rng = np.random.default_rng(seed)
    w = (rng.uniform(-1, 1, (n, k)) * 0.1).astype(np.float32)
    packed, scales = be.quantizeLinearWeight(w, g, scheme="int4-grouped")
    op, os_ = orc.quantize_linear_weight_int4(w, g)
    assert np.array_equal(packed, op) and np.array_equal(scales, os_)
    fmt = tb.StorageFormat("f16", tb.QuantPacking("int4-grouped", g, "f16"))
    return be.createQuantizedWeight(packed, scales, n, k, fmt), orc.dequantize_int4_to_f32(packed, scales, k, g), packed


@pytest.mark.parametrize("n,k,g", [(128, 128, 32), (300, 1024, 128), (33, 64, 8), (1024, 2048, 32)])
def test_int4_unpack_and_dequant_bit_exact(backend, n, k, g):
    be = backend
    w, ref, packed = _weight(be, n, k, g, seed=n + k)
    assert np.array_equal(be.unpackInt4(w, n, k), orc.unpack_int4(packed, k))
    d = be.dequantize(w, "f32")
    assert np.array_equal(be.ops.read(d).view(np.uint32), ref.view(np.uint32))
    h = be.dequantize(w, "f16")
    assert np.array_equal(be.ops.read(h), ref.astype(np.float16))
    for t in (d, h, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("act_dtype,out_dtype", [("f32", "f32"), ("f16", "f32"), ("f16", "f16"), ("bf16", "bf16")])
@pytest.mark.parametrize("m", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("n,k,g", [(128, 128, 32), (512, 1024, 128), (37, 264, 8)])
def test_int4_gemv_matches_oracle(backend, act_dtype, out_dtype, m, n, k, g):
    be = backend
    w, wref, _ = _weight(be, n, k, g, seed=7 * n + k + m)
    rng = np.random.default_rng(m)
    xv = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    if act_dtype == "f16":
        x = be.ops.tensorFromArray(xv.astype(np.float16), [m, k], "f16")
        xv = xv.astype(np.float16).astype(np.float32)
    elif act_dtype == "bf16":
        bits = orc.bf16_bits_rne(xv.reshape(-1))
        x = be.ops.tensorFromArray(bits, [m, k], "bf16")
        xv = orc.bf16_bits_to_f32(bits).reshape(m, k)
    else:
        x = be.ops.tensorFromArray(xv, [m, k], "f32")
    be.resetCounters()
    y = be.linear(x, w, None, None, out_dtype)
    assert be.getQuantGemvDispatchCount() == 1 and be.getDequantI8DispatchCount() == 0
    got = be.ops.read(y)
    got = orc.bf16_bits_to_f32(got) if out_dtype == "bf16" else np.asarray(got, np.float32)
    ref = orc.linear_reference(xv, wref)
    assert cases.rel_err(got, ref) <= (1e-3 if out_dtype == "f32" else 1e-2)
    for t in (x, y, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("act", [None, "relu", "gelu", "silu"])
def test_int4_gemv_epilogue(backend, act):
    be = backend
    n, k, g, m = 256, 512, 32, 4
    w, wref, _ = _weight(be, n, k, g, seed=99)
    rng = np.random.default_rng(5)
    xv = rng.uniform(-1, 1, (m, k)).astype(np.float16)
    bias = rng.uniform(-1, 1, n).astype(np.float32)
    x = be.ops.tensorFromArray(xv, [m, k], "f16")
    bt = be.ops.tensorFromArray(bias, [n], "f32")
    be.resetCounters()
    y = be.linear(x, w, bt, act, "f32")
    assert be.getGemvEpilogueDispatchCount() == 1
    ref = orc.linear_reference(xv.astype(np.float32), wref, bias, act)
    assert cases.rel_err(be.ops.read(y), ref) <= 1e-3
    for t in (x, bt, y, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
def test_int4_large_m_takes_the_dequant_plus_dense_route(backend, dtype):
    be = backend
    n, k, g, m = 256, 512, 128, 96
    w, wref, _ = _weight(be, n, k, g, seed=3)
    rng = np.random.default_rng(8)
    xv = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    if dtype == "f16":
        x = be.ops.tensorFromArray(xv.astype(np.float16), [m, k], "f16")
        xv = xv.astype(np.float16).astype(np.float32)
        wr = wref.astype(np.float16).astype(np.float32)   # the dense operand is the dequantized weight in the activation type
    elif dtype == "bf16":
        bits = orc.bf16_bits_rne(xv.reshape(-1))
        x = be.ops.tensorFromArray(bits, [m, k], "bf16")
        xv = orc.bf16_bits_to_f32(bits).reshape(m, k)
        wr = orc.bf16_bits_to_f32(orc.bf16_bits_rne(wref.reshape(-1))).reshape(n, k)
    else:
        x = be.ops.tensorFromArray(xv, [m, k], "f32")
        wr = wref
    be.resetCounters()
    y = be.linear(x, w, None, "relu", "f32")
    assert be.getQuantGemvDispatchCount() == 0 and be.getDequantI8DispatchCount() == 1
    ref = orc.linear_reference(xv, wr, None, "relu")
    assert cases.rel_err(be.ops.read(y), ref) <= 1e-3
    plan = be.planQuantizedMatmul(m, n, k, dtype, "f32", w.format.packing)
    assert plan["family"] == "gemm"
    assert be.planQuantizedMatmul(4, n, k, dtype, "f32", w.format.packing)["family"] == "gemv"
    for t in (x, y, w.scales, w):
        t.destroy()


def test_int4_argument_errors(backend):
    be = backend
    fmt = tb.StorageFormat("f16", tb.QuantPacking("int4-grouped", 32, "f16"))
    with pytest.raises(tb.TlError):
        be.createQuantizedWeight(np.zeros(10, np.uint32), np.zeros(4, np.uint16), 4, 36, fmt)  # K % 8
    with pytest.raises(tb.TlError):
        be.quantizeLinearWeight(np.zeros((2, 36), np.float32), 12, scheme="int4-grouped")


@pytest.mark.parametrize("m", [1, 8, 16])
@pytest.mark.parametrize("g", [128, 256, 1024])
def test_int4_tensor_core_and_simt_forms_agree(backend, m, g):
    """K and the group multiples of 128 take the mma.sync form; forcing {QGEMV, simt} takes the f32
    form.  Both against the oracle, and against each other within f32 summation-order noise."""
    be = backend
    n, k = 264, 1024
    w, wref, _ = _weight(be, n, k, g, seed=g + m)
    rng = np.random.default_rng(g)
    xv = rng.uniform(-1, 1, (m, k)).astype(np.float16)
    x = be.ops.tensorFromArray(xv, [m, k], "f16")
    y1 = be.linear(x, w, None, None, "f32")
    be.forceVariant((1, 1, 8, 1, 1, 0))
    try:
        y2 = be.linear(x, w, None, None, "f32")
    finally:
        be.forceVariant(None)
    ref = orc.linear_reference(xv.astype(np.float32), wref)
    a, b = be.ops.read(y1), be.ops.read(y2)
    assert cases.rel_err(a, ref) <= 1e-3 and cases.rel_err(b, ref) <= 1e-3
    assert cases.rel_err(a, b) <= 1e-4
    for t in (x, y1, y2, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("act", ["f16", "bf16"])
@pytest.mark.parametrize("g", [32, 64, 128, 384, 0])
@pytest.mark.parametrize("m,n,k", [(1, 1, 128), (1, 17, 384), (2, 500, 1536), (5, 33, 768), (8, 2400, 384), (9, 31, 1152), (16, 1000, 2304)])
def test_int4_ring_edges(backend, act, g, m, n, k):
    """Row tiles cut short, fewer k blocks than warps or ring stages, every group form, against the f32 form of the
    same product.  Both sum the same exact products in f32: K terms of relative size 2^-24 each, four roundings' worth."""
    be = backend
    g = g or k
    if k % g:
        pytest.skip("K is not whole groups")
    w, wref, _ = _weight(be, n, k, g, seed=n + m)
    rng = np.random.default_rng(k + m)
    xv = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    if act == "f16":
        x, xv = be.ops.tensorFromArray(xv.astype(np.float16), [m, k], "f16"), xv.astype(np.float16).astype(np.float64)
    else:
        bits = orc.bf16_bits_rne(xv.reshape(-1))
        x, xv = be.ops.tensorFromArray(bits, [m, k], "bf16"), orc.bf16_bits_to_f32(bits).reshape(m, k).astype(np.float64)
    y = be.linear(x, w, None, None, "f32")
    ref = xv @ wref.astype(np.float64).T
    size = np.abs(xv) @ np.abs(wref.astype(np.float64)).T
    assert (np.abs(be.ops.read(y) - ref) <= size * 2.0 ** -20).all()
    for t in (x, y, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("act", ["f16", "f32"])
@pytest.mark.parametrize("m,n,k,g", [(1, 1000, 4096, 128), (4, 3000, 2048, 128), (4, 12000, 1024, 128), (16, 3000, 2048, 128), (16, 12000, 1024, 1024),
                                     (16, 12000, 1024, 32), (1, 300, 128, 128), (3, 40, 136, 8)])
def test_int4_receipt_is_the_launch(backend, act, m, n, k, g):
    be = backend
    packing = tb.QuantPacking("int4-grouped", g, "f16")
    w = be.ops.empty([n, k // 8], "u32")
    w.scales = be.ops.empty([n, k // g], "u16")
    w.shape, w.dtype, w.format = [n, k], "f16", tb.StorageFormat("f16", packing)
    x, y = be.ops.empty([m, k], act), be.ops.empty([m, n], "f32")
    plan = be.planQuantizedMatmul(m, n, k, act, "f32", packing)
    got = launches(be, lambda: be.ops.matmul(x, be.ops.transpose(w), {"outBuffer": y}))
    assert (plan["grid"], plan["block"]) == got[0]
    for t in (x, y, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("m,n,k", [(11, 300, 1024), (16, 300, 1024), (16, 300, 4096)])
@pytest.mark.parametrize("warps,row_tiles,stages", [(16, 0, 0), (16, 1, 4), (8, 2, 4), (1, 2, 2)])
def test_int4_forced_shapes_run(backend, m, n, k, warps, row_tiles, stages):
    """Every forced CTA width, with stages to fit: the default's result up to the order of f32 sums."""
    be = backend
    w, wref, _ = _weight(be, n, k, 128, seed=m)
    xv = np.random.default_rng(k).uniform(-1, 1, (m, k)).astype(np.float16)
    x = be.ops.tensorFromArray(xv, [m, k], "f16")
    be.forceVariant((1, 9, warps, row_tiles, stages, 0))
    try:
        y = be.linear(x, w, None, None, "f32")
    finally:
        be.forceVariant(None)
    size = np.abs(xv.astype(np.float64)) @ np.abs(wref.astype(np.float64)).T
    assert (np.abs(be.ops.read(y) - xv.astype(np.float64) @ wref.astype(np.float64).T) <= size * 2.0 ** -20).all()
    for t in (x, y, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("out", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("m,n,k,g", [(9, 2400, 384, 32), (16, 2400, 1152, 64), (16, 4700, 256, 32), (9, 4700, 2304, 64), (1, 9500, 1024, 32), (1, 9500, 1024, 64),
                                     (1, 9500, 1024, 128), (16, 9500, 1024, 32), (16, 9500, 1024, 64), (16, 9500, 640, 128), (8, 9480, 128, 64)])
def test_int4_ring_of_few_warps(backend, out, m, n, k, g):
    """Tiles of 32 rows whose scales fold several times a block, and four warps a tile (16-bit outputs; f32 takes more warps), where rows,
    blocks and warps end.  Sums as above; a 16-bit result is rounded once more."""
    be = backend
    w, wref, _ = _weight(be, n, k, g, seed=n + m)
    xv = np.random.default_rng(k + m).uniform(-1, 1, (m, k)).astype(np.float32)
    if out == "bf16":
        bits = orc.bf16_bits_rne(xv.reshape(-1))
        x, xv = be.ops.tensorFromArray(bits, [m, k], "bf16"), orc.bf16_bits_to_f32(bits).reshape(m, k).astype(np.float64)
    else:
        x, xv = be.ops.tensorFromArray(xv.astype(np.float16), [m, k], "f16"), xv.astype(np.float16).astype(np.float64)
    y = be.linear(x, w, None, None, out)
    got = be.ops.read(y)
    got = orc.bf16_bits_to_f32(got.reshape(-1)).reshape(m, n) if out == "bf16" else np.asarray(got, np.float64)
    ref = xv @ wref.astype(np.float64).T
    bound = np.abs(xv) @ np.abs(wref.astype(np.float64)).T * 2.0 ** -20
    bound += {"f16": 2.0 ** -11, "bf16": 2.0 ** -8, "f32": 0.0}[out] * (np.abs(ref) + bound) + (2.0 ** -25 if out == "f16" else 0.0)
    assert (np.abs(got - ref) <= bound).all()
    for t in (x, y, w.scales, w):
        t.destroy()


@pytest.mark.parametrize("g", [32, 64, 0])
@pytest.mark.parametrize("m,n,k", [(5, 100, 640), (16, 300, 1024)])
@pytest.mark.parametrize("warps,row_tiles,stages", [(16, 1, 4), (8, 2, 4), (4, 1, 2), (1, 2, 2)])
def test_int4_forced_shapes_with_other_groups(backend, g, m, n, k, warps, row_tiles, stages):
    be = backend
    w, wref, _ = _weight(be, n, k, g or k, seed=m)
    xv = np.random.default_rng(k).uniform(-1, 1, (m, k)).astype(np.float16)
    x = be.ops.tensorFromArray(xv, [m, k], "f16")
    be.forceVariant((1, 9, warps, row_tiles, stages, 0))
    try:
        y = be.linear(x, w, None, None, "f32")
    finally:
        be.forceVariant(None)
    size = np.abs(xv.astype(np.float64)) @ np.abs(wref.astype(np.float64)).T
    assert (np.abs(be.ops.read(y) - xv.astype(np.float64) @ wref.astype(np.float64).T) <= size * 2.0 ** -20).all()
    for t in (x, y, w.scales, w):
        t.destroy()
