"""Small-batch products start while the kernels in front of them drain and ask for packed weights first, the CUDA-core kernel for scales
too.  Behind kernels that write these they must not: the edges of a capture say whether a dependency is a full one, with memory visibility."""
import ctypes as C

import numpy as np
import pytest

import cases
from oracle import oracle as orc
from torchlette_b200 import backend as tb

pytestmark = pytest.mark.gpu


def _edges(be, call):
    """The kernel edges of a capture of `call`, in order: True for a programmatic one."""
    from cuda.bindings import driver as cu

    def ok(result):
        assert result[0] == cu.CUresult.CUDA_SUCCESS, result
        return result[1] if len(result) == 2 else result[1:]

    ok(cu.cuStreamBeginCapture(be.stream(), cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    try:
        call()
    finally:
        graph = ok(cu.cuStreamEndCapture(be.stream()))
    nodes = ok(cu.cuGraphGetNodes(graph))[1]
    first, second, data, count = (C.c_void_p * nodes)(), (C.c_void_p * nodes)(), (C.c_ubyte * (8 * nodes))(), C.c_size_t(nodes)
    assert C.CDLL("libcuda.so.1").cuGraphGetEdges_v2(C.c_void_p(int(graph)), first, second, data, C.byref(count)) == 0
    assert count.value == nodes - 1  # one chain
    # CUgraphEdgeData: from_port, to_port, type (1: programmatic), reserved
    by_node = {first[i]: data[8 * i + 2] == 1 for i in range(count.value)}
    order, left = [], {first[i]: second[i] for i in range(count.value)}
    at = (set(left) - set(left.values())).pop()
    while at in left:
        order.append(by_node[at])
        at = left[at]
    cu.cuGraphDestroy(graph)
    return order


def _packed(be, n, k, g, scheme, act, bits):
    w = be.ops.empty([n, k * bits // 32], "u32")
    w.scales = be.ops.empty([n, k // g], "u16")
    w.shape, w.dtype, w.format = [n, k], act, tb.StorageFormat(act, tb.QuantPacking(scheme, g, "f16"))
    return w


@pytest.mark.parametrize("act,scheme,bits,k", [("f32", "int8-grouped", 8, 1024), ("f16", "int8-grouped", 8, 1024), ("bf16", "int8-grouped", 8, 4096),
                                               ("f16", "int4-grouped", 4, 1024)])
def test_a_product_waits_for_kernels_that_write_its_weights_or_scales(backend, act, scheme, bits, k):
    be, n, g = backend, 512, 64
    w = _packed(be, n, k, g, scheme, act, bits)
    x, y, full = be.ops.empty([1, k], act), be.ops.empty([1, n], "f32"), be.ops.empty([n, k], "f32")
    bytes8, row = be.ops.empty([n, k // 4], "u32"), be.ops.empty([1, n], "f32")

    def product():
        be.ops.matmul(x, be.ops.transpose(w), {"outBuffer": y})

    def quantize():
        be._calls.tl_quantize_linear_weight_device(be._handle, full.buffer, n, k, g, bytes8.buffer, w.scales.buffer)

    def unpack():
        unpack_kernel = be._lib.tl_unpack_int8 if bits == 8 else be._lib.tl_unpack_int4
        assert unpack_kernel(be._ctx, w.buffer, bytes8.buffer, n, k) == 0

    def relu(at, count, dtype):
        be._calls.tl_unary_op(be._handle, tb.B.TL_UNARY["relu"], at, tb.B.DTYPE_ID[dtype], at, tb.B.DTYPE_ID[dtype], count)

    def scales():
        relu(w.scales.buffer, n * (k // g), "f16")

    def other():  # writes nothing that the product asks for early
        relu(row.buffer, n, "f32")

    # taking the stream is the first thing a capture does here: the first product is an ordinary launch.  Only the CUDA-core kernel (f32
    # activations) asks for scales early.
    def each():
        for call in (product, product, quantize, product, product, unpack, product, other, product, scales, product, scales, other, product):
            call()
    early_scales = act != "f32"
    assert _edges(be, each) == [True, False, False, True, False, False, True, True, True, early_scales, True, True, True]
    for t in (x, y, full, bytes8, row, w.scales, w):
        t.destroy()


def test_scales_that_a_product_computes(backend):
    """The f32 scales of one weight are the output of the product in front, or of one in front of that."""
    be, n, k = backend, 512, 1024
    w = _packed(be, n, k, 64, "int8-grouped", "f32", 8)
    v = be.ops.empty([n, k // 4], "u32")
    v.scales, v.shape, v.dtype, v.format = be.ops.empty([1, n], "f32"), [n, k], "f32", tb.StorageFormat("f32", tb.QuantPacking("int8-grouped", k, "f32", "direct"))
    x, y = be.ops.empty([1, k], "f32"), be.ops.empty([1, n], "f32")

    def product(weight, out):
        return lambda: be.ops.matmul(x, be.ops.transpose(weight), {"outBuffer": out})

    def each():
        for call in (product(w, y), product(v, y), product(w, v.scales), product(v, y), product(w, v.scales), product(w, y), product(v, y), product(v, y)):
            call()
    assert _edges(be, each) == [True, True, False, True, True, False, True]
    for t in (x, y, w.scales, w, v.scales, v):
        t.destroy()


@pytest.mark.parametrize("act", ["f32", "f16"])
def test_device_quantizer_and_the_product_behind_it(backend, act):
    be, n, k = backend, 4096, 2048
    rng = np.random.default_rng(3)
    xv = rng.standard_normal((1, k)).astype(np.float32 if act == "f32" else np.float16)
    x = be.ops.tensorFromArray(xv, [1, k], act)
    for _ in range(12):
        wv = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
        full = be.ops.tensorFromArray(wv, [n, k], "f32")
        w = be.quantizeLinearWeightOnDevice(full, tb.resolveWeightFormat("int8-64"))
        y = be.linear(x, w, None, None, "f32")
        packed, scales = orc.quantize_linear_weight(wv, 64)
        ref = orc.linear_reference(xv.astype(np.float32), orc.dequantize_to_f32(packed, scales, k, 64))
        assert cases.rel_err(be.ops.read(y), ref) <= 1e-3
        for t in (full, y, w.scales, w):
            t.destroy()
    x.destroy()


def test_small_ops_behind_copies_and_a_joined_stream_in_a_capture(backend):
    """The attribute of an early launch where what is in front is no kernel, or more than one stream's work."""
    from cuda.bindings import driver as cu

    def ok(result):
        assert result[0] == cu.CUresult.CUDA_SUCCESS, result
        return result[1] if len(result) == 2 else result[1:]

    be, n = backend, 1024
    dt = tb.B.DTYPE_ID["f32"]
    xv = np.linspace(-1, 1, n, dtype=np.float32)
    x = be.ops.tensorFromArray(xv, [1, n], "f32")
    row, y, z, w = (be.ops.empty([1, n], "f32") for _ in range(4))
    s = be.stream()
    side = ok(cu.cuStreamCreate(cu.CUstream_flags.CU_STREAM_NON_BLOCKING))
    fork, join = (ok(cu.cuEventCreate(cu.CUevent_flags.CU_EVENT_DISABLE_TIMING)) for _ in range(2))
    be.sync()
    ok(cu.cuStreamBeginCapture(s, cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    try:
        ok(cu.cuEventRecord(fork, s))
        ok(cu.cuStreamWaitEvent(side, fork, 0))
        ok(cu.cuMemsetD32Async(w.buffer, int(np.float32(2.0).view(np.uint32)), n, side))
        ok(cu.cuEventRecord(join, side))
        be._calls.tl_copy2d(be._handle, row.buffer, 4 * n, x.buffer, 4 * n, 4 * n, 1)
        be._calls.tl_unary_op(be._handle, tb.B.TL_UNARY["relu"], row.buffer, dt, y.buffer, dt, n)  # behind a copy
        ok(cu.cuStreamWaitEvent(s, join, 0))
        be._calls.tl_binary_op(be._handle, tb.B.TL_BINARY["mul"], y.buffer, dt, w.buffer, dt, z.buffer, dt, 1, n, 0)  # behind a kernel and another stream
    finally:
        graph = ok(cu.cuStreamEndCapture(s))
    run = ok(cu.cuGraphInstantiate(graph, 0))
    ok(cu.cuGraphLaunch(run, s))
    be.sync()
    np.testing.assert_array_equal(be.ops.read(z).reshape(-1), np.maximum(xv, 0) * 2)
    cu.cuGraphExecDestroy(run)
    cu.cuGraphDestroy(graph)
    cu.cuEventDestroy(fork)
    cu.cuEventDestroy(join)
    cu.cuStreamDestroy(side)
    for t in (x, row, y, z, w):
        t.destroy()
