"""tl_alloc / tl_free: blocks are handed out again, but never while anything given to the device before still uses them."""
import threading

import numpy as np
import pytest
import torch

from torchlette_b200 import backend as tb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    own = tb.CudaBackend(0)  # a context of its own: the refusals below count as its errors
    yield own
    own.destroy()


class _Memory:
    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": "<f4", "version": 2}


def test_blocks_are_reused_and_live_ones_do_not_overlap(be):
    seen, live = set(), []
    rng = np.random.default_rng(0)
    again = 0
    for i in range(600):
        size = int(rng.choice([1, 100, 512, 4096, 70_000, 3_000_000]))
        p = be._alloc(size)
        assert p % 256 == 0
        again += p in seen
        seen.add(p)
        live.append((p, size))
        spans = sorted(live)
        assert all(a + s <= b for (a, s), (b, _) in zip(spans, spans[1:]))
        if len(live) > 5:
            be._free(live.pop(int(rng.integers(len(live))))[0])
    for p, _ in live:
        be._free(p)
    assert again > 100


def test_a_block_given_back_waits_for_other_streams(be):
    """torch reads the blocks on a stream of its own, long after they were given back; new results must not reach them."""
    count = 1 << 22
    side = torch.cuda.Stream()
    busy = torch.randn(4096, 4096, device="cuda")
    for _ in range(3):
        t = be.ops.tensorFromArray(np.full(count, 1.0, np.float32), [count], "f32")
        be.sync()
        with torch.cuda.stream(side):
            for _ in range(30):
                busy = (busy @ busy).clamp_(-1, 1)
            copy = torch.as_tensor(_Memory(t.buffer, count), device="cuda").clone()
        t.destroy()
        others = [be.ops.tensorFromArray(np.full(count, 2.0, np.float32), [count], "f32") for _ in range(70)]
        for o in others:
            o.destroy()
        side.synchronize()
        assert bool((copy == 1.0).all())


def test_errors(be):
    p = be._alloc(1000)
    be._free(p)
    with pytest.raises(tb.TlError):
        be._free(p)
    with pytest.raises(tb.TlError):
        be._alloc(1 << 50)
    q = be._alloc(1000)  # neither refusal spoils what follows
    be._free(q)


class _Capture(threading.Thread):
    """A capture on a thread of its own that stays open until `close`."""

    def __init__(self, begin, work, end):
        super().__init__()
        self.steps, self.opened, self.may_end, self.error, self.graph = (begin, work, end), threading.Event(), threading.Event(), None, None

    def run(self):
        begin, work, end = self.steps
        try:
            begin()
            self.opened.set()
            try:
                assert self.may_end.wait(60)
                work()
            finally:
                self.graph = end()
        except Exception as e:  # handed to the test
            self.error = e
        finally:
            self.opened.set()

    def close(self):
        self.may_end.set()
        self.join()


@pytest.mark.parametrize("size,count", [(100, 200), (30 << 20, 20)])
@pytest.mark.parametrize("other", ["context", "torch"])
def test_freeing_leaves_the_captures_of_others_alone(be, other, size, count):
    """More blocks than wait for one synchronization, given back while another context or torch captures on this device."""
    if other == "context":
        be2 = tb.CudaBackend(0)
        cache = be2.ops.tensorFromArray(np.zeros((1, 1, 4, 64), np.float32), [1, 1, 4, 64], "f32")
        new = be2.ops.tensorFromArray(np.full((1, 1, 1, 64), 3.0, np.float32), [1, 1, 1, 64], "f32")
        be2.sync()
        cap = _Capture(be2.beginCapture, lambda: be2.ops.kvAppend(cache, new, 2), be2.endCapture)
    else:
        stream, graph, x = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros(64, device="cuda")
        torch.cuda.synchronize()

        def begin():
            torch.cuda.set_stream(stream)
            graph.capture_begin(capture_error_mode="thread_local")

        cap = _Capture(begin, lambda: x.add_(3.0), graph.capture_end)
    blocks = [be._alloc(size) for _ in range(count)]
    cap.start()
    cap.opened.wait()
    try:
        for p in blocks:
            be._free(p)
        blocks = [be._alloc(size) for _ in range(count)]
    finally:
        cap.close()
    assert cap.error is None
    for p in blocks:
        be._free(p)
    if other == "context":
        be2.replay(cap.graph)
        got = be2.ops.read(cache)
        assert (got[0, 0, 2] == 3.0).all() and (got[0, 0, [0, 1, 3]] == 0.0).all()
        be2.destroyGraph(cap.graph)
        for t in (cache, new):
            t.destroy()
        be2.destroy()
    else:
        graph.replay()
        torch.cuda.synchronize()
        assert bool((x == 3.0).all())


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_a_capture_that_a_program_began_on_the_stream_refuses(be, mode):
    """The context's stream captured without tl_graph_begin: a block handed out or taken back there could be another tensor's
    by the time the graph runs."""
    from cuda.bindings import driver as cu

    kinds = cu.CUstreamCaptureMode
    mode = {"thread_local": kinds.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL, "relaxed": kinds.CU_STREAM_CAPTURE_MODE_RELAXED}[mode]
    held, kept = [be._alloc(1000) for _ in range(3)], [be._alloc(1000) for _ in range(70)]
    for p in kept:
        be._free(p)  # some are ready to be handed out again
    be.sync()

    def capture(call):
        assert cu.cuStreamBeginCapture(be.stream(), mode)[0] == cu.CUresult.CUDA_SUCCESS
        try:
            call()
        finally:
            err, graph = cu.cuStreamEndCapture(be.stream())
            if err == cu.CUresult.CUDA_SUCCESS:
                cu.cuGraphDestroy(graph)

    def free():
        with pytest.raises(tb.TlError):
            be._free(held[0])

    def alloc():
        if mode == kinds.CU_STREAM_CAPTURE_MODE_RELAXED:  # new memory is allowed there, another tensor's is not
            p = be._alloc(1000)
            assert p not in kept
            held.append(p)
        else:
            with pytest.raises(tb.TlError):
                be._alloc(1000)

    capture(free)
    capture(alloc)
    assert not set(be._alloc(1000) for _ in range(3)) & set(held)  # what was refused is still the caller's
    for p in held:
        be._free(p)


def test_a_graph_of_this_thread_on_another_context_refuses(be):
    be2 = tb.CudaBackend(0)
    p = be._alloc(1000)
    be2.beginCapture()
    with pytest.raises(tb.TlError):
        be._free(p)
    with pytest.raises(tb.TlError):
        be._alloc(1000)
    with pytest.raises(tb.TlError):  # what a cudaMalloc in the capturing thread does to the capture
        be2.endCapture()
    assert be._alloc(1000) != p
    be._free(p)
    be2.destroy()


def test_kept_bytes(be):
    """A program that needs the memory elsewhere: what is kept goes back at once, and with 0 nothing is kept."""
    assert be.getOption("kept_bytes") == 1 << 30
    blocks = [be._alloc(100 << 20) for _ in range(3)]
    for p in blocks:
        be._free(p)
    held = torch.cuda.mem_get_info()[0]
    be.setOption("kept_bytes", 0)
    assert torch.cuda.mem_get_info()[0] >= held + (300 << 20)
    free = torch.cuda.mem_get_info()[0]
    be._free(be._alloc(100 << 20))
    assert torch.cuda.mem_get_info()[0] >= free
    with pytest.raises(tb.TlError):
        be.setOption("kept_bytes", -1)
    be.setOption("kept_bytes", 1 << 30)


def _int4(be, n, k, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    packed = torch.randint(-2 ** 31, 2 ** 31 - 1, (n, k // 8), dtype=torch.int32, device="cuda", generator=gen)
    scales = torch.full((n, k // 128), 0.01, dtype=torch.float16, device="cuda")
    st = tb.CudaTensor(be, [n, k // 128], "u16", scales.data_ptr(), scales.nbytes, ownsBuffer=False)
    w = tb.CudaTensor(be, [n, k], "f16", packed.data_ptr(), packed.nbytes, ownsBuffer=False, scales=st,
                      format=tb.StorageFormat("f16", tb.QuantPacking("int4-grouped", 128, "f16")))
    x = torch.randn(20, k, device="cuda", generator=gen).half()
    xt = tb.CudaTensor(be, [20, k], "f16", x.data_ptr(), x.nbytes, ownsBuffer=False)
    y = torch.empty(20, n, device="cuda", dtype=torch.float32)
    yt = tb.CudaTensor(be, [20, n], "f32", y.data_ptr(), y.nbytes, ownsBuffer=False)
    torch.cuda.synchronize()

    def run():
        be.ops.matmul(xt, be.ops.transpose(w), {"outBuffer": yt})
        be.sync()
        return y
    run.keep = packed, scales, x
    return run


def test_scratch_takes_the_memory_that_freed_blocks_hold():
    """A nearly full GPU: the library's own scratch grows into what tl_free kept."""
    n, k = 16384, 16384  # 512 MB of scratch for the 16-bit copy
    own, hog = tb.CudaBackend(0), None
    try:
        _int4(own, 256, 256, 0)()  # its kernels are loaded
        run = _int4(own, n, k, 1)
        torch.cuda.empty_cache()
        blocks = [own._alloc(200 << 20) for _ in range(4)]
        for p in blocks:
            own._free(p)
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
        got = run().clone()
    finally:
        del hog
        torch.cuda.empty_cache()
        own.destroy()
    plenty = tb.CudaBackend(0)
    ref = _int4(plenty, n, k, 1)()
    plenty.destroy()
    assert bool(torch.isfinite(got).all()) and torch.equal(got, ref)


def test_dequantize_dense_without_memory_is_the_fused_kernel():
    """No room for the 16-bit copy of the weight: the fused kernel computes the call, unless the route was asked for by name."""
    m, n, k = 300, 16384, 16384
    gen = torch.Generator(device="cuda").manual_seed(2)
    q = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=gen)
    scales = torch.full((n, 1), 1e-3, device="cuda")
    x, y = torch.randn(m, k, device="cuda", generator=gen).half(), torch.empty(m, n, device="cuda")
    own, hog = tb.CudaBackend(0), None
    wrap = lambda t, dtype, **more: tb.CudaTensor(own, list(t.shape), dtype, t.data_ptr(), t.nbytes, ownsBuffer=False, **more)  # noqa: E731
    fmt = tb.perChannelFormat(k)
    w = own.ops.transpose(wrap(q, "f16", format=fmt, scales=wrap(scales, "f32")))
    xt, yt = wrap(x, "f16"), wrap(y, "f32")
    dense = (2, 2, 0, 0, 0, 0)

    def run(variant):
        own.forceVariant(variant)
        own.ops.matmul(xt, w, {"outBuffer": yt})
        own.sync()
        return y.clone()

    torch.cuda.synchronize()
    try:
        fused = [run((2, 0, 192, 128, 3, 8)), run((2, 0, 128, 128, 4, 8))]
        own.forceVariant(None)
        own.seedPerShapeMatmulChoice(m, n, k, "f16", fmt.packing, dense)
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (256 << 20), dtype=torch.uint8, device="cuda")
        with pytest.raises(tb.TlError, match="scratch"):
            run(dense)
        got = run(None)
    finally:
        del hog
        torch.cuda.empty_cache()
        own.destroy()
    assert any(torch.equal(got, r) for r in fused)
