"""The native calls (csrc/tl_pycall.cpp) against ctypes: every argument as the C function gets it, descriptors, what goes through
ctypes and what must not, the calls without the module, and a status as an exception.  No GPU: the functions called are Python callbacks with the library's signatures."""
import ctypes as C

import numpy as np
import pytest

from torchlette_b200 import backend as tb
from torchlette_b200 import binding as B

VALUES = {C.c_void_p: [0x7F0012345678, None], C.c_int32: [3, -1], C.c_int64: [1 << 40, -5], C.c_size_t: [1 << 40, 7], C.c_float: [0.5, -2.0]}


def _on_error(ctx, status):
    raise B.TlError(status, f"of {ctx}")


def _native(name, callback):
    """A native call of `callback`, a ctypes function of the library's signature for `name`, and the list of the calls that it sent
    through ctypes."""
    slow = []

    def through_ctypes(*args):
        slow.append(args)
        return callback(*args)

    return B._native_module().bind(name, C.cast(callback, C.c_void_p).value, through_ctypes, _on_error), slow


def test_the_module_has_the_calls_of_the_binding():
    assert set(B._native_module().names) == set(B.CALLS) == {n for n in vars(B.calls()) if n.startswith("tl_")}


@pytest.mark.parametrize("name", sorted(n for n in B.CALLS if n != "tl_alloc"))
@pytest.mark.parametrize("which", [0, 1])
def test_arguments_arrive_as_through_ctypes(name, which):
    kinds = [k if k in VALUES else C.c_void_p for k in B.SIGNATURES[name][1]]
    seen = []
    callback = C.CFUNCTYPE(C.c_int32, *kinds)(lambda *a: seen.append(a) or 0)
    call, slow = _native(name, callback)
    # different values in neighbouring places
    args = [VALUES[k][which] if k is C.c_float or VALUES[k][which] is None else VALUES[k][which] + (i if which == 0 else 0) for i, k in enumerate(kinds)]
    assert call(*args) is None
    callback(*args)
    assert seen[0] == seen[1] and not slow
    # each that is no plain number or address by itself: a ctypes pointer, an integer for a float, an integer of numpy
    for i, (a, k) in enumerate(zip(args, kinds)):
        mixed = list(args)
        mixed[i] = C.c_void_p(a) if k is C.c_void_p else int(a) if k is C.c_float else np.int64(a)
        assert call(*mixed) is None
        assert len(slow) == i + 1
        callback(*mixed)
        assert seen[-2] == seen[-1]
    with pytest.raises(TypeError):
        call(*args[:-1])
    with pytest.raises((TypeError, C.ArgumentError)):
        call(*([object()] + args[1:]))


def test_a_status_is_an_exception_and_alloc_gives_the_address():
    call, slow = _native("tl_free", C.CFUNCTYPE(C.c_int32, C.c_void_p, C.c_void_p)(lambda ctx, p: B.TL_ERR_CUDA))
    for pointer in (16, C.c_void_p(16)):
        with pytest.raises(B.TlError) as e:
            call(8, pointer)
        assert e.value.status == B.TL_ERR_CUDA
    assert len(slow) == 1

    def give(ctx, nbytes, out):
        out[0] = 4096 if nbytes else None
        return 0 if nbytes < 100 else B.TL_ERR_OOM

    callback = C.CFUNCTYPE(C.c_int32, C.c_void_p, C.c_size_t, C.POINTER(C.c_void_p))(give)
    lib = type("Lib", (), {"tl_alloc": callback})
    slow = []

    def through_ctypes(*args):
        slow.append(args)
        return B._alloc_through_ctypes(lib)(*args)

    alloc = B._native_module().bind("tl_alloc", C.cast(callback, C.c_void_p).value, through_ctypes, _on_error)
    assert alloc(8, 64) == 4096 and alloc(8, 0) is None
    with pytest.raises(B.TlError):
        alloc(8, 100)
    assert not slow
    assert alloc(C.c_void_p(8), 64) == 4096 and alloc(8, np.int64(64)) == 4096 and len(slow) == 2
    for bad in ((8,), (8, 1.5)):
        with pytest.raises((TypeError, C.ArgumentError)):
            alloc(*bad)


def _library(seen, status=0):
    """A fake of the library: each call notes the values that arrive, descriptors by their fields."""
    def value(a):
        if isinstance(a, C.POINTER(B.QuantDesc)):
            return tuple(getattr(a[0], f) for f, _ in B.QuantDesc._fields_) if a else None
        if isinstance(a, C.POINTER(B.Epilogue)):
            return (a[0].n_ops, [(o.kind, o.op, o.input_index, o.to_dtype) for o in a[0].ops], a[0].n_inputs, list(a[0].inputs)) if a else None
        return a

    lib = type("Lib", (), {})()
    for name in B.CALLS:
        kinds = B.SIGNATURES[name][1]

        def note(*args, name=name):
            seen.append((name,) + tuple(value(a) for a in args if not isinstance(a, C.POINTER(C.c_void_p))))
            if name == "tl_alloc":
                args[-1][0] = 4096
            return status
        setattr(lib, name, C.CFUNCTYPE(C.c_int32, *kinds)(note))
    return lib


def test_calls_without_the_module_are_the_same(monkeypatch):
    """Natively, natively with an argument for ctypes, and where the module has not been built: the same values and descriptors arrive."""
    seen = []
    lib = _library(seen)
    monkeypatch.setattr(B, "load", lambda: lib)
    made = []
    for path in (B.PYCALL_PATH, B.PYCALL_PATH + ".missing"):
        monkeypatch.setattr(B, "_calls", None)
        monkeypatch.setattr(B, "PYCALL_PATH", path)
        if path.endswith("missing"):
            with pytest.warns(UserWarning, match="not been built"):
                made.append(B.calls())
        else:
            made.append(B.calls())
    ops, inputs = ((1, 0, 0, 0), (2, 3, 0, 0)), (4096, None)
    for c in made:
        q, e = c.quant(1, np.int32(64), 2, -3), c.epilogue(ops, inputs)
        for x in (16, C.c_void_p(16)):
            c.tl_qmatmul_nt(8, x, 1, 32, 64, 128, 0, 2, 256, 512, q, 0.5, e)
            c.tl_qmatmul_nt(8, x, 1, 32, 64, 128, 0, 2, 256, 512, q, 0.5, None)
            c.tl_free(8, x)
        assert c.tl_alloc(8, 64) == 4096
        for short in (q[:-1], q + b"x", b""):
            with pytest.raises(C.ArgumentError):
                c.tl_qmatmul_nt(8, 16, 1, 32, 64, 128, 0, 2, 256, 512, short, 0.5, e)
    one = len(seen) // 2
    assert seen[:one] == seen[one:] and one == 7
    assert seen[0] == seen[3] and seen[0][11] == (1, 64, 2, -3) and seen[0][13][0] == 2 and seen[0][13][1][:2] == list(ops) and seen[0][13][3][:2] == [4096, None]
    bad = _library([], B.TL_ERR_OOM)
    bad.tl_last_error = lambda ctx: b"no room"
    monkeypatch.setattr(B, "load", lambda: bad)
    for call in (lambda c: c.tl_alloc(8, 64), lambda c: c.tl_free(8, 16)):
        with pytest.raises(B.TlError, match="no room"):
            call(B._ctypes_calls(bad))


def test_descriptors_have_the_layout_of_the_structures():
    calls = B.calls()
    q = B.QuantDesc.from_buffer_copy(calls.quant(1, 64, 2, -3))
    assert (q.scheme, q.group_size, q.scales_dtype, q.scale_convention) == (1, 64, 2, -3)
    ops = tuple((i, i + 1, i + 2, i + 3) for i in range(B.TL_EPI_MAX_OPS))
    e = B.Epilogue.from_buffer_copy(calls.epilogue(ops, (4096, None)))
    assert e.n_ops == len(ops) and tuple((o.kind, o.op, o.input_index, o.to_dtype) for o in e.ops) == ops
    assert e.n_inputs == 2 and list(e.inputs) == [4096, None, None, None]
    assert calls.quant(np.int64(1), np.uint8(64), True, -3) == calls.quant(1, 64, 1, -3)
    assert calls.epilogue(((1, np.int64(2), 3, 4),), ()) == calls.epilogue(((1, 2, 3, 4),), ())
    for make in (calls.epilogue, B._ctypes_calls(B.load()).epilogue):
        for bad in (((1, 2, 3),), ops + ops[:1], "x", ((1, 2, 3, 4.5),)):
            with pytest.raises(TypeError):
                make(bad, ())


def test_swiglu_states_the_chain_that_the_fusion_pass_finds():
    class Input:
        dtype = "f32"

    for out in ("f16", "f32"):
        seen = {}
        be = tb.CudaBackend.__new__(tb.CudaBackend)
        up = Input()
        up.destroy = lambda: None
        be.linear = lambda *a: up
        be.ops = type("Ops", (), {"transpose": staticmethod(lambda t: t), "matmul": staticmethod(lambda x, w, o: seen.update(o))})
        be.swiglu(None, None, None, out)
        config, inputs, _ = tb.detectMatmulEpilogue([("silu", None), ("mul", up)] + ([("cast", out)] if out != "f32" else []))
        assert seen["epilogue"] == config and seen["epilogueInputs"] == inputs
