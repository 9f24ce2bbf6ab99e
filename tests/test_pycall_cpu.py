"""The native calls (csrc/tl_pycall.cpp) against ctypes: every argument as the C function gets it, descriptors, what goes through
ctypes, and a status as an exception.  No GPU: the functions called are Python callbacks with the library's signatures."""
import ctypes as C

import pytest

from torchlette_b200 import backend as tb
from torchlette_b200 import binding as B

VALUES = {C.c_void_p: [0x7F0012345678, None], C.c_int32: [3, -1], C.c_int64: [1 << 40, -5], C.c_size_t: [1 << 40, 7], C.c_float: [0.5, -2.0]}


def _native(name, callback):
    """A native call of `callback`, a ctypes function of the library's signature for `name`."""
    import importlib.machinery
    import importlib.util

    loader = importlib.machinery.ExtensionFileLoader("_tlcall", B.PYCALL_PATH)
    mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("_tlcall", loader))
    loader.exec_module(mod)

    def on_error(ctx, status):
        raise B.TlError(status, f"of {ctx}")

    return mod.bind(name, C.cast(callback, C.c_void_p).value, callback, on_error), mod


@pytest.mark.parametrize("name", sorted(n for n in vars(B.calls()) if n.startswith("tl_") and n != "tl_alloc"))
@pytest.mark.parametrize("which", [0, 1])
def test_arguments_arrive_as_through_ctypes(name, which):
    kinds = [k if k in VALUES else C.c_void_p for k in B.SIGNATURES[name][1]]
    seen = []
    callback = C.CFUNCTYPE(C.c_int32, *kinds)(lambda *a: seen.append(a) or 0)
    call, _ = _native(name, callback)
    # different values in neighbouring places, integers for floats included (those go through ctypes)
    args = [VALUES[k][which] if k is C.c_float or VALUES[k][which] is None else VALUES[k][which] + (i if which == 0 else 0) for i, k in enumerate(kinds)]
    assert call(*args) is None
    callback(*args)
    assert seen[0] == seen[1]
    mixed = [C.c_void_p(a) if k is C.c_void_p else int(a) if k is C.c_float else a for a, k in zip(args, kinds)]
    assert call(*mixed) is None
    callback(*mixed)
    assert seen[2] == seen[3]
    with pytest.raises(TypeError):
        call(*args[:-1])
    with pytest.raises((TypeError, C.ArgumentError)):
        call(*([object()] + args[1:]))


def test_a_status_is_an_exception_and_alloc_gives_the_address():
    call, _ = _native("tl_free", C.CFUNCTYPE(C.c_int32, C.c_void_p, C.c_void_p)(lambda ctx, p: B.TL_ERR_CUDA))
    with pytest.raises(B.TlError) as e:
        call(8, 16)
    assert e.value.status == B.TL_ERR_CUDA

    def give(ctx, nbytes, out):
        out[0] = 4096 if nbytes else None
        return 0 if nbytes < 100 else B.TL_ERR_OOM

    alloc, _ = _native("tl_alloc", C.CFUNCTYPE(C.c_int32, C.c_void_p, C.c_size_t, C.POINTER(C.c_void_p))(give))
    assert alloc(8, 64) == 4096 and alloc(8, 0) is None
    with pytest.raises(B.TlError):
        alloc(8, 100)
    with pytest.raises(TypeError):
        alloc(8)


def test_descriptors_have_the_layout_of_the_structures():
    calls = B.calls()
    q = B.QuantDesc.from_buffer_copy(calls.quant(1, 64, 2, -3))
    assert (q.scheme, q.group_size, q.scales_dtype, q.scale_convention) == (1, 64, 2, -3)
    ops = tuple((i, i + 1, i + 2, i + 3) for i in range(B.TL_EPI_MAX_OPS))
    e = B.Epilogue.from_buffer_copy(calls.epilogue(ops, (4096, None)))
    assert e.n_ops == len(ops) and tuple((o.kind, o.op, o.input_index, o.to_dtype) for o in e.ops) == ops
    assert e.n_inputs == 2 and list(e.inputs) == [4096, None, None, None]
    for bad in (((1, 2, 3),), ops + ops[:1], "x"):
        with pytest.raises(TypeError):
            calls.epilogue(bad, ())


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
