"""Sixteen converter warps (two groups on alternate k steps) against eight, bit for bit: the operands and the order of the products are
the same.  Ragged shapes, one k step, odd numbers of them with several tiles a CTA (the groups change places from tile to tile) and a cut last
wave; per-channel scales and groups longer and shorter than a thread's share of a step, and of no power of two."""
import numpy as np
import pytest

import cases
from torchlette_b200 import backend as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn,stages", [(32, 8), (64, 6), (128, 4), (192, 3)])
@pytest.mark.parametrize("m,n,k,group,act", [(17, 130, 80, 0, "f16"), (70, 300, 1152, 48, "f16"), (40, 260, 640, 64, "bf16"), (33, 38000, 640, 128, "f16"),
                                             (130, 19000, 384, 192, "bf16"), (64, 200, 128, 16, "f16")])
def test_sixteen_converter_warps_give_the_bits_of_eight(backend, bn, stages, m, n, k, group, act):
    be = backend
    rng = np.random.default_rng(m + n)
    group = group or k
    q = rng.integers(-127, 128, (n, k), dtype=np.int8)
    scales = rng.uniform(0.001, 0.01, (n, k // group)).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    bits = x.astype(np.float16) if act == "f16" else (x.view(np.uint32) >> 16).astype(np.uint16)
    w = be.createQuantizedWeight(cases.pack_int8(q), scales, n, k, tb.StorageFormat(act, tb.QuantPacking("int8-grouped", group, "f32", "direct")))
    xt = be.ops.tensorFromArray(bits, [m, k], act)
    got = []
    for warps in (8, 16):
        be.forceVariant((2, 0, bn, 128, stages, warps))
        try:
            y = be.linear(xt, w)
        finally:
            be.forceVariant(None)
        got.append(be.ops.read(y))
        y.destroy()
    np.testing.assert_array_equal(got[0], got[1])
    for t in (xt, w.scales, w):
        t.destroy()
