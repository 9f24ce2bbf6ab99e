"""The CUDA-core small-batch kernel (f32 activations) where its steps end: k of one chunk, of part of a step, at and just past a
slice of activations (8192, 4096 and 2048 for one, two and four batch rows), rows that do not fill a CTA, groups of no power of two."""
import numpy as np
import pytest

import cases
from torchlette_b200 import backend as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 4])
@pytest.mark.parametrize("m,n,k,group", [(1, 33, 16, 0), (1, 5, 528, 48), (1, 64, 2048, 64), (1, 37, 8192, 64), (1, 19, 8208, 0), (1, 130, 14336, 128),
                                         (2, 19, 4112, 16), (3, 41, 2064, 48), (4, 29, 2048, 64), (4, 70, 6160, 80), (7, 18, 4096, 0), (16, 23, 1040, 208)])
def test_simt_against_f64(backend, rows, m, n, k, group):
    be = backend
    rng = np.random.default_rng(1000 * m + k)
    group = group or k
    q = rng.integers(-127, 128, (n, k), dtype=np.int8)
    scales = rng.uniform(0.001, 0.01, (n, k // group)).astype(np.float32)
    x = rng.standard_normal((m, k)).astype(np.float32)
    fmt = tb.StorageFormat("f32", tb.QuantPacking("int8-grouped", group, "f32", "direct"))
    w = be.createQuantizedWeight(cases.pack_int8(q), scales, n, k, fmt)
    xt = be.ops.tensorFromArray(x, [m, k], "f32")
    be.forceVariant((1, 1, 4, rows, 0, 0))
    try:
        y = be.linear(xt, w)
    finally:
        be.forceVariant(None)
    wv = q * np.repeat(scales, group, axis=1).astype(np.float64)
    # per lane sixteen products a step of 512, in one chain over all steps without groups; five shuffles, the scale, the convention factor
    steps = (k + 511) // 512
    bound = ((16 * steps if group == k else 16 + steps) + 5 + 3) * 2.0**-24 * (np.abs(x).astype(np.float64) @ np.abs(wv).T)
    assert (np.abs(be.ops.read(y) - x.astype(np.float64) @ wv.T) <= bound).all()
    for t in (y, xt, w.scales, w):
        t.destroy()
