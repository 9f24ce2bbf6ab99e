"""tl_attention against f64 attention at the edges of its kernels: key tiles and splits, query rows per KV head, head
dimensions, storage types, masks, caches longer than what is read."""
import numpy as np
import pytest

from torchlette_b200 import backend as tb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    assert tb.initCuda(0), tb.getCudaInitError()
    return tb.getBackend()


def to_bf16_bits(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


def store(be, a, dtype):
    """The tensor and the values it holds, as f64."""
    if dtype == "bf16":
        bits = to_bf16_bits(a)
        return be.ops.tensorFromArray(bits, list(a.shape), "bf16"), (bits.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    a = a.astype(np.float16 if dtype == "f16" else np.float32)
    return be.ops.tensorFromArray(a, list(a.shape), dtype), a.astype(np.float64)


def read(be, t):
    a = be.ops.read(t)
    return (a.astype(np.uint32) << 16).view(np.float32) if t.dtype == "bf16" else a


def reference(q, k, v, scale, causal, mask):
    h, s, n, rep = q.shape[1], q.shape[2], k.shape[2], q.shape[1] // k.shape[1]
    k, v = np.repeat(k, rep, axis=1), np.repeat(v, rep, axis=1)
    sc = np.matmul(q, k.transpose(0, 1, 3, 2)) * scale
    if mask is not None:
        sc = sc + mask
    if causal:
        sc = np.where(np.arange(n)[None, :] <= (n - s + np.arange(s))[:, None], sc, -np.inf)
    p = np.exp(sc - sc.max(-1, keepdims=True))
    o = np.matmul(p / p.sum(-1, keepdims=True), v)
    return o.transpose(0, 2, 1, 3).reshape(q.shape[0], s, h * q.shape[3])


# one rounding of an output below 2 to the storage type (half an ulp), plus 4e-6: f32 sums over up to 1e3 terms near 1, of which
# probabilities held to 23 bits (f16) or 24 are the smallest part
TOL = {"f16": 2.0 ** -11 + 4e-6, "bf16": 2.0 ** -8 + 4e-6, "f32": 4e-6}


def check(be, b, heads, kv_heads, d, s, n, dtype, causal=True, masked=False, capacity=None, seed=0):
    rng = np.random.default_rng(seed + 1000 * n + s)
    cap = capacity or n + 5
    q, qr = store(be, rng.standard_normal((b, heads, s, d)), dtype)
    kf, vf = rng.standard_normal((b, kv_heads, cap, d)), rng.standard_normal((b, kv_heads, cap, d))
    kf[:, :, n:], vf[:, :, n:] = np.nan, np.inf  # what lies behind the read prefix must not matter
    k, kr = store(be, kf, dtype)
    v, vr = store(be, vf, dtype)
    mask = np.where(rng.random((s, n)) < 0.3, -np.inf, rng.standard_normal((s, n))).astype(np.float32) if masked else None
    if masked:
        mask[:, 0] = 0.5  # every query sees something
    mt = be.ops.tensorFromArray(mask, [s, n], "f32") if masked else None
    scale = 1.0 / np.sqrt(d)
    out = be.ops.attention(q, k, v, n, scale, causal=causal, mask=mt)
    got = read(be, out).astype(np.float64)
    ref = reference(qr, kr[:, :, :n], vr[:, :, :n], scale, causal, mask)
    err = np.abs(got - ref) / np.maximum(1.0, np.abs(ref))
    assert np.isfinite(got).all() and err.max() <= TOL[dtype], (err.max(), np.unravel_index(err.argmax(), err.shape))
    for t in (q, k, v, out) + ((mt,) if masked else ()):
        t.destroy()


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,heads,kv_heads,s,n", [
    (1, 1, 1, 1, 1), (1, 4, 4, 1, 15), (2, 8, 2, 1, 16), (1, 8, 1, 1, 17), (3, 6, 2, 1, 129), (1, 4, 1, 1, 1000), (1, 16, 8, 1, 2051),
    (2, 4, 2, 3, 40), (1, 8, 2, 4, 4), (1, 16, 1, 1, 300), (1, 3, 1, 5, 260)])
def test_decode(be, dtype, d, b, heads, kv_heads, s, n):
    check(be, b, heads, kv_heads, d, s, n, dtype)


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("s,n,causal", [(1, 200, False), (2, 333, True), (4, 70, False)])
def test_decode_mask(be, dtype, s, n, causal):
    check(be, 2, 4, 2, 128, s, n, dtype, causal=causal, masked=True)


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
def test_decode_mask_of_lowest_values(be, dtype):
    """A row hidden altogether by the lowest f32 is the mean of all values, one hidden in part sees the rest."""
    rng = np.random.default_rng(7)
    low = np.finfo(np.float32).min
    q, qr = store(be, rng.standard_normal((1, 4, 2, 64)), dtype)
    k, kr = store(be, rng.standard_normal((1, 2, 300, 64)), dtype)
    v, vr = store(be, rng.standard_normal((1, 2, 300, 64)), dtype)
    mask = np.full((2, 300), low, np.float32)
    mask[1, 40:] = 0.0
    mt = be.ops.tensorFromArray(mask, [2, 300], "f32")
    out = be.ops.attention(q, k, v, 300, 0.125, causal=False, mask=mt)
    got = read(be, out).astype(np.float64)
    ref = np.empty_like(got)
    ref[:, 0] = np.repeat(vr.mean(2), 2, axis=1).reshape(1, -1)
    ref[:, 1] = reference(qr[:, :, 1:], kr[:, :, 40:], vr[:, :, 40:], 0.125, False, None)[:, 0]
    assert (np.abs(got - ref) / np.maximum(1.0, np.abs(ref))).max() <= TOL[dtype]
    for t in (q, k, v, mt, out):
        t.destroy()


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("s,n", [(3, 37), (3, 200)])
def test_decode_hidden_values_not_finite(be, dtype, s, n):
    """What the causal mask hides from a row does not reach it, infinite or not."""
    rng = np.random.default_rng(n)
    q, qr = store(be, rng.standard_normal((1, 4, s, 64)), dtype)
    k, kr = store(be, rng.standard_normal((1, 2, n, 64)), dtype)
    vf = rng.standard_normal((1, 2, n, 64))
    vf[:, 0, n - 1, :40], vf[:, 1, n - 1, 5] = np.inf, np.nan
    v, vr = store(be, vf, dtype)
    out = be.ops.attention(q, k, v, n, 0.125, causal=True)
    got = read(be, out).astype(np.float64)
    ref = reference(qr[:, :, :s - 1], kr[:, :, :n - 1], vr[:, :, :n - 1], 0.125, True, None)
    assert (np.abs(got[:, :s - 1] - ref) / np.maximum(1.0, np.abs(ref))).max() <= TOL[dtype]
    last = got[0, s - 1].reshape(4, 64)
    assert np.isinf(last[:2, :40]).all() and np.isfinite(last[:2, 40:]).all() and np.isnan(last[2:, 5]).all() and np.isfinite(last[2:, 6:]).all()
    for t in (q, k, v, out):
        t.destroy()


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("s,n,causal,masked", [(1, 1, False, False), (1, 16, False, False), (1, 17, False, False), (1, 64, True, False),
                                               (1, 333, False, True), (2, 50, False, False), (2, 64, False, True), (3, 37, True, False),
                                               (4, 600, True, False)])
@pytest.mark.parametrize("where", ["first", "middle", "last"])
def test_decode_visible_values_not_finite(be, dtype, d, s, n, causal, masked, where):
    """An infinite or NaN value of a key that every row sees comes out as what it is, wherever the key lies in its tile, and
    leaves the other dimensions and heads alone."""
    rng = np.random.default_rng(n + s)
    q, qr = store(be, rng.standard_normal((1, 4, s, d)), dtype)
    k, kr = store(be, rng.standard_normal((1, 2, n, d)), dtype)
    seen = n - s if causal else n - 1  # the last key that the first row sees
    vf = rng.standard_normal((1, 2, n, d))
    v_t, vr = store(be, vf, dtype)
    v_t.destroy()
    at = {"first": 0, "middle": seen // 2, "last": seen}[where]
    vf[:, 0, at, :20], vf[:, 0, at, 20:30], vf[:, 0, at, 30:33] = np.inf, -np.inf, np.nan
    v, _ = store(be, vf, dtype)
    mask = rng.standard_normal((s, n)).astype(np.float32) if masked else None
    mt = be.ops.tensorFromArray(mask, [s, n], "f32") if masked else None
    out = be.ops.attention(q, k, v, n, 0.125, causal=causal, mask=mt)
    got = read(be, out).astype(np.float64).reshape(s, 4, d)
    ref = reference(qr, kr, vr, 0.125, causal, mask).reshape(s, 4, d)  # of finite values: the other dimensions' results
    assert np.isposinf(got[:, :2, :20]).all() and np.isneginf(got[:, :2, 20:30]).all() and np.isnan(got[:, :2, 30:33]).all()
    for g, r in ((got[:, :2, 33:], ref[:, :2, 33:]), (got[:, 2:], ref[:, 2:])):
        assert (np.abs(g - r) / np.maximum(1.0, np.abs(r))).max() <= TOL[dtype]
    for t in (q, k, v, out) + ((mt,) if masked else ()):
        t.destroy()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("b,heads,kv_heads,d,s,n,causal", [
    (1, 4, 1, 128, 5, 5, True), (1, 8, 8, 64, 17, 17, True), (1, 8, 2, 128, 32, 32, True), (2, 8, 2, 128, 33, 200, True),
    (1, 4, 4, 64, 128, 128, True), (1, 4, 4, 128, 129, 130, True), (2, 6, 2, 64, 100, 511, True), (1, 3, 1, 128, 257, 300, True),
    (1, 8, 2, 128, 200, 333, False), (1, 4, 2, 64, 700, 700, True), (3, 14, 2, 128, 40, 1000, True), (2, 32, 8, 128, 640, 641, True),
    (4, 32, 8, 64, 300, 300, False)])
def test_prefill(be, dtype, b, heads, kv_heads, d, s, n, causal):
    check(be, b, heads, kv_heads, d, s, n, dtype, causal=causal)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_prefill_growing_scores(be, dtype):
    """Scores that climb from key to key: the running maximum moves at every step, by a little and by far."""
    rng = np.random.default_rng(3)
    s = n = 400
    q = np.abs(rng.standard_normal((1, 4, s, 64)))
    for slope in (0.01, 0.2):
        ramp = (np.arange(n) * slope / 8)[None, None, :, None]
        q_t, qr = store(be, q, dtype)
        k_t, kr = store(be, rng.standard_normal((1, 2, n, 64)) * 0.1 + ramp, dtype)
        v_t, vr = store(be, rng.standard_normal((1, 2, n, 64)), dtype)
        out = be.ops.attention(q_t, k_t, v_t, n, 0.125, causal=True)
        got = read(be, out).astype(np.float64)
        ref = reference(qr, kr, vr, 0.125, True, None)
        # scores up to 64 x 10 x 0.125 x 0.8: f32 products of that size are 2^-24 x 64 off, and exp turns that into a relative error
        top = (np.abs(qr).sum(-1).max() * np.abs(kr).max()) * 0.125
        assert (np.abs(got - ref) / np.maximum(1.0, np.abs(ref))).max() <= TOL[dtype] + 4 * top * 2.0 ** -23
        for t in (q_t, k_t, v_t, out):
            t.destroy()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_prefill_hidden_values_not_finite(be, dtype):
    rng = np.random.default_rng(11)
    s, n = 70, 150
    q, qr = store(be, rng.standard_normal((1, 4, s, 128)), dtype)
    k, kr = store(be, rng.standard_normal((1, 2, n, 128)), dtype)
    vf = rng.standard_normal((1, 2, n, 128))
    vf[:, 0, n - 1, :40], vf[:, 1, n - 1, 5] = np.inf, np.nan
    v, vr = store(be, vf, dtype)
    out = be.ops.attention(q, k, v, n, 0.1, causal=True)
    got = read(be, out).astype(np.float64)
    ref = reference(qr[:, :, :s - 1], kr[:, :, :n - 1], vr[:, :, :n - 1], 0.1, True, None)
    assert (np.abs(got[:, :s - 1] - ref) / np.maximum(1.0, np.abs(ref))).max() <= TOL[dtype]
    last = got[0, s - 1].reshape(4, 128)
    assert np.isinf(last[:2, :40]).all() and np.isfinite(last[:2, 40:]).all() and np.isnan(last[2:, 5]).all() and np.isfinite(last[2:, 6:]).all()
    for t in (q, k, v, out):
        t.destroy()
