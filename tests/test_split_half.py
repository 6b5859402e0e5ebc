"""GPU: the contractions in split float16 (gemm_half.cu, conv_halo.cu, the strided convolution's patches)
at the sizes where their tiling changes, and on operands that float16 pairs cannot hold: few such values,
which are multiplied apart, and many, which have to take the tf32 planes; the few-column products at the edges of their row and k tiles.

Bounds.  A value is carried to 2^-23 of itself, the product of two so carried to 2^-21, and the tensor core truncates once per addition into an accumulator
that takes at most 96 of them (tf32) or 64 (float16) before it is drained: 2^-24 each relative to the sum of
magnitudes so far.  96 * 2^-24 + 2^-21 < 6.3e-6 of sum |a||b|.  Float64 sums are rounded once: 2^-24.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 6.3e-6


@pytest.fixture(scope="module")
def T():
    from camel_b200 import tensor

    return tensor


def _product(T, a, b):
    out = T.matmul(T.from_numpy(a), T.from_numpy(b)).numpy()
    T.check_async()
    return out


def _check(got, a, b):
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    err = np.abs(got - a64 @ b64)
    assert np.all(err <= BOUND * (np.abs(a64) @ np.abs(b64)) + 1e-300)


# one tile and its edges; slices in a cluster, the last one empty (k = 570: nine groups of 64 over four slices;
# 1088: seventeen over eight); the drain after 1024 values of k; long columns (two passes over B); pairs of CTAs with a
# ragged last tile, also without slices beyond 2048; ten tiles and a long k (slices through the workspace); several
# tiles to a block over both accumulator sets; at most nine tiles or one row of them and k beyond 2048 (tf32 planes)
SHAPES = [(64, 64, 64), (128, 32, 128), (129, 33, 257), (128, 570, 128), (100, 1088, 130), (65, 1025, 130), (70, 1500, 66),
          (4100, 96, 1030), (2304, 1056, 2306), (1100, 2208, 2306), (1280, 5000, 128), (40000, 96, 100),
          (300, 2080, 260), (130, 4128, 131), (40, 9000, 70)]


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_product_narrow_scaled_and_wide_operands(T, m, k, n):
    rng = np.random.default_rng(m + 7 * k + n)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    plain = _product(T, a, b)
    _check(plain, a, b)
    # rows and columns of very different sizes, each narrow in itself
    ra = np.exp2(rng.integers(-50, 50, (m, 1))).astype(np.float32)
    cb = np.exp2(rng.integers(-50, 50, (1, n))).astype(np.float32)
    _check(_product(T, a * ra, b * cb), a * ra, b * cb)
    # rows that span ninety powers of two: no float16 scale fits them
    wide_a = a * np.exp2(rng.integers(-45, 45, (m, k))).astype(np.float32)
    wide_b = b * np.exp2(rng.integers(-45, 45, (k, n))).astype(np.float32)
    _check(_product(T, wide_a, b), wide_a, b)
    _check(_product(T, a, wide_b), a, wide_b)
    # one huge value that meets a zero must not cost the others their digits
    spike, gate = a.copy(), b.copy()
    spike[:, 3], gate[3, :] = 1e20, 0.0
    _check(_product(T, spike, gate), spike, gate)
    assert _product(T, a, b).tobytes() == plain.tobytes()  # nothing is left of the wide calls


def test_infinities_and_nan_stay_in_their_rows(T):
    rng = np.random.default_rng(5)
    a = rng.uniform(0.5, 1, (200, 96)).astype(np.float32)
    b = rng.uniform(0.5, 1, (96, 140)).astype(np.float32)
    clean = _product(T, a, b)
    a[7, 11], a[9, 3] = np.inf, np.nan
    got = _product(T, a, b)
    assert not np.isfinite(got[[7, 9]]).any()
    rest = np.setdiff1d(np.arange(200), [7, 9])
    assert got[rest].tobytes() == clean[rest].tobytes()


# k = 200: the dense layer is one launch that reads the weights themselves; 180: it reads packed ones
@pytest.mark.parametrize("k", [200, 180])
@pytest.mark.parametrize("wide", ["left", "weights", "both"])
def test_packed_weights_and_row_panels_agree_on_wide_operands(T, wide, k):
    import ctypes as C

    from camel_b200._lib import check, lib

    rng = np.random.default_rng(11)
    m, n = 384, 300
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    w = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    if wide in ("left", "both"):
        a *= np.exp2(rng.integers(-45, 45, a.shape)).astype(np.float32)
    if wide in ("weights", "both"):
        w *= np.exp2(rng.integers(-45, 45, w.shape)).astype(np.float32)
    ta, tw, out = T.from_numpy(a), T.from_numpy(w), T.zeros((m, n))
    ap, wp = C.c_void_p(), C.c_void_p()
    check(lib.ct_rows_pack(ta.ptr, m, k, C.byref(ap)))
    check(lib.ct_weights_pack(tw.ptr, k, n, C.byref(wp)))
    try:
        check(lib.ct_dense_packed(ta.ptr, tw.ptr, wp, None, m, k, n, 0, out.ptr, None))
        T.check_async()
        whole = out.numpy()
        _check(whole, a, w)
        for row0, rows in ((0, 128), (128, 256)):
            check(lib.ct_matmul_packed_rows(ap, row0, rows, wp, out.ptr + row0 * n * 4))
        T.check_async()
        _check(out.numpy(), a, w)
    finally:
        check(lib.ct_rows_free(ap))
        check(lib.ct_weights_free(wp))


def test_band_counts_where_every_block_walks_several_tiles_of_both_accumulator_sets(T):
    """n <= 64: half of the storing warps have nothing to store and run ahead of the others, over four tiles a block."""
    import ctypes as C

    import torch

    from camel_b200._lib import check, lib

    rng = np.random.default_rng(12)
    m, k, n = 4 * 148 * 128 - 60, 40, 64
    a, w = T.from_numpy(rng.uniform(-1, 1, (m, k)).astype(np.float32)), T.from_numpy(rng.uniform(-1, 1, (k, n)).astype(np.float32))
    want, got = T.zeros((m, n)), T.zeros((m, n))
    ap, wp = C.c_void_p(), C.c_void_p()
    check(lib.ct_rows_pack(a.ptr, m, k, C.byref(ap)))
    check(lib.ct_weights_pack(w.ptr, k, n, C.byref(wp)))
    try:
        check(lib.ct_matmul_packed_rows(ap, 0, m, wp, want.ptr))
        bands = [148 * 128, 2 * 148 * 128, m - 3 * 148 * 128]
        first = [0, bands[0], bands[0] + bands[1]]
        done, tiles = torch.zeros(3, dtype=torch.int32, device="cuda"), (C.c_uint32 * 3)()
        torch.cuda.synchronize()
        check(lib.ct_matmul_packed_bands(ap, wp, 3, (C.c_int64 * 3)(*bands),
                                         (C.c_void_p * 3)(*[got.ptr + f * n * 4 for f in first]), done.data_ptr(), tiles))
        T.check_async()
        assert list(tiles) == [148, 296, 148]
        assert done.cpu().tolist() == list(tiles)
        assert got.numpy().tobytes() == want.numpy().tobytes()
        _check(want.numpy(), a.numpy(), w.numpy())
    finally:
        check(lib.ct_rows_free(ap))
        check(lib.ct_weights_free(wp))


def _conv64(x, w, stride, pad):
    n, c, h, wd = x.shape
    ko, _, kh, kw = w.shape
    xp = np.pad(x.astype(np.float64), ((0, 0), (0, 0), (pad, pad), (pad, pad)))
    win = np.lib.stride_tricks.sliding_window_view(xp, (kh, kw), (2, 3))[:, :, ::stride, ::stride]
    return np.einsum("nchwrs,kcrs->nkhw", win, w.astype(np.float64), optimize=True)


# an output that depends on one product: both values to 2^-23, 2^-22 for the product of their low terms, which is left
# out, three additions cut off at 2^-23 each, two roundings of the sums and scales
SINGLE = 8 * 2.0**-23


def _beside_large(rng, shape, lowest):
    """Values from 2^(lowest - 16) to 2^-20 of a largest one that is 2^16."""
    return (rng.uniform(1, 2, shape) * np.exp2(rng.integers(lowest, -4, shape)) * rng.choice([-1, 1], shape)).astype(np.float32)


@pytest.mark.parametrize("size", [96, 288, 1100, 2300])
@pytest.mark.parametrize("side", ["left", "right"])
@pytest.mark.parametrize("lowest", [-9, -16, -44])
def test_small_values_keep_their_digits_beside_large_ones(T, size, side, lowest):
    rng = np.random.default_rng(size)
    a = _beside_large(rng, (size, size), lowest)
    a[:, 0] = 2.0**16
    b = np.diag(rng.uniform(1, 2, size)).astype(np.float32)
    b[0, 0] = 0.0
    got = _product(T, a, b) if side == "left" else _product(T, b, a.T.copy()).T
    want = a.astype(np.float64) * np.diag(b).astype(np.float64)
    assert np.all(np.abs(got - want) <= SINGLE * np.abs(want))


def _with_exceptions(rng, m, k, n, count):
    """Ordinary operands with `count` values in each that a float16 pair cannot hold, and the outputs that depend on
    one of those alone (or on one of each, at the same k)."""
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    rows, cols = rng.choice(m, count, replace=False), rng.choice(n, count, replace=False)
    ks = rng.choice(np.arange(1, k), count, replace=False)
    tiny = (rng.uniform(1, 2, (2, count)) * np.exp2(rng.integers(-50, -29, (2, count)))).astype(np.float32)
    a[:, 0] = rng.uniform(0.5, 1, m)
    a[rows, 0] = 0.0
    b[:, cols] = 0.0
    b[0, cols] = 0.75                    # keeps the column's scale; meets the zeros of a
    for t in range(count):
        a[rows[t], ks[t]] = tiny[0, t]
        b[ks[t], cols[t]] = tiny[1, t] if t % 2 else 0.5
        a[rows[t], ks[t - 1]] = a[rows[t], ks[t - 1]] or 0.25
    return a, b, rows, cols


# slices in a cluster; two passes over B; pairs; slices through the workspace; one wave of small tiles; more than a list holds;
# a tall left operand split inside the product, in four slices and in two
@pytest.mark.parametrize("m,k,n,count", [(128, 96, 200, 5), (300, 600, 300, 9), (600, 1500, 400, 12), (2600, 1100, 1500, 30),
                                         (1290, 4700, 128, 7), (1000, 300, 1000, 20), (700, 1200, 800, 40),
                                         (3200, 4100, 100, 12), (6500, 2100, 100, 30)])
@pytest.mark.parametrize("form", ["plain", "transposed", "weights", "rows"])
def test_values_that_float16_pairs_cannot_hold_are_put_right(T, m, k, n, count, form):
    import ctypes as C

    from camel_b200._lib import check, lib

    rng = np.random.default_rng(m + k + n)
    a, b, rows, cols = _with_exceptions(rng, m, k, n, count)
    bias = rng.uniform(-1, 1, n).astype(np.float32)
    bias[cols] = 0.0
    ta, tb, out = T.from_numpy(a), T.from_numpy(b), T.zeros((m, n))
    if form == "plain":
        check(lib.ct_dense(ta.ptr, tb.ptr, T.from_numpy(bias).ptr, m, k, n, 0, out.ptr, None))
    elif form == "transposed":
        out, bias = T.matmul_tn(T.from_numpy(a.T.copy()), tb), 0.0 * bias
    else:
        ap, wp, bias = C.c_void_p(), C.c_void_p(), 0.0 * bias
        check(lib.ct_weights_pack(tb.ptr, k, n, C.byref(wp)))
        check(lib.ct_rows_pack(ta.ptr, m, k, C.byref(ap)))
        if form == "weights":
            check(lib.ct_dense_packed(ta.ptr, tb.ptr, wp, None, m, k, n, 0, out.ptr, None))
        else:
            for row0 in range(0, m, 128):
                check(lib.ct_matmul_packed_rows(ap, row0, min(128, m - row0), wp, out.ptr + row0 * n * 4))
        T.check_async()
        check(lib.ct_rows_free(ap))
        check(lib.ct_weights_free(wp))
    got = out.numpy()
    T.check_async()
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    want = a64 @ b64 + bias
    assert np.all(np.abs(got - want) <= BOUND * (np.abs(a64) @ np.abs(b64) + np.abs(bias)))
    for t in range(count):  # column t holds 0.75 at k = 0, where row t is zero, and one value that meets the row's small one
        assert abs(got[rows[t], cols[t]] - want[rows[t], cols[t]]) <= SINGLE * abs(want[rows[t], cols[t]])


# patches; strided and unstrided halos; few channels from the input itself, from planes, and with a tile of odd rows
@pytest.mark.parametrize("shape", [(2, 49, 21, 23, 70, 3, 2, 1), (2, 48, 21, 23, 70, 3, 2, 1), (2, 64, 30, 28, 128, 3, 1, 1), (2, 32, 28, 28, 64, 3, 1, 1),
                                   (2, 20, 26, 27, 40, 3, 1, 1), (2, 20, 16, 18, 40, 3, 1, 0)])
@pytest.mark.parametrize("kind", ["input", "isolated", "filters"])
@pytest.mark.parametrize("lowest", [-9, -16, -44])
def test_convolution_keeps_small_values_beside_large_ones(T, shape, kind, lowest):
    n, c, h, wd, ko, kern, stride, pad = shape
    rng = np.random.default_rng(sum(shape))
    x, w = np.zeros((n, c, h, wd), np.float32), np.zeros((ko, c, kern, kern), np.float32)
    x[:, 1, 1::5, 2::5] = rng.uniform(1, 2, x[:, 1, 1::5, 2::5].shape)
    w[:, 1] = rng.uniform(1, 2, (ko, kern, kern))
    if kind == "input":  # a channel of large values that meets zero weights
        x[:, 1, 1::5, 2::5] = _beside_large(rng, x[:, 1, 1::5, 2::5].shape, lowest)
        x[:, 0] = 2.0**16
    elif kind == "isolated":  # one huge pixel beside one ordinary one
        x[:] = 0
        x[0, 0, 0, 0], x[0, 1, h - 2, wd - 2] = 1e16, 1.5
    else:  # a large weight that meets a channel of zeros
        w[:, 1], w[:, 0, 0, 0] = _beside_large(rng, (ko, kern, kern), lowest), 2.0**16
    want = _conv64(x, w, stride, pad)
    got = T.conv2d(T.from_numpy(x), T.from_numpy(w), None, stride, pad).numpy()
    T.check_async()
    assert np.all(np.abs(got - want) <= SINGLE * np.abs(want))


def _conv_at(T, x, w, stride, pad, off=0):
    """The layer on an input that starts `off` floats into its buffer."""
    from camel_b200._lib import check, lib

    n, c, h, wd = x.shape
    ko, _, kh, kw = w.shape
    tx = T.from_numpy(np.concatenate([np.zeros(off, np.float32), x.ravel()]))
    tw, out = T.from_numpy(w), T.zeros((n, ko, (h + 2 * pad - kh) // stride + 1, (wd + 2 * pad - kw) // stride + 1))
    check(lib.ct_conv2d(tx.ptr + 4 * off, tw.ptr, None, n, c, h, wd, ko, kh, kw, stride, pad, 0, out.ptr))
    T.check_async()
    return out.numpy()


# filters in tensor memory (tiles of seven rows, of six with the pool; of four), halos
@pytest.mark.parametrize("shape", [(5, 32, 16, 16, 64, 3), (4, 30, 28, 28, 60, 3), (3, 64, 30, 28, 128, 3)])
def test_bits_of_an_image_depend_on_that_image_alone(T, shape):
    """Not on the other images of the batch, on the fused pool, or on whether the input is read as it is or from planes."""
    n, c, h, wd, ko, kern = shape
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((n, c, h, wd)).astype(np.float32)
    w = rng.standard_normal((ko, c, kern, kern)).astype(np.float32)
    clean = _conv_at(T, x, w, 1, 1)
    wide = x.copy()
    wide[1, 3, h - 1, 2], wide[1, 2, 0, 0] = 2.0**-30, 2.0**3  # image 1 spans too much, its tiles do not
    wide[2, 0, h // 2] *= 2.0**-28                             # image 2 does inside a tile as well
    got = _conv_at(T, wide, w, 1, 1)
    others = [i for i in range(n) if i not in (1, 2)]
    assert got[others].tobytes() == clean[others].tobytes()
    for i in (1, 2):
        assert _conv_at(T, np.stack([wide[i]] * n), w, 1, 1)[0].tobytes() == got[i].tobytes()
    assert _conv_at(T, wide, w, 1, 1, off=1).tobytes() == got.tobytes()
    pooled = T.conv2d(T.from_numpy(wide), T.from_numpy(w), None, 1, 1, pool=2).numpy()
    assert pooled.tobytes() == T.maxpool2d(T.from_numpy(got), 2).numpy().tobytes()
    assert np.all(np.abs(got - _conv64(wide, w, 1, 1)) <= (384 * 2.0**-24 + 2.0**-21) * _conv64(np.abs(wide), np.abs(w), 1, 1))


def test_few_channel_layers_on_two_streams_share_no_state(T):
    """Wide and ordinary inputs side by side; neither layer uses the library's workspaces."""
    import ctypes as C

    from camel_b200._lib import check, lib

    rng = np.random.default_rng(21)
    x = [rng.standard_normal((40, 32, 28, 28)).astype(np.float32) for _ in range(2)]
    x[1] *= np.exp2(rng.integers(-45, 45, x[1].shape)).astype(np.float32)
    w = rng.standard_normal((64, 32, 3, 3)).astype(np.float32)
    want = [_conv_at(T, v, w, 1, 1).tobytes() for v in x]
    tx, tw = [T.from_numpy(v) for v in x], T.from_numpy(w)
    outs = [[T.zeros((40, 64, 28, 28)) for _ in range(6)] for _ in range(2)]
    streams = [C.c_void_p(), C.c_void_p()]
    T.sync()
    for s in streams:
        check(lib.ct_stream_create(C.byref(s)))
    try:
        for i in range(6):
            for j, s in enumerate(streams):
                check(lib.ct_set_stream(s))
                check(lib.ct_conv2d(tx[j].ptr, tw.ptr, None, 40, 32, 28, 28, 64, 3, 3, 1, 1, 0, outs[j][i].ptr))
        for s in streams:
            check(lib.ct_set_stream(s))
            check(lib.ct_sync())
    finally:
        check(lib.ct_set_stream(None))
        for s in streams:
            check(lib.ct_stream_destroy(s))
    T.check_async()
    for j in range(2):
        assert all(o.numpy().tobytes() == want[j] for o in outs[j])


# few channels, unstrided and strided halos, patches; a product of one wave and one with a conditional launch in front
@pytest.mark.parametrize("what", [(6, 32, 28, 28, 64, 3, 1, 1), (3, 64, 30, 28, 128, 3, 1, 1), (2, 48, 21, 23, 70, 3, 2, 1), (2, 49, 21, 23, 70, 3, 2, 1),
                                  (256, 200, 256), (1500, 700, 900)])
def test_recorded_calls_decide_on_every_replay(T, what):
    """The same graph over ordinary values, one small one, and values that need tf32 terms: the bytes of eager calls."""
    import ctypes as C

    from camel_b200._lib import check, lib

    rng = np.random.default_rng(sum(what))
    conv = len(what) > 3
    shape = what[:4] if conv else what[:2]
    plain = rng.standard_normal(shape).astype(np.float32)
    one, wide = plain.copy(), plain * np.exp2(rng.integers(-45, 45, shape)).astype(np.float32)
    one.flat[one.size // 3] = 1e-12
    w = rng.standard_normal((what[4], what[1], what[5], what[5]) if conv else what[1:]).astype(np.float32)
    inputs, tw = [T.from_numpy(v) for v in (plain, one, wide, plain)], T.from_numpy(w)
    if conv:
        n, c, h, wd, ko, kern, stride, pad = what
        out_shape = (n, ko, (h + 2 * pad - kern) // stride + 1, (wd + 2 * pad - kern) // stride + 1)
        call = lambda x, o: check(lib.ct_conv2d(x.ptr, tw.ptr, None, n, c, h, wd, ko, kern, kern, stride, pad, 1, o.ptr))  # noqa: E731
    else:
        out_shape = (what[0], what[2])
        call = lambda x, o: check(lib.ct_dense(x.ptr, tw.ptr, None, *what, 1, o.ptr, None))  # noqa: E731
    want = []
    for x in inputs:
        o = T.zeros(out_shape)
        call(x, o)
        want.append(o.numpy().tobytes())
    x, out, graph = T.from_numpy(plain), T.zeros(out_shape), C.c_void_p()
    call(x, out)
    check(lib.ct_graph_begin())
    call(x, out)
    check(lib.ct_graph_end(C.byref(graph)))
    try:
        for v, bytes_ in zip(inputs, want):
            check(lib.ct_d2d(x.ptr, v.ptr, plain.nbytes))
            check(lib.ct_graph_launch(graph))
            assert out.numpy().tobytes() == bytes_
        T.check_async()
    finally:
        check(lib.ct_graph_destroy(graph))


# (n, c, h, w, ko, kernel, stride, pad): patches in registers and read twice (k = 1200), odd sizes; halos with a stride, with a
# partial last tile, channels that do not fill a block, more than 128 filters, 1 x 1 and 5 x 5 taps
CONVS = [(3, 49, 21, 23, 70, 3, 2, 1), (3, 48, 21, 23, 70, 3, 2, 1), (2, 8, 33, 21, 20, 3, 2, 0), (2, 48, 15, 16, 40, 5, 3, 2), (2, 12, 24, 24, 65, 5, 1, 2),
         (2, 64, 30, 28, 128, 3, 1, 1), (3, 40, 14, 14, 136, 3, 1, 0), (2, 100, 17, 19, 72, 1, 1, 0), (2, 20, 57, 56, 72, 5, 1, 2)]


@pytest.mark.parametrize("shape", CONVS)
@pytest.mark.parametrize("kind", ["plain", "wide input", "wide filters"])
def test_convolution_narrow_and_wide(T, shape, kind):
    n, c, h, wd, ko, kern, stride, pad = shape
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((n, c, h, wd)).astype(np.float32)
    w = rng.standard_normal((ko, c, kern, kern)).astype(np.float32)
    if kind == "wide input":
        x *= np.exp2(rng.integers(-45, 45, x.shape)).astype(np.float32)
    if kind == "wide filters":
        w *= np.exp2(rng.integers(-45, 45, w.shape)).astype(np.float32)
    got = T.conv2d(T.from_numpy(x), T.from_numpy(w), None, stride, pad).numpy()
    T.check_async()
    # a halo layer's k (at most 1024) is one accumulation: up to 384 tf32 additions instead of 96
    bound = 384 * 2.0**-24 + 2.0**-21
    assert np.all(np.abs(got - _conv64(x, w, stride, pad)) <= bound * _conv64(np.abs(x), np.abs(w), stride, pad) + 1e-300)


# blocks of two and four rows, resident weights with four and (19001 rows) eight rows to a warp: up to six columns, and eight to twelve where the float64
# MMA has no room for its ring (1300 x 12, 1600 x 10, 1900 x 8) or only up to 18944 rows (1400 x 8); with that MMA (33 x 16, 785 x 10, 96 x 13);
# weights that leave room for a short ring (2300 x 10, 1400 x 16), for no ring (1600 x 16) and none at all (2700 x 12)
@pytest.mark.parametrize("m", [1, 2, 3, 297, 597, 2051, 4099, 19001])
@pytest.mark.parametrize("k,n", [(1, 3), (31, 1), (785, 4), (130, 6), (33, 16), (785, 10), (96, 13), (1400, 8), (1900, 8), (1600, 10), (1300, 12), (2300, 10), (1400, 16),
                                 (1600, 16), (2700, 12)])
def test_few_columns(T, m, k, n):
    rng = np.random.default_rng(m + k + n)
    x = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    w = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    b = rng.uniform(-1, 1, n).astype(np.float32)
    tx, tw, tb = T.from_numpy(x), T.from_numpy(w), T.from_numpy(b)
    z = x.astype(np.float64) @ w.astype(np.float64) + b
    # float64 sums in another order, rounded once
    g = rng.uniform(-1, 1, (m, n)).astype(np.float32)
    zt = x.astype(np.float64).T @ g.astype(np.float64)
    assert np.all(np.abs(T.matmul_tn(tx, T.from_numpy(g)).numpy() - zt) <= 2.0**-24 * np.abs(zt) + 1e-12)
    assert np.all(np.abs(T.dense(tx, tw, tb).numpy() - z) <= 2.0**-24 * np.abs(z) + 1e-13)
    logits = T.dense(tx, tw, tb).numpy()
    probs, arg = T.dense(tx, tw, tb, "softmax", with_argmax=True)
    assert np.array_equal(arg.numpy(), logits.argmax(1))  # first maximum wins in both
    e = np.exp(logits.astype(np.float64) - logits.max(1, keepdims=True))
    assert np.all(np.abs(probs.numpy() - e / e.sum(1, keepdims=True)) <= 4 * 2.0**-24)
