"""GPU: convolution layers at the edges of the halo and the paired-row kernels (strides, chunks of k, few filters, rows of
positions that fill an accumulator), small products computed in one launch, right operands in 64 x 64 blocks and the elements
behind the last vector of an elementwise operator.

Bounds.  Products and layers: 6.3e-6 of the sum of magnitudes (a value is carried to 2^-23 of itself, a product of two so
carried to 2^-21, at most 96 truncating additions of 2^-24 each into an accumulator).  bfloat16: 2^-8 per operand, 2^-7 of the
sum of magnitudes.  Elementwise float32 operators: exact.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

BOUND = 6.3e-6


@pytest.fixture(scope="module")
def T():
    from camel_b200 import tensor

    return tensor


@pytest.fixture(scope="module")
def port():
    oracle.build(ref=False)
    return oracle.port()


# n, c, h, w, ko, kh, kw, stride, pad.  Halo kernel: odd extents at strides 2 and 3 (sub-images of unequal size); taps that
# leave sub-images unread; half of a channel block, and one channel more; k of two and three drains (c = 97, 193 with
# nine taps; 33 with twenty-five); 17 and 129 filters; a tile of one row; partial last tiles.  Paired rows: an odd number of
# rows, a row of 128 positions, 16 and 64 filters, 8 channels, an even filter, rows that no tensor map covers, filters (4 x 3, 6 x 2) that fit
# single blocks or pairs of them only.  Halo again: more
# filters than have their bias in shared memory; 1 x 1 filters with and without a stride, a strided layer of one tile; filters that are streamed by rows of
# taps and, of a strided layer, by threes.
LAYERS = [(2, 48, 57, 57, 96, 3, 3, 2, 1), (1, 33, 20, 23, 70, 3, 3, 3, 1), (2, 40, 30, 33, 64, 1, 1, 2, 0), (1, 16, 41, 40, 65, 5, 5, 2, 2),
          (1, 97, 17, 30, 17, 3, 3, 1, 1), (1, 193, 15, 30, 129, 3, 3, 1, 0), (1, 33, 40, 61, 40, 5, 5, 1, 2), (1, 17, 20, 130, 80, 3, 3, 1, 1),
          (2, 9, 33, 64, 80, 3, 3, 1, 1), (2, 32, 28, 28, 64, 3, 3, 1, 1), (1, 8, 27, 33, 16, 3, 3, 1, 1), (1, 20, 16, 126, 33, 3, 3, 1, 1),
          (1, 31, 30, 29, 48, 2, 2, 1, 0), (1, 17, 12, 60, 17, 1, 5, 1, 0), (1, 40, 20, 30, 300, 3, 3, 1, 1),
          (2, 48, 30, 33, 64, 1, 1, 2, 0), (1, 16, 65, 64, 40, 3, 3, 2, 1), (1, 64, 9, 8, 70, 3, 3, 2, 1), (1, 70, 20, 30, 33, 1, 1, 1, 0),
          (1, 16, 40, 82, 48, 4, 3, 1, 1), (3, 32, 40, 46, 64, 6, 2, 1, 1), (1, 130, 30, 33, 100, 5, 5, 1, 2), (1, 100, 41, 37, 130, 5, 5, 2, 2), (1, 70, 20, 61, 130, 5, 5, 1, 0)]


@pytest.mark.parametrize("layer", LAYERS)
@pytest.mark.parametrize("kind", ["normal", "one image wide"])
def test_layers_at_the_edges_of_their_tiles(T, port, layer, kind):
    n, c, h, w, ko, kh, kw, stride, pad = layer
    rng = np.random.default_rng(sum(layer))
    x = rng.standard_normal((n, c, h, w)).astype(np.float32)
    if kind != "normal":  # the last image spans more powers of two than float16 pairs hold
        x[-1, 0, h // 2, w // 2] = 1e-20
    f = rng.standard_normal((ko, c, kh, kw)).astype(np.float32)
    b = rng.standard_normal(ko).astype(np.float32)
    got = T.conv2d(T.from_numpy(x), T.from_numpy(f), T.from_numpy(b), stride, pad, "relu")
    T.check_async()
    want = port.conv2d(x, f, b, stride, pad, 1)
    size = port.conv2d(np.abs(x), np.abs(f), np.abs(b), stride, pad, 0)
    assert np.all(np.abs(got.numpy() - want) <= BOUND * size)
    ho, wo = want.shape[2:]
    if stride == 1 and ho % 2 == 0 and wo % 2 == 0:  # the fused pool has the bytes of the two steps
        pooled = T.conv2d(T.from_numpy(x), T.from_numpy(f), T.from_numpy(b), stride, pad, "relu", pool=2)
        assert pooled.numpy().tobytes() == T.maxpool2d(got, 2).numpy().tobytes()


# Several passes to a pair of blocks: images of both forms next to each other, one tile to an image (the halves of a pair differ, and the
# last has no partner) and two; filters that stay in shared memory, in both layouts, and filters that are streamed, in two tiles.
@pytest.mark.parametrize("layer", [(161, 40, 10, 10, 40, 3, 3, 1, 1), (80, 40, 12, 12, 128, 3, 3, 1, 1), (45, 196, 13, 13, 130, 3, 3, 1, 1)])
def test_images_of_both_forms_in_one_batch(T, port, layer):
    n, c, h, w, ko, kh, kw, stride, pad = layer
    rng = np.random.default_rng(sum(layer))
    x = rng.standard_normal((n, c, h, w)).astype(np.float32)
    wide = rng.random(n) < 0.3
    wide[-1], wide[-2] = True, False
    x[wide, 0, 3, 3] = 1e-20
    f = rng.standard_normal((ko, c, kh, kw)).astype(np.float32)
    tf = T.from_numpy(f)
    got = T.conv2d(T.from_numpy(x), tf, None, stride, pad).numpy()
    T.check_async()
    assert np.all(np.abs(got - port.conv2d(x, f, None, stride, pad, 0)) <= BOUND * port.conv2d(np.abs(x), np.abs(f), None, stride, pad, 0))
    for i in (0, 7, n - 2, n - 1):  # an image's bytes do not depend on the others
        same = T.conv2d(T.from_numpy(np.stack([x[i]] * n)), tf, None, stride, pad).numpy()
        assert same[0].tobytes() == same[-1].tobytes() == got[i].tobytes()


# Few channels: five passes and more to a block or pair of blocks, an odd number of tiles, three to an image; by pairs from the input as it is and
# from planes, by single blocks so (up to 16 channels; filters that pairs would pad).  Images that no float16 pair holds stand alone, in
# pairs and in rows, so that every mixture of the two forms meets every accumulator set and stage; each image's bytes are those of the same image in a
# batch of its own, which single blocks compute.
@pytest.mark.parametrize("layer", [(301, 32, 26, 28, 64), (301, 20, 26, 29, 48), (251, 14, 26, 28, 40), (251, 14, 26, 29, 40), (301, 20, 26, 28, 48)])
def test_few_channel_layers_of_many_passes(T, port, layer):
    n, c, h, w, ko = layer
    rng = np.random.default_rng(sum(layer))
    kinds = rng.standard_normal((6, c, h, w)).astype(np.float32)
    kinds[4, 1, 9, 9] = 1e-20           # one tile spans too much
    kinds[5, 0, 2], kinds[5, 2, -2] = 1e-15, 2e10  # two do
    f = rng.standard_normal((ko, c, 3, 3)).astype(np.float32)
    tf = T.from_numpy(f)
    alone = np.concatenate([T.conv2d(T.from_numpy(kinds[i : i + 1]), tf, None, 1, 0).numpy() for i in range(6)])
    assert np.all(np.abs(alone - port.conv2d(kinds, f, None, 1, 0, 0)) <= BOUND * port.conv2d(np.abs(kinds), np.abs(f), None, 1, 0, 0))
    which = np.where(rng.random(n) < 0.4, rng.integers(4, 6, n), rng.integers(0, 4, n))
    which[100:110], which[-1] = 5, 4
    x = T.from_numpy(kinds[which])
    got, pooled = T.conv2d(x, tf, None, 1, 0).numpy(), T.conv2d(x, tf, None, 1, 0, pool=2).numpy()
    T.check_async()
    small = T.maxpool2d(T.from_numpy(alone), 2).numpy()
    for i in range(n):
        assert got[i].tobytes() == alone[which[i]].tobytes(), i
        assert pooled[i].tobytes() == small[which[i]].tobytes(), i


# Stride 3 takes its nine sub-images to the halo kernel from 16384 outputs per filter on: odd and unequal extents, padding, taps that leave five
# sub-images unread, rows and columns that no tap reaches, and images of both forms.
@pytest.mark.parametrize("layer", [(33, 48, 72, 72, 64, 3, 1), (33, 33, 73, 71, 70, 3, 1), (41, 40, 67, 70, 40, 2, 0), (30, 40, 71, 74, 40, 5, 2)])
def test_layers_at_stride_three(T, port, layer):
    n, c, h, w, ko, kern, pad = layer
    rng = np.random.default_rng(sum(layer))
    kinds = rng.standard_normal((3, c, h, w)).astype(np.float32)
    kinds[2, 1, 9, 7] = 1e-20
    f, b = (rng.standard_normal(shape).astype(np.float32) for shape in ((ko, c, kern, kern), (ko,)))
    which = rng.integers(0, 3, n)
    got = T.conv2d(T.from_numpy(kinds[which]), T.from_numpy(f), T.from_numpy(b), 3, pad).numpy()
    T.check_async()
    want = port.conv2d(kinds, f, b, 3, pad, 0)
    size = port.conv2d(np.abs(kinds), np.abs(f), np.abs(b), 3, pad, 0)
    for i, k in enumerate(which):
        assert np.all(np.abs(got[i] - want[k]) <= BOUND * size[k]), i
        assert got[i].tobytes() == got[np.flatnonzero(which == k)[0]].tobytes(), i


def test_a_batch_whose_planes_come_in_parts(T, port):
    """4.7 GB of planes where 4 are taken at a time: an odd batch in two unequal parts, each image as by itself."""
    rng = np.random.default_rng(3)
    kinds = rng.standard_normal((5, 64, 64, 64)).astype(np.float32)
    kinds[4, 0, 3, 3] = 1e-20
    f = rng.standard_normal((17, 64, 3, 3)).astype(np.float32)
    tf = T.from_numpy(f)
    alone = T.conv2d(T.from_numpy(kinds), tf, None, 1, 1).numpy()
    assert np.all(np.abs(alone - port.conv2d(kinds, f, None, 1, 1, 0)) <= BOUND * port.conv2d(np.abs(kinds), np.abs(f), None, 1, 1, 0))
    which = rng.integers(0, 5, 2101)
    got = T.conv2d(T.from_numpy(kinds[which]), tf, None, 1, 1).numpy()
    T.check_async()
    assert all(got[i].tobytes() == alone[k].tobytes() for i, k in enumerate(which))


# rows and columns that fill no tile, k at the edges of a slice and of its sixteen-value steps, an empty last slice
# (k = 770: eight slices of 112, the last one with none), rows and columns that are not 16-byte aligned
@pytest.mark.parametrize("m,k,n", [(1, 193, 33), (64, 784, 1024), (129, 257, 127), (128, 512, 512), (100, 770, 130), (65, 1023, 70), (30, 1024, 1800)])
@pytest.mark.parametrize("kind", ["plain", "small values", "ninety powers of two", "infinity"])
def test_small_products_in_one_launch(T, m, k, n, kind):
    rng = np.random.default_rng(m + 3 * k + n)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    if kind == "small values":
        a[m // 2, k // 3], b[k // 2, n // 3] = 1e-20, 1e-25
    if kind == "ninety powers of two":
        a *= np.exp2(rng.integers(-45, 45, (m, k))).astype(np.float32)
    if kind == "infinity":
        a[m // 2, k - 1], b[0, n // 2] = np.inf, np.nan
    got = T.matmul(T.from_numpy(a), T.from_numpy(b)).numpy()
    T.check_async()
    with np.errstate(invalid="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite)
    size = np.abs(np.where(np.isfinite(a), a, 0)).astype(np.float64) @ np.abs(np.where(np.isfinite(b), b, 0))
    assert np.all(np.abs(got[finite] - want[finite]) <= BOUND * size[finite])


# Many rows and eight to sixteen columns (the float64 MMA): columns beside the first eight, columns that there are not, tiles of eight
# and of sixteen rows that end ragged, k of less than a step, of one value more and of several steps.
# Bound: products are exact and summed in float64 (k additions of 2^-53 of the sum of magnitudes), rounded to float32 once.
@pytest.mark.parametrize("m,k,n", [(2401, 785, 13), (2403, 31, 8), (4741, 33, 10), (4740, 128, 12), (4739, 1, 9), (18951, 97, 16), (18949, 65, 7),
                                   (18945, 40, 8), (38001, 70, 11), (5001, 896, 15)])
@pytest.mark.parametrize("act", ["none", "softmax"])
def test_many_rows_of_few_columns(T, port, m, k, n, act):
    rng = np.random.default_rng(m + k + n)
    x, w, b = (rng.standard_normal(shape).astype(np.float32) for shape in ((m, k), (k, n), (n,)))
    if act == "none":
        x[m - 1, k - 1], x[m // 2, 0] = np.nan, np.inf
    got = T.dense(T.from_numpy(x), T.from_numpy(w), T.from_numpy(b), act).numpy()
    T.check_async()
    with np.errstate(invalid="ignore"):
        want = x.astype(np.float64) @ w.astype(np.float64) + b
    if act == "softmax":
        # a logit is off by half a unit in the last place, 2^-24 of it; its exponential, the sum and the quotient by 2^-21 in all, and below
        # the smallest normal value nothing is promised
        e = np.exp(want - want.max(axis=1, keepdims=True))
        want = e / e.sum(axis=1, keepdims=True)
        logit = np.abs(x.astype(np.float64) @ w + b).max()
        assert np.all(np.abs(got - want) <= want * (2.0**-21 + 2.0**-22 * logit) + 2.0**-126)
        return
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite) and np.array_equal(np.isnan(got), np.isnan(want))
    size = np.abs(np.where(np.isfinite(x), x, 0)).astype(np.float64) @ np.abs(w).astype(np.float64) + np.abs(b)
    assert np.all(np.abs(got[finite] - want[finite]) <= 2.0**-24 * np.abs(want[finite]) + (k + 1) * 2.0**-53 * size[finite])


# The transposed left operand with eight to sixteen columns: rows that end in each part of a warp's 64 and leave a warp without any,
# k of less than four values, of one more than a chunk and of several slices; single chunks that would nearly fill the machine, and pairs of them.
# The bound is the one above.
@pytest.mark.parametrize("m,k,n", [(1, 3, 8), (63, 33, 10), (65, 32, 9), (321, 500, 12), (785, 5003, 10), (257, 20001, 16), (130, 77, 7), (640, 129, 13),
                                   (100, 32999, 13), (250, 17003, 8), (190, 45001, 10)])
def test_transposed_operand_and_few_columns(T, m, k, n):
    rng = np.random.default_rng(m + k + n)
    x, y = (rng.standard_normal(shape).astype(np.float32) for shape in ((k, m), (k, n)))
    x[0, m - 1], x[k - 1, 0] = np.inf, np.nan
    got = T.matmul_tn(T.from_numpy(x), T.from_numpy(y)).numpy()
    T.check_async()
    with np.errstate(invalid="ignore"):
        want = x.T.astype(np.float64) @ y.astype(np.float64)
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite) and np.array_equal(np.isnan(got), np.isnan(want))
    size = np.abs(np.where(np.isfinite(x), x, 0)).T.astype(np.float64) @ np.abs(y).astype(np.float64)
    assert np.all(np.abs(got[finite] - want[finite]) <= 2.0**-24 * np.abs(want[finite]) + (k + 1) * 2.0**-53 * size[finite])


# one tile of columns: chunks of 128 values of k that end ragged, slices of unequal length, rows that are 16-byte aligned and rows that are
# not, and operands that are left to the product from planes; the first has too few tiles for it
@pytest.mark.parametrize("m,k,n", [(3300, 2100, 100), (4200, 4099, 128), (6500, 2050, 33), (6500, 2100, 100), (4200, 4100, 128)])
@pytest.mark.parametrize("kind", ["plain", "small value in A", "small value in B", "infinity", "ninety powers of two"])
def test_tall_products_with_one_tile_of_columns(T, m, k, n, kind):
    rng = np.random.default_rng(m + k + n)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    if kind == "small value in A":
        a[m // 2, k // 3] = 1e-20
    if kind == "small value in B":
        b[k // 2, n // 3] = 1e-20
    if kind == "infinity":
        a[m - 1, k - 1] = np.inf
    if kind == "ninety powers of two":
        a *= np.exp2(rng.integers(-45, 45, (m, k))).astype(np.float32)
    for _ in range(2):  # the mark of the first call is gone
        got = T.matmul(T.from_numpy(a), T.from_numpy(b)).numpy()
    T.check_async()
    with np.errstate(invalid="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite)
    size = np.abs(np.where(np.isfinite(a), a, 0)).astype(np.float64) @ np.abs(b).astype(np.float64)
    assert np.all(np.abs(got[finite] - want[finite]) <= BOUND * size[finite])


# the same as layers, with bias and relu, from the weights and from packed ones: panel product, the three launches behind it, and
# two that prepare the weights where they are not packed
@pytest.mark.parametrize("m,k,n", [(6500, 2100, 100), (4200, 4100, 128), (4200, 4099, 128), (6500, 2050, 33)])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("kind", ["plain", "small values", "infinity"])
def test_tall_layers_with_one_tile_of_columns(T, m, k, n, packed, kind):
    from camel_b200._lib import lib

    rng = np.random.default_rng(m + k + n)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    w = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    b = rng.uniform(-1, 1, n).astype(np.float32)
    if kind == "small values":
        a[m // 2, k // 3], w[k // 2, n // 3] = 1e-20, 1e-25
    if kind == "infinity":
        a[m - 1, k - 1] = np.inf
    ta, tw, tb = T.from_numpy(a), T.from_numpy(w), T.from_numpy(b)
    T.set_weight_cache(packed)
    try:
        first = T.dense(ta, tw, tb, "relu").numpy()
        launches = lib.ct_launch_count()
        got = T.dense(ta, tw, tb, "relu")
        launches = lib.ct_launch_count() - launches
        got = got.numpy()
    finally:
        T.set_weight_cache(True)
    T.check_async()
    assert launches == (4 if packed else 6) and got.tobytes() == first.tobytes()
    rows = np.isfinite(a).all(axis=1)
    a64, w64 = a[rows].astype(np.float64), w.astype(np.float64)
    assert np.all(np.abs(got[rows] - np.maximum(a64 @ w64 + b, 0.0)) <= BOUND * (np.abs(a64) @ np.abs(w64) + np.abs(b)))
    assert not np.isfinite(got[~rows]).any()


# rows of the result that begin anywhere in a line, one tile to a pair: a last tile of one, 33 and 129 columns, whole last tiles, rows
# that end inside a warp's 32
@pytest.mark.parametrize("m,k,n", [(1281, 65, 1793), (2305, 771, 1057), (1537, 100, 1665), (1280, 40, 2047), (4609, 130, 514)])
@pytest.mark.parametrize("kind", ["plain", "small value", "infinity"])
def test_results_whose_rows_are_not_aligned(T, m, k, n, kind):
    rng = np.random.default_rng(m + k + n)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    c = rng.uniform(-1, 1, n).astype(np.float32)
    if kind == "small value":
        a[m // 2, k // 3] = 1e-20
    if kind == "infinity":
        a[m - 1, k - 1] = np.inf
    got = T.dense(T.from_numpy(a), T.from_numpy(b), T.from_numpy(c), "relu").numpy()
    plain = T.matmul(T.from_numpy(a), T.from_numpy(b)).numpy()
    T.check_async()
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    product = a64 @ b64
    want, rows = np.maximum(product + c, 0.0), np.isfinite(a).all(axis=1)
    size = np.abs(a64[rows]) @ np.abs(b64) + np.abs(c)
    assert np.all(np.abs(got[rows] - want[rows]) <= BOUND * size)
    assert np.all(np.abs(plain[rows] - product[rows]) <= BOUND * size)
    # infinity, or NaN where the two terms of the other operand's value have opposite signs (inf - inf)
    assert not np.isfinite(plain[~rows]).any()


@pytest.mark.parametrize("k,n", [(1030, 130), (1100, 257), (2050, 64), (1088, 1)])
@pytest.mark.parametrize("precision", [0, 1])
def test_right_operands_in_blocks(T, k, n, precision):
    from camel_b200._lib import lib, check

    m = 2400  # several tiles of rows: no slices
    rng = np.random.default_rng(k + n)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, max(n, 33))).astype(np.float32)
    check(lib.ct_set_precision(precision))
    try:
        got = T.matmul(T.from_numpy(a), T.from_numpy(b)).numpy()
        T.check_async()
    finally:
        check(lib.ct_set_precision(0))
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    assert np.all(np.abs(got - a64 @ b64) <= (2.0 ** -7 if precision else BOUND) * (np.abs(a64) @ np.abs(b64)))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 4095, 4096, 4097, 16387])
def test_elements_behind_the_last_vector(T, port, n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    ta, tb = T.from_numpy(a), T.from_numpy(b)
    assert T.add(ta, tb).numpy().tobytes() == port.binary(oracle.ADD, a, b).tobytes()
    assert T.multiply(ta, tb).numpy().tobytes() == port.binary(oracle.MUL, a, b).tobytes()


def test_fused_pool_takes_its_window_in_the_order_of_maxpool2d(T):
    """A window (small, small, NaN, large): an output beyond the range of float32 is -infinity, which relu makes NaN, beside
    finite ones.  The largest value behind the NaN counts, in the fused form as in the two steps."""
    n, c, h, w, ko = 2, 32, 28, 32, 64
    rng = np.random.default_rng(5)
    x = rng.uniform(0.5, 1, (n, c, h, w)) * 2.0 ** 40
    x[:, :, 1::2, 0::2], x[:, :, 1::2, 1::2] = -1.99 * 2.0 ** 60, 1.99 * 2.0 ** 60
    f = np.zeros((ko, c, 1, 5))
    f[:, :, 0, 0], f[:, :, 0, 1] = 1.9 * 2.0 ** 60, -1.9 * 2.0 ** 60  # lower rows: -+ 3.2e38 in turn
    b = np.full(ko, -1e38)  # the negative ones leave the range, the positive ones are 2.2e38
    tx, tf, tb = (T.from_numpy(v.astype(np.float32)) for v in (x, f, b))
    full = T.conv2d(tx, tf, tb, 1, 0, "relu")
    values = full.numpy()
    assert np.isnan(values[:, :, 1::2, 0::2]).all() and (values[:, :, 1::2, 1::2] > 2e38).all()
    fused = T.conv2d(tx, tf, tb, 1, 0, "relu", pool=2).numpy()
    T.check_async()
    assert fused.tobytes() == T.maxpool2d(full, 2).numpy().tobytes()
    assert (fused > 2e38).all()


# the rows of the input that hold 2^-50, the others hold 2^-66: the image fits float16 pairs, tiles of its rows lie below 2^-60
@pytest.mark.parametrize("rows", [(0, 14), (20, 28)])
@pytest.mark.parametrize("pool", [0, 2])
def test_tiles_below_the_smallest_exponent_of_an_image_that_fits(T, port, rows, pool):
    from camel_b200._lib import check, lib

    n, c, h, w, ko = 3, 32, 28, 28, 64
    rng = np.random.default_rng(rows[0])
    x = rng.uniform(0.5, 1, (n, c, h, w)) * rng.choice([-1, 1], (n, c, h, w))
    x *= np.where((np.arange(h) >= rows[0]) & (np.arange(h) < rows[1]), 2.0 ** -50, 2.0 ** -66)[:, None]
    x, f = x.astype(np.float32), rng.uniform(0.1, 1, (ko, c, 3, 3)).astype(np.float32)
    want, size = port.conv2d(x, f, np.zeros(ko, np.float32), 1, 1, 0), port.conv2d(np.abs(x), f, np.zeros(ko, np.float32), 1, 1, 0)
    side = h // 2 if pool else h
    out = T.full((n, ko, side, side), 7.0)  # what a tile that nobody computes would keep
    tx, tf = T.from_numpy(x), T.from_numpy(f)
    check((lib.ct_conv2d_maxpool2 if pool else lib.ct_conv2d)(tx.ptr, tf.ptr, None, n, c, h, w, ko, 3, 3, 1, 1, 0, out.ptr))
    got = out.numpy()
    T.check_async()
    if pool:
        assert got.tobytes() == T.maxpool2d(T.conv2d(tx, tf, None, 1, 1, None), 2).numpy().tobytes()
        want, size = (v.reshape(n, ko, side, 2, side, 2).max(axis=(3, 5)) for v in (want, size))
    assert np.all(np.abs(got - want) <= BOUND * size)


@pytest.mark.parametrize("layer", [(65540, 8, 8, 9, 16, 3, 3, 1, 1), (65540, 17, 8, 9, 16, 3, 3, 1, 1)])
def test_more_images_than_a_pre_pass_takes(T, port, layer):
    n, c, h, w, ko, kh, kw, stride, pad = layer
    rng = np.random.default_rng(c)
    x = rng.standard_normal((n, c, h, w), dtype=np.float32)
    f, b = rng.standard_normal((ko, c, kh, kw)).astype(np.float32), rng.standard_normal(ko).astype(np.float32)
    got = T.conv2d(T.from_numpy(x), T.from_numpy(f), T.from_numpy(b), stride, pad, "relu").numpy()
    T.check_async()
    some = np.r_[0:6, 65530:n]
    want = port.conv2d(x[some], f, b, stride, pad, 1)
    size = port.conv2d(np.abs(x[some]), np.abs(f), np.abs(b), stride, pad, 0)
    assert np.all(np.abs(got[some] - want) <= BOUND * size)


@pytest.mark.parametrize("packed", [False, True])
def test_tall_products_add_what_float16_pairs_cannot_hold_in_order_of_k(T, packed):
    """Several such values in a column, from blocks of the pre-pass that finish in any order, and in a row.  The outputs that
    consist of them alone are the float32 sums in order of k, to the bit."""
    m, k, n, row, col = 3200, 4100, 100, 777, 41
    rng = np.random.default_rng(11)
    a, b = rng.uniform(-1, 1, (m, k)).astype(np.float32), (rng.integers(-255, 256, (k, n)) / 256).astype(np.float32)
    meet = np.arange(128, 1024, 128)  # in the first slice of k; what keeps the scales of row and column meets zeros there
    b[meet] = 0.0
    a[row] = 0.0
    a[row, meet] = 0.75
    ks_a = np.sort(np.concatenate([meet[:4] + d for d in (1, 40, 127)]))
    a[row, ks_a] = rng.uniform(1, 2, ks_a.size) * np.exp2(rng.integers(-40, -30, ks_a.size))
    rows = np.arange(100, 110)
    a[rows, 0] = 0.0
    b[:, col], b[0, col] = 0.0, 0.75
    ks_b = 66 * np.arange(1, 15)
    b[ks_b, col] = rng.uniform(1, 2, ks_b.size) * np.exp2(rng.integers(-40, -30, ks_b.size))
    ta, tb = T.from_numpy(a), T.from_numpy(b)
    T.set_weight_cache(packed)
    try:
        outs = [T.dense(ta, tb).numpy() for _ in range(10)]
    finally:
        T.set_weight_cache(True)
    T.check_async()
    assert all(o.tobytes() == outs[0].tobytes() for o in outs)
    for r in rows:
        want = np.float32(0)
        for kk in ks_b:
            want = np.float32(want + np.float32(a[r, kk] * b[kk, col]))
        assert outs[0][r, col] == want
    others = np.delete(np.arange(n), col)
    want = np.zeros(n - 1, np.float32)
    for kk in ks_a:  # one rounding: the product and the sum fit 53 bits
        want = (want.astype(np.float64) + a[row, kk].astype(np.float64) * b[kk, others].astype(np.float64)).astype(np.float32)
    assert np.array_equal(outs[0][row, others], want)


def test_pooled_layer_in_parts_of_the_batch(T):
    """More than 256 MB of activations: three parts of 190, 190 and 188 images, the bytes of the two steps over the whole batch.
    Images of wide range, which decide for themselves, lie on both sides of the cuts."""
    n, c, h, w, ko = 568, 33, 64, 64, 64
    rng = np.random.default_rng(8)
    x = rng.standard_normal((n, c, h, w), dtype=np.float32)
    x[[0, 189, 190, 380, 567], 5, 30, 20] = 1e-20
    f, b = (rng.standard_normal((ko, c, 3, 3)) / 17).astype(np.float32), rng.standard_normal(ko).astype(np.float32)
    tx, tf, tb = T.from_numpy(x), T.from_numpy(f), T.from_numpy(b)
    fused = T.conv2d(tx, tf, tb, 1, 1, "relu", pool=2).numpy()
    full = T.conv2d(tx, tf, tb, 1, 1, "relu")
    T.check_async()
    assert full.nbytes > 2 * (256 << 20) and fused.tobytes() == T.maxpool2d(full, 2).numpy().tobytes()
