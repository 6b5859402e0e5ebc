"""The calls whose speed this library is judged by.

Every case goes through the C ABI of libcamel_tensor_b200.so (include/camel_tensor_b200.h) on device
buffers that the program owns, which is how an operator body of the tensor module calls it.  Sizes are
those of the benchmark's own configurations (GEMM 512 and 16384, the 784-1024-1024-10 MLP, the 64 -> 128
channel convolution, the 28 x 28 CNN, the 60000 x 785 x 10 training step) and ragged ones of the same
ranges; `draw` spreads over those ranges.
"""
import ctypes as C
import math

import torch

from camel_b200 import _lib as L
from camel_b200._lib import check, lib

F32, I64, BOOL = L.F32, L.I64, L.BOOL


# ---- the cases --------------------------------------------------------------------------------------


def listed():
    return [
        # one product of the smallest benchmark configuration: launches and latency count
        dict(name="matmul_512", kind="matmul", m=512, k=512, n=512, bf16=False),
        # a product whose sizes fit no tile, as data sets give them
        dict(name="matmul_ragged", kind="matmul", m=1537, k=771, n=2050, bf16=False),
        # the largest product: the tensor pipe under the power cap
        dict(name="matmul_16384", kind="matmul", m=16384, k=16384, n=16384, bf16=False),
        # the reduced-precision option of the same entry point
        dict(name="matmul_bf16_8192", kind="matmul", m=8192, k=8192, n=8192, bf16=True),
        # a classifier answering a small request: three layers replayed as one recorded graph
        dict(name="mlp_64", kind="mlp", batch=64, width=1024, graph=True),
        # the same classifier over a full batch, layer by layer with packed weights
        dict(name="mlp_4096", kind="mlp", batch=4096, width=1024, graph=False),
        # a wide convolution layer with bias and relu
        dict(name="conv_64_128", kind="conv", batch=256, c=64, h=56, w=56, ko=128, kern=3, stride=1, pad=1),
        # a down-sampling layer on odd sizes
        dict(name="conv_stride2", kind="conv", batch=64, c=48, h=57, w=57, ko=96, kern=3, stride=2, pad=1),
        # a whole small network: two convolutions, pool, two dense layers
        dict(name="cnn_8192", kind="cnn", batch=8192),
        # one update step of softmax regression on an image data set with a bias column
        dict(name="train_60000", kind="train", rows=60000, d=785, classes=10, lr=1e-5),
        # a chain of elementwise operators on one large vector
        dict(name="elementwise_64m", kind="elementwise", n=1 << 26),
        # row and column operators on one large matrix
        dict(name="rows_8192", kind="rows", rows=8192, cols=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "mlp", "conv", "conv", "cnn", "train", "elementwise", "rows"])
    if kind == "matmul":
        return dict(kind=kind, m=_log_int(rng, 64, 16384), k=_log_int(rng, 64, 16384), n=_log_int(rng, 64, 16384),
                    bf16=rng.random() < 0.2)
    if kind == "mlp":
        batch = _log_int(rng, 1, 16384)
        return dict(kind=kind, batch=batch, width=rng.randint(16, 288) * 8, graph=batch <= 512)
    if kind == "conv":
        side, kern = rng.randint(12, 72), rng.choice([1, 3, 3, 5])
        return dict(kind=kind, batch=_log_int(rng, 4, 256), c=_log_int(rng, 8, 192), h=side, w=side + rng.choice([0, 0, 2, 3]),
                    ko=_log_int(rng, 16, 192), kern=kern, stride=rng.choice([1, 1, 1, 2]), pad=rng.choice([0, kern // 2]))
    if kind == "cnn":
        return dict(kind=kind, batch=_log_int(rng, 16, 8192))
    if kind == "train":
        return dict(kind=kind, rows=_log_int(rng, 500, 100000), d=_log_int(rng, 50, 1600), classes=rng.randint(2, 16), lr=1e-5)
    if kind == "elementwise":
        return dict(kind=kind, n=_log_int(rng, 1000, 1 << 27))
    return dict(kind=kind, rows=_log_int(rng, 16, 16384), cols=_log_int(rng, 8, 8192))


# ---- inputs -----------------------------------------------------------------------------------------


class _Packed:
    """Packed weights kept with the program's weights, freed with them."""

    def __init__(self, w):
        self.handle = C.c_void_p()
        check(lib.ct_weights_pack(w.data_ptr(), w.shape[0], w.shape[1], C.byref(self.handle)))

    def __del__(self):
        lib.ct_weights_free(self.handle)


class _Graph:
    """A recorded sequence of calls."""

    def __init__(self, calls):
        self.handle = C.c_void_p()
        calls()
        check(lib.ct_sync())
        check(lib.ct_graph_begin())
        try:
            calls()
        finally:
            check(lib.ct_graph_end(C.byref(self.handle)))

    def launch(self):
        check(lib.ct_graph_launch(self.handle))

    def __del__(self):
        lib.ct_graph_destroy(self.handle)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, device="cuda", generator=g) * (hi - lo) + lo


def _normal(g, std, *shape):
    return torch.randn(*shape, device="cuda", generator=g) * std


def _kaiming(g, fan_in, *shape):
    lim = math.sqrt(6.0 / fan_in)
    return _uniform(g, -lim, lim, *shape)


def _out(*shape, dtype=torch.float32):
    return torch.empty(*shape, device="cuda", dtype=dtype)


def _conv_out(case):
    side = lambda v: (v + 2 * case["pad"] - case["kern"]) // case["stride"] + 1  # noqa: E731
    return side(case["h"]), side(case["w"])


def _inputs(case, seed):
    """The tensors a program holds, from the seed alone."""
    g, kind = _gen(seed), case["kind"]
    if kind == "matmul":
        return dict(a=_uniform(g, -1, 1, case["m"], case["k"]), b=_uniform(g, -1, 1, case["k"], case["n"]))
    if kind == "mlp":
        dims = [784, case["width"], case["width"], 10]
        s = dict(x=_uniform(g, 0, 1, case["batch"], 784))
        for i in range(3):
            s["w%d" % i] = _kaiming(g, dims[i], dims[i], dims[i + 1])
            s["b%d" % i] = _uniform(g, -0.1, 0.1, dims[i + 1])
        return s
    if kind == "conv":
        fan = case["c"] * case["kern"] ** 2
        return dict(x=_normal(g, 1.0, case["batch"], case["c"], case["h"], case["w"]),
                    w=_normal(g, math.sqrt(2.0 / fan), case["ko"], case["c"], case["kern"], case["kern"]),
                    b=_normal(g, 0.1, case["ko"]))
    if kind == "cnn":
        return dict(x=_uniform(g, 0, 1, case["batch"], 1, 28, 28),
                    c1=_kaiming(g, 9, 32, 1, 3, 3), d1=_uniform(g, -0.1, 0.1, 32),
                    c2=_kaiming(g, 288, 64, 32, 3, 3), d2=_uniform(g, -0.1, 0.1, 64),
                    w1=_kaiming(g, 12544, 12544, 128), b1=_uniform(g, -0.1, 0.1, 128),
                    w2=_kaiming(g, 128, 128, 10), b2=_uniform(g, -0.1, 0.1, 10))
    if kind == "train":
        x = _uniform(g, 0, 1, case["rows"], case["d"])
        x[:, -1] = 1.0  # the bias column
        label = torch.randint(case["classes"], (case["rows"],), device="cuda", generator=g)
        y = torch.nn.functional.one_hot(label, case["classes"]).to(torch.float32).contiguous()
        return dict(x=x, y=y, w=_normal(g, 0.05, case["d"], case["classes"]))
    if kind == "elementwise":
        return dict(a=_uniform(g, -4, 4, case["n"]), b=_uniform(g, 0.1, 4, case["n"]))
    return dict(a=_normal(g, 2.0, case["rows"], case["cols"]), b=_normal(g, 1.0, case["rows"], 16))


def prepare(case, seed):
    check(lib.ct_set_precision(L.PREC_3XTF32))
    s, kind = _inputs(case, seed), case["kind"]
    s["case"] = case
    if kind == "matmul":
        s["out"] = _out(case["m"], case["n"])
    elif kind == "mlp":
        n, width = case["batch"], case["width"]
        s.update(p0=_Packed(s["w0"]), p1=_Packed(s["w1"]), h0=_out(n, width), h1=_out(n, width), probs=_out(n, 10),
                 arg=_out(n, dtype=torch.int64))
        if case["graph"]:
            s["graph"] = _Graph(lambda: _mlp(s))
    elif kind == "conv":
        s["out"] = _out(case["batch"], case["ko"], *_conv_out(case))
    elif kind == "cnn":
        n = case["batch"]
        s.update(p1=_Packed(s["w1"]), y1=_out(n, 32, 28, 28), y2=_out(n, 64, 14, 14), y3=_out(n, 128), probs=_out(n, 10),
                 arg=_out(n, dtype=torch.int64))
    elif kind == "train":
        r, d, c = case["rows"], case["d"], case["classes"]
        s.update(probs=_out(r, c), err=_out(r, c), grad=_out(d, c), new=_out(d, c))
    elif kind == "elementwise":
        n = case["n"]
        s.update(add=_out(n), mul=_out(n), scale=_out(n), relu=_out(n), exp=_out(n), log=_out(n), gt=_out(n, dtype=torch.uint8))
    else:
        r, c = case["rows"], case["cols"]
        s.update(softmax=_out(r, c), sum0=_out(c), sum1=_out(r), max1=_out(r), arg1=_out(r, dtype=torch.int64), t=_out(c, r),
                 cat=_out(r, c + 16))
    return s


# ---- one pass ---------------------------------------------------------------------------------------


def _p(t):
    return t.data_ptr()


def _mlp(s):
    n, width = s["case"]["batch"], s["case"]["width"]
    check(lib.ct_dense_packed(_p(s["x"]), _p(s["w0"]), s["p0"].handle, _p(s["b0"]), n, 784, width, L.ACT_RELU, _p(s["h0"]), None))
    check(lib.ct_dense_packed(_p(s["h0"]), _p(s["w1"]), s["p1"].handle, _p(s["b1"]), n, width, width, L.ACT_RELU, _p(s["h1"]), None))
    check(lib.ct_dense_packed(_p(s["h1"]), _p(s["w2"]), None, _p(s["b2"]), n, width, 10, L.ACT_SOFTMAX, _p(s["probs"]), _p(s["arg"])))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "matmul":
        check(lib.ct_set_precision(L.PREC_BF16 if case["bf16"] else L.PREC_3XTF32))
        check(lib.ct_matmul(F32, _p(s["a"]), F32, _p(s["b"]), case["m"], case["k"], case["n"], _p(s["out"])))
        check(lib.ct_set_precision(L.PREC_3XTF32))
        return s["out"]
    if kind == "mlp":
        if case["graph"]:
            s["graph"].launch()
        else:
            _mlp(s)
        return dict(h0=s["h0"], h1=s["h1"], probs=s["probs"], arg=s["arg"])
    if kind == "conv":
        check(lib.ct_conv2d(_p(s["x"]), _p(s["w"]), _p(s["b"]), case["batch"], case["c"], case["h"], case["w"], case["ko"],
                            case["kern"], case["kern"], case["stride"], case["pad"], L.ACT_RELU, _p(s["out"])))
        return s["out"]
    if kind == "cnn":
        n = case["batch"]
        check(lib.ct_conv2d(_p(s["x"]), _p(s["c1"]), _p(s["d1"]), n, 1, 28, 28, 32, 3, 3, 1, 1, L.ACT_RELU, _p(s["y1"])))
        check(lib.ct_conv2d_maxpool2(_p(s["y1"]), _p(s["c2"]), _p(s["d2"]), n, 32, 28, 28, 64, 3, 3, 1, 1, L.ACT_RELU, _p(s["y2"])))
        check(lib.ct_dense_packed(_p(s["y2"]), _p(s["w1"]), s["p1"].handle, _p(s["b1"]), n, 12544, 128, L.ACT_RELU, _p(s["y3"]), None))
        check(lib.ct_dense_packed(_p(s["y3"]), _p(s["w2"]), None, _p(s["b2"]), n, 128, 10, L.ACT_SOFTMAX, _p(s["probs"]), _p(s["arg"])))
        return dict(y1=s["y1"], y2=s["y2"], y3=s["y3"], probs=s["probs"], arg=s["arg"])
    if kind == "train":
        r, d, c = case["rows"], case["d"], case["classes"]
        check(lib.ct_dense(_p(s["x"]), _p(s["w"]), None, r, d, c, L.ACT_SOFTMAX, _p(s["probs"]), None))
        check(lib.ct_binary(L.SUB, F32, _p(s["probs"]), F32, _p(s["y"]), r * c, _p(s["err"])))
        check(lib.ct_matmul_tn(_p(s["x"]), _p(s["err"]), d, r, c, _p(s["grad"])))
        check(lib.ct_scaled_sub(_p(s["w"]), _p(s["grad"]), case["lr"], d * c, _p(s["new"])))
        return dict(probs=s["probs"], grad=s["grad"], new=s["new"])
    if kind == "elementwise":
        n, a, b = case["n"], _p(s["a"]), _p(s["b"])
        check(lib.ct_binary(L.ADD, F32, a, F32, b, n, _p(s["add"])))
        check(lib.ct_binary(L.MUL, F32, a, F32, b, n, _p(s["mul"])))
        check(lib.ct_binary_scalar(L.MUL, F32, a, 1.5, F32, 0, n, _p(s["scale"])))
        check(lib.ct_relu(a, n, _p(s["relu"])))
        check(lib.ct_compare(L.GT, F32, a, F32, b, n, _p(s["gt"])))
        check(lib.ct_exp(a, n, _p(s["exp"])))
        check(lib.ct_log(b, n, _p(s["log"])))  # waits for its own error word
        return dict((k, s[k]) for k in ("add", "mul", "scale", "relu", "gt", "exp", "log"))
    r, c, a = case["rows"], case["cols"], _p(s["a"])
    check(lib.ct_softmax_rows(a, r, c, _p(s["softmax"])))
    check(lib.ct_sum_axis(F32, a, r, c, 0, _p(s["sum0"])))
    check(lib.ct_sum_axis(F32, a, r, c, 1, _p(s["sum1"])))
    check(lib.ct_max_axis(F32, a, r, c, 1, _p(s["max1"])))
    check(lib.ct_argmax_axis(F32, a, r, c, 1, _p(s["arg1"])))
    check(lib.ct_transpose(F32, a, r, c, _p(s["t"])))
    check(lib.ct_concat(F32, a, _p(s["b"]), r, c, 16, 1, _p(s["cat"])))
    total = C.c_double()
    check(lib.ct_sum(F32, a, r * c, C.byref(total)))  # a host value: waits
    return dict(softmax=s["softmax"], sum0=s["sum0"], sum1=s["sum1"], max1=s["max1"], arg1=s["arg1"], t=s["t"], cat=s["cat"],
                total=total.value)


# ---- what a pass cannot do without ------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return dict(bytes=4 * (m * k + k * n + m * n), flops=2 * m * k * n)
    if kind == "mlp":
        n, d = case["batch"], case["width"]
        return dict(bytes=4 * (n * (784 + 2 * d + 10 + 2) + 784 * d + d * d + 10 * d + 2 * d + 10),
                    flops=2 * n * (784 * d + d * d + 10 * d))
    if kind == "conv":
        ho, wo = _conv_out(case)
        n, c, ko, t = case["batch"], case["c"], case["ko"], case["kern"] ** 2
        return dict(bytes=4 * (n * c * case["h"] * case["w"] + ko * c * t + ko + n * ko * ho * wo), flops=2 * n * ko * ho * wo * c * t)
    if kind == "cnn":
        n = case["batch"]
        # each activation is written once and read once by the next call
        return dict(bytes=4 * (n * (784 + 2 * 32 * 784 + 2 * 64 * 196 + 2 * 128 + 10 + 2) + 9 * 32 + 288 * 64 + 12544 * 128 + 1280 + 234),
                    flops=2 * n * (784 * 32 * 9 + 784 * 64 * 288 + 12544 * 128 + 1280))
    if kind == "train":
        r, d, c = case["rows"], case["d"], case["classes"]
        return dict(bytes=4 * (2 * r * d + 5 * r * c + 5 * d * c), flops=4 * r * d * c)
    if kind == "elementwise":
        return dict(bytes=case["n"] * (12 + 12 + 8 + 8 + 9 + 8 + 8), flops=0)
    r, c = case["rows"], case["cols"]
    return dict(bytes=4 * (8 * r * c + 3 * r * c + 32 * r) + 4 * c + 16 * r, flops=0)


def tolerance(case):
    kind = case["kind"]
    if kind == "matmul" and case["bf16"]:
        return dict(rel=1e-2, max=0.1)
    # a split-precision product is 1.8e-6 off its value in 64 bits, a convolution layer up to 4e-6 and
    # the second layer of a network 3.3e-6: four times that
    if kind == "matmul":
        return dict(rel=8e-6, max=8e-5)
    if kind == "conv":
        return dict(rel=1.6e-5, max=1.6e-4)
    if kind in ("mlp", "cnn"):
        return dict(rel=1.4e-5, max=2e-4, differ=2e-3)
    if kind == "train":
        return dict(rel=4e-6, max=1e-4)
    return dict(rel=1e-6, max=2e-6)


# ---- the same in 64 bits ----------------------------------------------------------------------------


def _conv64(x, w, b, stride, pad):
    n, c, h, wd = x.shape
    ko, _, kh, kw = w.shape
    ho, wo = (h + 2 * pad - kh) // stride + 1, (wd + 2 * pad - kw) // stride + 1
    out = torch.empty(n, ko, ho, wo, device="cuda", dtype=torch.float64)
    step = max(1, (1 << 28) // (c * kh * kw * ho * wo))
    w2 = w.double().reshape(ko, -1)
    for i in range(0, n, step):
        patches = torch.nn.functional.unfold(x[i:i + step].double(), (kh, kw), padding=pad, stride=stride)
        out[i:i + step] = (w2 @ patches + b.double()[:, None]).reshape(-1, ko, ho, wo)
    return out.relu_()


def exact(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    d = lambda k: s[k].double()  # noqa: E731
    if kind == "matmul":
        return d("a") @ d("b")
    if kind == "mlp":
        h0 = (d("x") @ d("w0") + d("b0")).relu()
        h1 = (h0 @ d("w1") + d("b1")).relu()
        z = h1 @ d("w2") + d("b2")
        return dict(h0=h0, h1=h1, probs=z.softmax(1), arg=z.argmax(1))
    if kind == "conv":
        return _conv64(s["x"], s["w"], s["b"], case["stride"], case["pad"])
    if kind == "cnn":
        y1 = _conv64(s["x"], s["c1"], s["d1"], 1, 1)
        y2 = torch.cat([torch.nn.functional.max_pool2d(_conv64(y1[i:i + 512], s["c2"], s["d2"], 1, 1), 2)
                        for i in range(0, case["batch"], 512)])
        y3 = (y2.reshape(case["batch"], -1) @ d("w1") + d("b1")).relu()
        z = y3 @ d("w2") + d("b2")
        return dict(y1=y1, y2=y2, y3=y3, probs=z.softmax(1), arg=z.argmax(1))
    if kind == "train":
        probs = (d("x") @ d("w")).softmax(1)
        grad = d("x").T @ (probs - d("y"))
        return dict(probs=probs, grad=grad, new=d("w") - case["lr"] * grad)
    if kind == "elementwise":
        a, b = d("a"), d("b")
        return dict(add=a + b, mul=a * b, scale=a * 1.5, relu=a.relu(), gt=None, exp=a.exp(), log=b.log())
    a = d("a")
    return dict(softmax=a.softmax(1), sum0=a.sum(0), sum1=a.sum(1), max1=a.amax(1), arg1=None, t=a.T.contiguous(),
                cat=torch.cat([a, d("b")], 1), total=float(a.sum()))
