"""The surrogate's fused training kernels against plain PyTorch in 64 bits, at batches that fill
no tile of rows and layers at both ends of the sizes they take."""

import ctypes as C

import pytest

from solprop_b200 import _lib, surrogate


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


# FP32 sums of m terms of either sign: their error is below m 2^-24 of the terms' norm, 2e-5 here;
# BF16 values carry 2^-9
@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 31, 32, 33, 200, 257, 1000])
@pytest.mark.parametrize("n", [32, 512])
def test_layer_backward(m, n):
    import torch

    g = torch.Generator(device="cuda").manual_seed(m)
    da = torch.randn(m, n, device="cuda", generator=g)
    pre = torch.randn(m, n, device="cuda", generator=g)
    x = torch.randn(m, 6, device="cuda", generator=g)
    rows = surrogate._pad64(m)
    z = pre.double()
    cdf = 0.5 * (1 + torch.erf(z / 2**0.5))
    dz = da.double() * (cdf + z * torch.exp(-0.5 * z * z) / (2 * torch.pi) ** 0.5)
    for p, want in ((pre, dz), (None, da.double())):
        dz16 = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        dz16t = torch.full((n, rows), float("nan"), dtype=torch.bfloat16, device="cuda")
        db = torch.empty(n, device="cuda")
        pre_ptr = None if p is None else p.data_ptr()
        _lib.check(_lib.library().sp_mlp_layer_backward(da.data_ptr(), pre_ptr, m, n, dz16.data_ptr(),
                                                        dz16t.data_ptr(), rows, db.data_ptr(), None))
        assert _rel(dz16, want) < 2**-8
        assert torch.equal(dz16t[:, :m], dz16.T) and not dz16t[:, m:].any()
        assert _rel(db, want.sum(0)) < 2e-5
        dw, db0 = torch.empty(n, 6, device="cuda"), torch.empty(n, device="cuda")
        _lib.check(_lib.library().sp_mlp_first_layer_backward(da.data_ptr(), pre_ptr, x.data_ptr(), 6, m, n, 6,
                                                              dw.data_ptr(), db0.data_ptr(), None))
        assert _rel(dw, want.T @ x.double()) < 2**-7
        assert _rel(db0, want.sum(0)) < 2e-5


@pytest.mark.gpu
def test_batched_conversion_and_adam():
    import torch

    g = torch.Generator(device="cuda").manual_seed(3)
    xs = [torch.randn(r, c, device="cuda", generator=g) for r, c in ((1, 6), (33, 64), (512, 6), (100, 512))]
    wide, pads = [64, 64, 64, 512], [64, 64, 512, 128]
    new = lambda r, c: torch.full((r, c), float("nan"), dtype=torch.bfloat16, device="cuda")  # noqa: E731
    copies = [new(x.shape[0], c) for x, c in zip(xs, wide)]
    transposes = [new(x.shape[1], r) for x, r in zip(xs, pads)]
    ints = lambda v: (C.c_int * 4)(*v)  # noqa: E731
    pointers = lambda ts: (C.c_void_p * 4)(*[t.data_ptr() for t in ts])  # noqa: E731
    _lib.check(_lib.library().sp_mlp_convert_batch(
        4, 0, pointers(xs), ints(x.shape[0] for x in xs), ints(x.shape[1] for x in xs), ints(x.stride(0) for x in xs),
        pointers(copies), ints(wide), pointers(transposes), ints(pads), None))
    for x, c, t in zip(xs, copies, transposes):
        r, k = x.shape
        assert torch.equal(c[:, :k], x.bfloat16()) and not c[:, k:].any()
        assert torch.equal(t[:, :r], x.bfloat16().T) and not t[:, r:].any()
    for x, pad in zip(xs, pads):  # one matrix on its own, rows of the transpose further apart
        for src in (x, x.bfloat16()):
            t = new(x.shape[1], pad + 3)
            _lib.check(_lib.library().sp_mlp_transpose_bf16(src.data_ptr(), int(src is not x), x.shape[1], *x.shape,
                                                            t.data_ptr(), pad + 3, pad, None))
            assert torch.equal(t[:, :x.shape[0]], x.bfloat16().T) and not t[:, x.shape[0]:pad].any()
            assert t[:, pad:].isnan().all()
            assert torch.equal(surrogate.transpose_bf16(src, pad), t[:, :pad])
    net, one = surrogate.Perceptron(7), surrogate.Perceptron(7)
    grads = [torch.randn(p.shape, device="cuda", generator=g) for p in net.params]
    net.adam(grads, 1e-3)
    for p, gr, m1, m2 in zip(one.params, grads, one.m1, one.m2):
        _lib.check(_lib.library().sp_mlp_adam(p.data_ptr(), gr.data_ptr(), m1.data_ptr(), m2.data_ptr(), p.numel(),
                                              1e-3, 0.9, 0.999, 1e-8, 1, None))
    for a, b in zip(net.params + net.m1 + net.m2, one.params + one.m1 + one.m2):
        assert torch.equal(a, b)


# ---- what the native passes are handed: they read rows by the weights' sizes alone, so a tensor
# of another shape is refused before the call (no GPU: a library that only records its calls)
class _Recorder:
    def __init__(self):
        self.calls = {}

    def __getattr__(self, name):
        def call(*args):
            self.calls[name] = args
            return 256 if name.endswith("scratch") else 0
        return call


def _cpu_member(sizes=(6, 32, 32, 16)):
    import torch

    net = object.__new__(surrogate.Perceptron)
    net.device, net.step = torch.device("cpu"), 0
    net.weights = [torch.zeros(b, a) for a, b in zip(sizes[:-1], sizes[1:])]
    net.biases = [torch.zeros(b) for b in sizes[1:]]
    net.params = [t for pair in zip(net.weights, net.biases) for t in pair]
    net.m1, net.m2 = ([torch.zeros_like(t) for t in net.params] for _ in range(2))
    return net


@pytest.fixture
def recorder(monkeypatch):
    lib = _Recorder()
    monkeypatch.setattr(surrogate, "_bind", lambda: lib)
    return lib


def _cache(net, m):
    import torch

    dims = [w.shape for w in net.weights]
    return [(torch.zeros(m, k, dtype=torch.bfloat16 if i else torch.float32),
             torch.zeros(m, n) if i + 1 < len(dims) else None) for i, (n, k) in enumerate(dims)]


@pytest.mark.parametrize("wrong", ["dy narrow", "dy wide", "dy short", "dy long", "inputs", "activations", "rows",
                                   "pre-activations", "cache"])
def test_backward_refuses_other_shapes(recorder, wrong):
    import torch

    net, m = _cpu_member(), 40
    cache, dy = _cache(net, m), torch.zeros(m, 16)
    net.gradients_tc(cache, dy)
    assert "sp_mlp_training_backward" in recorder.calls
    recorder.calls.clear()
    if wrong.startswith("dy"):
        dy = {"dy narrow": torch.zeros(m, 15), "dy wide": torch.zeros(m, 17), "dy short": torch.zeros(m - 1, 16),
              "dy long": torch.zeros(m + 1, 16)}[wrong]
    elif wrong == "inputs":
        cache[0] = (torch.zeros(m, 5), cache[0][1])
    elif wrong == "activations":
        cache[2] = (cache[2][0][:, :31], cache[2][1])
    elif wrong == "rows":
        cache[1] = (cache[1][0][:-1], cache[1][1])
    elif wrong == "pre-activations":
        cache[1] = (cache[1][0], cache[1][1][:-1])
    else:
        del cache[2]
    with pytest.raises((ValueError, IndexError)):
        net.gradients_tc(cache, dy)
    assert "sp_mlp_training_backward" not in recorder.calls


def test_forward_refuses_inputs_of_another_padded_width(recorder):
    import torch

    net = _cpu_member()
    net.forward_tc(torch.zeros(9, 6))
    assert "sp_mlp_training_forward" in recorder.calls
    recorder.calls.clear()
    for width in (0, 65):
        with pytest.raises(ValueError):
            net.forward_tc(torch.zeros(9, width))
    assert "sp_mlp_training_forward" not in recorder.calls


def test_adam_takes_no_more_gradients_than_parameters(recorder):
    import torch

    net = _cpu_member()
    grads = [torch.zeros_like(p) for p in net.params]
    net.adam(iter(grads + [torch.zeros(3)]), 1e-3)
    count, pointers = recorder.calls["sp_mlp_adam_batch"][:2]
    assert count == len(net.params) == len(pointers)


@pytest.mark.gpu
def test_training_pass_over_other_layouts():
    """Inputs of fewer or more columns, views and repeated rows, and the FP32 path's cache, against
    the same values laid out plainly: the same bits."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(5)
    net = surrogate.Perceptron(3)
    six = torch.randn(40, 6, device="cuda", generator=g)
    five = six.clone()
    five[:, 5] = 0
    seven = torch.cat([six, torch.ones(40, 1, device="cuda")], 1)
    repeated = six[:1].expand(40, 6)
    plain = {name: net.forward_tc(x.contiguous(), keep=True) for name, x in
             (("six", six), ("five", five), ("repeated", repeated))}
    for name, x in (("five", five[:, :5].contiguous()), ("five", six[:, :5]), ("six", seven), ("six", seven[:, :6]),
                    ("six", six.T.contiguous().T), ("repeated", repeated)):
        out, _, status = net.forward_tc(x, keep=True)
        assert int(status.item()) == 0 and torch.equal(out, plain[name][0]), (name, x.shape, x.stride())
    dy = torch.randn(40, surrogate.N_OUT, device="cuda", generator=g)
    _, cache, _ = plain["six"]
    want, _ = net.gradients_tc(cache, dy)
    wide = torch.zeros(40, surrogate.N_OUT + 4, device="cuda")
    wide[:, :surrogate.N_OUT] = dy
    strided = [(seven[:, :6], cache[0][1]), *cache[1:]]
    for c, d in ((cache, wide[:, :surrogate.N_OUT]), (strided, dy)):
        got, status = net.gradients_tc(c, d)
        assert int(status.item()) == 0 and all(torch.equal(a, b) for a, b in zip(got, want))
    _, fp32 = net.forward(six, keep=True)
    want, _ = net.gradients_tc([(a if i == 0 else a.bfloat16(), pre) for i, (a, pre) in enumerate(fp32)], dy)
    got, _ = net.gradients_tc(fp32, dy)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


# ---- the native passes themselves, beyond the surrogate's own network: one layer, a first layer
# wider than the small kernel takes, more layers than one batched launch takes, ragged batches
def _pass(sizes, m):
    """Random weights, the library's forward and backward over them; everything it wrote."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(m + len(sizes))
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    k, n = sizes[:-1], sizes[1:]
    layers, last = len(n), n[-1]
    w = [rand(b, a) / a**0.5 for a, b in zip(k, n)]
    b = [rand(c) for c in n]
    x, dy = rand(m, k[0]), rand(m, last)
    pre = [torch.empty(m, c, device="cuda") for c in n[:-1]]
    act = [torch.empty(m, c, dtype=torch.bfloat16, device="cuda") for c in n[:-1]]
    out = torch.empty(m, last, device="cuda")
    dw, db = [torch.empty_like(t) for t in w], [torch.empty_like(t) for t in b]
    lib, ptr = _lib.library(), surrogate._pointers
    cn, ck = (C.c_int * layers)(*n), (C.c_int * layers)(*k)
    size = lib.sp_mlp_training_scratch(layers, m, cn, ck)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(lib.sp_mlp_training_forward(layers, m, cn, ck, ptr(w), ptr(b), x.data_ptr(), k[0], ptr(pre), ptr(act),
                                           out.data_ptr(), scratch.data_ptr(), size, status.data_ptr(), None))
    _lib.check(lib.sp_mlp_training_backward(layers, m, cn, ck, ptr(w), x.data_ptr(), k[0], ptr([*pre, None]), ptr(act),
                                            dy.data_ptr(), ptr(dw), ptr(db), scratch.data_ptr(), size,
                                            status.data_ptr(), None))
    assert int(status.item()) == 0
    return w, b, x, dy, [*pre, out], act, dw, db


# Each layer from the library's own activations, in 64 bits with the operands' BF16 rounding: the
# FP32 sums' error, 1e-5; a gradient whose last bit turned its rounding to BF16 over in a layer
# above adds at most that rounding, 2^-9, for each of them
@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 63, 65])
@pytest.mark.parametrize("sizes", [(6, 256), (300, 256), (64, 256, 512), (8, 512, 256), (9, 256, 256),
                                   (6, *[256] * 12), (6, *[256] * 18)], ids=str)
def test_training_pass_layers(sizes, m):
    import torch

    w, b, x, dy, pre, act, dw, db = _pass(sizes, m)
    half = lambda t: t.bfloat16().double()  # noqa: E731
    inputs = [x, *act]
    for i, (wi, bi) in enumerate(zip(w, b)):
        assert _rel(pre[i], half(inputs[i]) @ half(wi).T + bi.double()) < 1e-5, i
    for p, a in zip(pre, act):
        z = p.double()
        assert _rel(a, z / 2 * torch.erfc(-z / 2**0.5)) < 2**-8
    g = dy.double()
    for i in reversed(range(len(w))):
        if i < len(w) - 1:
            z = pre[i].double()
            g = g * (0.5 * torch.erfc(-z / 2**0.5) + z * torch.exp(-0.5 * z * z) / (2 * torch.pi) ** 0.5)
        bound = 1e-5 + (len(w) - 1 - i) * 2**-9
        assert _rel(db[i], g.sum(0)) < bound, i
        assert _rel(dw[i], half(g).T @ half(inputs[i])) < bound, i
        g = half(g) @ half(w[i])


def test_training_pass_refusals():
    lib = _lib.library()
    n, k = (C.c_int * 2)(256, 256), (C.c_int * 2)(6, 256)
    size = lib.sp_mlp_training_scratch(2, 5, n, k)
    some = (C.c_void_p * 2)(256, 256)  # never read: every call is refused first
    forward = lambda layers, m, n, k, size: lib.sp_mlp_training_forward(  # noqa: E731
        layers, m, n, k, some, some, 256, 6, some, some, 256, 256, size, 256, None)
    backward = lambda layers, m, n, k, size: lib.sp_mlp_training_backward(  # noqa: E731
        layers, m, n, k, some, 256, 6, some, some, 256, some, some, 256, size, 256, None)
    apart = (C.c_int * 2)(6, 128)
    many = (C.c_int * 65)(*[256] * 65)
    assert size > 0 and lib.sp_mlp_training_scratch(64, 5, many, many) > 0
    argument = 1  # SP_ERR_ARGUMENT
    for call in (forward, backward):
        assert call(2, 0, n, k, size) == call(0, 5, n, k, size) == call(2, 5, n, apart, size) == argument
        assert call(65, 5, many, many, 1 << 40) == argument
        assert call(2, 5, n, k, 0) == argument
    assert backward(2, 5, n, k, size - 1) == argument  # the larger of the two
