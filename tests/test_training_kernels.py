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
    net, one = surrogate.Perceptron(7), surrogate.Perceptron(7)
    grads = [torch.randn(p.shape, device="cuda", generator=g) for p in net.params]
    net.adam(grads, 1e-3)
    for p, gr, m1, m2 in zip(one.params, grads, one.m1, one.m2):
        _lib.check(_lib.library().sp_mlp_adam(p.data_ptr(), gr.data_ptr(), m1.data_ptr(), m2.data_ptr(), p.numel(),
                                              1e-3, 0.9, 0.999, 1e-8, 1, None))
    for a, b in zip(net.params + net.m1 + net.m2, one.params + one.m1 + one.m2):
        assert torch.equal(a, b)
