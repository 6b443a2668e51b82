"""The FP64 kernels (32 x R outputs per warp with the lanes along a side, T x T with the lanes along
K, matrix-vector), K slices over warps and blocks at their edges, against extended-precision sums.

Tolerance: K fused multiply-adds and the slices' additions, each a relative rounding of 2^-53 of
a partial sum that is at most sum |a||b|; alpha and beta a few more.
"""
import numpy as np
import pytest
import torch

from pycc_gb300 import _lib, contract

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(2, 2, 1), (8, 8, 4), (9, 7, 5), (8, 33, 16), (33, 8, 17),
                                   (17, 16, 47), (5, 3000, 19), (3000, 6, 13), (40, 41, 1000),
                                   (300, 310, 19), (1, 700, 130), (2000, 1, 65), (1, 1, 5000)])
def test_edges(cuda, m, n, k):
    gen = torch.Generator(device=cuda).manual_seed(m * n + k)
    a, b, c = (torch.randn(s, dtype=torch.float64, device=cuda, generator=gen)
               for s in ((k, m), (n, k), (m, n)))
    got = c.clone()
    contract._launch([(m, 1, n)], [(n, k, 1)], [(k, m, 1)], -1.5, a.data_ptr(), b.data_ptr(), 0.5,
                     got.data_ptr(), _lib.stream_handle())
    A, B, C = (x.cpu().numpy().astype(np.longdouble) for x in (a.t(), b.t(), c))
    want = 0.5 * C - 1.5 * (A @ B)
    tol = 2.0 ** -53 * ((k + 8) * 1.5 * (abs(A) @ abs(B)) + 4 * abs(C))
    assert (abs(got.cpu().numpy() - want) <= tol).all()


@pytest.mark.parametrize("m,n,k", [(31, 2, 3), (32, 3, 4), (33, 4, 5), (64, 5, 33), (65, 6, 31),
                                   (1000, 7, 32), (1000, 11, 65), (4100, 13, 7), (3, 40, 9001),
                                   (3, 3, 128), (4, 5, 127), (9, 9, 4097), (13, 16, 500),
                                   (81, 82, 999), (255, 200, 300), (511, 9, 640), (1, 1023, 129),
                                   (1, 3000, 1000), (2, 1, 257)])
@pytest.mark.parametrize("order", ["mk,nk", "km,nk", "mk,kn", "km,kn"])
def test_orders(cuda, m, n, k, order):
    """Every order of the operands, K and the long side as products of two indices with gaps."""
    gen = torch.Generator(device=cuda).manual_seed(m + n * k)
    la, lb = order.split(",")
    ext = {"m": m, "n": n, "k": k}
    k0 = next(d for d in (7, 5, 3, 2, 1) if k % d == 0)
    a, b = (torch.randn(ext[x[0]] + 1, ext[x[1]] + 3, dtype=torch.float64, device=cuda,
                        generator=gen)[:-1, :-3] for x in (la, lb))
    st = lambda t, lab, c: t.stride(lab.index(c))
    c = torch.randn(n, m, dtype=torch.float64, device=cuda, generator=gen)
    got = c.clone()
    K = [(k // k0, k0 * st(a, la, "k"), k0 * st(b, lb, "k")), (k0, st(a, la, "k"), st(b, lb, "k"))]
    contract._launch([(m, st(a, la, "m"), 1)], [(n, st(b, lb, "n"), m)], K, 2.0, a.data_ptr(),
                     b.data_ptr(), -1.0, got.data_ptr(), _lib.stream_handle())
    A = (a if la == "mk" else a.t()).cpu().numpy().astype(np.longdouble)
    B = (b.t() if lb == "nk" else b).cpu().numpy().astype(np.longdouble)
    C = c.t().cpu().numpy()
    want = 2 * (A @ B) - C
    tol = 2.0 ** -53 * ((k + 40) * 2 * (abs(A) @ abs(B)) + 4 * abs(C))
    assert (abs(got.t().cpu().numpy() - want) <= tol).all()


@pytest.mark.parametrize("m,n,k", [(585, 7, 13), (586, 7, 13), (1365, 3, 255), (2049, 2, 256),
                                   (300, 2, 8192), (24, 2, 8193), (23, 2, 8193), (50, 7, 20001),
                                   (2, 2, 129), (7, 7, 1)])
@pytest.mark.parametrize("order", ["mk,nk", "km,kn"])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_short_sides(cuda, m, n, k, order, beta):
    """A side below eight, on both sides of the line between an output per warp and tiles."""
    gen = torch.Generator(device=cuda).manual_seed(m + n + k)
    la, lb = order.split(",")
    ext = {"m": m, "n": n, "k": k}
    a, b = (torch.randn(ext[x[0]], ext[x[1]], dtype=torch.float64, device=cuda, generator=gen)
            for x in (la, lb))
    c = torch.randn(m, n, dtype=torch.float64, device=cuda, generator=gen)
    got = c.clone() if beta else torch.full_like(c, float("nan"))
    st = lambda t, lab, x: t.stride(lab.index(x))
    contract._launch([(m, st(a, la, "m"), n)], [(n, st(b, lb, "n"), 1)],
                     [(k, st(a, la, "k"), st(b, lb, "k"))], -1.5, a.data_ptr(), b.data_ptr(), beta,
                     got.data_ptr(), _lib.stream_handle())
    A = (a if la == "mk" else a.t()).cpu().numpy().astype(np.longdouble)
    B = (b.t() if lb == "nk" else b).cpu().numpy().astype(np.longdouble)
    C = c.cpu().numpy()
    want = beta * C - 1.5 * (A @ B)
    tol = 2.0 ** -53 * ((k + 40) * 1.5 * (abs(A) @ abs(B)) + 4 * abs(C))
    assert (abs(got.cpu().numpy() - want) <= tol).all()
