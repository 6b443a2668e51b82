"""The FP64 kernel's warp tiles (8 x 8, 16 x 16, 8 x 32, 32 x 8), K slices over warps and blocks
and matrix-vector splits at their edges, against extended-precision sums.

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
