"""The residue-arithmetic contraction (csrc/contract_rns.cu) against extended-precision sums, at
the edges of its tiles, chunks and panels and over the operand forms it accepts.

Tolerance: the operands' rounding to integers gives at most sqrt(K) 2^-60 |a_i| |b_j| (each row
is scaled to a norm of at least 2^60.3 and rounded by at most one half), the conversion to FP64,
the scale and alpha / beta at most eight roundings of the terms.
"""
import math

import numpy as np
import pytest
import torch

from pycc_gb300 import _lib, contract
from pycc_gb300.contract import ContractPlan, contract_f64

pytestmark = pytest.mark.gpu


def rns(subs, a, b, out, alpha=1.0, beta=0.0, limit=contract.RNS_WORK_LIMIT):
    """One contraction on the residue path whatever the dispatch rule says."""
    M, N, K, batch, *_ = ContractPlan(subs, a, b).groups(a, b, out)
    assert not batch
    nbytes = contract._rns_work(*(math.prod(g[0] for g in G) for G in (M, N, K)), limit)
    assert 0 < nbytes <= limit
    work = torch.empty(nbytes, dtype=torch.uint8, device=out.device)
    contract._launch(M, N, K, alpha, a.data_ptr(), b.data_ptr(), beta, out.data_ptr(),
                     _lib.stream_handle(), work)
    return out


def sums(a, b, subs="mk,nk->mn"):
    """The contraction and its tolerance in extended precision."""
    A, B = (x.cpu().numpy().astype(np.longdouble) for x in (a, b))
    lhs, rhs = subs.split("->")
    la, lb = lhs.split(",")
    C = np.einsum(subs, A, B)
    ra, rb = ("".join(c for c in rhs if c in lab) for lab in (la, lb))
    norms = np.einsum("%s,%s->%s" % (ra, rb, rhs), np.sqrt(np.einsum(la + "->" + ra, A * A)),
                      np.sqrt(np.einsum(lb + "->" + rb, B * B)))
    k = math.prod(n for c, n in zip(la, A.shape) if c not in rhs)
    return C, np.sqrt(k) * 2.0 ** -60 * norms + 2.0 ** -50 * abs(C)


def spread(shape, gen, width):
    x = torch.randn(shape, dtype=torch.float64, device="cuda:0", generator=gen)
    return x * torch.exp(width * torch.randn(shape, dtype=torch.float64, device="cuda:0",
                                             generator=gen))


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (2, 3, 64), (127, 65, 63), (128, 64, 65),
                                   (129, 128, 960), (5, 129, 961), (130, 257, 1925),
                                   (13, 16, 30011), (400, 130, 70)])
def test_edges(cuda, m, n, k):
    gen = torch.Generator(device=cuda).manual_seed(m + n + k)
    a, b = spread((m, k), gen, 1.0), spread((n, k), gen, 1.0)
    ref, tol = sums(a, b)
    got = rns("mk,nk->mn", a, b, torch.full((m, n), float("nan"), dtype=torch.float64, device=cuda))
    assert (abs(got.cpu().numpy() - ref) <= tol).all()
    c0 = torch.randn(m, n, dtype=torch.float64, device=cuda, generator=gen)
    got = rns("mk,nk->mn", a, b, c0.clone(), alpha=-1.5, beta=0.25).cpu().numpy()
    want = 0.25 * c0.cpu().numpy().astype(np.longdouble) - 1.5 * ref
    assert (abs(got - want) <= 1.5 * tol + 2.0 ** -50 * (abs(want) + abs(ref))).all()


@pytest.mark.parametrize("subs", ["mk,nk->mn", "km,kn->mn", "mk,kn->nm", "km,nk->nm",
                                  "imae,mbej->ijab", "mief,maef->ia", "jnfb,mnef->mbej",
                                  "ijef,abef->ijab", "ma,mbij->ijab"])
def test_forms(cuda, subs):
    """Operand and output orders, and non-contiguous views that the output's rest survives."""
    ext = dict(zip("ijmnabefk", (5, 6, 7, 4, 17, 19, 13, 11, 70)))
    if subs.count("k"):
        ext.update(m=150, n=140)
    gen = torch.Generator(device=cuda).manual_seed(5)
    lhs, rhs = subs.split("->")
    ops = []
    for lab in lhs.split(","):
        big = torch.randn([ext[c] + 3 for c in lab], dtype=torch.float64, device=cuda,
                          generator=gen)
        ops.append(big[tuple(slice(2, 2 + ext[c]) for c in lab)])
    big = torch.randn([ext[c] + 1 for c in rhs], dtype=torch.float64, device=cuda, generator=gen)
    view = tuple(slice(1, None) for _ in rhs)
    one = big.clone()
    rns(subs, *ops, one[view], alpha=2.0, beta=1.0)
    ref, tol = sums(*ops, subs)
    want = big[view].cpu().numpy() + 2.0 * ref
    assert (abs(one[view].cpu().numpy() - want) <= 2 * tol + 2.0 ** -50 * abs(want)).all()
    keep = torch.ones_like(big, dtype=torch.bool)
    keep[view] = False
    assert torch.equal(one[keep], big[keep])


@pytest.mark.parametrize("limit", [40 << 20, 64 << 20])
def test_panels(cuda, limit):
    """Workspaces that hold panels of rows, columns and K only."""
    gen = torch.Generator(device=cuda).manual_seed(9)
    a, b = spread((900, 3000), gen, 1.0), spread((3000, 700), gen, 1.0)
    ref, tol = sums(a[::67], b.t()[::11])     # a sample: extended precision is slow
    c0 = torch.randn(900, 700, dtype=torch.float64, device=cuda, generator=gen)
    got = rns("mk,kn->mn", a, b, c0.clone(), beta=1.0, limit=limit).cpu().numpy()[::67, ::11]
    want = c0.cpu().numpy()[::67, ::11] + ref
    assert (abs(got - want) <= 2 * tol + 2.0 ** -50 * abs(want)).all()


def test_scales(cuda):
    """Rows of very different size, zero rows, subnormals, and products out of range."""
    gen = torch.Generator(device=cuda).manual_seed(2)
    a, b = spread((9, 130), gen, 1.0), spread((8, 130), gen, 1.0)
    for r, s in enumerate((1e-300, 1e-160, 1e-25, 1e-15, 1.0, 1e15, 1e25, 1e150, 0.0)):
        a[r] *= s
    b[0] *= 1e-140
    b[1] *= 1e140
    b[2] = 0.0
    b[3, 1:] = 0.0
    got = rns("mk,nk->mn", a, b, torch.empty(9, 8, dtype=torch.float64, device=cuda)).cpu().numpy()
    ref, tol = sums(a, b)
    assert (abs(got - ref) <= tol + 5e-324).all()
    big = rns("mk,nk->mn", a[7:8] * 1e150, b[1:2] * 1e20,
              torch.empty(1, 1, dtype=torch.float64, device=cuda))
    assert math.isinf(float(big))


def test_not_finite(cuda):
    """Infinities and NaN reach exactly the outputs that FP64 arithmetic gives them to."""
    gen = torch.Generator(device=cuda).manual_seed(3)
    a, b = (torch.randn(40, 100, dtype=torch.float64, device=cuda, generator=gen)
            for _ in range(2))
    a[3, 5], a[7, 0], b[11, 99], b[12, 5] = float("inf"), float("nan"), -float("inf"), 0.0
    got = rns("mk,nk->mn", a, b, torch.empty(40, 40, dtype=torch.float64, device=cuda)).cpu()
    ref = torch.einsum("mk,nk->mn", a, b).cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    inf = torch.isinf(ref)
    assert torch.equal(got[inf], ref[inf])
    rows, cols = [r for r in range(40) if r not in (3, 7)], [c for c in range(40) if c != 11]
    want, tol = sums(a[rows], b[cols])
    assert (abs(got[rows][:, cols].numpy() - want) <= tol).all()


def test_dispatch(cuda):
    """contract_f64 takes the residue path for a large contraction, on a side stream too, and
    the FP64 kernel when no scratch can be had."""
    gen = torch.Generator(device=cuda).manual_seed(4)
    a, b = (torch.randn(300, 2000, dtype=torch.float64, device=cuda, generator=gen)
            for _ in range(2))
    assert contract._takes_rns(300, 300, 2000) and not contract._takes_rns(20, 20, 20)
    ref, tol = sums(a[::23], b[::23])
    n0 = _lib.launch_count()
    got = contract_f64("mk,nk->mn", a, b)
    assert _lib.launch_count() - n0 == 5
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    side = contract_f64("mk,nk->mn", a, b, out=torch.zeros_like(got), stream=st)
    st.synchronize()
    assert torch.equal(got, side)
    assert (abs(got[::23, ::23].cpu().numpy() - ref) <= tol).all()


def graded(shape, gen, decades):
    """Random signs and mantissas, magnitudes over as many decades."""
    x = torch.randn(shape, dtype=torch.float64, device="cuda:0", generator=gen)
    return x * 10.0 ** (-decades * torch.rand(shape, dtype=torch.float64, device="cuda:0",
                                              generator=gen))


def check_products(got, a, b, subs, c0=None, alpha=1.0, beta=0.0):
    """Every output within the bound of FP64 multiply-adds: the residues' rounding gives at most
    sqrt(K) 2^-52 sum |a||b| where they are used, FP64 sums K 2^-53, and the rest eight roundings."""
    A, B = (x.cpu().numpy().astype(np.longdouble) for x in (a, b))
    S = np.einsum(subs, abs(A), abs(B))
    want = alpha * np.einsum(subs, A, B)
    k = math.prod(n for c, n in zip(subs, A.shape) if c not in subs.split("->")[1])
    tol = abs(alpha) * 2.0 ** -53 * (max(2 * math.sqrt(k), k) + 8) * S
    if c0 is not None:
        c = beta * c0.cpu().numpy().astype(np.longdouble)
        want, tol = want + c, tol + 2.0 ** -51 * abs(c)
    assert (abs(got.cpu().numpy() - want) <= tol).all()
    zero = (S == 0) if c0 is None else np.zeros_like(S, dtype=bool)
    assert (got.cpu().numpy()[zero] == 0).all()


@pytest.mark.parametrize("subs", ["mk,nk->mn", "km,kn->mn", "mk,kn->nm"])
@pytest.mark.parametrize("m,n,k,limit", [(3, 5, 2, None), (65, 33, 64, None), (130, 70, 961, None),
                                         (13, 16, 30011, None), (300, 260, 3000, 30 << 20)])
def test_graded_rows(cuda, subs, m, n, k, limit):
    """Magnitudes over twenty decades within the rows, some rows with zeros where the others are
    large: products that are far below the norms of their rows keep FP64's relative accuracy."""
    gen = torch.Generator(device=cuda).manual_seed(m + k)
    a, b = graded((m, k), gen, 20.0), graded((n, k), gen, 20.0)
    a[m // 2:, : k // 2] *= 1e30
    b[n // 2:, : k // 2] = 0.0
    a[0, k // 3:] = 0.0
    b[1, : k // 3] = 0.0
    la, lb = subs.split("->")[0].split(",")
    a = a if la == "mk" else a.t().contiguous()
    b = b if lb == "nk" else b.t().contiguous()
    shape = (m, n) if subs.endswith("mn") else (n, m)
    nan = torch.full(shape, float("nan"), dtype=torch.float64, device=cuda)
    kw = {} if limit is None else {"limit": limit}
    check_products(rns(subs, a, b, nan, **kw), a, b, subs)
    c0 = graded(shape, gen, 20.0)
    check_products(rns(subs, a, b, c0.clone(), alpha=-1.5, beta=0.25, **kw), a, b, subs, c0, -1.5,
                   0.25)


@pytest.mark.parametrize("s", [1e-9, 1e-15, 1e-18, 2.0 ** -70, 1e-100, 1e-300])
def test_small_products_of_large_rows(cuda, s):
    """(1, s, s, ...) times (0, 1-sized, ...): the rows' largest entries meet zeros."""
    gen = torch.Generator(device=cuda).manual_seed(6)
    a, b = (torch.randn(70, 512, dtype=torch.float64, device=cuda, generator=gen)
            for _ in range(2))
    a[:, 1:] *= s
    a[:, 0] = 1.0
    b[::2, 0] = 0.0
    out = torch.empty(70, 70, dtype=torch.float64, device=cuda)
    check_products(rns("mk,nk->mn", a, b, out), a, b, "mk,nk->mn")
    check_products(contract_f64("mk,nk->mn", a.repeat(8, 1), b), a.repeat(8, 1), b, "mk,nk->mn")
