"""The connected triples in residue arithmetic (csrc/triples_rns.cu) against the FP64 multi-term
contraction, at the edges of tiles and K blocks, and what non-finite operands give.

Tolerance: a partial sums four products of rows of length K = nv or no; the FP64 side rounds each
of its multiply-adds by 2^-53 of a partial sum of at most sum |a||b|, the residue side its scaled
operands by less than 2^-56 of the largest row norms' products.
"""
import ctypes as C

import pytest
import torch

from pycc_gb300 import _lib
from pycc_gb300.triples import contract_multi, orientation_terms

pytestmark = pytest.mark.gpu


def partials(V, O, t2, trips, batch):
    no, nv = t2.shape[0], t2.shape[2]
    nbytes = C.c_longlong(0)
    _lib.call("pcg_t3_rns_work", no, nv, batch, C.byref(nbytes))
    work = torch.empty(nbytes.value, dtype=torch.uint8, device=t2.device)
    _lib.call("pcg_t3_rns_pack", V.data_ptr(), O.data_ptr(), t2.data_ptr(), no, nv,
              work.data_ptr(), work.numel(), _lib.stream_handle())
    ijk = torch.tensor(trips, dtype=torch.int32, device=t2.device)
    out = torch.full((len(trips), 3, nv, nv, nv), float("nan"), dtype=torch.float64,
                     device=t2.device)
    for t0 in range(0, len(trips), batch):
        n = min(batch, len(trips) - t0)
        _lib.call("pcg_t3_rns_partials", no, nv, ijk[t0:].data_ptr(), n, out[t0].data_ptr(),
                  work.data_ptr(), work.numel(), _lib.stream_handle())
    return out


@pytest.mark.parametrize("no,nv", [(1, 1), (2, 3), (3, 19), (2, 64), (65, 5), (3, 65), (2, 130),
                                   (1, 257)])
def test_partials(cuda, no, nv):
    gen = torch.Generator(device=cuda).manual_seed(no + nv)
    rand = lambda *s: torch.randn(s, dtype=torch.float64, device=cuda, generator=gen)
    V, O, t2 = rand(nv, nv, nv, no), rand(no, nv, no, no), 0.1 * rand(no, no, nv, nv)
    trips = [(no - 1, no // 2, 0), (no - 1, no - 1, no // 3), (0, 0, 0)]
    got = partials(V, O, t2, trips, 2)
    for t, (i, j, k) in enumerate(trips):
        for q, (lab, terms) in enumerate(orientation_terms(i, j, k, t2, V, O)):
            ref, mag = torch.empty_like(got[t, q]), torch.empty_like(got[t, q])
            contract_multi(ref.permute(1, 2, 0), lab, terms)
            contract_multi(mag.permute(1, 2, 0), lab,
                           [(1.0, A.abs(), la, B.abs(), lb) for _, A, la, B, lb in terms])
            top = float(mag.max())
            tol = 2.0 ** -53 * (2 * (nv + no) + 8) * mag + 2.0 ** -56 * top
            assert bool(((got[t, q] - ref).abs() <= tol).all())


def test_not_finite(cuda):
    gen = torch.Generator(device=cuda).manual_seed(1)
    rand = lambda *s: torch.randn(s, dtype=torch.float64, device=cuda, generator=gen)
    V, O, t2 = rand(7, 7, 7, 3), rand(3, 7, 3, 3), rand(3, 3, 7, 7)
    t2[1, 2, 3, 4] = float("inf")
    assert bool(partials(V, O, t2, [(2, 1, 0)], 1).isnan().all())


@pytest.mark.parametrize("n,x,wide", [(1, 0.99, 0.0), (1, 1.99, 0.0), (2, 0.7, 0.0),
                                      (4, 0.4975, 0.0), (4, 0.489, 0.02), (16, 0.249, 0.0)])
def test_range(cuda, n, x, wide):
    """Collinear rows with norms just below a power of two: the four products of an orientation
    add up to the largest sum that the scales allow, which the moduli have to hold."""
    gen = torch.Generator(device=cuda).manual_seed(n)
    near = lambda *s: x * (1 + wide * (2 * torch.rand(s, dtype=torch.float64, device=cuda,
                                                      generator=gen) - 1))
    V, O, t2 = near(n, n, n, n), -near(n, n, n, n), near(n, n, n, n)
    trips = [(n - 1, n // 2, 0), (n - 1, n - 1, n - 1)]
    got = partials(V, O, t2, trips, 2)
    for t, (i, j, k) in enumerate(trips):
        for q, (lab, terms) in enumerate(orientation_terms(i, j, k, t2, V, O)):
            ref = torch.empty_like(got[t, q])
            contract_multi(ref.permute(1, 2, 0), lab, terms)
            # every product is positive: the sums of magnitudes are the sums
            tol = 2.0 ** -53 * (4 * n + 8) * ref + 2.0 ** -56 * float(ref.max())
            assert bool(((got[t, q] - ref).abs() <= tol).all())


def partials_of(V, O, t2, trips):
    no, nv = t2.shape[0], t2.shape[2]
    nbytes = C.c_longlong(0)
    _lib.call("pcg_t3_rns_work", no, nv, len(trips), C.byref(nbytes))
    work = torch.empty(nbytes.value, dtype=torch.uint8, device=t2.device)
    st = _lib.stream_handle()
    _lib.call("pcg_t3_rns_pack", V.data_ptr(), O.data_ptr(), t2.data_ptr(), no, nv,
              work.data_ptr(), work.numel(), st)
    ijk = torch.tensor(trips, dtype=torch.int32, device=t2.device)
    out = torch.full((len(trips), 3, nv, nv, nv), float("nan"), dtype=torch.float64,
                     device=t2.device)
    _lib.call("pcg_t3_rns_partials_of", V.data_ptr(), O.data_ptr(), t2.data_ptr(), no, nv,
              ijk.data_ptr(), len(trips), out.data_ptr(), work.data_ptr(), work.numel(), st)
    return out


@pytest.mark.parametrize("no,nv", [(1, 1), (3, 19), (2, 64), (34, 5), (3, 65), (2, 130)])
def test_graded_operands(cuda, no, nv):
    """Magnitudes over fifteen decades, and a slab of V that meets zeros only: each partial keeps
    FP64's accuracy relative to its own products, and exact zeros stay zero."""
    gen = torch.Generator(device=cuda).manual_seed(no + nv)
    def rand(*s):
        u = torch.rand(s, dtype=torch.float64, device=cuda, generator=gen)
        return torch.randn(s, dtype=torch.float64, device=cuda, generator=gen) * 10.0 ** (-15 * u)
    V, O, t2 = rand(nv, nv, nv, no), rand(no, nv, no, no), rand(no, no, nv, nv)
    V[:, :, 0] *= 1e20
    t2[..., 0] = 0.0
    O[:, nv // 2] = 0.0
    trips = [(no - 1, no // 2, 0), (no - 1, no - 1, no // 3), (0, 0, 0)]
    got = partials_of(V, O, t2, trips)
    for t, (i, j, k) in enumerate(trips):
        for q, (lab, terms) in enumerate(orientation_terms(i, j, k, t2, V, O)):
            ref, mag = torch.empty_like(got[t, q]), torch.empty_like(got[t, q])
            contract_multi(ref.permute(1, 2, 0), lab, terms)
            contract_multi(mag.permute(1, 2, 0), lab,
                           [(1.0, A.abs(), la, B.abs(), lb) for _, A, la, B, lb in terms])
            # (nv + no) 2^-51 on the residues' side, (nv + no + 8) 2^-52 on the reference's
            assert bool(((got[t, q] - ref).abs() <= 2.0 ** -51 * (2 * (nv + no) + 8) * mag).all())
            assert bool((got[t, q][mag == 0] == 0).all())


def test_not_finite_operands(cuda):
    """With the operands at hand, an infinity reaches the partials that FP64 arithmetic gives it to."""
    gen = torch.Generator(device=cuda).manual_seed(1)
    rand = lambda *s: torch.randn(s, dtype=torch.float64, device=cuda, generator=gen)
    V, O, t2 = rand(7, 7, 7, 3), rand(3, 7, 3, 3), rand(3, 3, 7, 7)
    t2[1, 2, 3, 4] = float("inf")
    got = partials_of(V, O, t2, [(2, 1, 0)])
    for q, (lab, terms) in enumerate(orientation_terms(2, 1, 0, t2, V, O)):
        ref = torch.empty_like(got[0, q])
        contract_multi(ref.permute(1, 2, 0), lab, terms)
        assert torch.equal(got[0, q].isnan(), ref.isnan())
        assert torch.equal(got[0, q].isinf(), ref.isinf())


def test_energy_with_a_large_idle_slab(cuda, monkeypatch):
    """E(T) when one virtual orbital's integrals are huge and its amplitudes zero."""
    import pycc_gb300 as pg
    from pycc_gb300 import triples
    no, nv = 4, 11
    fac = pg.SyntheticFactors(no, nv, 3)
    F, ERI, L = fac.hamiltonian()
    w = pg.CCwfn(pg.Hamiltonian.from_arrays(F, ERI, no, L=L, device=cuda))
    t2 = w.t2.clone()
    t2[:, :, 0, :] = 0.0
    t2[:, :, :, 0] = 0.0
    w.t2 = t2
    w.H.ERI[w.v, w.v, w.v, w.o][:, :, 0] *= 1e20
    got = triples.t_energy_fp64(w)
    monkeypatch.setattr(triples, "_t3_scratch", lambda *a: None)
    ref = triples.t_energy_fp64(w)
    assert ref != 0.0 and abs(got - ref) <= 1e-12 * abs(ref)


def wave_function(no, nv, device, seed=2):
    import pycc_gb300 as pg
    F, ERI, L = pg.SyntheticFactors(no, nv, seed).hamiltonian()
    return pg.CCwfn(pg.Hamiltonian.from_arrays(F, ERI, no, L=L, device=device))


@pytest.mark.parametrize("no,nv,c,batch", [(7, 12, 3, 1000), (7, 12, 2, 3), (5, 70, 1, 1),
                                           (9, 9, 4, 5)])
def test_windows(cuda, monkeypatch, no, nv, c, batch):
    """Windows of the occupied index, the last ragged, give the energy of one window for all."""
    from pycc_gb300 import triples
    w = wave_function(no, nv, cuda)
    full = triples.t_energy_fp64(w)
    monkeypatch.setattr(triples, "_t3_plan", lambda *a: (c, batch))
    assert abs(triples.t_energy_fp64(w) - full) <= 1e-13 * abs(full)


def test_scratch_limit(cuda, monkeypatch):
    """The scratch of an E(T) stays within T3_WORK_LIMIT where all residues (58 MB) do not fit."""
    from pycc_gb300 import triples
    w = wave_function(8, 40, cuda)
    full = triples.t_energy_fp64(w)
    monkeypatch.setattr(triples, "T3_WORK_LIMIT", 32 << 20)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    assert abs(triples.t_energy_fp64(w) - full) <= 1e-13 * abs(full)
    assert torch.cuda.max_memory_allocated() - before <= (32 << 20) + (2 << 20)
