"""What the FP64 calls in residue arithmetic do when the device has no room for their scratch: smaller
panels or windows first, then the FP64 kernels, with the same results."""
import pytest
import torch

from pycc_gb300 import _lib, contract, triples

pytestmark = pytest.mark.gpu


@pytest.fixture
def calls(monkeypatch):
    seen = []
    real = _lib.call

    def call(name, *args):
        seen.append(name)
        return real(name, *args)
    monkeypatch.setattr(_lib, "call", call)
    return seen


@pytest.fixture
def full_device(monkeypatch):
    """Makes allocations of scratch (uint8) of at least `least` bytes fail."""
    real = torch.empty
    refused = []

    def setup(least):
        def empty(*size, dtype=None, **kw):
            if dtype == torch.uint8 and size[0] >= least:
                refused.append(size[0])
                raise torch.cuda.OutOfMemoryError("no room")
            return real(*size, dtype=dtype, **kw)
        monkeypatch.setattr(torch, "empty", empty)
        return refused
    return setup


def products(m, n, k, device):
    gen = torch.Generator(device=device).manual_seed(m + k)
    a, b = (torch.randn(s, dtype=torch.float64, device=device, generator=gen)
            for s in ((m, k), (n, k)))
    # FP64 sums of K products on either side, K 2^-53 of the sum of their magnitudes each
    return a, b, torch.mm(a, b.t()), 2.0 ** -52 * (k + 8) * torch.mm(a.abs(), b.abs().t())


def test_contraction_without_scratch(cuda, calls, full_device):
    a, b, ref, tol = products(300, 300, 2000, cuda)
    refused = full_device(0)
    got = contract.contract_f64("mk,nk->mn", a, b)
    assert refused and calls.count("pcg_contract_f64") == 1
    assert "pcg_contract_rns_f64" not in calls
    assert bool(((got - ref).abs() <= tol).all())


def test_contraction_with_little_scratch(cuda, calls, full_device):
    m, n, k = 4000, 4000, 5000
    a, b, ref, tol = products(m, n, k, cuda)
    whole = contract._rns_work(m, n, k)
    assert whole // 4 >= 256 << 20
    refused = full_device(whole)
    got = contract.contract_f64("mk,nk->mn", a, b)
    assert refused == [whole] and "pcg_contract_f64" not in calls
    assert bool(((got - ref).abs() <= tol).all())


def test_energy_without_scratch(cuda, calls, full_device):
    import pycc_gb300 as pg
    F, ERI, L = pg.SyntheticFactors(5, 19, 0).hamiltonian()
    w = pg.CCwfn(pg.Hamiltonian.from_arrays(F, ERI, 5, L=L, device=cuda))
    full = triples.t_energy_fp64(w)
    c, batch = triples._t3_plan(5, 19, triples.T3_WORK_LIMIT)
    whole = triples._t3_bytes(5, 19, c, batch) - 24 * batch * 19 ** 3
    del calls[:]
    refused = full_device(whole)                    # smaller batches or windows
    assert abs(triples.t_energy_fp64(w) - full) <= 1e-13 * abs(full)
    assert refused == [whole] and "pcg_contract_multi_f64" not in calls
    del calls[:]
    full_device(0)                                  # not one triple
    assert abs(triples.t_energy_fp64(w) - full) <= 1e-12 * abs(full)
    assert "pcg_contract_multi_f64" in calls and "pcg_t3_rns_scales" not in calls
