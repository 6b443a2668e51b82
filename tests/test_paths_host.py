"""Host code that only a GPU run takes -- contractions with scratch for the residue path, the mixed
(T) with pitched partials -- on CPU, through the numpy model of the entry points."""
import pytest
import torch

import abi_model
import pycc_gb300 as pg
from pycc_gb300 import contract
from pycc_gb300.triples_tc import TriplesTC


@pytest.mark.parametrize("scratch", [True, False])
@pytest.mark.parametrize("subs", ["mk,nk->mn", "ijef,abef->ijab", "Qpr,Qqs->pqrs", "xmk,xnk->xmn"])
def test_contraction_routes(monkeypatch, subs, scratch):
    """A contraction above the line takes the residue entry point with its scratch (one for all its
    batch values), the FP64 one when there is none; below the line scratch is not asked for."""
    model = abi_model.install(monkeypatch)
    asked = []

    def room(m, n, k, device, stream):
        asked.append((m, n, k))
        return torch.empty(64, dtype=torch.uint8) if scratch else None
    monkeypatch.setattr(contract, "_rns_scratch", room)
    ext = dict(zip("ijefabmnkQpqrsx", (12, 13, 40, 41, 14, 15, 170, 160, 1500, 300, 21, 22, 23, 24, 3)))
    lhs, rhs = subs.split("->")
    gen = torch.Generator().manual_seed(1)
    a, b = (torch.randn([ext[c] for c in lab], dtype=torch.float64, generator=gen)
            for lab in lhs.split(","))
    big = torch.randn([ext[c] + 1 for c in rhs], dtype=torch.float64, generator=gen)
    out = big[tuple(slice(1, None) for _ in rhs)]
    want = 0.5 * out + 2.0 * torch.einsum(subs, a, b)
    contract.contract_f64(subs, a, b, out=out, alpha=2.0, beta=0.5)
    assert torch.allclose(out, want, rtol=1e-12, atol=1e-10)
    batch = 3 if "x" in rhs else 1
    used = "pcg_contract_rns_f64" if scratch else "pcg_contract_f64"
    assert model.calls == [used] * batch and len(asked) == 1
    assert torch.allclose(contract.contract_f64("ij,kj->ik", a.reshape(-1, 2)[:4], b.reshape(-1, 2)[:5]),
                          torch.einsum("ij,kj->ik", a.reshape(-1, 2)[:4], b.reshape(-1, 2)[:5]))
    assert len(asked) == 1


@pytest.mark.parametrize("pitch", [20, 24])
@pytest.mark.parametrize("batch", [32, 7, 1])
def test_pitched_partials(monkeypatch, ham_o5v19, golden_o5v19, pitch, batch):
    """Group offsets, runs of rows and the padded copies at a pitch above nv = 19."""
    model = abi_model.install(monkeypatch)
    _, F, ERI, L = ham_o5v19
    w = pg.CCwfn(pg.Hamiltonian.from_arrays(F, ERI, 5, L=L, device="cpu"))
    t1, t2 = (torch.from_numpy(golden_o5v19[k].copy()) for k in ("t1", "t2"))
    t = TriplesTC(w, t1, t2, batch=batch)
    t.pitch = pitch
    assert abs(t.energy() - float(golden_o5v19["et_tjl"])) < 1e-9
    assert "pcg_tc_grouped_gemm_pitched" in model.calls
    assert "pcg_triples_energy_pitched" in model.calls and "pcg_triples_energy" not in model.calls
