"""FP64 (T) in windows of the occupied index: the plan's scratch, the windows' triples, and the
host code that goes through them (``tests/abi_model.py``), on CPU."""
import ctypes as C

import numpy as np
import pytest
import torch

import abi_model
import pycc_gb300 as pg
from pycc_gb300 import triples


@pytest.mark.parametrize("no,nv", [(5, 19), (7, 45), (9, 70), (20, 180), (30, 240), (40, 300),
                                   (1, 250), (60, 200)])
def test_scratch_within_the_limit(no, nv):
    for limit in (triples.T3_WORK_LIMIT, triples.T3_WORK_LIMIT // 4):
        c, batch = triples._t3_plan(no, nv, limit)
        assert triples._t3_bytes(no, nv, c, batch) <= max(limit, triples._t3_bytes(no, nv, 1, 1))
        # a triple's products, partials and four blocks of residues
        assert triples._t3_bytes(no, nv, 1, 1) <= 136 * nv ** 2 * (nv + no + 72) + 80 * (nv + 16) ** 3


@pytest.mark.parametrize("no,c", [(1, 1), (5, 1), (5, 2), (7, 3), (7, 7), (8, 4)])
def test_windows_cover_every_triple_once(no, c):
    slots, seen = [None] * 3, []
    for first, changed, trips in triples._t3_windows(no, c):
        for q in range(3):
            if changed >> q & 1:
                slots[q] = first[q]
            assert slots[q] == first[q] and first[q] % c == 0
        assert first[0] >= first[1] >= first[2]
        assert all(first[q] <= t[q] < first[q] + c for t in trips for q in range(3))
        seen += trips
    assert sorted(seen) == triples.triples_list(no) and len(seen) == len(set(seen))
    if c == no:
        assert seen == triples.triples_list(no)


@pytest.mark.parametrize("c,batch", [(5, 35), (5, 4), (2, 3), (1, 1)])
def test_energy_in_windows(monkeypatch, ham_o5v19, golden_o5v19, c, batch):
    model = abi_model.install(monkeypatch)
    _, F, ERI, L = ham_o5v19
    w = pg.CCwfn(pg.Hamiltonian.from_arrays(F, ERI, 5, L=L, device="cpu"))
    w.t1 = torch.from_numpy(golden_o5v19["t1"].copy())
    w.t2 = torch.from_numpy(golden_o5v19["t2"].copy())
    monkeypatch.setattr(triples, "_t3_scratch", lambda no, nv, device, stream: (
        torch.empty(16, dtype=torch.uint8),
        torch.full((batch, 3, nv, nv, nv), float("nan"), dtype=torch.float64), c, batch))
    assert abs(triples.t_energy_fp64(w) - float(golden_o5v19["et_tjl"])) < 1e-13
    assert "pcg_contract_multi_f64" not in model.calls
    assert model.calls.count("pcg_t3_rns_scales") == 1


def test_window_arguments_are_checked():
    from pycc_gb300 import _lib
    p = C.c_void_p(256)
    def call(no, nv, c, first, length):
        _lib.call("pcg_t3_rns_window_pack", p, p, p, no, nv, c, (C.c_int * 3)(*first), 7, p, length,
                  None)
    for bad in ((4, 9, 2, (0, 2, 0)), (4, 9, 2, (1, 0, 0)), (4, 9, 2, (4, 0, 0)), (4, 9, 0, (0, 0, 0)),
                (4, 9, 5, (0, 0, 0))):
        with pytest.raises(_lib.EngineError):
            call(*bad, 1 << 40)
    with pytest.raises(_lib.EngineError):
        call(4, 9, 2, (2, 0, 0), 256)
    assert _lib.load().pcg_t3_rns_window_work(4, 9, 5, 1, C.byref(C.c_longlong(0))) == 0
