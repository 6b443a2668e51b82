"""(T) correction on the GPU (the reference's ``t_tjl``, ``pycc/cctriples.py:177-240``).

For every triple i >= j >= k the connected triples W[a,b,c] (``t3c_ijk``, :27-72) are
built as three partial tensors, one per output orientation of the twelve t3 terms:

* orientation 1, P1[a,b,c]: t2_kj <ba|ei>, t2_ki <ab|ej>, -t2_imab <mc|jk>, -t2_jmba <mc|ik>
* orientation 2, P2[a,c,b]: t2_jk <ca|ei>, t2_ji <ac|ek>, -t2_imac <mb|kj>, -t2_kmca <mb|ij>
* orientation 3, P3[b,c,a]: t2_ij <bc|ek>, t2_ik <cb|ej>, -t2_kmcb <ma|ji>, -t2_jmbc <ma|ki>

so each partial is written once by one multi-term contraction.  A partial is stored with its
last (column) index slowest, P[z][x][y] for the logical P[x,y,z], the layout in which the
tensor-core GEMM writes it with coalesced stores.  The energy kernel
(``csrc/triples.cu``) adds the partials, the disconnected triples (``t3d_ijk``) and the
Lee-Rendell weights, and accumulates E(T) in FP64.

``precision='DP'`` builds batches of triples in residue arithmetic on the tensor cores (or, without
scratch for a batch, one triple at a time by the FP64 multi-term contraction); the mixed path
(``t_energy_tc``) builds the partials for batches of triples with the grouped tcgen05 GEMM.
"""
from __future__ import annotations

import contextlib
import ctypes as C
import functools

import torch

from . import _lib

MAX_SUB = 4


def orientation_terms(i, j, k, t2, V, O):
    """The four terms of each orientation: (alpha, A, A labels, B, B labels).

    V = <pq|ex> (the vvvo block), O = <mp|xy> (the ovoo block).
    """
    return [
        ("abc", [(1.0, V[:, :, :, i], "bae", t2[k, j], "ce"),
                 (1.0, V[:, :, :, j], "abe", t2[k, i], "ce"),
                 (-1.0, t2[i], "mab", O[:, :, j, k], "mc"),
                 (-1.0, t2[j], "mba", O[:, :, i, k], "mc")]),
        ("acb", [(1.0, V[:, :, :, i], "cae", t2[j, k], "be"),
                 (1.0, V[:, :, :, k], "ace", t2[j, i], "be"),
                 (-1.0, t2[i], "mac", O[:, :, k, j], "mb"),
                 (-1.0, t2[k], "mca", O[:, :, i, j], "mb")]),
        ("bca", [(1.0, V[:, :, :, k], "bce", t2[i, j], "ae"),
                 (1.0, V[:, :, :, j], "cbe", t2[i, k], "ae"),
                 (-1.0, t2[k], "mcb", O[:, :, j, i], "ma"),
                 (-1.0, t2[j], "mbc", O[:, :, k, i], "ma")]),
    ]


def contract_multi(out, out_labels, terms, beta=0.0, stream=None):
    """out = beta*out + sum_t alpha_t einsum(A_t, B_t) on the FP64 multi-term kernel."""
    nt = len(terms)
    if not 1 <= nt <= 4:
        raise ValueError("contract_multi: 1..4 terms")
    ost = dict(zip(out_labels, out.stride()))
    oext = dict(zip(out_labels, out.shape))
    alab0, blab0 = terms[0][2], terms[0][4]
    Ml = [c for c in out_labels if c in alab0]
    Nl = [c for c in out_labels if c in blab0]
    m_sa, n_sb, k_n, k_ext, k_sa, k_sb, alphas, As, Bs = [], [], [], [], [], [], [], [], []
    for alpha, A, alab, B, blab in terms:
        if [c for c in out_labels if c in alab] != Ml or [c for c in out_labels if c in blab] != Nl:
            raise ValueError("contract_multi: terms disagree on the output index split")
        ast = dict(zip(alab, A.stride()))
        bst = dict(zip(blab, B.stride()))
        aex = dict(zip(alab, A.shape))
        m_sa += [ast[c] for c in Ml] + [0] * (MAX_SUB - len(Ml))
        n_sb += [bst[c] for c in Nl] + [0] * (MAX_SUB - len(Nl))
        kl = [c for c in alab if c in blab and c not in out_labels]
        kl.sort(key=lambda c: -ast[c])
        k_n.append(len(kl))
        k_ext += [aex[c] for c in kl] + [1] * (MAX_SUB - len(kl))
        k_sa += [ast[c] for c in kl] + [0] * (MAX_SUB - len(kl))
        k_sb += [bst[c] for c in kl] + [0] * (MAX_SUB - len(kl))
        alphas.append(float(alpha))
        As.append(A.data_ptr())
        Bs.append(B.data_ptr())
    i64 = _lib.i64s
    _lib.call("pcg_contract_multi_f64", nt, len(Ml), i64([oext[c] for c in Ml]),
              i64([ost[c] for c in Ml]), i64(m_sa), len(Nl), i64([oext[c] for c in Nl]),
              i64([ost[c] for c in Nl]), i64(n_sb), (C.c_int * nt)(*k_n), i64(k_ext), i64(k_sa),
              i64(k_sb), (C.c_double * nt)(*alphas), (C.c_void_p * nt)(*As),
              (C.c_void_p * nt)(*Bs), float(beta), out.data_ptr(), _lib.stream_handle(stream))
    return out


def triples_list(no):
    return [(i, j, k) for i in range(no) for j in range(i + 1) for k in range(j + 1)]


# Bytes of scratch (residues, products and partials) of one E(T), or, where that is more, what one
# triple needs: 136 nv^2 (nv + no) of residues and 75 nv^3 of products and partials.
T3_WORK_LIMIT = 8 << 30


@functools.lru_cache(maxsize=4096)
def _t3_bytes(no, nv, c, batch):
    """Scratch for windows of c occupied orbitals a slot and batches of triples (0: sizes refused)."""
    out = C.c_longlong(0)
    _lib.call("pcg_t3_rns_window_work", no, nv, c, batch, C.byref(out))
    return out.value and out.value + 24 * batch * nv ** 3


def _t3_plan(no, nv, limit):
    """(c, batch): the window width and the triples of a batch that fit ``limit`` bytes, at least one
    orbital and one triple; None for sizes that the residue path refuses.

    All orbitals in one window where that leaves room for about 16e6 elements of partials (fewer keep
    the launches longer than the work), else the widest windows: the packs of a slot are repeated for
    each window that it is in."""
    if not _t3_bytes(no, nv, 1, 1):
        return None
    ntrip = no * (no + 1) * (no + 2) // 6
    for c in [no] + list(range((no - 1) // 2, 0, -1)):
        most = min(4096, ntrip, c ** 3 if c < no else ntrip)
        want = max(1, min(most, 2 ** 24 // (3 * nv ** 3)))
        if not 0 < _t3_bytes(no, nv, c, want) <= limit:
            continue
        each = _t3_bytes(no, nv, c, 4096) - _t3_bytes(no, nv, c, 4095)
        return c, min(most, want + (limit - _t3_bytes(no, nv, c, want)) // each)
    return 1, 1


def _t3_scratch(no, nv, device, stream):
    """(work, partials, c, batch) for the residue path on ``device``, owned by the launching stream,
    or None when it cannot run there or the device has no room even for one triple."""
    if device.type != "cuda":
        return None
    with torch.cuda.stream(stream) if stream is not None else contextlib.nullcontext():
        limit = T3_WORK_LIMIT
        while (plan := _t3_plan(no, nv, limit)) is not None:
            c, batch = plan
            nbytes = _t3_bytes(no, nv, c, batch) - 24 * batch * nv ** 3
            try:
                return (torch.empty(nbytes, dtype=torch.uint8, device=device),
                        torch.empty((batch, 3, nv, nv, nv), dtype=torch.float64, device=device),
                        c, batch)
            except torch.cuda.OutOfMemoryError:
                if plan == (1, 1):
                    break
                limit = min(limit, nbytes) // 4
    return None


def _t3_windows(no, c):
    """The triples i >= j >= k in windows of c orbitals a slot: (first orbitals of the slots, which
    slots differ from the window before, triples)."""
    last = None
    for i0 in range(0, no, c):
        for j0 in range(0, i0 + 1, c):
            for k0 in range(0, j0 + 1, c):
                first = (i0, j0, k0)
                trips = [(i, j, k) for i in range(i0, min(i0 + c, no))
                         for j in range(j0, min(j0 + c, i + 1)) for k in range(k0, min(k0 + c, j + 1))]
                changed = 7 if last is None else sum((first[r] != last[r]) << r for r in range(3))
                last = first
                yield first, changed, trips


def t_energy_fp64(w, t1=None, t2=None):
    """E(T) with FP64 partials and FP64 energy arithmetic.

    The partials of a batch of triples come from one launch of the residue GEMM on the tensor
    cores (``csrc/triples_rns.cu``), in windows of the occupied index where the residues of all
    would exceed ``T3_WORK_LIMIT``; without room for one triple, from the FP64 multi-term
    contraction, one triple and orientation at a time."""
    t1 = (w.t1 if t1 is None else t1).contiguous()
    t2 = (w.t2 if t2 is None else t2).contiguous()
    no, nv = w.no, w.nv
    o, v = w.o, w.v
    V = w.H.ERI[v, v, v, o]
    O = w.H.ERI[o, v, o, o]
    dev = t2.device
    st = _lib.stream_handle(w.stream)
    scratch = _t3_scratch(no, nv, dev, w.stream)
    windows = list(_t3_windows(no, no if scratch is None else scratch[2]))
    trips = [t for window in windows for t in window[2]]
    part = torch.empty((len(trips), nv), dtype=torch.float64, device=dev)
    ijk = torch.tensor(trips, dtype=torch.int32, device=dev)
    fov = w.H.F[o, v].contiguous()
    fov_ptr = fov.data_ptr() if bool(fov.abs().max() > 0) else None
    eoovv = w.H.ERI[o, o, v, v].contiguous()

    def energy(t0, n, P):
        _lib.call("pcg_triples_energy", 0, P[0, 0].data_ptr(), P[0, 1].data_ptr(),
                  P[0, 2].data_ptr(), 3 * nv ** 3, ijk[t0:].data_ptr(), n, w.H.eps.data_ptr(),
                  eoovv.data_ptr(), t1.data_ptr(), t2.data_ptr(), fov_ptr, no, nv,
                  part[t0:].data_ptr(), st)

    if scratch is None:
        P = torch.empty((1, 3, nv, nv, nv), dtype=torch.float64, device=dev)
        for t, (i, j, k) in enumerate(trips):
            for q, (lab, terms) in enumerate(orientation_terms(i, j, k, t2, V, O)):
                contract_multi(P[0, q].permute(1, 2, 0), lab, terms, stream=w.stream)
            energy(t, 1, P)
    else:
        work, P, c, batch = scratch
        V, O = V.contiguous(), O.contiguous()
        ops = (V.data_ptr(), O.data_ptr(), t2.data_ptr(), no, nv, c)
        room = (work.data_ptr(), work.numel(), st)
        _lib.call("pcg_t3_rns_scales", *ops, *room)
        t0 = 0
        for first, changed, of_window in windows:
            slots = (C.c_int * 3)(*first)
            _lib.call("pcg_t3_rns_window_pack", *ops, slots, changed, *room)
            for n in [min(batch, len(of_window) - q) for q in range(0, len(of_window), batch)]:
                _lib.call("pcg_t3_rns_window_partials", *ops, slots, ijk[t0:].data_ptr(), n,
                          P.data_ptr(), *room)
                energy(t0, n, P)
                t0 += n
    out = torch.zeros((), dtype=torch.float64, device=dev)
    _lib.call("pcg_reduce_sum_f64", part.data_ptr(), part.numel(), out.data_ptr(), st)
    return float(out)


def t_energy(w, t1=None, t2=None):
    """E(T) for the converged amplitudes of ``w`` in ``w``'s precision."""
    if w.precision == 'DP':
        return t_energy_fp64(w, t1, t2)
    from .triples_tc import t_energy_tc
    return t_energy_tc(w, t1, t2)


def t_tjl(ccwfn):
    """The reference's entry point ``t_tjl(ccwfn) -> float`` (``pycc/cctriples.py:177-240``):
    E(T) at ``ccwfn``'s amplitudes, in its precision (``t_energy``)."""
    return t_energy(ccwfn)


def t_vikings(ccwfn):
    """``t_vikings(ccwfn) -> float`` (``pycc/cctriples.py:243-308``): the reference's
    full-(i,j,k) formulation of the same E(T); the engine evaluates it over i >= j >= k with
    the Lee-Rendell weights, which gives the same value (``t_energy``)."""
    return t_energy(ccwfn)
