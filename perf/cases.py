"""The calls that a user of the CCSD engine makes, over their sizes, for timing and comparison.

Kinds of call:

* ``solve``: a whole ``CCwfn.solve_cc`` in FP64, the call every user makes, at molecule sizes
  where launches and host work count;
* ``residual``: one ``CCwfn.residuals`` (what real-time propagation, derivative drivers and the
  solver's own loop call), in FP64, in the mixed engine's first and final precision stage, and
  in the single-precision-class mode;
* ``wmbej``: one o^3 v^3 intermediate builder, the block a driver that keeps its own equations
  calls by name;
* ``contract``: one pairwise contraction through the einsum backend;
* ``triples``: the (T) energy of given amplitudes, FP64 and mixed;
* ``lambda``: one reverse sweep of the residual (J^T lambda), the body of a Lambda iteration.

Hamiltonians are seeded synthetic ones: <pq|rs> = sum_Q B_Qpr B_Qqs with a random symmetric
three-index factor scaled to a convergent correlation strength, occupied orbital energies in
[-1.2, -0.4] and virtual ones in [0.3, 2.5].
"""
import math

import torch

import pycc_gb300 as pg
from pycc_gb300.adjoint import CCSDAdjoint
from pycc_gb300.contract import ContractionBackend
from pycc_gb300.hamiltonian import ERI_BLOCKS, L_BLOCKS, BlockTensor, Hamiltonian
from pycc_gb300.triples import t_tjl

DEVICE = "cuda:0"

# contractions of the residual, by what they stress: the ladder and the rings (large K), a
# short K with an o^2 v^2 output, a small output with a long K
SUBSCRIPTS = {"ladder": "ijef,abef->ijab", "ring": "imae,mbej->ijab", "hole": "mnab,mnij->ijab",
              "dress": "ijae,be->ijab", "t1": "ie,abej->ijab", "small": "mnaf,mnef->ae"}


def listed():
    return [
        # a water-sized molecule from the guess to convergence: about a dozen iterations of
        # small kernels
        {"name": "solve o5v19", "kind": "solve", "no": 5, "nv": 19},
        # residual of a small molecule in a larger basis, odd sizes
        {"name": "residual DP o9v53", "kind": "residual", "precision": "DP", "no": 9, "nv": 53},
        # the largest FP64 residual that users of the CPU reference can still compare with
        {"name": "residual DP o20v180", "kind": "residual", "precision": "DP", "no": 20,
         "nv": 180},
        # final (most exact) stage of the mixed engine where launches weigh as much as work
        {"name": "residual MIXED o10v80", "kind": "residual", "precision": "MIXED",
         "stage": "final", "no": 10, "nv": 80},
        # final stage at production size, where the tensor cores' work dominates
        {"name": "residual MIXED o28v220", "kind": "residual", "precision": "MIXED",
         "stage": "final", "no": 28, "nv": 220},
        # first stage (FP8 ladder, BF16) of a solve, odd sizes
        {"name": "residual MIXED first o17v133", "kind": "residual", "precision": "MIXED",
         "stage": "first", "no": 17, "nv": 133},
        # single-precision-class residual
        {"name": "residual SP o12v71", "kind": "residual", "precision": "SP", "no": 12,
         "nv": 71},
        # a ring intermediate called by name
        {"name": "wmbej DP o14v110", "kind": "wmbej", "no": 14, "nv": 110},
        # one ragged ladder contraction through the einsum backend
        {"name": "contract ladder o7v113", "kind": "contract", "term": "ladder", "no": 7,
         "nv": 113},
        # (T) in FP64 after a small CCSD
        {"name": "triples DP o7v45", "kind": "triples", "precision": "DP", "no": 7, "nv": 45},
        # (T) on the tensor cores, odd sizes
        {"name": "triples MIXED o15v121", "kind": "triples", "precision": "MIXED", "no": 15,
         "nv": 121},
        # the backward direction: one Lambda sweep in FP64
        {"name": "lambda DP o11v83", "kind": "lambda", "no": 11, "nv": 83},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "residual", "residual", "residual", "wmbej", "contract",
                       "triples", "triples", "lambda"])
    if kind == "solve":
        return {"kind": kind, "no": rng.randint(3, 8), "nv": rng.randint(12, 40)}
    if kind == "residual":
        prec = rng.choice(["DP", "MIXED", "MIXED", "SP"])
        if prec == "DP":
            return {"kind": kind, "precision": prec, "no": _log(rng, 5, 18),
                    "nv": _log(rng, 30, 160)}
        if prec == "SP":
            return {"kind": kind, "precision": prec, "no": _log(rng, 7, 16),
                    "nv": _log(rng, 50, 110)}
        return {"kind": kind, "precision": prec, "stage": rng.choice(["first", "final"]),
                "no": _log(rng, 8, 26), "nv": _log(rng, 60, 200)}
    if kind == "wmbej":
        return {"kind": kind, "no": _log(rng, 6, 16), "nv": _log(rng, 40, 130)}
    if kind == "contract":
        return {"kind": kind, "term": rng.choice(sorted(SUBSCRIPTS)), "no": _log(rng, 5, 20),
                "nv": _log(rng, 30, 150)}
    if kind == "triples":
        if rng.random() < 0.5:
            return {"kind": kind, "precision": "DP", "no": rng.randint(4, 9),
                    "nv": _log(rng, 20, 70)}
        return {"kind": kind, "precision": "MIXED", "no": rng.randint(8, 18),
                "nv": _log(rng, 60, 150)}
    return {"kind": kind, "no": _log(rng, 5, 14), "nv": _log(rng, 30, 110)}


# -- inputs -------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=torch.float64, device=DEVICE)


def _factor(no, nv, g):
    """Orbital energies and the factor B of one Hamiltonian, scaled so that
    o^2 v^2 var(<ij|ab>) is half of the value at no=5, nv=19 with sigma = 0.35/sqrt(72)."""
    n = no + nv
    naux = min(3 * n, 160)
    u = torch.rand(n, generator=g, dtype=torch.float64, device=DEVICE)
    eps = torch.cat([torch.sort(-1.2 + 0.8 * u[:no])[0], torch.sort(0.3 + 2.2 * u[no:])[0]])
    sigma = (0.94 / (no * no * nv * nv * naux)) ** 0.25
    B = torch.triu(sigma * _randn(g, naux, n, n))
    return eps, B + torch.triu(B, 1).transpose(1, 2)


def _block(B, no, pat, alpha=1.0):
    """alpha <pq|rs> = alpha sum_Q B_Qpr B_Qqs over o/v ranges, contiguous."""
    n = B.shape[1]
    p, q, r, s = (slice(0, no) if c == "o" else slice(no, n) for c in pat)
    X, Y = B[:, p, r], B[:, q, s]
    out = torch.mm((alpha * X).reshape(X.shape[0], -1).t(), Y.reshape(Y.shape[0], -1))
    out = out.view(X.shape[1], X.shape[2], Y.shape[1], Y.shape[2])
    return out.permute(0, 2, 1, 3).contiguous()


def _blocks(no, nv, g):
    eps, B = _factor(no, nv, g)
    eri = {pat: _block(B, no, pat) for pat in ERI_BLOCKS}
    ll = {}
    for pat in L_BLOCKS:
        sw = pat[0] + pat[1] + pat[3] + pat[2]
        ll[pat] = 2.0 * eri[pat] - _block(B, no, sw).transpose(2, 3)
    # a Fock matrix close to diagonal: small coupling off the diagonal, as a finite field or a
    # non-canonical basis leaves it
    n = no + nv
    X = 0.005 * _randn(g, n, n)
    return torch.diag(eps) + X + X.t(), eri, ll


def _amplitudes(F, eri, no, nv, g):
    """Amplitudes near a solution: MP2 doubles with some noise, small singles."""
    eo, ev = torch.diagonal(F)[:no], torch.diagonal(F)[no:]
    t2 = eri["oovv"] / (eo.view(-1, 1, 1, 1) + eo.view(-1, 1, 1) - ev.view(-1, 1) - ev)
    rms = float(t2.square().mean().sqrt())
    t2 = t2 + 0.1 * rms * _randn(g, no, no, nv, nv)
    t2 = 0.5 * (t2 + t2.permute(1, 0, 3, 2))
    t1 = 0.1 / math.sqrt(no * nv) * _randn(g, no, nv)
    return t1, t2.contiguous()


def _wfn(case, F, eri, ll):
    no, nv = case["no"], case["nv"]
    H = Hamiltonian(F, BlockTensor("ERI", no, nv, eri), BlockTensor("L", no, nv, ll), no, nv,
                    torch.device(DEVICE))
    return pg.CCwfn(H, precision=case.get("precision", "DP"))


def _operands(case, seed):
    """Operands of a ``contract`` case: amplitude-like and integral-like random tensors."""
    subs = SUBSCRIPTS[case["term"]]
    lhs = subs.split("->")[0]
    g = _gen(seed)
    out = []
    for lab in lhs.split(","):
        shape = [case["no"] if c in "ijmn" else case["nv"] for c in lab]
        # a spread of magnitudes, as amplitudes and integrals have
        out.append(0.05 * _randn(g, *shape) * torch.exp(_randn(g, *shape)))
    return subs, out


def prepare(case, seed):
    kind, no, nv = case["kind"], case["no"], case["nv"]
    if kind == "contract":
        subs, (a, b) = _operands(case, seed)
        return {"case": case, "subs": subs, "a": a, "b": b, "contract": ContractionBackend()}
    g = _gen(seed)
    F, eri, ll = _blocks(no, nv, g)
    if kind == "solve":
        F = torch.diag(torch.diagonal(F))          # a canonical SCF solution
    w = _wfn(case, F, eri, ll)
    t1, t2 = _amplitudes(F, eri, no, nv, g)
    st = {"case": case, "w": w, "t1": t1, "t2": t2}
    if kind == "solve":
        st["guess"] = w.t2.clone()
    elif kind == "residual" and case.get("stage") == "final":
        w.mixed_engine().select_mode(0.0)          # the stage that fixes the energy
    elif kind == "triples":
        w.t1, w.t2 = t1, t2
    elif kind == "lambda":
        w.t1, w.t2 = t1, t2
        st["adj"] = CCSDAdjoint(w)
        st["l1"], st["l2"] = _lambda_input(t1, t2, g)
        st["g1"], st["g2"] = _lambda_input(t1, t2, g)
    return st


def _lambda_input(t1, t2, g):
    l2 = 2.0 * t2 - t2.transpose(2, 3) + 0.1 * t2.square().mean().sqrt() * _randn(g, *t2.shape)
    l2 = 0.5 * (l2 + l2.permute(1, 0, 3, 2))
    return 2.0 * t1 + 0.01 * _randn(g, *t1.shape) / math.sqrt(t1.numel()), l2.contiguous()


# -- one pass -----------------------------------------------------------------------------
def run(state):
    kind = state["case"]["kind"]
    if kind == "contract":
        return state["contract"](state["subs"], state["a"], state["b"])
    w = state["w"]
    if kind == "solve":
        w.t1 = torch.zeros_like(state["t1"])
        w.t2 = state["guess"]
        e = w.solve_cc(e_conv=1e-10, r_conv=1e-10, maxiter=100)
        return {"e": e, "t1": w.t1.clone(), "t2": w.t2.clone()}
    if kind == "residual":
        r1, r2 = w.residuals(w.H.F, state["t1"], state["t2"])
        return {"r1": r1, "r2": r2}
    if kind == "wmbej":
        return w.build_Wmbej(w.o, w.v, w.H.ERI, w.H.L, state["t1"], state["t2"])
    if kind == "triples":
        return t_tjl(w)
    g1, g2 = state["adj"].jt_lambda(state["l1"], state["l2"], state["g1"], state["g2"])
    return {"g1": g1, "g2": g2}


# -- what a pass cannot do without ----------------------------------------------------------
def work(case):
    kind, o, v = case["kind"], float(case["no"]), float(case["nv"])
    t = o * v + o * o * v * v
    size = {"o": o, "v": v}

    def blocks(pats):
        return sum(math.prod(size[c] for c in p) for p in pats)

    ints = blocks(ERI_BLOCKS) + blocks(L_BLOCKS)
    iteration = 2 * o**2 * v**4 + 18 * o**3 * v**3 + 10 * o**2 * v**3 + 4 * o**4 * v**2
    if kind == "contract":
        lhs, rhs = SUBSCRIPTS[case["term"]].split("->")
        ext = {c: (o if c in "ijmn" else v) for c in lhs if c != ","}
        n = sum(math.prod(ext[c] for c in s) for s in lhs.split(",") + [rhs])
        return {"bytes": 8 * n, "flops": 2 * math.prod(ext.values())}
    if kind == "solve":
        # about ten iterations
        return {"bytes": 10 * 8 * (ints + 2 * t), "flops": 10 * iteration}
    if kind == "residual":
        return {"bytes": 8 * (ints + 2 * t), "flops": iteration}
    if kind == "wmbej":
        n = blocks(["ovvo", "ovvv", "oovo", "oovv", "oovv", "ovvo"]) + t
        return {"bytes": 8 * n, "flops": 4 * o**3 * v**3 + 2 * o**2 * v**3}
    if kind == "triples":
        trip = o * (o + 1) * (o + 2) / 6
        return {"bytes": 8 * (blocks(["vvvo", "ovoo", "oovv"]) + t),
                "flops": trip * 12 * (v**4 + o * v**3)}
    return {"bytes": 8 * (ints + 4 * t), "flops": 2 * iteration}


# -- the same in plain torch, 64 bits -------------------------------------------------------
def _residual(F, E, L, no, t1, t2):
    """The RHF-CCSD residual with its equations written out over o/v blocks."""
    e = torch.einsum
    Foo, Fov, Fvv = F[:no, :no], F[:no, no:], F[no:, no:]
    tau = t2 + e("ia,jb->ijab", t1, t1)
    taut = t2 + 0.5 * e("ia,jb->ijab", t1, t1)
    tah = 0.5 * t2 + e("ia,jb->ijab", t1, t1)
    Fae = Fvv - 0.5 * e("me,ma->ae", Fov, t1) + e("mf,mafe->ae", t1, L["ovvv"])
    Fae = Fae - e("mnaf,mnef->ae", taut, L["oovv"])
    Fmi = Foo + 0.5 * e("ie,me->mi", t1, Fov) + e("ne,mnie->mi", t1, L["ooov"])
    Fmi = Fmi + e("inef,mnef->mi", taut, L["oovv"])
    Fme = Fov + e("nf,mnef->me", t1, L["oovv"])
    Wmnij = E["oooo"] + e("je,mnie->mnij", t1, E["ooov"]) + e("ie,mnej->mnij", t1, E["oovo"])
    Wmnij = Wmnij + e("ijef,mnef->mnij", tau, E["oovv"])
    Wmbej = _wmbej(E, L, t1, t2)
    Wmbje = -E["ovov"] - e("jf,mbfe->mbje", t1, E["ovvv"]) + e("nb,mnje->mbje", t1, E["ooov"])
    Wmbje = Wmbje + e("jnfb,mnfe->mbje", tah, E["oovv"])
    Zmbij = e("mbef,ijef->mbij", E["ovvv"], tau)

    t2s = 2.0 * t2 - t2.transpose(2, 3)
    r1 = F[no:, :no].t() + e("ie,ae->ia", t1, Fae) - e("mi,ma->ia", Fmi, t1)
    r1 = r1 + e("imae,me->ia", t2s, Fme) + e("nf,nafi->ia", t1, L["ovvo"])
    r1 = r1 + e("mief,maef->ia", t2s, E["ovvv"]) - e("mnae,nmei->ia", t2, L["oovo"])

    r = 0.5 * E["vvoo"].permute(2, 3, 0, 1)
    r = r + e("ijae,be->ijab", t2, Fae - 0.5 * e("mb,me->be", t1, Fme))
    r = r - e("imab,mj->ijab", t2, Fmi + 0.5 * e("je,me->mj", t1, Fme))
    r = r + 0.5 * e("mnab,mnij->ijab", tau, Wmnij) + 0.5 * e("ijef,abef->ijab", tau, E["vvvv"])
    r = r - e("ma,mbij->ijab", t1, Zmbij)
    r = r + e("imae,mbej->ijab", t2 - t2.transpose(2, 3), Wmbej)
    r = r + e("imae,mbej->ijab", t2, Wmbej + Wmbje.transpose(2, 3))
    r = r + e("mjae,mbie->ijab", t2, Wmbje)
    r = r - e("ma,imbj->ijab", t1, e("ie,mbej->imbj", t1, E["ovvo"]))
    r = r - e("mb,imaj->ijab", t1, e("ie,maje->imaj", t1, E["ovov"]))
    r = r + e("ie,abej->ijab", t1, E["vvvo"]) - e("ma,mbij->ijab", t1, E["ovoo"])
    return r1, r + r.permute(1, 0, 3, 2)


def _wmbej(E, L, t1, t2):
    e = torch.einsum
    tah = 0.5 * t2 + e("ia,jb->ijab", t1, t1)
    W = E["ovvo"] + e("jf,mbef->mbej", t1, E["ovvv"]) - e("nb,mnej->mbej", t1, E["oovo"])
    W = W - e("jnfb,mnef->mbej", tah, E["oovv"])
    return W + 0.5 * e("njfb,mnef->mbej", t2, L["oovv"])


def _energy(F, L, no, t1, t2):
    tau = t2 + torch.einsum("ia,jb->ijab", t1, t1)
    return 2.0 * (F[:no, no:] * t1).sum() + (tau * L["oovv"]).sum()


def _solve(F, E, L, no, nv):
    """Jacobi iterations with DIIS to 1e-13; (energy, t1, t2)."""
    eo, ev = torch.diagonal(F)[:no], torch.diagonal(F)[no:]
    D1 = eo.view(-1, 1) - ev
    D2 = eo.view(-1, 1, 1, 1) + eo.view(-1, 1, 1) - ev.view(-1, 1) - ev
    t1, t2 = torch.zeros_like(D1), E["oovv"] / D2
    xs, es = [], []
    for _ in range(200):
        r1, r2 = _residual(F, E, L, no, t1, t2)
        step = torch.cat([(r1 / D1).reshape(-1), (r2 / D2).reshape(-1)])
        x = torch.cat([t1.reshape(-1), t2.reshape(-1)]) + step
        if float(step.norm()) < 1e-13:
            break
        xs, es = (xs + [x])[-8:], (es + [step])[-8:]
        k = len(es)
        S = torch.stack(es)
        A = -torch.ones(k + 1, k + 1, dtype=torch.float64, device=x.device)
        A[k, k] = 0.0
        A[:k, :k] = S @ S.t() / float(step.square().sum())
        rhs = torch.zeros(k + 1, dtype=torch.float64, device=x.device)
        rhs[k] = -1.0
        c = torch.linalg.lstsq(A.cpu(), rhs.cpu().unsqueeze(1), driver="gelsd").solution
        x = (c[:k].to(x.device) * torch.stack(xs)).sum(0)
        t1, t2 = x[:no * nv].view(no, nv), x[no * nv:].view(no, no, nv, nv)
    return _energy(F, L, no, t1, t2), t1, t2


def _triples(F, E, no, t1, t2):
    """The Lee-Rendell (T) energy over i >= j >= k with whole v^3 arrays."""
    e = torch.einsum
    nv = t1.shape[1]
    V, O, W2 = E["vvvo"], E["ovoo"], E["oovv"]
    eps, Fov = torch.diagonal(F), F[:no, no:]
    ev = eps[no:]
    Dv = ev.view(-1, 1, 1) + ev.view(-1, 1) + ev
    a = torch.arange(nv, device=t1.device)
    A, B, C = a.view(-1, 1, 1), a.view(1, -1, 1), a.view(1, 1, -1)
    wt = 1.0 + (A == B) + (A == C) + (B == C)
    tri = ((A >= B) & (B >= C)).double()
    V = V.permute(3, 0, 1, 2).contiguous()
    total = torch.zeros((), dtype=torch.float64, device=t1.device)
    for i in range(no):
        for j in range(i + 1):
            for k in range(j + 1):
                W = e("bae,ce->abc", V[i], t2[k, j]) + e("cae,be->abc", V[i], t2[j, k])
                W = W + e("ace,be->abc", V[k], t2[j, i]) + e("bce,ae->abc", V[k], t2[i, j])
                W = W + e("cbe,ae->abc", V[j], t2[i, k]) + e("abe,ce->abc", V[j], t2[k, i])
                W = W - e("mc,mab->abc", O[:, :, j, k], t2[i])
                W = W - e("mb,mac->abc", O[:, :, k, j], t2[i])
                W = W - e("mb,mca->abc", O[:, :, i, j], t2[k])
                W = W - e("ma,mcb->abc", O[:, :, j, i], t2[k])
                W = W - e("ma,mbc->abc", O[:, :, k, i], t2[j])
                W = W - e("mc,mba->abc", O[:, :, i, k], t2[j])
                D = e("ab,c->abc", W2[i, j], t1[k]) + e("ac,b->abc", W2[i, k], t1[j])
                D = D + e("bc,a->abc", W2[j, k], t1[i]) + e("ab,c->abc", t2[i, j], Fov[k])
                D = D + e("ac,b->abc", t2[i, k], Fov[j]) + e("bc,a->abc", t2[j, k], Fov[i])
                X = (W + D) / wt
                p = [(0, 1, 2), (1, 2, 0), (2, 0, 1), (0, 2, 1), (1, 0, 2), (2, 1, 0)]
                Wp, Xp = [W.permute(q) for q in p], [X.permute(q) for q in p]
                S = 3.0 * sum(x * y for x, y in zip(Wp, Xp))
                Y, Z = Xp[0] + Xp[1] + Xp[2], Xp[3] + Xp[4] + Xp[5]
                S = S + (Y - 2.0 * Z) * (Wp[0] + Wp[1] + Wp[2])
                S = S + (Z - 2.0 * Y) * (Wp[3] + Wp[4] + Wp[5])
                fac = 2.0 - ((i == j) + (i == k) + (j == k))
                total = total + fac * (S * tri / (eps[i] + eps[j] + eps[k] - Dv)).sum()
    return total


def exact(case, seed):
    kind, no, nv = case["kind"], case["no"], case["nv"]
    if kind == "contract":
        subs, (a, b) = _operands(case, seed)
        return torch.einsum(subs, a, b)
    g = _gen(seed)
    F, E, L = _blocks(no, nv, g)
    if kind == "solve":
        F = torch.diag(torch.diagonal(F))
        e, t1, t2 = _solve(F, E, L, no, nv)
        return {"e": float(e), "t1": t1, "t2": t2}
    t1, t2 = _amplitudes(F, E, no, nv, g)
    if kind == "residual":
        r1, r2 = _residual(F, E, L, no, t1, t2)
        return {"r1": r1, "r2": r2}
    if kind == "wmbej":
        return _wmbej(E, L, t1, t2)
    if kind == "triples":
        return float(_triples(F, E, no, t1, t2))
    l1, l2 = _lambda_input(t1, t2, g)
    g1, g2 = _lambda_input(t1, t2, g)
    t1.requires_grad_()
    t2.requires_grad_()
    r1, r2 = _residual(F, E, L, no, t1, t2)
    d1, d2 = torch.autograd.grad((l1 * r1).sum() + (l2 * r2).sum(), (t1, t2))
    return {"g1": g1 + d1, "g2": g2 + d2}
