"""numpy model of the FP64 C-ABI entry points, for CPU tests of the host logic only.

Each function restates the documented semantics of one entry point of
``include/pycc_gb300.h`` on tensors in host memory (``data_ptr()`` of a CPU tensor is a host
address).  Tests install it in place of ``pycc_gb300._lib.call`` to run the host code of the
engine -- the builders' contraction plans, the mixed engine's operand definitions and output
maps, the (T) drivers' layouts and batches, the adjoint tape and its sweeps, the solver loops,
DIIS -- without a GPU.  The (T) energy entry point is modelled with the oracle's per-triple
Lee-Rendell energy.  The
tensor-core pack and GEMM are modelled in exact FP64 (no format rounding), so a residual
planned by the mixed engine must equal the FP64 residual to rounding.  The CUDA kernels
themselves are checked against the oracle in the ``-m gpu`` tests; nothing here says anything
about them, and nothing outside ``tests/`` imports this module.
"""
from __future__ import annotations

import ctypes as C

import numpy as np


def _ints(arr, n):
    return [int(arr[i]) for i in range(n)]


def view(ptr, shape, strides, dtype=np.float64):
    """A strided numpy view of host memory at ``ptr`` (strides in elements, non-negative)."""
    if not ptr:
        raise AssertionError("null pointer")
    dt = np.dtype(dtype)
    span = 1 + sum((e - 1) * s for e, s in zip(shape, strides)) if all(e > 0 for e in shape) else 0
    base = np.frombuffer((C.c_char * (max(span, 1) * dt.itemsize)).from_address(ptr), dtype=dt)
    return np.lib.stride_tricks.as_strided(base, shape=tuple(shape),
                                           strides=tuple(s * dt.itemsize for s in strides))


def flat(ptr, n, dtype=np.float64):
    return view(ptr, (n,), (1,), dtype)


class ABIModel:
    """Callable with the signature of ``_lib.call(name, *args)``."""

    def __init__(self):
        self.calls = []
        self.packs = {}           # hi buffer address -> the FP64 values a pack would convert

    def __call__(self, name, *a):
        self.calls.append(name)
        fn = getattr(self, name[4:], None)        # strip "pcg_"
        if fn is None:
            raise AssertionError("no model of %s" % name)
        fn(*a)
        return 0

    # C[m,n] = beta C + alpha sum_k A[m,k] B[n,k]
    def contract_f64(self, m_n, m_ext, m_sa, m_sc, n_n, n_ext, n_sb, n_sc, k_n, k_ext, k_sa,
                     k_sb, alpha, A, B, beta, Cp, _st):
        me, ne, ke = _ints(m_ext, m_n), _ints(n_ext, n_n), _ints(k_ext, k_n)
        Av = view(A, me + ke, _ints(m_sa, m_n) + _ints(k_sa, k_n))
        Bv = view(B, ne + ke, _ints(n_sb, n_n) + _ints(k_sb, k_n))
        Cv = view(Cp, me + ne, _ints(m_sc, m_n) + _ints(n_sc, n_n))
        prod = np.tensordot(Av, Bv, axes=(list(range(m_n, m_n + k_n)),
                                          list(range(n_n, n_n + k_n))))
        res = alpha * prod if beta == 0.0 else beta * Cv + alpha * prod
        Cv[...] = res

    def contract_rns_f64(self, m_n, m_ext, m_sa, m_sc, n_n, n_ext, n_sb, n_sc, k_n, k_ext, k_sa,
                         k_sb, alpha, A, B, beta, Cp, work, length, _st):
        """The same contraction with scratch."""
        assert work and length > 0
        self.contract_f64(m_n, m_ext, m_sa, m_sc, n_n, n_ext, n_sb, n_sc, k_n, k_ext, k_sa, k_sb,
                          alpha, A, B, beta, Cp, _st)

    def combine4_f64(self, ext4, a, X, xs4, b, Y, ys4, out, os4, _st):
        ext = _ints(ext4, 4)
        res = a * view(X, ext, _ints(xs4, 4))
        if Y:
            res = res + b * view(Y, ext, _ints(ys4, 4))
        view(out, ext, _ints(os4, 4))[...] = res

    def tau_f64(self, t1, t2, no, nv, f1, f2, out, _st):
        T1 = view(t1, (no, nv), (nv, 1))
        T2 = flat(t2, no * no * nv * nv).reshape(no, no, nv, nv)
        res = f1 * T2 + f2 * np.einsum("ia,jb->ijab", T1, T1)
        flat(out, no * no * nv * nv).reshape(no, no, nv, nv)[...] = res

    def symmetrize_f64(self, h, no, nv, out, _st):
        Hh = flat(h, no * no * nv * nv).reshape(no, no, nv, nv)
        flat(out, no * no * nv * nv).reshape(no, no, nv, nv)[...] = Hh + Hh.transpose(1, 0, 3, 2)

    def energy_f64(self, fov, fs2, L, ls4, t1, t2, no, nv, _work, _wl, out, _st):
        f = view(fov, (no, nv), _ints(fs2, 2))
        Lv = view(L, (no, no, nv, nv), _ints(ls4, 4))
        T1 = view(t1, (no, nv), (nv, 1))
        T2 = flat(t2, no * no * nv * nv).reshape(no, no, nv, nv)
        tau = T2 + np.einsum("ia,jb->ijab", T1, T1)
        flat(out, 1)[0] = 2.0 * np.sum(f * T1) + np.sum(tau * Lv)

    def inv_denominators_f64(self, eps, no, nv, inv1, inv2, _st):
        e = flat(eps, no + nv)
        eo, ev = e[:no], e[no:]
        flat(inv1, no * nv)[...] = (1.0 / (eo[:, None] - ev[None, :])).ravel()
        d2 = eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, :, None] - ev
        flat(inv2, no * no * nv * nv)[...] = (1.0 / d2).ravel()

    def update_inv_f64(self, t, r, inv, n, _work, _wl, out, _st):
        step = flat(r, n) * flat(inv, n)
        flat(t, n)[...] += step
        flat(out, 1)[0] = np.dot(step, step)

    def update_amps_f64(self, t1, t2, r1, r2, eps, no, nv, _work, _wl, out, _st):
        e = flat(eps, no + nv)
        eo, ev = e[:no], e[no:]
        d1 = (eo[:, None] - ev[None, :]).ravel()
        d2 = (eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, :, None]
              - ev).ravel()
        s1 = flat(r1, no * nv) / d1
        s2 = flat(r2, no * no * nv * nv) / d2
        flat(t1, no * nv)[...] += s1
        flat(t2, no * no * nv * nv)[...] += s2
        flat(out, 1)[0] = np.dot(s1, s1) + np.dot(s2, s2)

    def _diis_error(self, dt, x, old, e, ys, k, n, out):
        E = flat(e, n, dt)
        E[...] = (flat(x, n) - flat(old, n)).astype(dt)
        e64 = E.astype(np.float64)
        o = flat(out, k)
        for j in range(k - 1):
            o[j] = np.dot(e64, flat(ys[j], n, dt).astype(np.float64))
        o[k - 1] = np.dot(e64, e64)

    def diis_error_f64(self, x, old, e, ys, k, n, _work, _wl, out, _st):
        assert 1 <= k <= 16
        self._diis_error(np.float64, x, old, e, ys, k, n, out)

    def diis_error_f32(self, x, old, e, ys, k, n, _work, _wl, out, _st):
        assert 1 <= k <= 16
        self._diis_error(np.float32, x, old, e, ys, k, n, out)

    def lincomb_f64(self, xs, c, k, n, out, _st):
        assert 1 <= k <= 16 and all(xs[j] != out for j in range(k))
        acc = np.zeros(n)
        for j in range(k):
            acc = acc + c[j] * flat(xs[j], n)
        flat(out, n)[...] = acc

    lincomb_f64_df = lincomb_f64

    # -- the tensor-core engine, modelled in exact FP64 --------------------------------------
    # A pack records the FP64 values it would convert (keyed by its hi buffer); the GEMM
    # multiplies those.  The model so checks which operand combinations, layouts and output
    # maps the host plans, independently of the GEMM formats' rounding.
    @staticmethod
    def _offsets(ext, strides):
        off = np.zeros(1, dtype=np.int64)
        for e, s in zip(ext, strides):
            off = (off[:, None] + np.arange(e, dtype=np.int64)[None, :] * s).ravel()
        return off

    def pack_operand(self, fmt, r_n, r_ext, r_str, k_n, k_ext, k_str, Kp, a, X, b, Y, c, P, Q,
                     d, R_, S_, hi, mid, lo, scale, row_tab, rows, k_tab, k_w, kcount, _st):
        re_, ke = _ints(r_ext, r_n), _ints(k_ext, k_n)
        rs, ks = _ints(r_str, 24), _ints(k_str, 24)
        K = kcount if k_tab else (int(np.prod(ke)) if ke else 1)
        assert K <= Kp and Kp % (128 if fmt == 2 else 64) == 0
        assert not k_w or k_tab
        if row_tab:
            rtab = flat(row_tab, 6 * rows, np.int64).reshape(6, rows)
        if k_tab:
            ktab = flat(k_tab, 6 * kcount, np.int64).reshape(6, kcount)
        R = rows if row_tab else (int(np.prod(re_)) if re_ else 1)

        def source(s, ptr):
            koff = ktab[s] if k_tab else self._offsets(ke, ks[4 * s:4 * s + k_n])
            roff = rtab[s] if row_tab else self._offsets(re_, rs[4 * s:4 * s + r_n])
            idx = roff[:, None] + koff[None, :]
            return flat(ptr, int(idx.max()) + 1)[idx]

        v = np.zeros((R, K))
        if X:
            v += a * source(0, X)
        if Y:
            v += b * source(1, Y)
        if P:
            v += c * source(2, P) * source(3, Q)
        if R_:
            v += d * source(4, R_) * source(5, S_)
        if k_w:
            v *= flat(k_w, K, np.float32).astype(np.float64)[None, :]
        self.packs[hi] = v

    def tc_gemm(self, fmt, A_hi, A_mid, A_lo, M, lda, B_hi, B_mid, B_lo, N, ldb, Kp, a_scale,
                b_scale, m_n, m_ext, m_sc, n_n, n_ext, n_sc, col_map, col_scale, alpha, beta, Cp,
                _status, _st):
        A, B = self.packs[A_hi], self.packs[B_hi]
        assert A.shape[0] == M and B.shape[0] == N and A.shape[1] == B.shape[1]
        offm = self._offsets(_ints(m_ext, m_n), _ints(m_sc, m_n))
        assert offm.size == M
        if col_map:
            offn = flat(col_map, N, np.int64).copy()
        else:
            offn = self._offsets(_ints(n_ext, n_n), _ints(n_sc, n_n))
        assert offn.size == N and 0 <= offn.min() and offn.max() < 2 ** 31
        S = alpha * (A @ B.T)
        if col_scale:
            S = S * flat(col_scale, N)[None, :]
        idx = offm[:, None] + offn[None, :]
        assert np.unique(idx).size == idx.size, "output map is not injective"
        Cf = flat(Cp, int(idx.max()) + 1)
        Cf[idx] = S if beta == 0.0 else beta * Cf[idx] + S


    def ladder_pm_assemble(self, Gp, Gm, no, nv, h, _st):
        """h[i,j,a,b] += G+ (+-) G- over the a <= b triangle of the pairs (i <= j) and their
        transposed pairs, as pcg_ladder_pm_assemble documents."""
        P, Q = nv * (nv + 1) // 2, nv * (nv - 1) // 2
        gp = flat(Gp, (no * (no + 1) // 2) * P).reshape(-1, P)
        gm = flat(Gm, (no * (no - 1) // 2) * Q).reshape(-1, Q) if Gm else None
        H = view(h, (no, no, nv, nv), (no * nv * nv, nv * nv, nv, 1))
        a, b = np.triu_indices(nv)
        strict = b > a
        qm = 0
        for q, (i, j) in enumerate(zip(*np.triu_indices(no))):
            g = gp[q].copy()
            if j > i:
                m = np.zeros(P)
                if gm is not None:
                    m[strict] = gm[qm]
                qm += 1
                H[i, j][a, b] += g + m
                H[j, i][a[strict], b[strict]] += (g - m)[strict]
            else:
                H[i, i][a, b] += np.where(strict, g, 0.5 * g)

    def pair_pm_assemble(self, Gp, Gm, no, nrow, Z, _st):
        """Z[r, i, j] += G+ + G-, Z[r, j, i] += G+ - G- (i < j), Z[r, i, i] += G+, as
        pcg_pair_pm_assemble documents."""
        gp = flat(Gp, (no * (no + 1) // 2) * nrow).reshape(-1, nrow)
        gm = flat(Gm, (no * (no - 1) // 2) * nrow).reshape(-1, nrow) if Gm else None
        Zv = view(Z, (nrow, no, no), (no * no, no, 1))
        qm = 0
        for q, (i, j) in enumerate(zip(*np.triu_indices(no))):
            if j > i:
                m = gm[qm] if gm is not None else 0.0
                qm += 1
                Zv[:, i, j] += gp[q] + m
                Zv[:, j, i] += gp[q] - m
            else:
                Zv[:, i, i] += gp[q]

    # -- the (T) density entry points -----------------------------------------------------
    def t3_ijk_f64(self, P, eps, i, j, k, no, nv, Woovv, t1, t2, fov, M3, N3, _st):
        v = nv
        Pv = flat(P, 3 * v ** 3).reshape(3, v, v, v)
        # W[a,b,c] = P1[c][a][b] + P2[b][a][c] + P3[a][b][c]
        W = np.einsum('cab->abc', Pv[0]) + np.einsum('bac->abc', Pv[1]) + Pv[2]
        e = flat(eps, no + nv)
        ev = e[no:]
        D = e[i] + e[j] + e[k] - ev[:, None, None] - ev[None, :, None] - ev[None, None, :]
        Wo = flat(Woovv, no * no * v * v).reshape(no, no, v, v)
        T1 = flat(t1, no * v).reshape(no, v)
        T2 = flat(t2, no * no * v * v).reshape(no, no, v, v)
        n = (Wo[i, j][:, :, None] * T1[k][None, None, :] + Wo[i, k][:, None, :] * T1[j][None, :, None]
             + Wo[j, k][None, :, :] * T1[i][:, None, None])
        if fov:
            Fo = flat(fov, no * v).reshape(no, v)
            n = n + (T2[i, j][:, :, None] * Fo[k][None, None, :] + T2[i, k][:, None, :] * Fo[j][None, :, None]
                     + T2[j, k][None, :, :] * Fo[i][:, None, None])
        flat(M3, v ** 3)[...] = (W / D).ravel()
        flat(N3, v ** 3)[...] = (n / D).ravel()

    def t3_density_terms_f64(self, M3, N3, nv, A, S, Z, Ma, Mb, Mc, _st):
        v = nv
        M = flat(M3, v ** 3).reshape(v, v, v)
        N = flat(N3, v ** 3).reshape(v, v, v)

        def sym(X):   # 8 X_abc - 4 X_bac - 4 X_acb - 4 X_cba + 2 X_cab + 2 X_bca
            return (8 * X - 4 * X.transpose(1, 0, 2) - 4 * X.transpose(0, 2, 1)
                    - 4 * X.transpose(2, 1, 0) + 2 * np.einsum('cab->abc', X)
                    + 2 * np.einsum('bca->abc', X))
        sm, sn = sym(M), sym(N)
        flat(A, v ** 3)[...] = (2 * sm + sn).ravel()
        flat(S, v ** 3)[...] = (sm + sn).ravel()
        flat(Z, v ** 3)[...] = (2 * M - 2 * M.transpose(0, 2, 1) - M.transpose(1, 0, 2)
                                + np.einsum('bca->abc', M)).ravel()
        flat(Ma, v ** 3)[...] = (M - M.transpose(2, 1, 0)).ravel()
        flat(Mb, v ** 3)[...] = (2 * M - M.transpose(0, 2, 1) - M.transpose(2, 1, 0)).ravel()
        flat(Mc, v ** 3)[...] = (2 * M - 2 * M.transpose(1, 0, 2)).ravel()

    # -- the (T) entry points ------------------------------------------------------------------
    PART_LEN = 4              # the model's per-triple partial-sum length in FP32 mode

    def contract_multi_f64(self, nt, m_n, m_ext, m_sc, m_sa, n_n, n_ext, n_sc, n_sb, k_n, k_ext,
                           k_sa, k_sb, alpha, A, B, beta, Cp, _st):
        me, ne = _ints(m_ext, m_n), _ints(n_ext, n_n)
        Cv = view(Cp, me + ne, _ints(m_sc, m_n) + _ints(n_sc, n_n))
        acc = 0.0
        for t in range(nt):
            kn = int(k_n[t])
            ke = [int(k_ext[4 * t + q]) for q in range(kn)]
            sa = [int(m_sa[4 * t + q]) for q in range(m_n)] + [int(k_sa[4 * t + q]) for q in range(kn)]
            sb = [int(n_sb[4 * t + q]) for q in range(n_n)] + [int(k_sb[4 * t + q]) for q in range(kn)]
            Av, Bv = view(A[t], me + ke, sa), view(B[t], ne + ke, sb)
            acc = acc + alpha[t] * np.tensordot(Av, Bv, axes=(list(range(m_n, m_n + kn)),
                                                                list(range(n_n, n_n + kn))))
        Cv[...] = acc if beta == 0.0 else beta * Cv + acc

    # -- FP64 (T) in residue arithmetic: the same partials, from slots that were packed ----------
    def t3_rns_scales(self, V, O, t2, no, nv, c, work, length, _st):
        self.t3_slots = [None] * 3

    def t3_rns_window_pack(self, V, O, t2, no, nv, c, first, changed, work, length, _st):
        for q in range(3):
            assert 0 <= first[q] < no and first[q] % c == 0 and (q == 0 or first[q] <= first[q - 1])
            if changed >> q & 1:
                self.t3_slots[q] = first[q]

    def t3_rns_window_partials(self, V, O, t2, no, nv, c, first, ijk, ntrip, P, work, length, _st):
        assert self.t3_slots == [first[q] for q in range(3)]
        from pycc_gb300.triples import orientation_terms
        import torch
        arr = [torch.from_numpy(flat(p, int(np.prod(s))).reshape(s).copy()) for p, s in
               ((V, (nv, nv, nv, no)), (O, (no, nv, no, no)), (t2, (no, no, nv, nv)))]
        out = flat(P, 3 * ntrip * nv ** 3).reshape(ntrip, 3, nv, nv, nv)
        for t, (i, j, k) in enumerate(flat(ijk, 3 * ntrip, np.int32).reshape(ntrip, 3)):
            assert all(0 <= x - f < c for x, f in zip((i, j, k), self.t3_slots))
            for q, (lab, terms) in enumerate(orientation_terms(i, j, k, arr[2], arr[0], arr[1])):
                W = sum(a * torch.einsum("%s,%s->%s" % (la, lb, lab), A, B)
                        for a, A, la, B, lb in terms)
                out[t, q] = W.permute(2, 0, 1).numpy()   # [z][x][y]

    def tc_grouped_gemm(self, na, a_ptr, a_rows, a_ld, nb, b_ptr, b_rows, b_ld, groups, ngroups,
                        M, N, Cp, ldm, ldn, _status, _st):
        from pycc_gb300.triples_tc import GROUP_DTYPE
        g = np.frombuffer((C.c_char * (ngroups * GROUP_DTYPE.itemsize)).from_address(groups),
                          dtype=GROUP_DTYPE)
        As = [self.packs[a_ptr[q]] for q in range(na)]
        Bs = [self.packs[b_ptr[q]] for q in range(nb)]
        m, n = np.arange(M), np.arange(N)
        for rec in g:
            acc = np.zeros((M, N))
            for s in range(int(rec["nseg"])):
                A = As[rec["amap"][s]][rec["arow"][s] + m]
                B = Bs[rec["bmap"][s]][rec["brow"][s] + n]
                assert A.shape[1] <= 64 * rec["nkb"][s]
                acc += A @ B.T
            idx = int(rec["out"]) + m[:, None] * ldm + n[None, :] * ldn
            flat(Cp, int(idx.max()) + 1, np.float32)[idx] = acc.astype(np.float32)

    def tc_grouped_gemm_pitched(self, na, a_ptr, a_rows, a_ld, nb, b_ptr, b_rows, b_ld, groups,
                                ngroups, M, N, Cp, inner, outer, ldn, _status, _st):
        """Row m of a group at (m / inner) * outer + m % inner."""
        assert M % inner == 0 and outer >= inner
        tmp = np.zeros((ngroups, N, M), dtype=np.float32)
        from pycc_gb300.triples_tc import GROUP_DTYPE
        g = np.frombuffer((C.c_char * (ngroups * GROUP_DTYPE.itemsize)).from_address(groups),
                          dtype=GROUP_DTYPE).copy()
        outs = g["out"].copy()
        g["out"] = np.arange(ngroups) * N * M
        self.tc_grouped_gemm(na, a_ptr, a_rows, a_ld, nb, b_ptr, b_rows, b_ld, g.ctypes.data,
                             ngroups, M, N, tmp.ctypes.data, 1, M, _status, _st)
        for o, block in zip(outs, tmp):
            view(Cp + 4 * int(o), (N, M // inner, inner), (ldn, outer, 1), np.float32)[...] = \
                block.reshape(N, M // inner, inner)

    def triples_energy_pitched(self, P, pitch, ijk, ntrip, eps, eoovv, t1, t2, fov, no, nv, part,
                               _status, _st):
        assert pitch >= nv and pitch % 4 == 0
        rows = lambda p, lead: np.ascontiguousarray(
            view(p, (lead, nv, nv), (nv * pitch, pitch, 1), np.float32))
        dense = np.ascontiguousarray(
            view(P, (ntrip, 3, nv, nv, nv),
                 (3 * nv * nv * pitch, nv * nv * pitch, nv * pitch, pitch, 1), np.float32))
        e, t = rows(eoovv, no * no), rows(t2, no * no)
        self.triples_energy(1, dense.ctypes.data, dense.ctypes.data + 4 * nv ** 3,
                            dense.ctypes.data + 8 * nv ** 3, 3 * nv ** 3, ijk, ntrip, eps,
                            e.ctypes.data, t1, t.ctypes.data, fov, no, nv, part, _st)

    def triples_energy(self, fp32, P1, P2, P3, pstride, ijk, ntrip, eps, eoovv, t1, t2, fov,
                       no, nv, part, _st):
        from oracle.triples import ijk_energy
        dt = np.float32 if fp32 else np.float64
        v3 = nv ** 3
        tri = flat(ijk, 3 * ntrip, np.int32).reshape(ntrip, 3)
        e = flat(eps, no + nv)
        F = np.diag(e)
        if fov:
            F[:no, no:] = flat(fov, no * nv).reshape(no, nv)
        V = flat(eoovv, no * no * nv * nv, dt).astype(np.float64).reshape(no, no, nv, nv)
        T1 = flat(t1, no * nv).reshape(no, nv)
        T2 = flat(t2, no * no * nv * nv, dt).astype(np.float64).reshape(no, no, nv, nv)
        plen = self.PART_LEN if fp32 else nv
        out = flat(part, ntrip * plen)
        o, v = slice(0, no), slice(no, no + nv)
        for t in range(ntrip):
            # a partial is stored [z][x][y] for the logical P[x, y, z]
            P = [flat(p + t * pstride * np.dtype(dt).itemsize, v3, dt).astype(np.float64)
                 .reshape(nv, nv, nv).transpose(1, 2, 0) for p in (P1, P2, P3)]
            W = P[0] + P[1].transpose(0, 2, 1) + P[2].transpose(2, 0, 1)
            i, j, k = (int(x) for x in tri[t])
            out[t * plen:(t + 1) * plen] = 0.0
            out[t * plen] = ijk_energy(o, v, i, j, k, W, T1, T2, V, F)

    def reduce_sum_f64(self, x, n, out, _st):
        flat(out, 1)[0] += flat(x, n).sum()


class _LibStub:
    """The two size queries the host makes on the library object itself."""

    @staticmethod
    def pcg_triples_part_len(fp32, nv):
        return ABIModel.PART_LEN if fp32 else nv

    @staticmethod
    def pcg_tc_group_desc_size():
        return 96


def install(monkeypatch):
    """Route the engine's library calls to the model (CPU tensors accepted)."""
    from pycc_gb300 import _lib, contract
    model = ABIModel()
    monkeypatch.setattr(_lib, "call", model)
    monkeypatch.setattr(_lib, "load", lambda *a, **k: _LibStub)
    monkeypatch.setattr(_lib, "stream_handle", lambda stream=None: None)

    def check(t, name):
        import torch
        if not isinstance(t, torch.Tensor) or t.dtype != torch.float64:
            raise TypeError("contract: %s must be a float64 tensor" % name)
    monkeypatch.setattr(contract, "_check", check)
    return model
